// Himeno 19-point variable-coefficient Jacobi sweep on GB300 (sm_103a),
// with the residual (gosa = sum of ss*ss) fused into the same pass.
//
// Semantics: the Physis Himeno kernel (examples/himeno/himenobmtxpa_physis.c:
// 331-361), i = x fastest, over the interior domain; cells outside the domain
// are never written.  The residual follows the original benchmark's loop
// (examples/himeno/himenobmtxpa_original.c:331-334), which the Physis port
// dropped; here it costs no extra HBM traffic.
//
// Design (persistent, like the 7-point kernel: (z-chunk, tile) work items in
// chunk-major order taken round-robin by SMs x occupancy CTAs, so resident
// CTAs march the same z-chunk of neighbouring tiles; a tile is 128 x warps
// cells in x,y, or 64 or 32 cells wide and higher, see himeno19_lanes):
// * p planes with a one-cell y halo and a 4-cell (16-byte) x halo arrive by
//   TMA into a ring of `ns` stages; the sweep at plane z reads planes z-1, z
//   and z+1 from the ring (the 19-point stencil needs xy neighbours on all
//   three planes, so a register queue alone does not suffice);
// * the 12 centre-only coefficient arrays (a0..a3, b0..b2, c0..c2, bnd,
//   wrk1) arrive as 12 TMA boxes of the tile per plane into a second ring
//   of `ns2` stages, all signalled by one mbarrier per stage;
// * a producer warp fills both rings, on into the CTA's next item; consumer
//   warps release stages one by one, so nothing drains between items;
// * one thread per 4 consecutive x cells: 16-byte shared loads, x neighbours
//   by warp shuffles, one 16-byte store;
// * the arithmetic keeps the reference's expression order, round-to-nearest
//   without FMA contraction, so p matches the REF target bit for bit;
// * residual: FP32 per thread, FP32 warp-shuffle + block tree, one FP64
//   partial per CTA, and the last CTA to finish (atomic ticket) adds the
//   partials in FP64 in a fixed order (deterministic run to run).
// Bound: HBM, 14 arrays of 4 bytes a cell; 257 x 257 x 513 takes 290 us with the
// residual, 270 at the copy rate.  Against 128-cell tiles filled by a consumer
// between CTA barriers, a sweep with its residual read back: 200^3 100 against
// 114 us, 142 x 245 x 97 57 and 74, 65^3 28 and 37.  All coefficients loaded before any is
// used takes 155 registers for 96, one CTA of three per SM and 4 % more time.
#include "himeno_body.cuh"

namespace psg {
namespace {

struct HimenoMaps {
  CUtensorMap p;               // p0 with the tile's halo box
  CUtensorMap coef[kHimCoef];  // the tile's box
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <bool GOSA, int LX>
__global__ void __maxnreg__(128)
himeno19_kernel(const __grid_constant__ HimenoMaps maps, const HParams p) {
  const int warps = blockDim.y - 1;  // consumers; the last warp is the producer
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  const HimSmem h = him_smem(smem, p.nsp, p.nsc, warps);
  __shared__ float red[32];
  __shared__ int last_cta;

  const int lane = threadIdx.x, row = threadIdx.y;
  const int tid = row * 32 + lane;
  if (tid == 0) {
    prefetch_tmap(&maps.p);
    him_init(h, p.nsp, p.nsc, warps);
  }
  __syncthreads();
  // dependents are not let in early: CTAs that take places as they fall free lose
  // the neighbours they share p's halos with (257 x 257 x 513, sweep after sweep:
  // 298 us against 292)
  wait_for_predecessors();

  HRing pprod, cprod, pcons, prel, ccons;
  bool ok = true;
  float acc = 0.0f;
  if (row < warps || lane == 0) {
    for (int64_t item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
      const int chunk = (int)(item / p.tiles);
      const int tile = (int)(item - (int64_t)chunk * p.tiles);
      const int zs = p.dmin2 + chunk * p.zlen;
      const int ze = min(zs + p.zlen, p.dmax2);
      ok = row < warps ? himeno_consume<GOSA, LX>(p, h, warps, tile, zs, ze, pcons, prel, ccons, acc)
                       : himeno_produce(&maps.p, maps.coef, p, h, warps, LX, tile, zs, ze, pprod,
                                        cprod);
    }
  }
  if (!__syncthreads_and(ok)) {
    if (tid == 0) him_drain(h, p.nsp, p.nsc);
    return;
  }
  if (!GOSA) return;

  // Residual: FP32 block tree, FP64 partial per CTA, FP64 final combine.
  acc = warp_sum(acc);
  if (lane == 0 && row < warps) red[row] = acc;
  __syncthreads();
  if (tid == 0) {
    float bs = 0.0f;
    for (int w = 0; w < warps; ++w) bs = __fadd_rn(bs, red[w]);
    p.partials[blockIdx.x] = (double)bs;
    __threadfence();
    const unsigned prev = atomicAdd(p.ticket, 1u);
    last_cta = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (last_cta && row == 0) {
    __threadfence();
    double v = 0.0;
    for (unsigned i = lane; i < gridDim.x; i += 32) v = __dadd_rn(v, __ldcg(&p.partials[i]));
    v = warp_sum(v);
    if (lane == 0) {
      *p.result = v;
      *p.ticket = 0u;
    }
  }
}

}  // namespace

size_t himeno19_smem_bytes(const MarchConfig &cfg) {
  // 128 bytes of slack for aligning the dynamic shared-memory base
  return 128 + (size_t)h_bar_bytes(2 * (cfg.ns + cfg.ns2)) +
         (size_t)cfg.ns * h_align128((uint32_t)(kHimW * (cfg.warps + 2) * 4)) +
         (size_t)cfg.ns2 * kHimCoef * kHimTX * cfg.warps * 4;
}

// Lanes side by side in x: all tiles hold the same cells, so the widest is
// taken unless a narrower one covers the domain with 3 % fewer (a batch of 24
// problems 39 to 160 wide: 271 us a step, 299 with 128-cell tiles and no producer).
int himeno19_lanes(const Box &dom, int warps) {
  const int nx = dom.max[0] - dom.min[0] / 4 * 4, ny = dom.max[1] - dom.min[1];
  int best = 32;
  double cost = 0;
  for (int lx = 32; lx >= 8; lx /= 2) {
    const int tx = 4 * lx, ty = him_rows(warps, lx);
    const double c = (double)((nx + tx - 1) / tx) * ((ny + ty - 1) / ty);
    if (lx == 32 || c < 0.97 * cost) {
      best = lx;
      cost = c;
    }
  }
  return best;
}

void himeno19_boxes(int lx, int warps, int p_box[2], int c_box[2]) {
  c_box[0] = 4 * lx;
  c_box[1] = him_rows(warps, lx);
  p_box[0] = c_box[0] + 8;
  p_box[1] = c_box[1] + 2;
}

namespace {
template <int LX>
auto him_kernel(bool gosa) {
  return gosa ? himeno19_kernel<true, LX> : himeno19_kernel<false, LX>;
}
}  // namespace

cudaError_t launch_himeno19(const Himeno19Args &a, const MarchConfig &cfg,
                            const CUtensorMap *tmaps, const ResidualSink &sink,
                            int *dev_err, int sm_count, cudaStream_t s) {
  HimenoMaps maps;
  maps.p = tmaps[0];
  for (int i = 0; i < kHimCoef; ++i) maps.coef[i] = tmaps[1 + i];
  HParams p;
  const GridView &out = a.g[1];
  p.out = static_cast<float *>(out.ptr);
  p.row = out.pitch / 4;
  p.plane = p.row * out.ny;
  p.dmin0 = a.dom.min[0];
  p.dmin1 = a.dom.min[1];
  p.dmin2 = a.dom.min[2];
  p.dmax0 = a.dom.max[0];
  p.dmax1 = a.dom.max[1];
  p.dmax2 = a.dom.max[2];
  p.xbase = (a.dom.min[0] / 4) * 4;
  p.nsp = cfg.ns;
  p.nsc = cfg.ns2;
  p.omega = a.omega;
  p.partials = sink.partials;
  p.ticket = sink.ticket;
  p.result = sink.result;
  p.err = dev_err;
  const int ex = a.dom.max[0] - p.xbase;
  const int ey = a.dom.max[1] - a.dom.min[1];
  const int ez = a.dom.max[2] - a.dom.min[2];
  if (ex <= 0 || ey <= 0 || ez <= 0) return cudaSuccess;
  if (cfg.warps < 1 || cfg.warps > 8 || cfg.ns < 3 || cfg.ns > 16 || cfg.ns2 < 1 ||
      cfg.ns2 > 8)
    return cudaErrorInvalidConfiguration;
  const int lx = himeno19_lanes(a.dom, cfg.warps);
  const int tx = 4 * lx, ty = him_rows(cfg.warps, lx);
  p.tiles_x = (ex + tx - 1) / tx;
  p.tiles = p.tiles_x * ((ey + ty - 1) / ty);
  const size_t smem = himeno19_smem_bytes(cfg);
  // Opt in to the dynamic shared memory this launch needs (the kernel also
  // has a little static shared memory, so the opt-in is the exact size).
  static size_t attr_set[2][3] = {};
  static int occ[2][3][9][17][9];  // [gosa][lanes][warps][ns][ns2] -> CTAs per SM
  const int gi = a.gosa ? 1 : 0, li = lx == 32 ? 0 : lx == 16 ? 1 : 2;
  auto kern = lx == 32 ? him_kernel<32>(a.gosa) : lx == 16 ? him_kernel<16>(a.gosa)
                                                           : him_kernel<8>(a.gosa);
  const int threads = 32 * (cfg.warps + 1);
  size_t &have = attr_set[gi][li];
  if (smem > have) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    have = smem;
  }
  // The round-robin schedule assumes every CTA is resident: never launch
  // more per SM than fit.
  int &oc = occ[gi][li][cfg.warps][cfg.ns][cfg.ns2];
  if (oc == 0) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&oc, kern, threads, smem);
    if (e != cudaSuccess) return e;
    if (oc < 1) oc = 1;
  }
  const int per_sm = (cfg.ctas_per_sm > 0 && cfg.ctas_per_sm < oc) ? cfg.ctas_per_sm : oc;
  const int resident = sm_count * per_sm;
  p.zlen = choose_zchunk(p.tiles, ez, resident);
  p.items = (int64_t)p.tiles * ((ez + p.zlen - 1) / p.zlen);
  int64_t grid = resident;
  if (grid > p.items) grid = p.items;
  if (a.gosa && grid > sink.max_partials) grid = sink.max_partials;
  return launch_kernel(kern, (unsigned)grid, dim3(32, cfg.warps + 1, 1), smem, s, a.overlap, maps, p);
}

}  // namespace psg
