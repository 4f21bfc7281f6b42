// Batched execution of many independent stencil runs in one persistent
// launch per time step (GB300, sm_103a).  No counterpart in the reference,
// which runs every PSStencilRun by itself.
//
// Every problem (one run: a grid pair and its maps) is cut into (z-chunk,
// tile) work items, tiles as its single-run kernel would cut them.  The items
// of all problems form one list, problem after problem and chunk-major within
// a problem; a persistent grid of SMs x occupancy CTAs takes items
// round-robin, so small problems fill the GPU together and large ones keep
// the chunk-major locality of the single-run kernels.  A CTA's items ascend, so
// it looks for an item's problem from the last one's on, and runs the
// shared per-item body (s7_body.cuh / himeno_body.cuh) with that
// problem's parameters and tensor maps, both read from global memory.
// Problem kinds: the 7-point family (DIFFUSION7, SUM7, COPY; 1, 2 or 4 rows
// per thread) and the plain Himeno sweep, float grids.  Each family has its own
// kernel so that each launch carries only its family's registers and shared
// memory; a batch holding both families launches one of each per step, side by
// side (both ask for the largest shared-memory carveout: an SM holding CTAs of
// one does not otherwise take the other's until it is idle).  Himeno's comes
// first: its items are the longer ones, and CTAs of it that found their places
// taken would make the tail (48 grids up to 320 x 320 x 512 161.7 GLUPS, 155.7 with
// the 7-point family first, in turn on one box; other boxes gave 157 to 163).
// In each kernel the last warp is a producer that fills the ring on into the
// CTA's next item, and consumer warps release stages one by one.
// Bound: the Himeno family HBM (216 of the 24-problem batch's 256 us a step), the
// 7-point family issue slots and latency of small items.  Per step, with 128-cell
// tiles and rings drained between items: 24 problems 32 to 160 wide 299 us, 26
// problems 16 to 80 wide 70 (50 now), 6 problems 16 to 48 wide 9.1 (6.0).
#include "batch.h"
#include "himeno_body.cuh"
#include "s7_body.cuh"

namespace psg {
namespace {

// A consumer warp releases a stage on its "empty" mbarrier.
struct B7Sync {
  static constexpr bool kIssues = false;
  uint64_t *empty;
  int ns;
  RingPos rel;
  __device__ __forceinline__ void last() {
    __syncwarp();
    if (threadIdx.x == 0) mbar_arrive(&empty[rel.stage]);
    rel.advance(ns);
  }
  __device__ __forceinline__ bool done(bool ok) {
    ok = __all_sync(0xffffffffu, ok);
    if (ok) last();
    return ok;
  }
};

template <int K>
__device__ __forceinline__ bool s7_rows(const BatchProblem &bp, int parity, uint64_t *full,
                                        float *ring, int stage_elems, int warps, int tile, int zs,
                                        int ze, RingPos &cons, B7Sync &sync) {
  const S7Params<float> &p = bp.s7[parity];
  if (bp.rows == 1)
    return s7_item<float, K, 1, true>(p, full, ring, stage_elems, warps, tile, zs, ze, cons, sync);
  if (bp.rows == 2)
    return s7_item<float, K, 2, true>(p, full, ring, stage_elems, warps, tile, zs, ze, cons, sync);
  return s7_item<float, K, 4, true>(p, full, ring, stage_elems, warps, tile, zs, ze, cons, sync);
}

// Problem of an item at or after those of problem `q`: items of a CTA ascend.
// Often still q; else found by bisection, as each look at a problem waits for L2.
__device__ __forceinline__ int batch_problem(const BatchProblem *__restrict__ probs, int nprob,
                                             int64_t item, int q) {
  if (q + 1 >= nprob || probs[q + 1].item_begin > item) return q;
  int lo = q + 1, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].item_begin <= item) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __maxnreg__(112)
batch7_kernel(const BatchProblem *__restrict__ probs, int nprob, const CUtensorMap *tmaps,
              int64_t total_items, int parity, int ns7, int stage_elems) {
  const int warps = blockDim.y - 1;  // consumers; the last warp is the producer
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + ns7;
  float *ring = reinterpret_cast<float *>(smem + s7_bar_bytes(2 * ns7));
  const int lane = threadIdx.x, row = threadIdx.y, tid = row * 32 + lane;
  if (tid == 0) {
    for (int s = 0; s < ns7; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], warps);
    }
    fence_barrier_init();
  }
  __syncthreads();

  RingPos prod, cons;
  B7Sync sync{empty, ns7};
  bool ok = true;
  int q = 0;
  if (row < warps || lane == 0) {
    for (int64_t item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
      q = batch_problem(probs, nprob, item, q);
      const BatchProblem &bp = probs[q];
      const int local = (int)(item - bp.item_begin);
      const int chunk = local / bp.tiles, tile = local - chunk * bp.tiles;
      const int zs = bp.dmin2 + chunk * bp.zlen;
      const int ze = min(zs + bp.zlen, bp.dmax2);
      if (row == warps) {
        const S7Params<float> &p = bp.s7[parity];
        const CUtensorMap *map = tmaps + bp.tmap[parity];
        const int tx = 4 * bp.lx, ty = warps * bp.rows * (32 / bp.lx);
        const int x = p.xbase + (tile % p.tiles_x) * tx - 4;
        const int y = p.dmin1 + (tile / p.tiles_x) * ty - 1;
        const uint32_t bytes = (uint32_t)((tx + 8) * (ty + 2) * 4);
        for (int z = zs - 1; z <= ze && ok; ++z) {
          const int s = prod.stage;
          ok = mbar_wait(&empty[s], prod.phase ^ 1u, p.err);
          if (!ok) break;
          mbar_arrive_expect_tx(&full[s], bytes);
          tma_load_3d(ring + s * stage_elems, map, x, y, z, &full[s]);
          prod.advance(ns7);
        }
      } else {
        switch (bp.kind) {
          case kKernelDiffusion7:
            ok = s7_rows<kKernelDiffusion7>(bp, parity, full, ring, stage_elems, warps, tile, zs,
                                            ze, cons, sync);
            break;
          case kKernelSum7:
            ok = s7_rows<kKernelSum7>(bp, parity, full, ring, stage_elems, warps, tile, zs, ze,
                                      cons, sync);
            break;
          default:
            ok = s7_rows<kKernelCopy>(bp, parity, full, ring, stage_elems, warps, tile, zs, ze,
                                      cons, sync);
            break;
        }
      }
    }
  }
  if (!__syncthreads_and(ok) && tid == 0) {
    // Give copies still in flight a bounded chance to land before exit.
    for (int s = 0; s < ns7; ++s) mbar_wait(&full[s], 0, nullptr, 1024);
  }
}

__global__ void __maxnreg__(112)
batch_himeno_kernel(const BatchProblem *__restrict__ probs, int nprob, const CUtensorMap *tmaps,
                    int64_t total_items, int parity, int nsp, int nsc) {
  const int warps = blockDim.y - 1;  // consumers; the last warp is the producer
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  const HimSmem h = him_smem(smem, nsp, nsc, warps);
  const int lane = threadIdx.x, row = threadIdx.y, tid = row * 32 + lane;
  if (tid == 0) him_init(h, nsp, nsc, warps);
  __syncthreads();

  HRing pprod, cprod, pcons, prel, ccons;
  float acc = 0.0f;
  bool ok = true;
  int q = 0;
  if (row < warps || lane == 0) {
    for (int64_t item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
      q = batch_problem(probs, nprob, item, q);
      const BatchProblem &bp = probs[q];
      const HParams &p = bp.him[parity];
      const int local = (int)(item - bp.item_begin);
      const int chunk = local / bp.tiles, tile = local - chunk * bp.tiles;
      const int zs = bp.dmin2 + chunk * bp.zlen;
      const int ze = min(zs + bp.zlen, bp.dmax2);
      if (row == warps)
        ok = himeno_produce(tmaps + bp.tmap[parity], tmaps + bp.cmap, p, h, warps, bp.lx, tile, zs,
                            ze, pprod, cprod);
      else if (bp.lx == 32)
        ok = himeno_consume<false, 32>(p, h, warps, tile, zs, ze, pcons, prel, ccons, acc);
      else if (bp.lx == 16)
        ok = himeno_consume<false, 16>(p, h, warps, tile, zs, ze, pcons, prel, ccons, acc);
      else
        ok = himeno_consume<false, 8>(p, h, warps, tile, zs, ze, pcons, prel, ccons, acc);
    }
  }
  if (!__syncthreads_and(ok) && tid == 0) him_drain(h, nsp, nsc);
}

}  // namespace

size_t batch_stage7(const BatchShape &sh) {
  return sh.stage7 ? (size_t)sh.stage7
                   : s7_stage_bytes((uint32_t)(34 * 4 * (sh.warps * sh.max_rows + 2) * 4));
}

size_t batch_smem_bytes(const BatchShape &sh, int fam) {
  const size_t r7 = (size_t)sh.ns7 * batch_stage7(sh);
  const size_t rh = (size_t)sh.nsp * h_align128((uint32_t)(kHimW * (sh.warps + 2) * 4)) +
                    (size_t)sh.nsc * kHimCoef * kHimTX * sh.warps * 4;
  return 128 + (fam == kBatch7 ? (size_t)s7_bar_bytes(2 * sh.ns7) + r7
                               : (size_t)h_bar_bytes(2 * (sh.nsp + sh.nsc)) + rh);
}

namespace {
const void *batch_fn(int fam) {
  return fam == kBatch7 ? reinterpret_cast<const void *>(batch7_kernel)
                        : reinterpret_cast<const void *>(batch_himeno_kernel);
}
}  // namespace

int batch_occupancy(const BatchShape &sh, int fam) {
  int oc = 0;
  const size_t smem = batch_smem_bytes(sh, fam);
  if (cudaFuncSetAttribute(batch_fn(fam), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(batch_fn(fam), cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&oc, batch_fn(fam),
                                                    32 * (sh.warps + 1), smem) !=
          cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return oc;
}

cudaError_t launch_batch(const BatchProblem *probs_dev, int nprob, const CUtensorMap *tmaps_dev,
                         int64_t total_items, int parity, const BatchShape &sh, int grid, int fam,
                         cudaStream_t s) {
  const size_t smem = batch_smem_bytes(sh, fam);
  const dim3 block(32, sh.warps + 1, 1);  // the last warp is the producer
  if (fam == kBatch7)
    batch7_kernel<<<grid, block, smem, s>>>(probs_dev, nprob, tmaps_dev, total_items, parity,
                                            sh.ns7, (int)(batch_stage7(sh) / 4));
  else
    batch_himeno_kernel<<<grid, block, smem, s>>>(probs_dev, nprob, tmaps_dev, total_items, parity,
                                                  sh.nsp, sh.nsc);
  return cudaGetLastError();
}

}  // namespace psg
