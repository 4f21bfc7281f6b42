// Batched execution of many independent stencil runs in one persistent
// launch per time step (GB300, sm_103a).  No counterpart in the reference,
// which runs every PSStencilRun by itself.
//
// Every problem (one run: a grid pair and its maps) is cut into (z-chunk,
// tile) work items exactly as its single-run kernel would cut it.  The items
// of all problems form one list, problem after problem and chunk-major within
// a problem; a persistent grid of SMs x occupancy CTAs takes items
// round-robin, so small problems fill the GPU together and large ones keep
// the chunk-major locality of the single-run kernels.  A CTA's items ascend, so
// it finds an item's problem by stepping on from the last one's, and runs the
// shared per-item body (s7_body.cuh / himeno_body.cuh) with that
// problem's parameters and tensor maps, both read from global memory.
// Problem kinds: the 7-point family (DIFFUSION7, SUM7, COPY; 1, 2 or 4 rows
// per thread) and the plain Himeno sweep, float grids.  Each family has its own
// kernel so that each launch carries only its family's registers and shared memory; a batch holding both families
// launches one of each per step.
#include "batch.h"
#include "himeno_body.cuh"
#include "s7_body.cuh"

namespace psg {
namespace {

template <int K>
__device__ __forceinline__ bool s7_rows(const BatchProblem &bp, int parity,
                                        const CUtensorMap *tmaps, uint64_t *full, float *ring,
                                        int tile, int zs, int ze, RingPos &prod,
                                        RingPos &cons) {
  constexpr int W = 34 * 4;
  const S7Params<float> &p = bp.s7[parity];
  const CUtensorMap *tin = tmaps + bp.tmap[parity];
  const int TY = blockDim.y * bp.rows;
  const uint32_t plane_bytes = (uint32_t)(W * (TY + 2) * 4);
  const int plane_elems = (int)(s7_stage_bytes(plane_bytes) / 4);
  if (bp.rows == 1)
    return s7_item<float, K, 1>(tin, p, full, ring, plane_elems, plane_bytes, TY, tile, zs, ze,
                                prod, cons);
  if (bp.rows == 2)
    return s7_item<float, K, 2>(tin, p, full, ring, plane_elems, plane_bytes, TY, tile, zs, ze,
                                prod, cons);
  return s7_item<float, K, 4>(tin, p, full, ring, plane_elems, plane_bytes, TY, tile, zs, ze,
                              prod, cons);
}

// Problem of an item at or after those of problem `q`: items of a CTA ascend.
__device__ __forceinline__ int batch_problem(const BatchProblem *__restrict__ probs, int nprob,
                                             int64_t item, int q) {
  while (q + 1 < nprob && probs[q + 1].item_begin <= item) ++q;
  return q;
}

__global__ void __launch_bounds__(256, 1)
batch7_kernel(const BatchProblem *__restrict__ probs, int nprob, const CUtensorMap *tmaps,
              int64_t total_items, int parity, int ns7) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  float *ring = reinterpret_cast<float *>(smem + s7_bar_bytes(ns7));
  const int tid = threadIdx.y * 32 + threadIdx.x;
  if (tid == 0) {
    for (int s = 0; s < ns7; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  __syncthreads();

  RingPos prod, cons;
  bool ok = true;
  int q = 0;
  for (int64_t item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
    q = batch_problem(probs, nprob, item, q);
    const BatchProblem &bp = probs[q];
    const int64_t local = item - bp.item_begin;
    const int chunk = (int)(local / bp.tiles);
    const int tile = (int)(local - (int64_t)chunk * bp.tiles);
    const int zs = bp.dmin2 + chunk * bp.zlen;
    const int ze = min(zs + bp.zlen, bp.dmax2);
    switch (bp.kind) {
      case kKernelDiffusion7:
        ok = s7_rows<kKernelDiffusion7>(bp, parity, tmaps, full, ring, tile, zs, ze, prod, cons);
        break;
      case kKernelSum7:
        ok = s7_rows<kKernelSum7>(bp, parity, tmaps, full, ring, tile, zs, ze, prod, cons);
        break;
      default:
        ok = s7_rows<kKernelCopy>(bp, parity, tmaps, full, ring, tile, zs, ze, prod, cons);
        break;
    }
  }
  if (!ok && tid == 0) {
    for (int s = 0; s < ns7; ++s) mbar_wait(&full[s], 0, nullptr, 1024);
  }
}

__global__ void __maxnreg__(128)
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

size_t batch_smem_bytes(const BatchShape &sh, int fam) {
  const size_t r7 = (size_t)sh.ns7 * s7_stage_bytes((uint32_t)(34 * 4 * (sh.warps * sh.max_rows + 2) * 4));
  const size_t rh = (size_t)sh.nsp * h_align128((uint32_t)(kHimW * (sh.warps + 2) * 4)) +
                    (size_t)sh.nsc * kHimCoef * kHimTX * sh.warps * 4;
  return 128 + (fam == kBatch7 ? (size_t)s7_bar_bytes(sh.ns7) + r7
                               : (size_t)h_bar_bytes(2 * (sh.nsp + sh.nsc)) + rh);
}

namespace {
const void *batch_fn(int fam) {
  return fam == kBatch7 ? reinterpret_cast<const void *>(batch7_kernel)
                        : reinterpret_cast<const void *>(batch_himeno_kernel);
}
// Himeno CTAs have a producer warp besides.
int batch_warps(const BatchShape &sh, int fam) { return sh.warps + (fam == kBatchHimeno ? 1 : 0); }
}  // namespace

int batch_occupancy(const BatchShape &sh, int fam) {
  int oc = 0;
  const size_t smem = batch_smem_bytes(sh, fam);
  if (cudaFuncSetAttribute(batch_fn(fam), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&oc, batch_fn(fam),
                                                    32 * batch_warps(sh, fam), smem) !=
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
  const dim3 block(32, batch_warps(sh, fam), 1);
  if (fam == kBatch7)
    batch7_kernel<<<grid, block, smem, s>>>(probs_dev, nprob, tmaps_dev, total_items, parity,
                                            sh.ns7);
  else
    batch_himeno_kernel<<<grid, block, smem, s>>>(probs_dev, nprob, tmaps_dev, total_items, parity,
                                                  sh.nsp, sh.nsc);
  return cudaGetLastError();
}

}  // namespace psg
