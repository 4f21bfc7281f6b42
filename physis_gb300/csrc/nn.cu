// Kernels of the learned warm start for the 19-point Jacobi (Himeno) solve:
// a 3D convolutional network of 3x3x3 layers with 16 channels, BF16 weights
// and activations, FP32 accumulation, trained on the GPU.  No counterpart in
// the reference.
//
// Tensors are channels-last, [batch, z, y, x, 16] BF16 (16 channels: 32
// bytes per voxel).  A convolution is an implicit GEMM per tap: rows are
// voxels, K the 16 input channels, N the 16 output channels.  Three forms:
// conv_pad_kernel (tcgen05 over zero-padded slabs) wherever a padded plane has
// at most 1024 voxels, conv_tc_kernel (tcgen05, gathered tiles) for larger
// planes, and conv_kernel (mma.sync.m16n8k16: each warp owns 16 voxels and
// accumulates 27 taps x 2 n-tiles) when PS_WARMSTART_TC=0 asks for it.  The
// backward-data pass is the same kernel with the weights flipped in space and
// transposed in channels; the weight gradient is a K = voxels GEMM per tap
// (wgrad_run_kernel; wgrad_kernel for unaligned tensors), split over CTAs
// and reduced in a fixed order (deterministic).
// Pooling (fine grids -> coarse network input), the MSE gradient, Adam and
// cubic upsampling (coarse prediction -> fine warm start) complete the
// set.  Every kernel is checked against oracle/nn_oracle.py.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdlib.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ps_device.cuh"
#include "ps_internal.h"

namespace psg {
namespace {

int *g_err = nullptr;  // the runtime's device error word (bounded waits)

constexpr int kC = 16;       // channels
constexpr int kTaps = 27;
constexpr int kPoolChannels = 9;  // network input channels in use
constexpr int kConvWarps = 8;

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4],
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct Dims {
  int B, Z, Y, X;
  long long nvox;
};

// Voxel coordinates of flattened index v (x fastest).
struct Vox {
  int b, z, y, x;
  bool ok;
};
__device__ __forceinline__ Vox vox_of(long long v, const Dims &d) {
  Vox r;
  r.ok = v < d.nvox;
  if (!r.ok) v = 0;
  r.x = (int)(v % d.X);
  long long t = v / d.X;
  r.y = (int)(t % d.Y);
  t /= d.Y;
  r.z = (int)(t % d.Z);
  r.b = (int)(t / d.Z);
  return r;
}

// Flattened index of the neighbour of `p` at tap t, or -1 outside.
__device__ __forceinline__ long long nbr(const Vox &p, int t, const Dims &d) {
  const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
  const int z = p.z + dz, y = p.y + dy, x = p.x + dx;
  if (!p.ok || z < 0 || z >= d.Z || y < 0 || y >= d.Y || x < 0 || x >= d.X) return -1;
  return (((long long)p.b * d.Z + z) * d.Y + y) * d.X + x;
}

__device__ __forceinline__ uint32_t ld_pair(const __nv_bfloat16 *base, long long v, int c) {
  return v < 0 ? 0u : *reinterpret_cast<const uint32_t *>(base + v * kC + c);
}
__device__ __forceinline__ uint32_t pack2(const __nv_bfloat16 *base, long long v0, long long v1,
                                          int c) {
  const uint16_t lo = v0 < 0 ? 0 : reinterpret_cast<const uint16_t *>(base)[v0 * kC + c];
  const uint16_t hi = v1 < 0 ? 0 : reinterpret_cast<const uint16_t *>(base)[v1 * kC + c];
  return (uint32_t)lo | ((uint32_t)hi << 16);
}

// Y = epilogue(conv(X, W) + bias): relu, or times (mask > 0).  W is
// [27][out][in] BF16.  yf (optional) receives channel 0 in FP32.
__global__ void __launch_bounds__(32 * kConvWarps)
conv_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
            const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask,
            int relu, __nv_bfloat16 *__restrict__ y, float *__restrict__ yf, Dims d) {
  __shared__ __align__(16) __nv_bfloat16 ws[kTaps * kC * kC];
  for (int i = threadIdx.x; i < kTaps * kC * kC / 8; i += blockDim.x)
    reinterpret_cast<uint4 *>(ws)[i] = reinterpret_cast<const uint4 *>(w)[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const long long v0 = ((long long)blockIdx.x * kConvWarps + warp) * 16;
  if (v0 >= d.nvox) return;
  const Vox pa = vox_of(v0 + g, d), pb = vox_of(v0 + g + 8, d);
  float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};
  for (int t = 0; t < kTaps; ++t) {
    const long long na = nbr(pa, t, d), nb = nbr(pb, t, d);
    const uint32_t a[4] = {ld_pair(x, na, 2 * q), ld_pair(x, nb, 2 * q),
                           ld_pair(x, na, 2 * q + 8), ld_pair(x, nb, 2 * q + 8)};
    const uint32_t *wt = reinterpret_cast<const uint32_t *>(ws + t * kC * kC);
    // B (k = in, n = out) from ws[t][out][in]: two consecutive in-channels
    mma_16816(acc0, a, wt[(g * kC + 2 * q) / 2], wt[(g * kC + 2 * q + 8) / 2]);
    mma_16816(acc1, a, wt[((g + 8) * kC + 2 * q) / 2], wt[((g + 8) * kC + 2 * q + 8) / 2]);
  }
  // C: c0,c1 -> (voxel g, out 2q, 2q+1); c2,c3 -> (voxel g+8, ...)
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const Vox &p = half ? pb : pa;
    if (!p.ok) continue;
    const long long v = v0 + g + 8 * half;
#pragma unroll
    for (int tile = 0; tile < 2; ++tile) {
      const float *acc = tile ? acc1 : acc0;
      const int co = 2 * q + 8 * tile;
      float r0 = acc[2 * half], r1 = acc[2 * half + 1];
      if (bias) {
        r0 += bias[co];
        r1 += bias[co + 1];
      }
      if (relu) {
        r0 = fmaxf(r0, 0.f);
        r1 = fmaxf(r1, 0.f);
      }
      if (mask) {
        const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(mask + v * kC + co);
        if (!(__bfloat162float(m.x) > 0.f)) r0 = 0.f;
        if (!(__bfloat162float(m.y) > 0.f)) r1 = 0.f;
      }
      *reinterpret_cast<__nv_bfloat162 *>(y + v * kC + co) = __floats2bfloat162_rn(r0, r1);
      if (yf && co == 0) yf[v] = r0;
    }
  }
}

// ---- tcgen05 implicit GEMM -------------------------------------------------
//
// One CTA: M = 128 consecutive voxels, N = 16 output channels, K = 27 taps x
// 16 input channels, in three phases of 9 taps (one z offset each).  Per
// phase all 256 threads gather the 9 A tiles (each voxel's neighbour row of
// 16 BF16 channels, zero outside) into shared memory in the canonical
// no-swizzle K-major layout of 8-row x 16-byte core matrices (K-adjacent core
// matrices 128 B apart, M-adjacent ones 256 B apart); one thread issues the 9
// tcgen05.mma (kind::f16, BF16 x BF16 -> FP32 in tensor memory) and commits
// them to an mbarrier; everyone waits (bounded) before the buffer is reused.
// The 27 B tiles (the layer's [tap][out][in] weights) are staged once.  After
// the last phase warps 0-3 and 4-7 read columns 0-7 and 8-15 of the 128 x 16
// accumulator with tcgen05.ld and apply the epilogue.  52 KB of shared
// memory: 4 CTAs per SM.  Tensor memory (32 columns) is allocated and freed
// by warp 0 on every path.
constexpr int kTcM = 128;
constexpr int kTcThreads = 256;
constexpr int kTcPhaseTaps = 9;
constexpr int kTcATile = kTcM * kC * 2;   // 4096 B per tap
constexpr int kTcBTile = kC * kC * 2;     // 512 B per tap
constexpr size_t kTcSmem = 1024 + (size_t)kTcPhaseTaps * kTcATile + (size_t)kTaps * kTcBTile + 64;

// Shared-memory matrix descriptor: start, leading (K) and stride (M/N) byte
// offsets >> 4, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor: FP32 accumulate, BF16 A and B, both K-major,
// N = 16, M = 128.
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kC >> 3) << 17) |
                              ((uint32_t)(kTcM >> 4) << 24);

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__global__ void __launch_bounds__(kTcThreads, 4)
conv_tc_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
               const float *__restrict__ bias, const __nv_bfloat16 *__restrict__ mask, int relu,
               __nv_bfloat16 *__restrict__ y, float *__restrict__ yf, Dims d, int *err) {
  extern __shared__ __align__(1024) unsigned char tc_raw[];
  unsigned char *smem = tc_raw + ((1024u - (smem_u32(tc_raw) & 1023u)) & 1023u);
  unsigned char *sa = smem;
  unsigned char *sb = sa + kTcPhaseTaps * kTcATile;
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sb + kTaps * kTcBTile);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long v0 = (long long)blockIdx.x * kTcM;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(
                     smem_u32(tslot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  // B tiles: row n (out channel) of 16 in-channels = two 16-byte halves
  for (int i = tid; i < kTaps * kC * 2; i += kTcThreads) {
    const int t = i / (kC * 2), n = (i / 2) % kC, c = i & 1;
    const uint4 v = *reinterpret_cast<const uint4 *>(w + (t * kC + n) * kC + c * 8);
    *reinterpret_cast<uint4 *>(sb + t * kTcBTile + (n >> 3) * 256 + c * 128 + (n & 7) * 16) = v;
  }
  // this thread's A row (voxel m, 16-byte half c) and its neighbour bounds
  const int m = tid & (kTcM - 1), c = tid >> 7;
  const Vox p = vox_of(v0 + m, d);
  const long long vm = v0 + m;
  const long long YX = (long long)d.Y * d.X;
  const bool ylo = p.y > 0, yhi = p.y < d.Y - 1, xlo = p.x > 0, xhi = p.x < d.X - 1;
  unsigned char *dst = sa + (m >> 3) * 256 + c * 128 + (m & 7) * 16;
  const __nv_bfloat16 *src = x + vm * kC + c * 8;

  bool ok = true;
  uint32_t tmem = 0;
  for (int g = 0; g < 3; ++g) {
    const int dz = g - 1;
    const bool zok = p.ok && (dz < 0 ? p.z > 0 : (dz > 0 ? p.z < d.Z - 1 : true));
#pragma unroll
    for (int k = 0; k < kTcPhaseTaps; ++k) {
      const int dy = k / 3 - 1, dx = k % 3 - 1;
      const bool in = zok && (dy < 0 ? ylo : (dy > 0 ? yhi : true)) &&
                      (dx < 0 ? xlo : (dx > 0 ? xhi : true));
      uint4 v = make_uint4(0, 0, 0, 0);
      if (in) v = *reinterpret_cast<const uint4 *>(src + (dz * YX + dy * d.X + dx) * kC);
      *reinterpret_cast<uint4 *>(dst + k * kTcATile) = v;
    }
    // make the generic-proxy writes visible to the tensor core (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = *tslot;
    if (tid == 0) {
      const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
      for (int k = 0; k < kTcPhaseTaps; ++k) {
        const int t = g * kTcPhaseTaps + k;
        const uint64_t ad = umma_desc(a0 + k * kTcATile, 128, 256);
        const uint64_t bd = umma_desc(b0 + t * kTcBTile, 128, 256);
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(kTcIdesc), "r"((uint32_t)(t > 0))
            : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              smem_u32(bar))
          : "memory");
    }
    // the A buffer is reused by the next phase only after these MMAs are done
    if (!mbar_wait(bar, (uint32_t)(g & 1), err)) ok = false;
    tc_fence_after();
  }
  // epilogue: warp quadrant q = rows 32q..32q+31, column half h
  {
    const int q = warp & 3, h = warp >> 2;
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(8 * h)));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    const long long v = v0 + 32 * q + lane;
    if (ok && v < d.nvox) {
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int co = 8 * h + i;
        float a = __uint_as_float(r[i]);
        if (bias) a += bias[co];
        if (relu) a = fmaxf(a, 0.f);
        if (mask && !(__bfloat162float(mask[v * kC + co]) > 0.f)) a = 0.f;
        f[i] = a;
      }
      uint4 o;
      __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) ob[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      *reinterpret_cast<uint4 *>(y + v * kC + 8 * h) = o;
      if (yf && h == 0) yf[v] = f[0];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem)
                 : "memory");
  }
}

// ---- padded slabs ---------------------------------------------------------------
//
// The kernels below stage a slab of z planes of one instance as zero-padded
// planes: rows of X + 1 voxels, Y + 1 rows, the last column and row zero, so
// that the neighbour of padded voxel m at tap (dz, dy, dx) is voxel
// m + dz P + dy (X + 1) + dx (P = (Y + 1)(X + 1)) whatever m is: one voxel's
// left pad is the previous row's last column.  A slab arrives as one TMA box
// per 8-channel half of [batch, z, y, x, channel]; TMA fills what lies
// outside the tensor with zeros, which is the padding.  A half plane holds 16
// bytes per voxel, so a tap of 8 or 128 consecutive voxels is contiguous
// shared memory at a shifted start address: nothing is gathered per tap.
struct PadGeom {
  int px, P;       // row and plane pitch in padded voxels
  int zs, nslab;   // planes per slab, slabs per instance
  int pre;         // bytes in front of a half plane (zeros: the first row's upper-left taps)
};

// Planes per slab: at most zmax, fewer while there are not `want` slabs,
// then evened out over the slabs of an instance.
PadGeom pad_geom(const Dims &d, int zmax, long long want) {
  PadGeom g;
  g.px = d.X + 1;
  g.P = (d.Y + 1) * g.px;
  g.pre = ((g.px + 1) * 16 + 127) / 128 * 128;
  const long long spread = ((long long)d.B * d.Z + want - 1) / want;
  int zs = zmax < d.Z ? zmax : d.Z;
  if (spread < zs) zs = (int)spread;
  g.nslab = (d.Z + zs - 1) / zs;
  g.zs = (d.Z + g.nslab - 1) / g.nslab;
  g.nslab = (d.Z + g.zs - 1) / g.zs;
  return g;
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, int c, int x,
                                            int y, int z, int b, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c), "r"(x), "r"(y), "r"(z), "r"(b),
      "r"(bar)
      : "memory");
}

// ---- tcgen05 convolution over padded slabs --------------------------------------
//
// As conv_tc_kernel (M = 128, N = 16, 27 taps of K = 16 in the same order, so
// the same bits), with the A operand of every tap read straight from the
// padded half planes: tap t of 128 consecutive padded voxels is the no-swizzle
// K-major matrix whose 8-voxel core matrices lie 128 bytes apart and whose two
// 8-channel halves one half plane apart, at a start address shifted by the
// tap.  Rows that are padding compute values nobody stores (19 % of 9 x 9
// planes).  Warp 4 issues the TMA boxes and all MMAs, one commit per tile of
// 128; warps 0-3 read each finished tile's 16 accumulator columns and apply
// the epilogue while later tiles are still running.
// Bound: every MMA reads its 4 KB A tile from shared memory, 27 * 32 cycles
// per 128 voxels (46 us of the case below).  Measured on 1024 x 17 x 9 x 9
// voxels: 73 us (267 TFLOP/s, tensor pipe 86 % active) against 187 us of
// conv_tc_kernel, which gathers every tap's tile through registers; on 32
// instances 9.6 against 12.5 us.
constexpr int kPcThreads = 160;
constexpr int kPcMaxTiles = 8;                     // 8 x 16 accumulator columns
constexpr int kPcCols = kPcMaxTiles * kC;          // tensor memory columns
constexpr int kPcHead = 256;                       // barriers, tensor memory address, bias
constexpr int kPcB = kTaps * kTcBTile;             // weights
constexpr size_t kPcMinSmem = 46 * 1024;           // at most 4 CTAs x 128 columns per SM

__host__ __device__ constexpr int pc_tiles(int zs, int P) { return (zs * P + kTcM - 1) / kTcM; }
// Bytes of one half plane: the zeros in front, then every row a tile's taps read.
__host__ __device__ constexpr int pc_half(int zs, int P, int px, int pre) {
  return pre + ((pc_tiles(zs, P) * kTcM + 2 * P + px + 1) * 16 + 127) / 128 * 128;
}
// The largest pc_smem: 1024 rows of tiles, planes of up to 1024 voxels in rows of
// up to 256.  The kernel is always allowed this much, not each launch's own size,
// which another thread's launch could lower in between.
constexpr size_t kPcMaxSmem =
    128 + kPcHead + kPcB + 2 * (size_t)(257 * 16 + 112 + (1024 + 2 * 1024 + 257) * 16 + 112);
size_t pc_smem(const PadGeom &g) {
  const size_t n = 128 + kPcHead + kPcB + 2 * (size_t)pc_half(g.zs, g.P, g.px, g.pre);
  return n < kPcMinSmem ? kPcMinSmem : n;
}

__global__ void __launch_bounds__(kPcThreads)
conv_pad_kernel(const __grid_constant__ CUtensorMap tmx, const __nv_bfloat16 *w,
                const float *bias, const __nv_bfloat16 *mask, int relu, __nv_bfloat16 *y,
                float *yf, Dims d, PadGeom g, int *err) {
  extern __shared__ __align__(128) unsigned char pc_raw[];
  unsigned char *smem = pc_raw + ((128u - (smem_u32(pc_raw) & 127u)) & 127u);
  unsigned long long *bars = reinterpret_cast<unsigned long long *>(smem);  // load, tiles
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + 128);
  float *sbias = reinterpret_cast<float *>(smem + 192);
  unsigned char *sb = smem + kPcHead;
  unsigned char *sx = sb + kPcB;
  const int half = pc_half(g.zs, g.P, g.px, g.pre);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x / g.nslab;
  const int z0 = (blockIdx.x - b * g.nslab) * g.zs;
  const int nz = min(g.zs, d.Z - z0);
  const int rows = nz * g.P;
  const int ntiles = (rows + kTcM - 1) / kTcM;

  if (warp == 4) {
    if (lane == 0) {
      for (int i = 0; i <= kPcMaxTiles; ++i) mbar_init(&bars[i], 1);
      fence_barrier_init();
    }
    wait_for_predecessors();
    if (lane == 0) {
      // planes z0 - 1 .. z0 + zs of both halves
      mbar_arrive_expect_tx(&bars[0], 2u * (unsigned)((g.zs + 2) * g.P * 16));
      for (int h = 0; h < 2; ++h)
        tma_load_5d(smem_u32(sx + h * half + g.pre), &tmx, 8 * h, 0, 0, z0 - 1, b,
                    smem_u32(&bars[0]));
    }
    __syncwarp();
    // after the wait: columns held while waiting could be ones that the kernel
    // waited for, the caller's own, has yet to allocate
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(kPcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    wait_for_predecessors();
    // weights: out channel n's 16 in-channels as two 16-byte halves
    for (int i = tid; i < kTaps * kC * 2; i += 128) {
      const int t = i / (kC * 2), n = (i / 2) % kC, c = i & 1;
      const uint4 v = *reinterpret_cast<const uint4 *>(w + (t * kC + n) * kC + c * 8);
      *reinterpret_cast<uint4 *>(sb + t * kTcBTile + (n >> 3) * 256 + c * 128 + (n & 7) * 16) = v;
    }
    for (int i = tid; i < g.pre / 8; i += 128)
      *reinterpret_cast<uint4 *>(sx + (i >= g.pre / 16 ? half - g.pre : 0) + i * 16) =
          make_uint4(0u, 0u, 0u, 0u);
    if (tid < kC) sbias[tid] = bias ? bias[tid] : 0.f;
    // generic-proxy writes visible to the tensor core (async proxy)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;

  if (warp == 4) {
    if (lane == 0) {
      const bool ok = mbar_wait(&bars[0], 0, err);
      const uint32_t a0 = smem_u32(sx) + g.pre, b0 = smem_u32(sb);
      for (int i = 0; i < ntiles && ok; ++i) {
        // row m of the tile is padded voxel m of the slab's first own plane,
        // one plane into the staged ones
        const uint32_t base = a0 + i * kTcM * 16;
#pragma unroll
        for (int t = 0; t < kTaps; ++t) {
          const int dz = t / 9, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
          const uint64_t ad = umma_desc(base + (dz * g.P + dy * g.px + dx) * 16, half, 128);
          const uint64_t bd = umma_desc(b0 + t * kTcBTile, 128, 256);
          asm volatile(
              "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem + i * kC),
              "l"(ad), "l"(bd), "r"(kTcIdesc), "r"((uint32_t)(t > 0))
              : "memory");
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&bars[1 + i]))
            : "memory");
      }
    }
    __syncwarp();
  } else {
    const long long vox0 = ((long long)b * d.Z + z0) * d.Y * d.X;
    // padded voxel of this thread's row: coordinates advanced by 128 per tile
    int m = tid;
    int zz = m / g.P, r = m - zz * g.P;
    int yy = r / g.px, xx = r - yy * g.px;
    const int sz = kTcM / g.P, sr = kTcM - sz * g.P, sy = sr / g.px, sxx = sr - sy * g.px;
    for (int i = 0; i < ntiles; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bars[1 + i], 0, err))) break;
      tc_fence_after();
      uint32_t a[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
          "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]),
            "=r"(a[7]), "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]),
            "=r"(a[13]), "=r"(a[14]), "=r"(a[15])
          : "r"(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(i * kC)));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (zz < nz && yy < d.Y && xx < d.X) {
        const long long v = vox0 + ((long long)zz * d.Y + yy) * d.X + xx;
        float f[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          f[k] = __uint_as_float(a[k]);
          if (bias) f[k] += sbias[k];
          if (relu) f[k] = fmaxf(f[k], 0.f);
        }
        if (mask) {
          uint4 mv[2];
          mv[0] = *reinterpret_cast<const uint4 *>(mask + v * kC);
          mv[1] = *reinterpret_cast<const uint4 *>(mask + v * kC + 8);
          const __nv_bfloat16 *mb = reinterpret_cast<const __nv_bfloat16 *>(mv);
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (!(__bfloat162float(mb[k]) > 0.f)) f[k] = 0.f;
        }
        uint4 o[2];
        __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(o);
#pragma unroll
        for (int k = 0; k < 8; ++k) ob[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
        *reinterpret_cast<uint4 *>(y + v * kC) = o[0];
        *reinterpret_cast<uint4 *>(y + v * kC + 8) = o[1];
        if (yf) yf[v] = f[0];
      }
      xx += sxx;
      yy += sy;
      zz += sz;
      if (xx >= g.px) {
        xx -= g.px;
        ++yy;
      }
      if (yy > d.Y) {
        yy -= d.Y + 1;
        ++zz;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kPcCols)
                 : "memory");
  }
}

// ---- weight gradient -----------------------------------------------------------
//
// dW[t][in][out] = sum over voxels v of X[v + d_t][in] * dY[v][out]: a GEMM
// per tap with M = N = 16 and K = voxels.  M = 16 is below tcgen05's smallest
// tile, so the products run on mma.sync.m16n8k16.
//
// CTAs (g, s) make the nine taps of z offset g - 1 for split s.  Split s takes
// every S-th run of 128 voxels; its warp w the w-th 16 of each run, in ascending
// order, so each FP32 accumulator sees the products in the order that
// wgrad_kernel gives them, and the results are the same bits (a training run is
// sensitive to the last one: it decides BF16 roundings of the weights).  X rows
// of a run and of its y and x neighbours are one contiguous stretch of memory
// (three, one per y offset, where rows of the grid are longer than a run); they
// and the run's dY rows arrive by cp.async, three runs ahead.  They sit in two
// planes of 8-channel halves, so the eight 16-byte rows of an ldmatrix phase
// are 128 contiguous bytes (no bank conflicts); ldmatrix.trans turns
// [voxel][channel] rows into K = voxel fragments.  A lane follows the
// coordinates of the voxel whose row it hands to ldmatrix, and hands it a row
// of zeros where the tap leaves the grid.
// Bound: 54 products per 16 voxels, about 10 cycles each on a sub-partition's
// mma.sync pipe (40 us of the case below were the CTAs even over the SMs).
// Measured, 1024 x 17 x 9 x 9 voxels, 64 splits: 135 us (167 with eight-warp
// CTAs; wgrad_kernel, two-byte gathers from L2 for every tap, 1760); 32
// instances 13 us (60).
// A split's eight warps are two CTAs of four (a cluster, whose sums are added
// through distributed shared memory): 384 of them even out better over the SMs
// than 192 of eight.
constexpr int kWgHalves = 2;
constexpr int kWgWarps = kConvWarps / kWgHalves;
constexpr int kWgThreads = 32 * kWgWarps;
constexpr int kWgRun = 16 * kWgWarps;     // voxels of a CTA's half run
constexpr int kWgStages = 4;

// Staging of a run's X rows: `segs` stretches of `len` rows, a tap's y offset
// being `pitch` staged rows.
struct WgRows {
  int segs, len, pitch;
};
__host__ __device__ inline WgRows wg_rows(int X) {
  const int run = kWgRun + 2;
  return X <= run ? WgRows{1, run + 2 * X, X} : WgRows{3, run, run};
}
__host__ __device__ inline int wg_stage_bytes(const WgRows &r) {
  return (r.segs * r.len + kWgRun) * 32;
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ void cp_async16_to(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
               "l"(__cvta_generic_to_global(src))
               : "memory");
}

__global__ void __cluster_dims__(kWgHalves, 1, 1) __launch_bounds__(kWgThreads, 4)
wgrad_run_kernel(const __nv_bfloat16 *x, const __nv_bfloat16 *dy, float *part, float *bpart, Dims d,
                 WgRows rows) {
  extern __shared__ __align__(128) unsigned char wg_smem[];
  __shared__ float bred[kWgWarps][kC];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = blockIdx.x / kWgHalves, half = blockIdx.x % kWgHalves;
  const int s = blockIdx.y, S = gridDim.y;
  const int dz = g - 1;
  const long long YX = (long long)d.Y * d.X;
  constexpr int kFull = kWgHalves * kWgRun;
  const long long runs = (d.nvox + kFull - 1) / kFull;
  const int n = s < runs ? (int)((runs - s + S - 1) / S) : 0;  // this split's runs
  const int XR = rows.segs * rows.len;                          // staged X rows
  const uint32_t sbytes = wg_stage_bytes(rows);
  const uint32_t zero_row = smem_u32(wg_smem), sm0 = zero_row + 16;
  if (tid < 4) reinterpret_cast<uint32_t *>(wg_smem)[tid] = 0u;
  wait_for_predecessors();

  // Staging: 16-byte unit i of a stretch is half i & 1 of row i >> 1.  Rows
  // outside the tensor are left alone (no lane reads them).
  const uint32_t xdst = ((tid & 1) * XR + (tid >> 1)) * 16;
  const uint32_t ydst = XR * 32 + ((tid & 1) * kWgRun + (tid >> 1)) * 16;
  const long long hop = (long long)S * kFull;  // voxels from one run to the next
  const long long v_first = (long long)s * kFull + half * kWgRun;
  long long v_next = v_first;  // first voxel of the next run to stage
  const char *ysrc = reinterpret_cast<const char *>(dy) + v_next * 32 + tid * 16;
  long long x_next = v_next + dz * YX - d.X - 1;  // its first X row
  const char *xsrc = reinterpret_cast<const char *>(x) + x_next * 32 + tid * 16;
  auto load = [&](int stage) {
    uint32_t dst = sm0 + stage * sbytes;
    const bool whole = x_next >= 0 && v_next + kWgRun <= d.nvox &&
                       x_next + (long long)(rows.segs - 1) * d.X + rows.len <= d.nvox;
    if (whole || v_next + (tid >> 1) < d.nvox) cp_async16_to(dst + ydst, ysrc);
    dst += xdst;
    const char *src = xsrc;
    if (whole) {
      // 132 units or more: one per thread, one more for some, rarely others
      const int units = 2 * rows.len;
      for (int sg = 0; sg < rows.segs; ++sg) {
        cp_async16_to(dst, src);
        if (tid + kWgThreads < units) cp_async16_to(dst + kWgThreads * 8, src + kWgThreads * 16);
#pragma unroll 1
        for (int i = tid + 2 * kWgThreads; i < units; i += kWgThreads)
          cp_async16_to(dst + (i - tid) * 8, src + (i - tid) * 16);
        dst += rows.len * 16;
        src += (long long)d.X * 32;
      }
    } else {
      long long row = x_next;
#pragma unroll 1
      for (int sg = 0; sg < rows.segs; ++sg) {
#pragma unroll 1
        for (int i = tid; i < 2 * rows.len; i += kWgThreads) {
          const long long k = row + (i >> 1);
          if (k >= 0 && k < d.nvox) cp_async16_to(dst + (i - tid) * 8, src + (i - tid) * 16);
        }
        dst += rows.len * 16;
        src += (long long)d.X * 32;
        row += d.X;
      }
    }
    v_next += hop;
    x_next += hop;
    ysrc += hop * 32;
    xsrc += hop * 32;
  };

  // This lane's row of an ldmatrix.x4: voxel lv of its warp's 16, channel half
  // lh.  Coordinates of that voxel, advanced by S runs at a time.
  const int lv = (lane & 7) + ((lane >> 4) << 3), lh = (lane >> 3) & 1;
  long long v = v_first + warp * 16 + lv;
  int cx, cy, cz;
  {
    const long long q = v / d.X;
    cx = (int)(v - q * d.X);
    cy = (int)(q % d.Y);
    cz = (int)((q / d.Y) % d.Z);
  }
  const int sx = (int)(hop % d.X), sy = (int)((hop / d.X) % d.Y), sz = (int)((hop / YX) % d.Z);
  const uint32_t xrow = (lh * XR + warp * 16 + lv) * 16;
  const uint32_t yrow = XR * 32 + (lh * kWgRun + warp * 16 + lv) * 16;
  const uint32_t ypitch = rows.pitch * 16;

  float acc[9][2][4] = {};
  float bsum0 = 0.f, bsum1 = 0.f;
#pragma unroll
  for (int t = 0; t < kWgStages - 1; ++t) {
    if (t < n) load(t);
    cp_async_commit();
  }
  int stage = 0, fill = kWgStages - 1;
  for (int t = 0; t < n; ++t) {
    cp_async_wait<kWgStages - 2>();
    __syncthreads();  // the run has landed; the stage read a run ago is free
    if (t + kWgStages - 1 < n) load(fill);
    cp_async_commit();
    if (++fill == kWgStages) fill = 0;
    const uint32_t st = sm0 + stage * sbytes;
    if (++stage == kWgStages) stage = 0;

    const bool in = v < d.nvox;
    const bool z = in && (unsigned)(cz + dz) < (unsigned)d.Z;
    const bool yok[3] = {z && cy > 0, z, z && cy < d.Y - 1};
    const bool xok[3] = {cx > 0, true, cx < d.X - 1};
    uint32_t b[4];
    ldmatrix_x4_trans(b, in ? st + yrow : zero_row);
    uint32_t xa = st + xrow;
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      uint32_t a[3][4];
#pragma unroll
      for (int k = 0; k < 3; ++k)
        ldmatrix_x4_trans(a[k], yok[ky] && xok[k] ? xa + 16 * k : zero_row);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        mma_16816(acc[ky * 3 + k][0], a[k], b[0], b[2]);
        mma_16816(acc[ky * 3 + k][1], a[k], b[1], b[3]);
      }
      xa += ypitch;
    }
    if (g == 1) {
      const uint32_t bb[4] = {b[0], b[2], b[1], b[3]};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float lo = __uint_as_float(bb[i] << 16), hi = __uint_as_float(bb[i] & 0xffff0000u);
        if (i < 2) bsum0 += lo + hi;
        else bsum1 += lo + hi;
      }
    }
    v += hop;
    cx += sx;
    cy += sy;
    cz += sz;
    if (cx >= d.X) {
      cx -= d.X;
      ++cy;
    }
    if (cy >= d.Y) {
      cy -= d.Y;
      ++cz;
    }
    if (cz >= d.Z) cz -= d.Z;
  }
  cp_async_wait<0>();  // only empty groups can remain

  // warps' sums, added in warp order over the cluster, three taps at a time
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  float *red = reinterpret_cast<float *>(wg_smem);
  constexpr int kSums = 3 * kC * kC;
  const int gq = lane >> 2, q = lane & 3;
  bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, 1);
  bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, 2);
  bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, 1);
  bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, 2);
  if (q == 0) {
    bred[warp][gq] = bsum0;
    bred[warp][gq + 8] = bsum1;
  }
#pragma unroll
  for (int ky = 0; ky < 3; ++ky) {
    if (ky == 0) __syncthreads();  // the stages are free
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<float2 *>(red + warp * kSums + k * kC * kC + (gq + i * 8) * kC +
                                      m * 8 + 2 * q) =
              make_float2(acc[ky * 3 + k][m][2 * i], acc[ky * 3 + k][m][2 * i + 1]);
    cl.sync();
    for (int i = tid + half * kWgThreads; i < kSums; i += kWgHalves * kWgThreads) {
      float f = 0.f;
#pragma unroll
      for (int r = 0; r < kWgHalves; ++r) {
        const float *from = cl.map_shared_rank(red, r);
#pragma unroll
        for (int w = 0; w < kWgWarps; ++w) f += from[w * kSums + i];
      }
      part[((long long)s * kTaps + g * 9 + ky * 3) * kC * kC + i] = f;
    }
    if (ky == 0 && g == 1 && half == 0 && tid < kC) {
      float f = 0.f;
      for (int r = 0; r < kWgHalves; ++r) {
        const float *from = cl.map_shared_rank(&bred[0][0], r);
        for (int w = 0; w < kWgWarps; ++w) f += from[w * kC + tid];
      }
      bpart[s * kC + tid] = f;
    }
    cl.sync();  // read before it is overwritten, or the CTA leaves
  }
}

// Partial weight gradients: block (t, s) sums over the s-th share of the
// 16-voxel chunks dW[t][in][out] = sum_v X[v + d_t][in] * dY[v][out] into
// part[s][t][in][out]; blocks of the centre tap also sum dY into
// bpart[s][out] (the bias gradient).
__global__ void __launch_bounds__(32 * kConvWarps)
wgrad_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy,
             float *__restrict__ part, float *__restrict__ bpart, Dims d) {
  __shared__ float red[kConvWarps][kC * kC];
  __shared__ float bred[kConvWarps][kC];
  const int t = blockIdx.x, s = blockIdx.y, S = gridDim.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};
  float bsum0 = 0.f, bsum1 = 0.f;
  const long long nchunks = (d.nvox + 15) / 16;
  for (long long c = (long long)s * kConvWarps + warp; c < nchunks; c += (long long)S * kConvWarps) {
    const long long k0 = c * 16 + 2 * q;  // this lane's voxels: k0, k0+1, k0+8, k0+9
    const long long vk[4] = {k0, k0 + 1, k0 + 8, k0 + 9};
    long long nb[4], dv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const Vox p = vox_of(vk[i], d);
      nb[i] = nbr(p, t, d);
      dv[i] = p.ok ? vk[i] : -1;
    }
    // A = X^T (rows in-channel, k voxel)
    const uint32_t a[4] = {pack2(x, nb[0], nb[1], g), pack2(x, nb[0], nb[1], g + 8),
                           pack2(x, nb[2], nb[3], g), pack2(x, nb[2], nb[3], g + 8)};
    // B = dY (k voxel, n out-channel)
    const uint32_t b00 = pack2(dy, dv[0], dv[1], g), b01 = pack2(dy, dv[2], dv[3], g);
    const uint32_t b10 = pack2(dy, dv[0], dv[1], g + 8), b11 = pack2(dy, dv[2], dv[3], g + 8);
    mma_16816(acc0, a, b00, b01);
    mma_16816(acc1, a, b10, b11);
    if (t == 13) {
      const uint32_t bb[4] = {b00, b01, b10, b11};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float lo = __uint_as_float(bb[i] << 16), hi = __uint_as_float(bb[i] & 0xffff0000u);
        if (i < 2) bsum0 += lo + hi;
        else bsum1 += lo + hi;
      }
    }
  }
  // C tile layout: (row in g / g+8, col out 2q, 2q+1 [+8 for tile 1])
#pragma unroll
  for (int tile = 0; tile < 2; ++tile) {
    const float *acc = tile ? acc1 : acc0;
    const int co = 2 * q + 8 * tile;
    red[warp][g * kC + co] = acc[0];
    red[warp][g * kC + co + 1] = acc[1];
    red[warp][(g + 8) * kC + co] = acc[2];
    red[warp][(g + 8) * kC + co + 1] = acc[3];
  }
  bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, 1);
  bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, 2);
  bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, 1);
  bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, 2);
  if (q == 0) {
    bred[warp][g] = bsum0;
    bred[warp][g + 8] = bsum1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kC * kC; i += blockDim.x) {
    float v = 0.f;
    for (int w = 0; w < kConvWarps; ++w) v += red[w][i];
    part[((long long)s * kTaps + t) * kC * kC + i] = v;
  }
  if (t == 13 && threadIdx.x < kC) {
    float v = 0.f;
    for (int w = 0; w < kConvWarps; ++w) v += bred[w][threadIdx.x];
    bpart[s * kC + threadIdx.x] = v;
  }
}

// Sums the splits' partials in split order: 64 gradients per CTA, four threads
// fetching each one's partials of 64 splits, one adding them (one thread
// walking through memory took 5.1 us for 64 splits).
__global__ void __launch_bounds__(256)
wgrad_reduce_kernel(const float *part, const float *bpart, int S, float *dw, float *db) {
  wait_for_predecessors();
  __shared__ float buf[64][65];
  const int c = threadIdx.x & 63, k = threadIdx.x >> 6;
  const int i = blockIdx.x * 64 + c;
  const int n = kTaps * kC * kC;
  const bool on = i < n || (i < n + kC && db);
  const float *src = i < n ? part + i : bpart + (i - n);
  const int step = i < n ? n : kC;
  float v = 0.f;
  for (int s0 = 0; s0 < S; s0 += 64) {
    float u[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int s = s0 + k * 16 + j;
      u[j] = on && s < S ? src[(long long)s * step] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) buf[k * 16 + j][c] = u[j];
    __syncthreads();
    if (on && k == 0) {
      const int m = min(64, S - s0);
      if (m == 64) {
#pragma unroll
        for (int j = 0; j < 64; ++j) v += buf[j][c];
      } else {
        for (int j = 0; j < m; ++j) v += buf[j][c];
      }
    }
    __syncthreads();
  }
  if (!on || k) return;
  if (i < n) dw[i] = v;
  else db[i - n] = v;
}

// FP32 master [27][in][out] -> BF16 forward [27][out][in] and backward-data
// [27][in][out] with taps reversed (the adjoint convolution).
__global__ void prep_weights_kernel(const float *w, __nv_bfloat16 *wf, __nv_bfloat16 *wb) {
  wait_for_predecessors();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kTaps * kC * kC) return;
  const int t = i / (kC * kC), ci = (i / kC) % kC, co = i % kC;
  const __nv_bfloat16 v = __float2bfloat16_rn(w[i]);
  wf[(t * kC + co) * kC + ci] = v;
  wb[((kTaps - 1 - t) * kC + ci) * kC + co] = v;
}

// One Adam update (Kingma & Ba 2015) with bias corrections c1 = 1/(1 - b1^t),
// c2 = 1/(1 - b2^t); returns the new weight.
__device__ __forceinline__ float adam_step(float w, float gi, float &m, float &v, float lr,
                                           float b1, float b2, float eps, float c1, float c2) {
  const float mi = b1 * m + (1.f - b1) * gi;
  const float vi = b2 * v + (1.f - b2) * gi * gi;
  m = mi;
  v = vi;
  return w - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ g,
                            float *__restrict__ m, float *__restrict__ v, long long n, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  w[i] = adam_step(w[i], g[i], m[i], v[i], lr, b1, b2, eps, c1, c2);
}

// The Adam step of a whole network (layers x [27][in][out] weights, then
// layers x 16 biases) and the BF16 copies of its new weights: what twelve
// adam_kernel and six prep_weights_kernel launches of 3 us each did for six
// layers, latency-bound at 1.7 MB of traffic, in one.
__global__ void adam_layers_kernel(float *w, const float *g, float *m, float *v, int layers, float lr,
                                   float b1, float b2, float eps, float c1, float c2,
                                   __nv_bfloat16 *wf, __nv_bfloat16 *wb) {
  wait_for_predecessors();
  constexpr int per = kTaps * kC * kC;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= layers * (per + kC)) return;
  const float nw = adam_step(w[i], g[i], m[i], v[i], lr, b1, b2, eps, c1, c2);
  w[i] = nw;
  if (i >= layers * per) return;
  const int l = i / per, k = i - l * per;
  const int t = k / (kC * kC), ci = (k / kC) % kC, co = k % kC;
  const __nv_bfloat16 h = __float2bfloat16_rn(nw);
  wf[l * per + (t * kC + co) * kC + ci] = h;
  wb[l * per + ((kTaps - 1 - t) * kC + ci) * kC + co] = h;
}

// dY (channel 0) = 2 (pred - target) / n; per-block FP64 sums of the
// squared error in part[blockIdx.x].
__global__ void mse_kernel(const float *pred, const float *tgt, long long n, __nv_bfloat16 *dy,
                           double *part) {
  wait_for_predecessors();
  __shared__ double red[256];
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double e2 = 0.0;
  if (i < n) {
    const float e = pred[i] - tgt[i];
    e2 = (double)e * (double)e;
    uint4 z = make_uint4(0, 0, 0, 0);
    uint4 *row = reinterpret_cast<uint4 *>(dy + i * kC);
    row[0] = z;
    row[1] = z;
    dy[i * kC] = __float2bfloat16_rn(2.f * e / (float)n);
  }
  red[threadIdx.x] = e2;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// Fine stacked grids -> coarse network input.  Instance b sits at fine
// origin ((b % nsx) * inx, 0, (b / nsx) * inz) of float grids with row pitch
// `pitch` bytes and ny rows per plane; coarse cell (zc, yc, xc) averages the
// fine cells [zc f, zc f + f) x ... inside the instance.
//
// `flip` selects one of the 16 mirror images of an instance that are
// instances of the same problem family: bit 0/1/2 mirror x/y/z, bit 3 swaps
// x and y (with a2 and a1, the x and y coefficients; needs inx == iny).  The 19-point operator with
// c_i = a_i and b = 0 weighs both neighbours of a cell along an axis with
// that cell's own a_i, and the Dirichlet faces are symmetric, so the mirrored
// fields' solution is the mirrored solution: one solve gives 16 training
// pairs.  Coordinates below are those of the mirror image; vmap takes them
// back to the stored instance.
struct PoolArgs {
  const float *a0, *a1, *a2, *wrk1, *bnd, *p;
  long long pitch_e;  // row pitch in floats
  int ny;             // rows per plane of the stacked grids
  int inx, iny, inz;  // instance size
  int nsx;            // instances along x
  int f;              // pooling factor
  int zc, yc, xc;     // coarse size
  int batch;
  int flip;
  float wscale, pscale;
  const float *inst_scale;  // per-instance source/solution scale (NULL: 1)
  const float *p_sub;       // pool_target: subtract this grid from p (NULL: none)
};

__device__ __forceinline__ float inst_scale_of(const PoolArgs &a, int b) {
  return a.inst_scale ? a.inst_scale[b] : 1.f;
}

__device__ __forceinline__ long long fine_index(const PoolArgs &a, int b, int z, int y, int x) {
  const int ox = (b % a.nsx) * a.inx, oz = (b / a.nsx) * a.inz;
  return ((long long)(oz + z) * a.ny + y) * a.pitch_e + ox + x;
}

// Index of mirror-image cell (z, y, x) of instance b in the stored grids.
__device__ __forceinline__ long long vmap(const PoolArgs &a, int b, int z, int y, int x) {
  if (a.flip & 1) x = a.inx - 1 - x;
  if (a.flip & 2) y = a.iny - 1 - y;
  if (a.flip & 4) z = a.inz - 1 - z;
  if (a.flip & 8) {
    const int t = x;
    x = y;
    y = t;
  }
  return fine_index(a, b, z, y, x);
}

// Channels (means over the block): 0-2 ln a0, ln a1, ln a2; 3 wrk1 * wscale;
// 4 bnd; 5 wrk1 * 3 / (a0 + a1 + a2) * wscale (the source over the local
// coefficient, whose block mean the means of wrk1 and a do not give);
// 6-8 -ln mean(1 / a_i) (log harmonic means: a block's series
// conductance); 9-15 zeros.  a1/a2 are those of the mirror image.
__global__ void pool_inputs_kernel(PoolArgs a, __nv_bfloat16 *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)a.batch * a.zc * a.yc * a.xc;
  if (i >= n) return;
  const int xc = (int)(i % a.xc), yc = (int)((i / a.xc) % a.yc);
  const int zc = (int)((i / ((long long)a.xc * a.yc)) % a.zc);
  const int b = (int)(i / ((long long)a.xc * a.yc * a.zc));
  // a0 weighs the z neighbours, a1 the y and a2 the x neighbours
  const float *ay = (a.flip & 8) ? a.a2 : a.a1;
  const float *ax = (a.flip & 8) ? a.a1 : a.a2;
  float s[kPoolChannels] = {};
  int cnt = 0;
  for (int z = zc * a.f; z < min(zc * a.f + a.f, a.inz); ++z)
    for (int y = yc * a.f; y < min(yc * a.f + a.f, a.iny); ++y)
      for (int x = xc * a.f; x < min(xc * a.f + a.f, a.inx); ++x) {
        const long long k = vmap(a, b, z, y, x);
        const float c0 = a.a0[k], c1 = ay[k], c2 = ax[k], w = a.wrk1[k];
        s[0] += logf(c0);
        s[1] += logf(c1);
        s[2] += logf(c2);
        s[3] += w;
        s[4] += a.bnd[k];
        s[5] += w * 3.f / (c0 + c1 + c2);
        s[6] += 1.f / c0;
        s[7] += 1.f / c1;
        s[8] += 1.f / c2;
        ++cnt;
      }
  const float inv = 1.f / (float)cnt;
  const float ws = a.wscale * inst_scale_of(a, b);
  __nv_bfloat16 *row = out + i * kC;
  row[0] = __float2bfloat16_rn(s[0] * inv);
  row[1] = __float2bfloat16_rn(s[1] * inv);
  row[2] = __float2bfloat16_rn(s[2] * inv);
  row[3] = __float2bfloat16_rn(s[3] * inv * ws);
  row[4] = __float2bfloat16_rn(s[4] * inv);
  row[5] = __float2bfloat16_rn(s[5] * inv * ws);
  for (int c = 6; c < 9; ++c) row[c] = __float2bfloat16_rn(-logf(s[c] * inv));
  for (int c = kPoolChannels; c < kC; ++c) row[c] = __float2bfloat16_rn(0.f);
}

// Training target: p at each block's centre (c + 0.5) f - 0.5, the mean of
// the fine cells nearest to it (two per axis for even f), times pscale; in
// the mirror image's coordinates.
__global__ void pool_target_kernel(PoolArgs a, float *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)a.batch * a.zc * a.yc * a.xc;
  if (i >= n) return;
  const int xc = (int)(i % a.xc), yc = (int)((i / a.xc) % a.yc);
  const int zc = (int)((i / ((long long)a.xc * a.yc)) % a.zc);
  const int b = (int)(i / ((long long)a.xc * a.yc * a.zc));
  // nearest fine cells to the centre: lo = floor, hi = ceil of (c + 0.5) f - 0.5
  auto near = [&](int c, int nf, int &lo, int &hi) {
    lo = min((2 * c * a.f + a.f - 1) / 2, nf - 1);
    hi = min((2 * c * a.f + a.f) / 2, nf - 1);
  };
  int z0, z1, y0, y1, x0, x1;
  near(zc, a.inz, z0, z1);
  near(yc, a.iny, y0, y1);
  near(xc, a.inx, x0, x1);
  const int zs[2] = {z0, z1}, ys[2] = {y0, y1}, xs[2] = {x0, x1};
  float s = 0.f;
  for (int k = 0; k < 2; ++k)
    for (int j = 0; j < 2; ++j)
      for (int m = 0; m < 2; ++m) {
        const long long c = vmap(a, b, zs[k], ys[j], xs[m]);
        s += a.p_sub ? a.p[c] - a.p_sub[c] : a.p[c];
      }
  out[i] = s * 0.125f * a.pscale * inst_scale_of(a, b);
}

// Catmull-Rom weights of points -1, 0, 1, 2 at t in [0, 1] past point 0
// (Catmull & Rom 1974).
__device__ __forceinline__ void catmull_rom(float t, float (&w)[4]) {
  const float t2 = t * t, t3 = t2 * t;
  w[0] = 0.5f * (-t3 + 2.f * t2 - t);
  w[1] = 0.5f * (3.f * t3 - 5.f * t2 + 2.f);
  w[2] = 0.5f * (-3.f * t3 + 4.f * t2 + t);
  w[3] = 0.5f * (t3 - t2);
}

// Coarse prediction (FP32, one value per coarse cell) -> fine p:
// Catmull-Rom cubic interpolation per axis from coarse centres at
// (c + 0.5) f - 0.5 (positions clamped to [0, nc - 1], neighbour indices to
// the coarse grid), divided by pscale, times bnd.  Writes (or, with add,
// adds to) every fine cell of every instance.  With a mirror (flip != 0) the
// coarse grid is a prediction for that mirror image: stored cell (z, y, x)
// reads it at its mirror-image coordinates.
__global__ void upsample_kernel(PoolArgs a, const float *__restrict__ coarse,
                                float *__restrict__ p, bool add) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)a.batch * a.inz * a.iny * a.inx;
  if (i >= n) return;
  const int x = (int)(i % a.inx), y = (int)((i / a.inx) % a.iny);
  const int z = (int)((i / ((long long)a.inx * a.iny)) % a.inz);
  const int b = (int)(i / ((long long)a.inx * a.iny * a.inz));
  // mirror-image coordinates of stored cell (z, y, x): undo vmap
  int xm = (a.flip & 8) ? y : x, ym = (a.flip & 8) ? x : y, zm = z;
  if (a.flip & 1) xm = a.inx - 1 - xm;
  if (a.flip & 2) ym = a.iny - 1 - ym;
  if (a.flip & 4) zm = a.inz - 1 - zm;
  auto axis = [&](int j, int nc, int (&idx)[4], float (&w)[4]) {
    float pos = ((float)j + 0.5f) / (float)a.f - 0.5f;
    pos = fminf(fmaxf(pos, 0.f), (float)(nc - 1));
    const int i0 = min((int)floorf(pos), nc - 1);
    catmull_rom(pos - (float)i0, w);
    for (int k = 0; k < 4; ++k) idx[k] = min(max(i0 - 1 + k, 0), nc - 1);
  };
  int iz[4], iy[4], ix[4];
  float wz[4], wy[4], wx[4];
  axis(zm, a.zc, iz, wz);
  axis(ym, a.yc, iy, wy);
  axis(xm, a.xc, ix, wx);
  const float *c = coarse + (long long)b * a.zc * a.yc * a.xc;
  float v = 0.f;
  for (int kz = 0; kz < 4; ++kz) {
    float vy = 0.f;
    for (int ky = 0; ky < 4; ++ky) {
      const float *row = c + ((long long)iz[kz] * a.yc + iy[ky]) * a.xc;
      float vx = 0.f;
      for (int kx = 0; kx < 4; ++kx) vx += wx[kx] * row[ix[kx]];
      vy += wy[ky] * vx;
    }
    v += wz[kz] * vy;
  }
  const long long k = fine_index(a, b, z, y, x);
  const float sc = inst_scale_of(a, b);
  const float u = sc != 0.f ? v / (a.pscale * sc) * a.bnd[k] : 0.f;
  p[k] = add ? p[k] + u : u;
}

// Residual source of the current pressure p, for the correction problem:
// with c_i = a_i and b = 0 the 19-point Himeno residual is
// ss = (s0 a3 - p) bnd with s0 = sum_i a_i (p(x + e_i) + p(x - e_i)) + wrk1
// and a3 = 1 / (2 (a0 + a1 + a2)), so r = ss / a3 =
// (s0 - 2 (a0 + a1 + a2) p) bnd is the source (in wrk1's units) of the
// equation the error p* - p satisfies.  Cells on an instance's faces (and
// bnd = 0 cells) get r = 0 and read no neighbours.  r is written in the
// stacked layout of the fields.  Grid (G, batch): block (g, b) strides over
// instance b's cells and stores its FP64 partial sum of r^2 at
// part[b * G + g] (fixed assignment, so the per-instance sums are
// deterministic).
__global__ void residual_source_kernel(PoolArgs a, float *__restrict__ r,
                                       double *__restrict__ part) {
  const int b = blockIdx.y;
  const long long n = (long long)a.inz * a.iny * a.inx;
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % a.inx), y = (int)((i / a.inx) % a.iny);
    const int z = (int)(i / ((long long)a.inx * a.iny));
    const long long k = fine_index(a, b, z, y, x);
    float v = 0.f;
    const bool inner = x > 0 && x < a.inx - 1 && y > 0 && y < a.iny - 1 && z > 0 &&
                       z < a.inz - 1;
    if (inner && a.bnd[k] != 0.f) {
      const long long py = a.pitch_e, pz = (long long)a.ny * a.pitch_e;
      const float pc = a.p[k];
      const float c0 = a.a0[k], c1 = a.a1[k], c2 = a.a2[k];
      float s0 = c0 * (a.p[k + pz] + a.p[k - pz]);
      s0 += c1 * (a.p[k + py] + a.p[k - py]);
      s0 += c2 * (a.p[k + 1] + a.p[k - 1]);
      s0 += a.wrk1[k];
      v = (s0 - 2.f * (c0 + c1 + c2) * pc) * a.bnd[k];
    }
    r[k] = v;
    acc += (double)v * v;
  }
  __shared__ double red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(long long)b * gridDim.x + blockIdx.x] = red[0];
}

// p = p_scale * p + delta at every cell of every instance (stored layout;
// delta may be NULL): one rounding of p per restart, whatever number of
// mirror predictions delta sums.
__global__ void add_correction_kernel(PoolArgs a, const float *__restrict__ delta,
                                      float p_scale, float *__restrict__ p) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)a.batch * a.inz * a.iny * a.inx;
  if (i >= n) return;
  const int x = (int)(i % a.inx), y = (int)((i / a.inx) % a.iny);
  const int z = (int)((i / ((long long)a.inx * a.iny)) % a.inz);
  const int b = (int)(i / ((long long)a.inx * a.iny * a.inz));
  const long long k = fine_index(a, b, z, y, x);
  const float v = p_scale == 1.f ? p[k] : __fmul_rn(p_scale, p[k]);
  p[k] = delta ? __fadd_rn(v, delta[k]) : v;
}

// scale[b] = target_rms / rms(r of instance b) over its interior cells
// (0 when r vanishes); the partials are summed in a fixed order.
__global__ void inst_scale_kernel(const double *__restrict__ part, int G, int batch,
                                  long long cells, float target_rms,
                                  float *__restrict__ scale) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  double s = 0.0;
  for (int g = 0; g < G; ++g) s += part[(long long)b * G + g];
  const double rms = sqrt(s / (double)cells);
  scale[b] = rms > 0.0 ? (float)(target_rms / rms) : 0.f;
}

}  // namespace

void nn_set_error_word(int *err) { g_err = err; }

static bool use_tcgen05() {
  const char *e = getenv("PS_WARMSTART_TC");
  return !(e && e[0] == '0');
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return n;
}

// Tensor map of x [batch, z, y, x, 16] BF16 with a box of 8 channels x bx x by
// x bz voxels of one instance; false if the driver cannot encode it.
static bool tmap_slab(CUtensorMap *m, const void *x, const Dims &d, int bx, int by, int bz) {
  typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                             const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<Encode>(fn);
  }();
  if (!encode) return false;
  const cuuint64_t dims[5] = {(cuuint64_t)kC, (cuuint64_t)d.X, (cuuint64_t)d.Y, (cuuint64_t)d.Z,
                              (cuuint64_t)d.B};
  const cuuint64_t row = (cuuint64_t)kC * 2;
  const cuuint64_t strides[4] = {row, row * d.X, row * d.X * d.Y,
                                 row * d.X * d.Y * (cuuint64_t)d.Z};
  const cuuint32_t box[5] = {8, (cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bz, 1};
  const cuuint32_t one[5] = {1, 1, 1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(x), dims, strides, box,
                one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A launch may start as the last CTAs of the stream's previous kernel leave (its
// kernel waits for their writes), except while the stream is captured: the
// captured edge would be one.  A training step of 27 launches takes 256 us with
// it, 282 without; a layer's forward, data and weight gradients of 1024 instances
// 283 and 291.  No kernel here lets its dependents in before its CTAs leave, and
// none allocates tensor memory before its wait: the kernel ahead, which may be the
// caller's and let dependents in early, could still want those columns.  What
// these kernels read is not __restrict__, as read-only loads could be moved ahead of the wait.
static bool may_overlap(cudaStream_t s) {
  const char *e = getenv("PS_OVERLAP");
  if (e && e[0] == '0') return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
    return true;
  cudaGetLastError();
  return false;
}

// conv_pad_kernel over slabs, or false if a slab of one plane does not fit
// (more than 1024 padded voxels per plane), a pointer is not aligned for TMA
// and 16-byte accesses, or the map cannot be encoded.
static bool launch_conv_pad(const void *x, const void *w, const float *bias, const void *mask,
                            int relu, void *y, float *yf, const Dims &d, cudaStream_t s,
                            cudaError_t *e) {
  const long long P = (long long)(d.X + 1) * (d.Y + 1);
  if (d.X > 255 || d.Y > 255 || P > kPcMaxTiles * kTcM || !aligned16(x) || !aligned16(w) ||
      !aligned16(mask) || !aligned16(y))
    return false;
  int zmax = (int)(kPcMaxTiles * kTcM / P);
  if (zmax > 254) zmax = 254;
  const PadGeom g = pad_geom(d, zmax, 4LL * sm_count());
  const long long items = (long long)d.B * g.nslab;
  if (items > 0x7fffffff) return false;
  // A few slabs of wide planes: one CTA makes a slab's tiles one after the other,
  // 3.6 us and 1 us a tile, where conv_tc_kernel's CTAs share all tiles out, 8.5 us
  // and 1.4 us for each tile an SM gets (2 x 10 x 4 x 200 voxels, 20 slabs of 8 tiles:
  // 11.7 against 9.3 us; 4 x 20 x 4 x 200: 11.8 against 14.4).
  const int sms = sm_count();
  if (items <= sms && 3.6 + pc_tiles(g.zs, g.P) >
                          8.5 + 1.4 * (double)((d.nvox + kTcM - 1) / kTcM) / sms)
    return false;
  CUtensorMap tm;
  if (!tmap_slab(&tm, x, d, g.px, d.Y + 1, g.zs + 2)) return false;
  const size_t smem = pc_smem(g);
  *e = cudaFuncSetAttribute(conv_pad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kPcMaxSmem);
  if (*e != cudaSuccess) return true;
  *e = launch_kernel(conv_pad_kernel, dim3((unsigned)items), dim3(kPcThreads), smem, s, may_overlap(s),
                     tm, static_cast<const __nv_bfloat16 *>(w), bias,
                     static_cast<const __nv_bfloat16 *>(mask), relu,
                     static_cast<__nv_bfloat16 *>(y), yf, d, g, g_err);
  return true;
}

int nn_conv(const void *x, const void *w, const float *bias, const void *mask, int relu,
            void *y, float *yf, int B, int Z, int Y, int X, cudaStream_t s) {
  Dims d{B, Z, Y, X, (long long)B * Z * Y * X};
  if (d.nvox <= 0) return 0;
  if (use_tcgen05()) {
    cudaError_t e = cudaSuccess;
    if (launch_conv_pad(x, w, bias, mask, relu, y, yf, d, s, &e)) return (int)e;
    static bool attr = false;
    if (!attr) {
      const cudaError_t e = cudaFuncSetAttribute(
          conv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
      if (e != cudaSuccess) return (int)e;
      attr = true;
    }
    const long long blocks = (d.nvox + kTcM - 1) / kTcM;
    conv_tc_kernel<<<(unsigned)blocks, kTcThreads, kTcSmem, s>>>(
        static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(w), bias,
        static_cast<const __nv_bfloat16 *>(mask), relu, static_cast<__nv_bfloat16 *>(y), yf, d,
        g_err);
    return (int)cudaGetLastError();
  }
  const long long blocks = (d.nvox + 16 * kConvWarps - 1) / (16 * kConvWarps);
  conv_kernel<<<(unsigned)blocks, 32 * kConvWarps, 0, s>>>(
      static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(w), bias,
      static_cast<const __nv_bfloat16 *>(mask), relu, static_cast<__nv_bfloat16 *>(y), yf, d);
  return (int)cudaGetLastError();
}

int nn_wgrad(const void *x, const void *dy, float *part, int S, float *dw, float *db, int B,
             int Z, int Y, int X, cudaStream_t s) {
  Dims d{B, Z, Y, X, (long long)B * Z * Y * X};
  if (S < 1) return -1;
  float *bpart = part + (long long)S * kTaps * kC * kC;
  const __nv_bfloat16 *xb = static_cast<const __nv_bfloat16 *>(x);
  const __nv_bfloat16 *yb = static_cast<const __nv_bfloat16 *>(dy);
  const bool overlap = may_overlap(s);
  // wgrad_kernel's two-byte loads take any pointer, cp.async 16-byte ones
  if (aligned16(x) && aligned16(dy)) {
    const WgRows rows = wg_rows(X);
    const int stages = 16 + kWgStages * wg_stage_bytes(rows);
    const int sums = kWgWarps * 3 * kC * kC * 4;
    const int smem = stages > sums ? stages : sums;
    // at most 33552 bytes: under what a launch may use without asking
    const cudaError_t e = launch_kernel(wgrad_run_kernel, dim3(3 * kWgHalves, S), dim3(kWgThreads),
                                        smem, s, overlap, xb, yb, part, bpart, d, rows);
    if (e != cudaSuccess) return (int)e;
  } else {
    wgrad_kernel<<<dim3(kTaps, S), 32 * kConvWarps, 0, s>>>(xb, yb, part, bpart, d);
  }
  const int n = kTaps * kC * kC + kC;
  const cudaError_t e = launch_kernel(wgrad_reduce_kernel, dim3((n + 63) / 64), dim3(256), 0, s,
                                      overlap, part, bpart, S, dw, db);
  return (int)e;
}

int nn_prep_weights(const float *w, void *wf, void *wb, cudaStream_t s) {
  return (int)launch_kernel(prep_weights_kernel, dim3((kTaps * kC * kC + 255) / 256), dim3(256), 0, s,
                            may_overlap(s), w, static_cast<__nv_bfloat16 *>(wf),
                            static_cast<__nv_bfloat16 *>(wb));
}

int nn_adam(float *w, const float *g, float *m, float *v, long long n, float lr, float b1,
            float b2, float eps, int step, cudaStream_t s) {
  if (n <= 0 || step < 1) return -1;
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, step)));
  const float c2 = (float)(1.0 / (1.0 - pow((double)b2, step)));
  adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, g, m, v, n, lr, b1, b2, eps, c1, c2);
  return (int)cudaGetLastError();
}

int nn_adam_layers(float *w, const float *g, float *m, float *v, int layers, float lr, float b1,
                   float b2, float eps, int step, void *wf, void *wb, cudaStream_t s) {
  if (layers < 1 || layers > 4096 || step < 1) return -1;
  const float c1 = (float)(1.0 / (1.0 - pow((double)b1, step)));
  const float c2 = (float)(1.0 / (1.0 - pow((double)b2, step)));
  const int n = layers * (kTaps * kC * kC + kC);
  return (int)launch_kernel(adam_layers_kernel, dim3((n + 255) / 256), dim3(256), 0, s,
                            may_overlap(s), w, g, m, v, layers, lr, b1, b2, eps, c1, c2,
                            static_cast<__nv_bfloat16 *>(wf), static_cast<__nv_bfloat16 *>(wb));
}

int nn_mse(const float *pred, const float *tgt, long long n, void *dy, double *part,
           cudaStream_t s) {
  if (n <= 0) return -1;
  return (int)launch_kernel(mse_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, s,
                            may_overlap(s), pred, tgt, n, static_cast<__nv_bfloat16 *>(dy), part);
}

static PoolArgs pool_args(const NNFields &f) {
  PoolArgs a{};
  a.a0 = f.a0;
  a.a1 = f.a1;
  a.a2 = f.a2;
  a.wrk1 = f.wrk1;
  a.bnd = f.bnd;
  a.p = f.p;
  a.pitch_e = f.pitch / 4;
  a.ny = f.ny;
  a.inx = f.inx;
  a.iny = f.iny;
  a.inz = f.inz;
  a.nsx = f.nsx;
  a.f = f.factor;
  a.zc = (f.inz + f.factor - 1) / f.factor;
  a.yc = (f.iny + f.factor - 1) / f.factor;
  a.xc = (f.inx + f.factor - 1) / f.factor;
  a.batch = f.batch;
  a.flip = f.flip;
  a.wscale = f.wscale;
  a.pscale = f.pscale;
  a.inst_scale = f.inst_scale;
  a.p_sub = f.p_sub;
  return a;
}

int nn_pool_inputs(const NNFields &f, void *out, cudaStream_t s) {
  const PoolArgs a = pool_args(f);
  const long long n = (long long)a.batch * a.zc * a.yc * a.xc;
  if (n <= 0) return -1;
  pool_inputs_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(
      a, static_cast<__nv_bfloat16 *>(out));
  return (int)cudaGetLastError();
}

int nn_pool_target(const NNFields &f, float *out, cudaStream_t s) {
  const PoolArgs a = pool_args(f);
  const long long n = (long long)a.batch * a.zc * a.yc * a.xc;
  if (n <= 0 || !a.p) return -1;
  pool_target_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(a, out);
  return (int)cudaGetLastError();
}

int nn_upsample(const NNFields &f, const float *coarse, float *p, bool add, cudaStream_t s) {
  const PoolArgs a = pool_args(f);
  const long long n = (long long)a.batch * a.inz * a.iny * a.inx;
  if (n <= 0) return -1;
  upsample_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, coarse, p, add);
  return (int)cudaGetLastError();
}

int nn_residual_source(const NNFields &f, float *r, float *inst_scale, float target_rms,
                       double *work, int work_len, cudaStream_t s) {
  const PoolArgs a = pool_args(f);
  if (!a.p || !r || !inst_scale || !work || a.batch < 1) return -1;
  const int G = work_len / a.batch;
  if (G < 1) return -1;
  const int g = G < 64 ? G : 64;
  residual_source_kernel<<<dim3((unsigned)g, (unsigned)a.batch), 256, 0, s>>>(a, r, work);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  const long long cells = (long long)(a.inz - 2) * (a.iny - 2) * (a.inx - 2);
  inst_scale_kernel<<<(unsigned)((a.batch + 127) / 128), 128, 0, s>>>(
      work, g, a.batch, cells > 0 ? cells : 1, target_rms, inst_scale);
  return (int)cudaGetLastError();
}

int nn_add_correction(const NNFields &f, const float *delta, float p_scale, float *p,
                      cudaStream_t s) {
  const PoolArgs a = pool_args(f);
  const long long n = (long long)a.batch * a.inz * a.iny * a.inx;
  if (n <= 0 || !p) return -1;
  add_correction_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, delta, p_scale, p);
  return (int)cudaGetLastError();
}

}  // namespace psg
