// Whole runs of the clamped 7-point diffusion over grids that fit on chip
// (GB300, sm_103a): one cooperative launch makes every time step.
//
// The reference launches one kernel per map per step
// (translator/cuda_runtime_builder.cc:1512-1583).  A small grid's step is then
// all launch and latency: 2.6 us at 64^3 replayed from a CUDA graph, for 0.2 us
// of L2 traffic.
//
// Design.  The grid is cut into bricks, full rows in x and by x bz rows in y
// and z, one per CTA (at most one CTA per SM, all resident: a cooperative
// launch).  A CTA keeps its brick and a halo of k rows in shared memory, two
// copies, and makes k steps on its own, its valid region shrinking by one row
// per step (as temporal7.cu does with tiles).  Then it needs its neighbours'
// rows again.
// * Exchange.  A CTA publishes the rows within k of its faces as 16-byte
//   packets of 8 bytes of cells and the epoch's number, written and read
//   whole (.b128 accesses are single-copy atomic), and a reader polls the
//   packets themselves until they carry the number it expects: one trip
//   through L2 instead of three (data and fence, flag, data).  Numbers count
//   upwards over all launches (`base`), so nothing is reset.  Two buffers
//   alternate: a CTA overwrites what it published two epochs ago, which its
//   neighbours had read before they published the last one.
// * A thread computes 2 x 2 rows (y, z) of 16 bytes (12 shared loads serve four
//   vectors), or 1 x 2 where that keeps more threads busy; x neighbours come
//   from shuffles.  At the grid's faces the
//   kept region ends, so clamping row indices to it is the boundary rule.
// * The last two steps go to the two grids, where a plain run leaves them.
// * Each cell's arithmetic is the plain sweep's, so the result has the same
//   bits.
// * Polls are bounded; a CTA whose wait gives up sets the error word and
//   leaves, and its neighbours' waits then give up too.
// Bound: the exchange's latency against the steps' issue slots, which grow
// with k; choose_resident7 weighs the two.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "ps_device.cuh"
#include "ps_internal.h"

namespace psg {
namespace {

constexpr int kResThreads = 512;
constexpr int kResBatch = 3;             // vectors of halo a thread polls together
constexpr size_t kResSmem = 220 * 1024;   // most dynamic shared memory of a CTA
constexpr unsigned kResPolls = 1u << 20;  // packet reads (about 0.7 us each) before a wait gives up

template <typename T>
struct RParams {
  T *g[2];             // g1 (step 0 on entry), g2
  int64_t row, plane;  // elements
  int nx, ny, nz;
  int by, bz, nby, k;
  int steps;
  unsigned base;       // no packet carries a larger number on entry
  uint4 *packets;      // [2][nz][ny][nvec][2]
  T cc, cw, ce, cs, cn, cb, ct;
  int *err;
};

// 16 bytes in one access.
__device__ __forceinline__ void st_packet(uint4 *p, unsigned long long data, unsigned seq) {
  asm volatile(
      "{\n\t.reg .b128 v;\n\t.reg .b64 s;\n\tmov.b64 s, {%2, %2};\n\tmov.b128 v, {%1, s};\n\t"
      "st.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p),
      "l"(data), "r"(seq)
      : "memory");
}
__device__ __forceinline__ bool ld_packet(const uint4 *p, unsigned seq, unsigned long long &data) {
  unsigned long long d, f;
  asm volatile(
      "{\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%2];\n\tmov.b128 {%0, %1}, v;\n\t}"
      : "=l"(d), "=l"(f)
      : "l"(p)
      : "memory");
  data = d;
  return (unsigned)f == seq;
}

// Division of n < 2^16 by d < 2^16 through a multiply.
struct FastDiv {
  unsigned d, m;
};
__device__ __forceinline__ FastDiv fast_div(int d) {
  return FastDiv{(unsigned)d, d > 1 ? 0xffffffffu / (unsigned)d + 1u : 0u};
}
__device__ __forceinline__ void split(const FastDiv &f, int n, int &q, int &r) {
  q = f.d > 1 ? (int)__umulhi((unsigned)n, f.m) : n;
  r = n - q * (int)f.d;
}

// The 16 bytes of one row at x, given its neighbours' rows; lanes of a warp
// hold consecutive vectors (row after row).
template <typename T, int VEC>
__device__ __forceinline__ void res_row(const RParams<T> &p, const T (&c)[VEC], const T (&n)[VEC],
                                        const T (&s)[VEC], const T (&b)[VEC], const T (&t)[VEC],
                                        const T *at, bool left_edge, int east, bool load_left,
                                        bool load_right, bool cross, T (&o)[VEC]) {
  typedef RN<T> R;
  T left = shfl_up1(c[VEC - 1]), right = shfl_down1(c[0]);
  if (cross) {  // a row may start or end inside a warp: its first or last lane reads on
    ld_shared_if(load_left, at - 1, left);
    ld_shared_if(load_right, at + VEC, right);
  }
  if (left_edge) left = c[0];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const T w = i == 0 ? left : c[i - 1];
    T e = i == VEC - 1 ? right : c[i + 1];
    if (i == east) e = c[i];
    // cc*c + cw*w + ce*e + cs*s + cn*n + cb*b + ct*t, left to right
    T v = R::mul(p.cc, c[i]);
    v = R::add(v, R::mul(p.cw, w));
    v = R::add(v, R::mul(p.ce, e));
    v = R::add(v, R::mul(p.cs, s[i]));
    v = R::add(v, R::mul(p.cn, n[i]));
    v = R::add(v, R::mul(p.cb, b[i]));
    v = R::add(v, R::mul(p.ct, t[i]));
    o[i] = v;
  }
}

template <typename T, int YB>
__global__ void __launch_bounds__(kResThreads, 1) resident7_kernel(const RParams<T> p) {
  constexpr int VEC = 16 / (int)sizeof(T);
  extern __shared__ __align__(128) unsigned char res_smem[];
  __shared__ FastDiv ydiv[kResident7MaxK + 1];  // blocks per y extent of step j
  const int tid = threadIdx.x, lane = tid & 31;
  const int iy = blockIdx.x % p.nby, iz = blockIdx.x / p.nby;
  const int nvec = (p.nx + VEC - 1) / VEC;
  const int P = nvec * VEC;
  // own rows, and the extended region kept in shared memory
  const int y0 = iy * p.by, y1 = min(y0 + p.by, p.ny);
  const int z0 = iz * p.bz, z1 = min(z0 + p.bz, p.nz);
  const int ye0 = max(0, y0 - p.k), ye1 = min(p.ny, y1 + p.k);
  const int ze0 = max(0, z0 - p.k), ze1 = min(p.nz, z1 + p.k);
  const int EY = ye1 - ye0, EZ = ze1 - ze0;
  const int zstride = EY * P;
  T *cur = reinterpret_cast<T *>(res_smem);
  T *nxt = cur + EZ * zstride;
  // rows of step j in the extended region's coordinates: [ya(j), yb(j))
  auto ya_of = [&](int j) { return ye0 == 0 ? 0 : j; };
  auto yb_of = [&](int j) { return ye1 == p.ny ? EY : EY - j; };
  auto za_of = [&](int j) { return ze0 == 0 ? 0 : j; };
  auto zb_of = [&](int j) { return ze1 == p.nz ? EZ : EZ - j; };
  if (tid <= p.k && tid >= 1) ydiv[tid] = fast_div((yb_of(tid) - ya_of(tid) + YB - 1) / YB);
  const FastDiv vdiv = fast_div(nvec), ediv = fast_div(EY);
  const bool cross = (32 % nvec) != 0;
  const int64_t half = (int64_t)p.nz * p.ny * nvec * 2;  // packets per buffer

  // step 0: the extended region from g1
  for (int i = tid; i < EZ * EY * nvec; i += kResThreads) {
    int r, v, z, y;
    split(vdiv, i, r, v);
    split(ediv, r, z, y);
    reinterpret_cast<uint4 *>(cur)[i] =
        __ldcg(reinterpret_cast<const uint4 *>(p.g[0] + (int64_t)(ze0 + z) * p.plane +
                                               (int64_t)(ye0 + y) * p.row) + v);
  }
  __syncthreads();

  int t = 0;
  for (unsigned e = 0;; ++e) {
    const int kk = min(p.k, p.steps - t);
    uint4 *const pub = p.packets + (e & 1) * half;
    const unsigned seq = p.base + e + 1;
    for (int j = 1; j <= kk; ++j) {
      ++t;
      // where this step's own brick goes besides shared memory
      T *const out = t == p.steps ? p.g[0] : (t == p.steps - 1 ? p.g[1] : nullptr);
      const bool publish = j == kk && t < p.steps;
      const int ya = ya_of(j), yb = yb_of(j), za = za_of(j), zb = zb_of(j);
      const FastDiv yd = ydiv[j];
      const int items = nvec * (int)yd.d * ((zb - za + 1) / 2);
      for (int i0 = tid - lane; i0 < items; i0 += kResThreads) {
        const bool active = i0 + lane < items;
        int r, xv, zi, yi;
        split(vdiv, min(i0 + lane, items - 1), r, xv);
        split(yd, r, zi, yi);
        const int y = ya + YB * yi, z = za + 2 * zi, x = xv * VEC;
        // rows y - 1 .. y + YB and planes z - 1 .. z + 2, kept inside the region
        int yo[YB + 2];
#pragma unroll
        for (int q = 0; q < YB + 2; ++q) yo[q] = min(max(y + q - 1, 0), EY - 1) * P;
        const T *zm = cur + max(z - 1, 0) * zstride + x, *zc = cur + z * zstride + x,
                *zc1 = cur + min(z + 1, EZ - 1) * zstride + x,
                *zp = cur + min(z + 2, EZ - 1) * zstride + x;
        // rows q = 0 .. YB + 1 (the first and last only as neighbours)
        T c0[YB + 2][VEC], c1[YB + 2][VEC], b[YB][VEC], u[YB][VEC], o[2][YB][VEC];
#pragma unroll
        for (int q = 0; q < YB + 2; ++q) {
          ld16_shared<T>(c0[q], zc + yo[q]);
          ld16_shared<T>(c1[q], zc1 + yo[q]);
        }
#pragma unroll
        for (int q = 0; q < YB; ++q) {
          ld16_shared<T>(b[q], zm + yo[q + 1]);
          ld16_shared<T>(u[q], zp + yo[q + 1]);
        }
        const bool ledge = x == 0;
        const int east = p.nx - 1 - x;  // element that clamps east
        const bool ll = lane == 0 && x > 0, lr = lane == 31 && xv < nvec - 1;
#pragma unroll
        for (int q = 0; q < YB; ++q) {
          res_row<T, VEC>(p, c0[q + 1], c0[q], c0[q + 2], b[q], c1[q + 1], zc + yo[q + 1], ledge,
                          east, ll, lr, cross, o[0][q]);
          res_row<T, VEC>(p, c1[q + 1], c1[q], c1[q + 2], c0[q + 1], u[q], zc1 + yo[q + 1], ledge,
                          east, ll, lr, cross, o[1][q]);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int q = 0; q < YB; ++q) {
            if (!active || y + q >= yb || z + a >= zb) continue;
            *reinterpret_cast<uint4 *>(nxt + (z + a) * zstride + (y + q) * P + x) =
                *reinterpret_cast<const uint4 *>(o[a][q]);
          }
        if (!out && !publish) continue;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int q = 0; q < YB; ++q) {
            const int gy = ye0 + y + q, gz = ze0 + z + a;
            if (!active || gy < y0 || gy >= y1 || gz < z0 || gz >= z1) continue;
            if (out) {
              T *d = out + (int64_t)gz * p.plane + (int64_t)gy * p.row + x;
              if (x + VEC <= p.nx) {
                st16_global<T>(d, o[a][q]);
              } else {
#pragma unroll
                for (int i = 0; i < VEC; ++i)
                  if (i <= east) d[i] = o[a][q][i];
              }
            }
            // rows that some neighbour keeps
            if (publish && (gy - y0 < p.k || y1 - gy <= p.k || gz - z0 < p.k || z1 - gz <= p.k)) {
              uint4 *d = pub + (((int64_t)gz * p.ny + gy) * nvec + xv) * 2;
              const unsigned long long *w =
                  reinterpret_cast<const unsigned long long *>(o[a][q]);
              st_packet(d, w[0], seq);
              st_packet(d + 1, w[1], seq);
            }
          }
      }
      T *const sw = cur;
      cur = nxt;
      nxt = sw;
      __syncthreads();
    }
    if (t == p.steps) return;
    // read the halo the neighbours published in this epoch
    bool ok = true;
    const int n = EZ * EY * nvec;
    for (int i0 = tid; i0 < n && ok; i0 += kResBatch * kResThreads) {
      // the packets of up to kResBatch vectors in flight together
      const uint4 *src[kResBatch];
      unsigned need = 0;
#pragma unroll
      for (int q = 0; q < kResBatch; ++q) {
        const int i = min(i0 + q * kResThreads, n - 1);
        int r, v, z, y;
        split(vdiv, i, r, v);
        split(ediv, r, z, y);
        const int gy = ye0 + y, gz = ze0 + z;
        src[q] = pub + (((int64_t)gz * p.ny + gy) * nvec + v) * 2;
        if (i0 + q * kResThreads < n && !(gy >= y0 && gy < y1 && gz >= z0 && gz < z1))
          need |= 1u << q;
      }
      for (unsigned polls = 0; need && polls < kResPolls; ++polls) {
        unsigned long long w[kResBatch][2];
        bool have[kResBatch];
#pragma unroll
        for (int q = 0; q < kResBatch; ++q) {
          have[q] = false;
          if ((need >> q) & 1u) {
            const bool h0 = ld_packet(src[q], seq, w[q][0]), h1 = ld_packet(src[q] + 1, seq, w[q][1]);
            have[q] = h0 && h1;
          }
        }
#pragma unroll
        for (int q = 0; q < kResBatch; ++q)
          if (have[q]) {
            reinterpret_cast<ulonglong2 *>(cur)[i0 + q * kResThreads] =
                make_ulonglong2(w[q][0], w[q][1]);
            need &= ~(1u << q);
          }
      }
      ok = need == 0;
    }
    if (!ok) atomicOr(p.err, kDevErrWaitTimeout);
    if (!__syncthreads_and(ok)) return;
  }
}

template <typename T>
cudaError_t launch_t(const Resident7Args &a, cudaStream_t s) {
  RParams<T> p;
  p.g[0] = static_cast<T *>(a.g1.ptr);
  p.g[1] = static_cast<T *>(a.g2.ptr);
  p.row = a.g1.pitch / (int64_t)sizeof(T);
  p.plane = p.row * a.g1.ny;
  p.nx = a.g1.nx;
  p.ny = a.g1.ny;
  p.nz = a.g1.nz;
  p.by = a.plan.by;
  p.bz = a.plan.bz;
  p.nby = (p.ny + p.by - 1) / p.by;
  p.k = a.plan.k;
  p.steps = a.steps;
  p.base = a.base;
  p.packets = static_cast<uint4 *>(a.packets);
  p.ce = (T)a.coef[0];
  p.cw = (T)a.coef[1];
  p.cn = (T)a.coef[2];
  p.cs = (T)a.coef[3];
  p.ct = (T)a.coef[4];
  p.cb = (T)a.coef[5];
  p.cc = (T)a.coef[6];
  p.err = a.err;
  // two rows per thread reuse more of what they load; one row, where that would
  // leave threads without work, halves a step's latency
  const int ry = p.by + 2 * (p.k - 1), rz = (p.bz + 2 * (p.k - 1) + 1) / 2;
  const bool one = (long long)(p.nx * (int)sizeof(T) + 15) / 16 * ry * rz <= kResThreads;
  auto kern = one ? resident7_kernel<T, 1> : resident7_kernel<T, 2>;
  const size_t smem = resident7_smem(a.plan, p.nx, p.ny, p.nz, (int)sizeof(T));
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kResSmem);
  if (e != cudaSuccess) return e;
  void *args[] = {&p};
  return cudaLaunchCooperativeKernel(
      reinterpret_cast<void *>(kern), dim3((unsigned)(p.nby * ((p.nz + p.bz - 1) / p.bz))),
      dim3(kResThreads), args, smem, s);
}

}  // namespace

size_t resident7_packet_bytes(int nx, int ny, int nz, int esz) {
  return 2 * (size_t)nz * ny * (((size_t)nx * esz + 15) / 16) * 2 * 16;
}

size_t resident7_smem(const Resident7Plan &q, int nx, int ny, int nz, int esz) {
  const int vec = 16 / esz;
  const size_t row = (size_t)(nx + vec - 1) / vec * 16;
  const int ey = q.by + 2 * q.k < ny ? q.by + 2 * q.k : ny;
  const int ez = q.bz + 2 * q.k < nz ? q.bz + 2 * q.k : nz;
  return 2 * row * (size_t)ey * ez;
}

// Cost per epoch, fitted on GB300 to 32^3 .. 128^3: 1.1 us for the exchange,
// 0.33 us of latency per step, and per 16-byte vector 0.83 ns computed (7.7 ns
// in double precision, whose pipe is the bound) and 0.6 ns of halo.  Measured
// per step against sweeps replayed from a graph: 32^3 0.9 against 2.6 us, 64^3 1.5
// against 2.6 (k = 2, bricks of 5 x 6 rows), 96^3 3.0 against 4.9, 120^3 5.0
// against 5.8, 128^3 5.4 and 5.4; double 32^3 3.1 against 6.1, 64^3 9.4 against
// 10.2.
bool choose_resident7(int nx, int ny, int nz, int esz, int sms, Resident7Plan *best) {
  const int vec = 16 / esz, nvec = (nx + vec - 1) / vec;
  // fewer rows than four per SM make bricks thinner than their halo
  if ((long long)ny * nz < 4LL * sms) return false;
  best->us = 1e30;
  for (int k = 1; k <= kResident7MaxK; ++k)
    for (int by = 1; by <= ny; ++by) {
      const int nby = (ny + by - 1) / by;
      if (nby > sms) continue;
      const int nbz_max = sms / nby;
      Resident7Plan q;
      q.k = k;
      q.by = by;
      q.bz = (nz + nbz_max - 1) / nbz_max;
      if (resident7_smem(q, nx, ny, nz, esz) > kResSmem) continue;
      double vecs = 0;  // 16-byte vectors computed per epoch
      for (int j = 1; j <= k; ++j)
        vecs += (double)nvec * (by + 2 * (k - j)) * (q.bz + 2 * (k - j));
      const double halo = (double)nvec * ((by + 2.0 * k) * (q.bz + 2.0 * k) - (double)by * q.bz);
      q.us = (1.1 + 0.33 * k + (esz == 4 ? 0.00083 : 0.0077) * vecs + 0.0006 * halo) / k;
      if (q.us < best->us) *best = q;
    }
  return best->us < 1e29;
}

// The plan's time per step with what the cost above leaves out: blocks of rows
// that a brick's extent cuts, and passes over more blocks than threads.  Fitted to
// the same sizes and 140 random boxes of 8 to 400 cells a side: 0.75 to 1.2 of
// the measured time (the cost above: 0.47 to 1.2).
double resident7_us(const Resident7Plan &q, int nx, int ny, int nz, int esz) {
  const int vec = 16 / esz, nvec = (nx + vec - 1) / vec, k = q.k;
  const int ry = q.by + 2 * (k - 1), rz = (q.bz + 2 * (k - 1) + 1) / 2;
  const int yb = (long long)nvec * ry * rz <= kResThreads ? 1 : 2;  // as launch_t chooses
  double vecs = 0, passes = 0;
  for (int j = 1; j <= k; ++j) {
    const int hy = std::min(q.by + 2 * (k - j), ny), hz = std::min(q.bz + 2 * (k - j), nz);
    const double items = (double)nvec * ((hy + yb - 1) / yb) * ((hz + 1) / 2);
    vecs += 2 * yb * items;
    passes += std::max(0.0, std::ceil(items / kResThreads) - 1);
  }
  const double halo = (double)nvec * ((q.by + 2.0 * k) * (q.bz + 2.0 * k) - (double)q.by * q.bz);
  return (esz == 4 ? 1.33 + 0.28 * k + 0.00072 * vecs + 0.35 * passes + 0.00053 * halo
                   : 0.55 + 1.355 * k + 0.00655 * vecs + 0.002 * halo) / k;
}

cudaError_t launch_resident7(const Resident7Args &a, cudaStream_t s) {
  return a.g1.type == kFloat ? launch_t<float>(a, s) : launch_t<double>(a, s);
}

}  // namespace psg
