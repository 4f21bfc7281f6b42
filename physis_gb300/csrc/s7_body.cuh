// The per-item body of the 7-point z-march (stencil7.cu's kernel and the
// batched kernel in batch.cu both run it).  One item is one tile of one grid
// marched over planes [zs, ze).  See stencil7.cu for the design.
#pragma once

#include "ps_device.cuh"
#include "ps_internal.h"

namespace psg {

template <typename T>
struct S7Params {
  T *out;
  int64_t row;    // out pitch in elements
  int64_t plane;  // out elements per z-plane
  int nx, ny, nz;
  int dmin0, dmin1, dmin2, dmax0, dmax1, dmax2;
  int lx;         // lanes side by side in x: 32, 16 or 8 (the others take rows further down)
  int xbase;      // x of the first tile (multiple of VEC)
  int tiles_x;    // tiles per y-band
  int tiles;      // tiles_x * tiles per x-column
  int zlen;       // planes per z-chunk
  int64_t items;  // tiles * chunks
  int ns;
  int early;      // the next launch's CTAs may take places while this one runs
  T cc, cw, ce, cs, cn, cb, ct;  // expression order of DIFFUSION7
  int *err;
};

__host__ __device__ constexpr int s7_bar_bytes(int ns) { return 128 * ((8 * ns + 127) / 128); }
__host__ __device__ constexpr uint32_t s7_stage_bytes(uint32_t b) { return (b + 127u) & ~127u; }

// Position in a ring of mbarrier-signalled stages used in issue order.
struct RingPos {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance(int n) {
    if (++stage == n) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

// How a CTA's threads agree and refill the ring.  S7Block: no producer; thread 0
// issues an item's planes, each when a CTA barrier shows that every thread is
// done with its stage.  Other kinds (batch.cu) have done(ok), called by each
// thread when it is done with a plane, and last() when it is done with the
// item's last one besides, and fill the ring themselves.
struct S7Block {
  static constexpr bool kIssues = true;
  const CUtensorMap *tin;
  RingPos prod;
};

// Marches tile `tile` of p over planes [zs, ze).  `full` are the ring's ns
// mbarriers, `ring` its stages (stride plane_elems elements).  Tiles are LX
// vectors of 16 bytes wide (LX = 32, or p.lx if NARROW) and warps * RY * 32 / LX
// rows high.  cons and sync persist across items.  Returns false if a bounded
// wait gave up.
template <typename T, int K, int RY, bool NARROW, class Sync>
__device__ __forceinline__ bool s7_item(const S7Params<T> &p, uint64_t *full, T *ring,
                                        int plane_elems, int warps, int tile, int zs, int ze,
                                        RingPos &cons, Sync &sync) {
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr bool kClamp = (K == kKernelDiffusion7);
  typedef RN<T> R;
  const int LX = NARROW ? p.lx : 32;
  const int TX = LX * VEC, W = TX + 2 * VEC;  // W: shared row width in elements
  const int TY = warps * RY * (32 / LX);
  const int ns = p.ns;
  const int lane = threadIdx.x, warp = threadIdx.y;
  const int tid = warp * 32 + lane;
  const int xl = NARROW ? lane & (LX - 1) : lane;
  const int rows0 = NARROW ? (warp * (32 / LX) + lane / LX) * RY : warp * RY;  // first own row in the tile
  const int cen0 = (rows0 + 1) * W + VEC + xl * VEC;  // own first row, centre
  bool ok = true;

  const int x0 = p.xbase + (tile % p.tiles_x) * TX;
  const int y0 = p.dmin1 + (tile / p.tiles_x) * TY;

  const int nplanes = ze - zs + 2;  // planes zs-1 .. ze

  // Issues plane q (global plane zs-1+q) into the producer's next stage.
  auto issue = [&](int q) {
    if constexpr (Sync::kIssues) {
      mbar_arrive_expect_tx(&full[sync.prod.stage], (uint32_t)(W * (TY + 2) * sizeof(T)));
      tma_load_3d(ring + sync.prod.stage * plane_elems, sync.tin, x0 - VEC, y0 - 1, zs - 1 + q,
                  &full[sync.prod.stage]);
      sync.prod.advance(ns);
    }
  };
  // Agreement after a plane.
  auto done = [&]() {
    if constexpr (Sync::kIssues) ok = __syncthreads_and(ok);
    else ok = sync.done(ok);
  };
  if constexpr (Sync::kIssues) {
    if (tid == 0) {
      const int n0 = min(ns, nplanes);
      for (int q = 0; q < n0; ++q) issue(q);
    }
  }
  // Waits for the next plane in issue order; returns its stage.
  auto wait_next = [&]() -> const T * {
    if (!mbar_wait(&full[cons.stage], cons.phase, p.err)) ok = false;
    const T *pl = ring + cons.stage * plane_elems;
    cons.advance(ns);
    return pl;
  };

  T b[RY][VEC], c[RY][VEC], t[RY][VEC];
  const T *pm = wait_next();   // plane zs-1
  const T *cur = wait_next();  // plane zs
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    ld16_shared<T>(c[r], cur + cen0 + r * W);
    ld16_shared<T>(b[r], pm + cen0 + r * W);
    if (kClamp && zs == 0) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) b[r][i] = c[r][i];
    }
  }
  done();
  if (!ok) return false;
  if (Sync::kIssues && tid == 0 && ns < nplanes) issue(ns);

  const int x = x0 + xl * VEC;
  const int y = y0 + rows0;  // first own row
  const int ywarp = y0 + warp * RY * (32 / LX);  // the warp's first row
  const bool vec_in = (x >= p.dmin0) && (x + VEC <= p.dmax0);
  const bool west_face = kClamp && (x == 0);            // element 0 clamps west
  const int east_elem = kClamp ? (p.nx - 1 - x) : -1;  // element clamping east

  for (int z = zs; z < ze; ++z) {
    const T *nxt = wait_next();
    T n[VEC], s[VEC];
#pragma unroll
    for (int r = 0; r < RY; ++r) ld16_shared<T>(t[r], nxt + cen0 + r * W);
    if (K != kKernelCopy) {
      ld16_shared<T>(n, cur + cen0 - W);       // row above the column
      ld16_shared<T>(s, cur + cen0 + RY * W);  // row below the column
    }
    if (kClamp && z == p.nz - 1) {
#pragma unroll
      for (int r = 0; r < RY; ++r)
#pragma unroll
        for (int i = 0; i < VEC; ++i) t[r][i] = c[r][i];
    }
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      // double precision is short of FP64 issue: nothing for rows outside
      if (sizeof(T) == 8 && ywarp + r >= p.dmax1) break;
      T o[VEC];
      if (K == kKernelCopy) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) o[i] = c[r][i];
      } else {
        T nn[VEC], ss[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          nn[i] = (r == 0) ? n[i] : c[r - 1][i];
          ss[i] = (r == RY - 1) ? s[i] : c[r + 1][i];
        }
        if (kClamp) {
          if (y + r == 0) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) nn[i] = c[r][i];
          }
          if (y + r == p.ny - 1) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) ss[i] = c[r][i];
          }
        }
        T left = shfl_up1(c[r][VEC - 1]);
        T right = shfl_down1(c[r][0]);
        if (xl == 0) left = cur[cen0 + r * W - 1];
        if (xl == LX - 1) right = cur[cen0 + r * W + VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          T w = (i == 0) ? left : c[r][i - 1];
          T e = (i == VEC - 1) ? right : c[r][i + 1];
          if (kClamp) {
            if (i == 0 && west_face) w = c[r][0];
            if (i == east_elem) e = c[r][i];
            // cc*c + cw*w + ce*e + cs*s + cn*n + cb*b + ct*t, left to right
            T v = R::mul(p.cc, c[r][i]);
            v = R::add(v, R::mul(p.cw, w));
            v = R::add(v, R::mul(p.ce, e));
            v = R::add(v, R::mul(p.cs, ss[i]));
            v = R::add(v, R::mul(p.cn, nn[i]));
            v = R::add(v, R::mul(p.cb, b[r][i]));
            v = R::add(v, R::mul(p.ct, t[r][i]));
            o[i] = v;
          } else {
            // c + e + w + s + n + b + t, left to right
            T v = R::add(c[r][i], e);
            v = R::add(v, w);
            v = R::add(v, ss[i]);
            v = R::add(v, nn[i]);
            v = R::add(v, b[r][i]);
            v = R::add(v, t[r][i]);
            o[i] = v;
          }
        }
      }
      if (ok && y + r < p.dmax1) {
        T *dst = p.out + (int64_t)z * p.plane + (int64_t)(y + r) * p.row + x;
        if (vec_in) {
          st16_global<T>(dst, o);
        } else {
#pragma unroll
          for (int i = 0; i < VEC; ++i)
            if (x + i >= p.dmin0 && x + i < p.dmax0) dst[i] = o[i];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RY; ++r)
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        b[r][i] = c[r][i];
        c[r][i] = t[r][i];
      }
    cur = nxt;
    done();
    if (!ok) return false;
    // Plane q is consumed by every thread: refill its stage with q + ns.
    const int q = z - zs + 1;
    if (Sync::kIssues && tid == 0 && q + ns < nplanes) issue(q + ns);
  }
  if constexpr (!Sync::kIssues) sync.last();  // plane ze, in registers since the last step
  return true;
}

}  // namespace psg
