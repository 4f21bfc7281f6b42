// The per-item body of the Himeno 19-point sweep (himeno19.cu's kernel and
// the batched kernel in batch.cu both run it).  One item is one tile of one
// problem swept over planes [zs, ze).  See himeno19.cu for the design.
#pragma once

#include "ps_device.cuh"
#include "ps_internal.h"

namespace psg {

constexpr int kHimTX = 128;      // widest tile in cells (32 lanes x float4)
constexpr int kHimW = kHimTX + 8;  // its shared p row width (4-cell halo each side)
constexpr int kHimCoef = 12;     // a0 a1 a2 a3 b0 b1 b2 c0 c1 c2 bnd wrk1

// Tiles of LX lanes side by side (32, 16 or 8): 4 LX cells by warps * 32 / LX rows.
// All hold the same cells, so coefficient stages have one size; no p stage is
// larger than the widest tile's (up to 8 warps).
__host__ __device__ constexpr int him_rows(int warps, int lx) { return warps * (32 / lx); }

struct HParams {
  float *out;
  int64_t row, plane;  // out pitch / plane in elements
  int dmin0, dmin1, dmin2, dmax0, dmax1, dmax2;
  int xbase, tiles_x, tiles, zlen;
  int64_t items;
  int nsp, nsc;
  float omega;
  double *partials;
  unsigned *ticket;
  double *result;
  int *err;
};

__host__ __device__ constexpr int h_bar_bytes(int n) { return 128 * ((8 * n + 127) / 128); }
// Every TMA destination starts on a 128-byte boundary.
__host__ __device__ constexpr uint32_t h_align128(uint32_t b) { return (b + 127u) & ~127u; }

// The lane's four cells of a row and the ones beside them.
template <int LX>
__device__ __forceinline__ void him_row6(const float *pl, int idx, int xl, float (&r)[6]) {
  float v[4];
  ld16_shared<float>(v, pl + idx);
  float l = shfl_up1(v[3]);
  float rr = shfl_down1(v[0]);
  ld_shared_if(xl == 0, pl + idx - 1, l);
  ld_shared_if(xl == LX - 1, pl + idx + 4, rr);
  r[0] = l;
  r[1] = v[0];
  r[2] = v[1];
  r[3] = v[2];
  r[4] = v[3];
  r[5] = rr;
}

// Position in a ring of mbarrier-signalled stages used in issue order.
struct HRing {
  int stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance(int n) {
    if (++stage == n) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

// The two rings of a CTA.  The last warp is the producer: one lane issues the
// boxes of every plane of the CTA's items in one sequence, so an item's first
// planes arrive while the one before it is computed.  Each plane lands on its
// stage's "full" mbarrier; consumer warps release stages one by one on "empty".
struct HimSmem {
  uint64_t *pfull, *cfull, *pempty, *cempty;
  float *pring, *cring;
  int p_elems, c_elems;  // stage strides
};
__device__ __forceinline__ HimSmem him_smem(unsigned char *smem, int nsp, int nsc, int warps) {
  HimSmem h;
  h.pfull = reinterpret_cast<uint64_t *>(smem);
  h.cfull = h.pfull + nsp;
  h.pempty = h.cfull + nsc;
  h.cempty = h.pempty + nsp;
  h.p_elems = (int)(h_align128((uint32_t)(kHimW * (warps + 2) * 4)) / 4);
  h.c_elems = kHimCoef * kHimTX * warps;
  h.pring = reinterpret_cast<float *>(smem + h_bar_bytes(2 * (nsp + nsc)));
  h.cring = h.pring + nsp * h.p_elems;
  return h;
}
__device__ __forceinline__ void him_init(const HimSmem &h, int nsp, int nsc, int warps) {
  for (int s = 0; s < nsp; ++s) {
    mbar_init(&h.pfull[s], 1);
    mbar_init(&h.pempty[s], warps);
  }
  for (int s = 0; s < nsc; ++s) {
    mbar_init(&h.cfull[s], 1);
    mbar_init(&h.cempty[s], warps);
  }
  fence_barrier_init();
}
// A bounded wait for copies still in flight, once a wait has given up.
__device__ __forceinline__ void him_drain(const HimSmem &h, int nsp, int nsc) {
  for (int s = 0; s < nsp; ++s) mbar_wait(&h.pfull[s], 0, nullptr, 1024);
  for (int s = 0; s < nsc; ++s) mbar_wait(&h.cfull[s], 0, nullptr, 1024);
}

// Producer, one lane: tile `tile` of p over planes [zs, ze).  pmap is p0's halo
// map, cmaps the 12 coefficient maps in order.  False if a bounded wait gave up.
__device__ __forceinline__ bool himeno_produce(const CUtensorMap *pmap, const CUtensorMap *cmaps,
                                               const HParams &p, const HimSmem &h, int warps,
                                               int lx, int tile, int zs, int ze, HRing &pprod,
                                               HRing &cprod) {
  const int tx = 4 * lx, ty = him_rows(warps, lx);
  const uint32_t p_bytes = (uint32_t)((tx + 8) * (ty + 2) * 4);
  const int c_tile = tx * ty;
  const int x0 = p.xbase + (tile % p.tiles_x) * tx;
  const int y0 = p.dmin1 + (tile / p.tiles_x) * ty;
  // planes zs-1 and zs, then for each step the plane above and the coefficients
  for (int q = -2; q < ze - zs; ++q) {
    const int s = pprod.stage;
    if (!mbar_wait(&h.pempty[s], pprod.phase ^ 1u, p.err)) return false;
    mbar_arrive_expect_tx(&h.pfull[s], p_bytes);
    tma_load_3d(h.pring + s * h.p_elems, pmap, x0 - 4, y0 - 1, zs + 1 + q, &h.pfull[s]);
    pprod.advance(p.nsp);
    if (q < 0) continue;
    const int c = cprod.stage;
    if (!mbar_wait(&h.cempty[c], cprod.phase ^ 1u, p.err)) return false;
    mbar_arrive_expect_tx(&h.cfull[c], (uint32_t)(h.c_elems * 4));
    float *dst = h.cring + c * h.c_elems;
#pragma unroll 1
    for (int a = 0; a < kHimCoef; ++a)
      tma_load_3d(dst + a * c_tile, cmaps + a, x0, y0, zs + q, &h.cfull[c]);
    cprod.advance(p.nsc);
  }
  return true;
}

// Consumer warp: sweeps the tile; acc accumulates ss*ss when GOSA.  False if a
// bounded wait gave up (the producer's waits for this warp then give up too).
template <bool GOSA, int LX>
__device__ __forceinline__ bool himeno_consume(const HParams &p, const HimSmem &h, int warps,
                                               int tile, int zs, int ze, HRing &pcons,
                                               HRing &prel, HRing &ccons, float &acc) {
  typedef RN<float> R;
  constexpr int kTX = 4 * LX, kW = kTX + 8, kNumCoef = kHimCoef;
  const int TY = him_rows(warps, LX), c_tile = kTX * TY;
  const int lane = threadIdx.x, xl = lane % LX;
  const int row = threadIdx.y * (32 / LX) + lane / LX;
  const int cen = (row + 1) * kW + 4 + xl * 4;
  const int cidx = row * kTX + xl * 4;

  const int x = p.xbase + (tile % p.tiles_x) * kTX + xl * 4;
  const int y = p.dmin1 + (tile / p.tiles_x) * TY + row;
  const bool row_in = (y < p.dmax1);
  const bool vec_in = (x >= p.dmin0) && (x + 4 <= p.dmax0);

  auto wait_p = [&](const float *&pl) {
    pl = h.pring + pcons.stage * h.p_elems;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&h.pfull[pcons.stage], pcons.phase, p.err));
    pcons.advance(p.nsp);
    return ok;
  };
  auto release_p = [&]() {
    if (lane == 0) mbar_arrive(&h.pempty[prel.stage]);
    prel.advance(p.nsp);
  };
  const float *pm, *pc, *pp;
  if (!wait_p(pm) || !wait_p(pc)) return false;  // planes zs-1 and zs
  for (int z = zs; z < ze; ++z) {
    if (!wait_p(pp)) return false;  // plane z+1
    const float *cf = h.cring + ccons.stage * h.c_elems;  // coefficients of plane z
    if (!__all_sync(0xffffffffu, mbar_wait(&h.cfull[ccons.stage], ccons.phase, p.err)))
      return false;

    float Zc[6], Zym[6], Zyp[6], Zpc[6], Zmc[6];
    float Zpyp[4], Zpym[4], Zmyp[4], Zmym[4];
    him_row6<LX>(pc, cen, xl, Zc);
    him_row6<LX>(pc, cen - kW, xl, Zym);
    him_row6<LX>(pc, cen + kW, xl, Zyp);
    him_row6<LX>(pp, cen, xl, Zpc);
    him_row6<LX>(pm, cen, xl, Zmc);
    ld16_shared<float>(Zpyp, pp + cen + kW);
    ld16_shared<float>(Zpym, pp + cen - kW);
    ld16_shared<float>(Zmyp, pm + cen + kW);
    ld16_shared<float>(Zmym, pm + cen - kW);
    float co[kNumCoef][4];
#pragma unroll
    for (int a = 0; a < kNumCoef; ++a) ld16_shared<float>(co[a], cf + a * c_tile + cidx);

    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // s0 = a0*p(k+1) + a1*p(j+1) + a2*p(i+1) + b0*(..) + b1*(..) + b2*(..)
      //    + c0*p(k-1) + c1*p(j-1) + c2*p(i-1) + wrk1   (left to right)
      float s0 = R::mul(co[0][i], Zpc[i + 1]);
      s0 = R::add(s0, R::mul(co[1][i], Zyp[i + 1]));
      s0 = R::add(s0, R::mul(co[2][i], Zc[i + 2]));
      float t0 = R::add(R::sub(R::sub(Zpyp[i], Zpym[i]), Zmyp[i]), Zmym[i]);
      s0 = R::add(s0, R::mul(co[4][i], t0));
      float t1 = R::add(R::sub(R::sub(Zyp[i + 2], Zym[i + 2]), Zyp[i]), Zym[i]);
      s0 = R::add(s0, R::mul(co[5][i], t1));
      float t2 = R::add(R::sub(R::sub(Zpc[i + 2], Zmc[i + 2]), Zpc[i]), Zmc[i]);
      s0 = R::add(s0, R::mul(co[6][i], t2));
      s0 = R::add(s0, R::mul(co[7][i], Zmc[i + 1]));
      s0 = R::add(s0, R::mul(co[8][i], Zym[i + 1]));
      s0 = R::add(s0, R::mul(co[9][i], Zc[i]));
      s0 = R::add(s0, co[11][i]);
      // ss = (s0*a3 - p) * bnd ; p1 = p + omega*ss
      const float ss = R::mul(R::sub(R::mul(s0, co[3][i]), Zc[i + 1]), co[10][i]);
      o[i] = R::add(Zc[i + 1], R::mul(p.omega, ss));
      if (GOSA) {
        const bool in = row_in && (x + i >= p.dmin0) && (x + i < p.dmax0);
        if (in) acc = R::add(acc, R::mul(ss, ss));
      }
    }
    __syncwarp();
    release_p();  // plane z-1
    if (lane == 0) mbar_arrive(&h.cempty[ccons.stage]);
    ccons.advance(p.nsc);
    if (row_in) {
      float *dst = p.out + (int64_t)z * p.plane + (int64_t)y * p.row + x;
      if (vec_in) {
        st16_global<float>(dst, o);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (x + i >= p.dmin0 && x + i < p.dmax0) dst[i] = o[i];
      }
    }
    pm = pc;
    pc = pp;
  }
  __syncwarp();
  release_p();  // planes ze-1 and ze
  release_p();
  return true;
}

}  // namespace psg
