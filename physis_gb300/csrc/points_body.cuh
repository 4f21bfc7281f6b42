// The point-list stencil sweep, written once for two builds:
//  * points.cu compiles it with a run-time point table (PtsTableSpec): one
//    kernel serves every registered stencil;
//  * jit.cpp compiles it with NVRTC for one stencil at a time, with a
//    generated spec whose offsets, plane lags, weights and tile geometry are
//    compile-time constants (the point loop unrolls into 16-byte shared loads
//    at immediate offsets, each issued once for all the cells that use it).
// No header dependencies beyond ps_arith.cuh, so NVRTC can compile it from
// memory.  See points.cu for the design.
#pragma once

#include "ps_arith.cuh"

namespace psg {

constexpr int kPtsVX = 4;         // cells per lane and row; a tile is kPtsVX * lx cells wide
constexpr int kPtsMaxPoints = 64;
// Shared memory: point table (run-time spec only: offsets, lags, weights),
// then the ring's mbarriers (full, empty, raw), then the ring (128-byte
// aligned stages).
constexpr int kPtsTableBytes = kPtsMaxPoints * (4 + 4 + 8);
constexpr int kPtsMaxStages = 16;
constexpr int kPtsRingOffset = kPtsTableBytes + 24 * kPtsMaxStages;
// Opaque TMA descriptor (the layout of CUtensorMap: 128 bytes, 64-aligned).
struct alignas(64) PtsTmap {
  unsigned long long opaque[16];
};
enum { kPtsNone = 0, kPtsPeriodic = 1, kPtsClamp = 2 };

template <typename T>
struct PtsParams {
  const T *in;
  T *out;            // may equal in (red/black)
  long long row;     // pitch in elements
  long long plane;   // elements per z-plane
  int nx, ny, nz;
  int dmin0, dmin1, dmin2, dmax0, dmax1, dmax2;
  int boundary;      // kPtsNone / kPtsPeriodic / kPtsClamp
  int color;         // -1 every cell, 0 red, 1 black
  int n;             // points
  int rxl, rxh, ryl, ryh, rzl, rzh;  // extent of the offsets per axis
  int lp, w, rows_h, nstage, plane_elems;
  int pstride;       // ring stage stride in elements (128-byte multiple)
  int lx;            // lanes side by side in x: 32, 16 or 8 (the others take rows further down)
  int xbase, tiles_x, tiles, zlen;
  long long items;
  int early;         // the next launch's CTAs may take places while this one runs
  int *err;          // device error word (bounded waits that give up)
  int off[kPtsMaxPoints];  // shared offset of point i relative to the cell
  int lag[kPtsMaxPoints];  // rzl + dz_i: the point's plane relative to z - rzl
  T wt[kPtsMaxPoints];
};

// Grid index of coordinate i on an axis of n cells.  Periodic: i mod n, which
// equals the reference's (i + n) % n for every i >= -n (the host admits only
// offsets with |d| <= n, so every read that is used has i >= -n; halo cells
// that are never read may lie further out and still land inside the grid).
// Clamp, and the never-read halo of boundary "none": the nearest face.
__device__ __forceinline__ int pts_map_axis(int i, int n, int boundary) {
  if (boundary == kPtsPeriodic) {
    if ((unsigned)i < (unsigned)n) return i;
    const int m = i % n;
    return m < 0 ? m + n : m;
  }
  return min(max(i, 0), n - 1);
}

// The cells of a tile's TMA box that lie outside the grid and that some cell
// of the tile can read (at most the offsets' extent beyond a face): whole rows
// beyond a y face, then the columns beyond an x face of the other rows.  TMA
// filled them with zeros; cell e is rewritten with the value the boundary rule
// maps it to.  Only edge tiles of periodic and clamped stencils have any.
struct PtsHalo {
  int xs, ys;              // box origin
  int c0, ncol, r0, rtop;  // outside rows: columns c0 .. c0 + ncol, rtop rows from r0, then from rin1
  int rin0, rin1;          // rows inside the grid
  int clow, cin1, nc;      // outside columns: clow from c0, then from cin1, nc in all
  int rows, total;         // cells in outside rows, cells in all
};
template <typename T>
__device__ __forceinline__ PtsHalo pts_halo(const PtsParams<T> &p, int x0, int y0, int W) {
  PtsHalo h;
  h.xs = x0 - p.lp;
  h.ys = y0 - p.ryl;
  h.c0 = max(0, -p.rxl - h.xs);
  const int c1 = min(W, p.nx + p.rxh - h.xs);
  h.ncol = c1 - h.c0;
  h.r0 = max(0, -p.ryl - h.ys);
  const int r1 = min(p.rows_h, p.ny + p.ryh - h.ys);
  h.rin0 = max(h.r0, -h.ys);
  h.rin1 = min(r1, p.ny - h.ys);
  h.rtop = h.rin0 - h.r0;
  h.clow = max(h.c0, -h.xs) - h.c0;
  h.cin1 = min(c1, p.nx - h.xs);
  h.nc = h.clow + (c1 - h.cin1);
  h.rows = (h.rtop + (r1 - h.rin1)) * h.ncol;
  h.total = h.rows + h.nc * (h.rin1 - h.rin0);
  return h;
}
// Cell e of the halo: its offset in the box (return value) and in the grid
// plane that its values come from.
template <typename T>
__device__ __forceinline__ int pts_halo_cell(const PtsParams<T> &p, const PtsHalo &h, int e, int W,
                                             long long *src) {
  int r, c;
  if (e < h.rows) {
    const int k = e / h.ncol;
    c = h.c0 + (e - k * h.ncol);
    r = k < h.rtop ? h.r0 + k : h.rin1 + (k - h.rtop);
  } else {
    const int k = (e - h.rows) / h.nc, m = (e - h.rows) - k * h.nc;
    r = h.rin0 + k;
    c = m < h.clow ? h.c0 + m : h.cin1 + (m - h.clow);
  }
  *src = (long long)pts_map_axis(h.ys + r, p.ny, p.boundary) * p.row +
         pts_map_axis(h.xs + c, p.nx, p.boundary);
  return r * W + c;
}

// The run-time spec: the point table travels in the kernel parameters and is
// copied to shared memory; the tile geometry comes from the parameters.
struct PtsTableSpec {
  static constexpr bool kStatic = false, kWideHalo = true;
  template <typename T>
  static __device__ __forceinline__ int lx(const PtsParams<T> &p) { return p.lx; }
  template <typename T>
  static __device__ __forceinline__ int w(const PtsParams<T> &p) { return p.w; }
  template <typename T>
  static __device__ __forceinline__ int nstage(const PtsParams<T> &p) { return p.nstage; }
  template <typename T>
  static __device__ __forceinline__ int pstride(const PtsParams<T> &p) { return p.pstride; }
};

// 16 bytes of a shared row as VEC cells.
template <typename T>
struct PtsVec {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};
template <typename T>
__device__ __forceinline__ PtsVec<T> pts_ld16(const T *src) {
  union { uint4 u; PtsVec<T> v; } c;
  c.u = *reinterpret_cast<const uint4 *>(src);
  return c.v;
}

// Compiled spec.  acc[r][c] (+)= w * the point's value for the cells of row r:
// lane l of the LX side by side owns the VEC = 16 / sizeof(T) consecutive cells
// from LX VEC j + VEC l of each of the 4 / VEC column groups j.  Every read is an
// aligned 16-byte shared load (conflict-free, as a load goes by quarter warps
// and eight lanes are always consecutive); a point's row and x offset only
// select cells of such vectors, and the compiler issues each vector once per
// step however many points and rows use it (a 27-point stencil needs 3 planes
// x 6 rows x 3 vectors for 16 cells, 3.4 loads a cell).
template <typename T, int RY, bool UNIT, class S, int K>
__device__ __forceinline__ void pts_point(T (&acc)[RY][kPtsVX], const T *const *pl, int cell0) {
  typedef RN<T> R;
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int DX = S::kDx[K], DY = S::kDy[K], LAG = S::kLag[K];
  constexpr T wk = (T)S::kWt[K];
#pragma unroll
  for (int r = 0; r < RY; ++r)
#pragma unroll
    for (int c = 0; c < kPtsVX; ++c) {
      const int j = c / VEC, i = c % VEC + DX;
      const int vi = (i + 8 * VEC) / VEC - 8, e = i - vi * VEC;
      const T v = pts_ld16<T>(pl[LAG] + cell0 + (r + DY) * S::kW + j * S::kLX * VEC + vi * VEC)
                      .v[e];
      const T t = UNIT ? v : R::mul(wk, v);
      acc[r][c] = K == 0 ? t : R::add(acc[r][c], t);
    }
}
template <typename T, int RY, bool UNIT, class S, int K>
__device__ __forceinline__ void pts_points(T (&acc)[RY][kPtsVX], const T *const *pl, int cell0) {
  if constexpr (K < S::kN) {
    pts_point<T, RY, UNIT, S, K>(acc, pl, cell0);
    pts_points<T, RY, UNIT, S, K + 1>(acc, pl, cell0);
  }
}

// Table spec: acc[r][j] (+)= w * src[r*W + LX*j]; `first` starts the sum.
template <typename T, int RY, bool UNIT>
__device__ __forceinline__ void pts_term(T (&acc)[RY][kPtsVX], const T *src, int W, int LX, T wk,
                                         bool first) {
  typedef RN<T> R;
#pragma unroll
  for (int r = 0; r < RY; ++r)
#pragma unroll
    for (int j = 0; j < kPtsVX; ++j) {
      const T v = src[r * W + LX * j];
      const T t = UNIT ? v : R::mul(wk, v);
      acc[r][j] = first ? t : R::add(acc[r][j], t);
    }
}

// Position of an item (tile column, tile row, z-chunk), advanced by a fixed
// number of items without divisions.
struct PtsPos {
  int tx, ty, chunk;
};
__device__ __forceinline__ PtsPos pts_split(unsigned item, unsigned tiles_x, unsigned tiles) {
  const unsigned chunk = item / tiles, tile = item - chunk * tiles, ty = tile / tiles_x;
  PtsPos q;
  q.chunk = (int)chunk;
  q.ty = (int)ty;
  q.tx = (int)(tile - ty * tiles_x);
  return q;
}
__device__ __forceinline__ void pts_advance(PtsPos &q, const PtsPos &step, int tiles_x,
                                            int tiles_y) {
  q.tx += step.tx;
  q.ty += step.ty;
  q.chunk += step.chunk;
  if (q.tx >= tiles_x) {
    q.tx -= tiles_x;
    ++q.ty;
  }
  if (q.ty >= tiles_y) {
    q.ty -= tiles_y;
    ++q.chunk;
  }
}

// The sweep: persistent (z-chunk, tile) items, a ring of planes, the points
// summed in order.  The last warp of the CTA is the producer, the others
// consume.  Each plane of a tile arrives by one TMA box load on its stage's
// "full" mbarrier; a consumer warp that is done with a stage arrives on its
// "empty" mbarrier, so warps run up to a ring apart and no step ends in a CTA
// barrier.  Planes are loaded in one sequence over all of the CTA's items: an
// item's first planes arrive while the previous item is being computed (a 2D
// grid is one plane per item).  On the edge tiles of periodic and clamped
// stencils the out-of-grid cells of the box are rewritten through the boundary
// map by the producer warp before it completes the stage's "full" barrier (the
// box then lands on a barrier of its own, "raw"; with boundary "none" those
// cells are never read).  A consumer whose bounded wait gives up computes and
// stores nothing more, but keeps its arrivals going so that the CTA ends.
// `smem_raw` is the dynamic shared memory, `tmap` the TMA descriptor of `in`.
template <typename T, int RY, bool UNIT, class S>
__device__ __forceinline__ void pts_body(const PtsParams<T> &p, const void *tmap,
                                         unsigned char *smem_raw) {
  constexpr int VEC = 16 / (int)sizeof(T);
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  int *s_off = reinterpret_cast<int *>(smem);
  int *s_lag = s_off + kPtsMaxPoints;
  T *s_w = reinterpret_cast<T *>(smem + kPtsMaxPoints * 8);
  unsigned long long *full = reinterpret_cast<unsigned long long *>(smem + kPtsTableBytes);
  unsigned long long *empty = full + kPtsMaxStages, *raw = empty + kPtsMaxStages;
  T *ring = reinterpret_cast<T *>(smem + kPtsRingOffset);
  const int W = S::w(p), NST = S::nstage(p), PS = S::pstride(p), LX = S::lx(p);
  const int TX = kPtsVX * LX;

  const int lane = threadIdx.x, warp = threadIdx.y;
  const int consumers = blockDim.y - 1;  // warps
  const int tid = warp * 32 + lane;
  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], consumers);
      mbar_init(&raw[s], 1);
    }
    fence_barrier_init();
  }
  if (!S::kStatic) {
    for (int i = tid; i < p.n; i += blockDim.x * blockDim.y) {
      s_off[i] = p.off[i];
      s_lag[i] = p.lag[i];
      s_w[i] = p.wt[i];
    }
  }
  __syncthreads();
  if (p.early) launch_dependents();
  wait_for_predecessors();

  const int TY = consumers * RY * (32 / LX);
  const int zext = p.rzl + p.rzh;
  const int tiles_y = p.tiles / p.tiles_x;
  PtsPos pos = pts_split(blockIdx.x, p.tiles_x, p.tiles);
  const PtsPos step = pts_split(gridDim.x, p.tiles_x, p.tiles);

  if (warp == consumers) {
    const unsigned bytes = (unsigned)(p.plane_elems * (int)sizeof(T));
    int slot = 0, fslot = 0;    // next slot to fill, next slot whose halo is to be rewritten
    unsigned phase = 0;         // bit s: parity of slot s's next fill
    unsigned raws = 0;          // bit s: parity of the next box landing on raw[s]
    bool used = false;          // every slot has been filled once
    for (long long item = blockIdx.x; item < p.items; item += gridDim.x) {
      const int zs = p.dmin2 + pos.chunk * p.zlen;
      const int n = min(p.zlen, p.dmax2 - zs) + zext;
      const int x0 = p.xbase + pos.tx * TX, y0 = p.dmin1 + pos.ty * TY;
      pts_advance(pos, step, p.tiles_x, tiles_y);
      PtsHalo h;
      h.total = 0;
      if (p.boundary != kPtsNone &&
          !(x0 - p.rxl >= 0 && x0 + TX + p.rxh <= p.nx && y0 - p.ryl >= 0 &&
            y0 - p.ryl + p.rows_h <= p.ny))
        h = pts_halo(p, x0, y0, W);
      const bool fix = h.total > 0;
      // this lane's first halo cells, the same ones in every plane
      constexpr int kBatch = 5;
      int dst[kBatch];
      long long src[kBatch];
      if (fix) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int e = lane + 32 * i;
          dst[i] = e < h.total ? pts_halo_cell(p, h, e, W, &src[i]) : -1;
        }
      }
      // their values in plane q, fetched a plane ahead of the rewrite
      T v[kBatch];
      auto fetch = [&](int q) {
        const T *plane = p.in + (long long)pts_map_axis(zs - p.rzl + q, p.nz, p.boundary) * p.plane;
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
          if (dst[i] >= 0) v[i] = plane[src[i]];
      };
      if (fix) fetch(0);
      int filled = 0, done = 0;  // planes whose box was issued / whose stage is complete
      while (done < n) {
        // fill free stages; block for one only when there is nothing to rewrite
        while (filled < n && filled - done < NST) {
          bool free = !used;
          if (used) {
            void *e = &empty[slot];
            const unsigned par = ((phase >> slot) & 1u) ^ 1u;  // the last fill's readers
            if (fix && filled > done) {
              free = __all_sync(0xffffffffu, mbar_test_wait(e, par));
              if (!free) break;
            } else if (!__all_sync(0xffffffffu, mbar_wait(e, par, p.err))) {
              return;
            }
          }
          if (lane == 0) {
            void *bar = fix ? &raw[slot] : &full[slot];
            mbar_arrive_expect_tx(bar, bytes);
            tma_load_3d(ring + slot * PS, tmap, x0 - p.lp, y0 - p.ryl,
                        pts_map_axis(zs - p.rzl + filled, p.nz, p.boundary), bar);
          }
          phase ^= 1u << slot;
          if (++slot == NST) {
            slot = 0;
            used = true;
          }
          ++filled;
          if (!fix) {
            ++done;
            if (++fslot == NST) fslot = 0;
          }
        }
        if (!fix) continue;
        // rewrite the halo of plane `done`
        T *box = ring + fslot * PS;
        if (!__all_sync(0xffffffffu, mbar_wait(&raw[fslot], (raws >> fslot) & 1u, p.err))) return;
        raws ^= 1u << fslot;
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
          if (dst[i] >= 0) box[dst[i]] = v[i];
        const T *plane =
            p.in + (long long)pts_map_axis(zs - p.rzl + done, p.nz, p.boundary) * p.plane;
        // the rest of a wide halo, kMore loads of a lane in flight at a time
        constexpr int kMore = S::kWideHalo ? 4 : 1;
        for (int e0 = lane + 32 * kBatch; e0 < h.total; e0 += 32 * kMore) {
          int to[kMore];
          T u[kMore];
#pragma unroll
          for (int i = 0; i < kMore; ++i) {
            const int e = e0 + 32 * i;
            long long from = 0;
            to[i] = e < h.total ? pts_halo_cell(p, h, e, W, &from) : -1;
            u[i] = plane[from];
          }
#pragma unroll
          for (int i = 0; i < kMore; ++i)
            if (to[i] >= 0) box[to[i]] = u[i];
        }
        // these writes precede the consumers' reads (the arrival below) and
        // the box that reuses the stage (the proxy fence)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[fslot]);
        if (++fslot == NST) fslot = 0;
        if (++done < n) fetch(done);
      }
    }
    // the last copies land before the CTA may end (the consumers see to that
    // themselves unless one of them gave up)
    for (int s = 0; s < NST; ++s)
      if (used || s < slot) mbar_wait(&full[s], ((phase >> s) & 1u) ^ 1u, nullptr, 1u << 16);
    return;
  }

  // first cell of the lane's first row relative to a plane: its vector
  // (compiled spec) or its first lane-strided cell (table spec)
  const int xl = lane % LX, row0 = (warp * (32 / LX) + lane / LX) * RY;
  const int cell0 = S::kStatic ? (row0 + p.ryl) * W + p.lp + xl * VEC : row0 * W + xl;
  bool ok = true;
  // Slot of plane z - rzl of the current step, the next slot to wait for, and
  // the parity of each slot's next completion (bit s).
  int cs = 0, wslot = 0;
  unsigned phase = 0;
  for (long long item = blockIdx.x; item < p.items; item += gridDim.x) {
    const int zs = p.dmin2 + pos.chunk * p.zlen;
    const int ze = min(zs + p.zlen, p.dmax2);
    const int x0 = p.xbase + pos.tx * TX;
    const int y0 = p.dmin1 + pos.ty * TY;
    pts_advance(pos, step, p.tiles_x, tiles_y);
    // cells of the lane in the domain: bit c of colmask, bit r of rowmask
    unsigned colmask = 0, rowmask = 0;
#pragma unroll
    for (int c = 0; c < kPtsVX; ++c) {
      const int x = S::kStatic ? x0 + (c / VEC) * LX * VEC + xl * VEC + c % VEC
                               : x0 + xl + LX * c;
      if (x >= p.dmin0 && x < p.dmax0) colmask |= 1u << c;
    }
#pragma unroll
    for (int r = 0; r < RY; ++r)
      if (y0 + row0 + r < p.dmax1) rowmask |= 1u << r;
    const bool whole = colmask == (1u << kPtsVX) - 1u && rowmask == (1u << RY) - 1u;
    const bool any = __any_sync(0xffffffffu, colmask && rowmask);  // else nothing to do
    T *dst = p.out + (long long)zs * p.plane + (long long)(y0 + row0) * p.row + x0 +
             xl * (S::kStatic ? VEC : 1);

    int waited = 0;  // planes of this item that have landed
    for (int z = zs; z < ze; ++z, dst += p.plane) {
      const int need = z - zs + zext;  // newest plane this step reads
      while (waited <= need) {
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&full[wslot], (phase >> wslot) & 1u, p.err));
        phase ^= 1u << wslot;
        ++waited;
        if (++wslot == NST) wslot = 0;
      }

      if (ok && any) {
        T acc[RY][kPtsVX];
        if constexpr (S::kStatic) {
          const T *pl[S::kPlanes];
#pragma unroll
          for (int l = 0; l < S::kPlanes; ++l) {
            int s = cs + l;
            if (s >= NST) s -= NST;
            pl[l] = ring + s * PS;
          }
          pts_points<T, RY, UNIT, S, 0>(acc, pl, cell0);
          if (p.color >= 0) {
            // the lane's other-colour cells keep their value: nothing writes
            // them in this launch, so a whole vector can be stored
#pragma unroll
            for (int r = 0; r < RY; ++r)
#pragma unroll
              for (int c = 0; c < kPtsVX; ++c) {
                const int x = x0 + (c / VEC) * LX * VEC + xl * VEC + c % VEC;
                const T own =
                    pts_ld16<T>(pl[S::kCentre] + cell0 + r * S::kW + (c / VEC) * LX * VEC)
                        .v[c % VEC];
                if ((x + y0 + row0 + r + z + p.color) & 1) acc[r][c] = own;
              }
          }
#pragma unroll
          for (int r = 0; r < RY; ++r) {
            if (!whole && !((rowmask >> r) & 1u)) continue;
#pragma unroll
            for (int j = 0; j < kPtsVX / VEC; ++j) {
              const unsigned m = (colmask >> (j * VEC)) & ((1u << VEC) - 1u);
              T *d = dst + r * p.row + j * LX * VEC;
              if (whole || m == (1u << VEC) - 1u) {
                union { uint4 u; T t[VEC]; } c;
#pragma unroll
                for (int i = 0; i < VEC; ++i) c.t[i] = acc[r][j * VEC + i];
                *reinterpret_cast<uint4 *>(d) = c.u;
              } else {
#pragma unroll
                for (int i = 0; i < VEC; ++i)
                  if ((m >> i) & 1u) d[i] = acc[r][j * VEC + i];
              }
            }
          }
        } else {
          for (int k = 0; k < p.n; ++k) {
            int s = cs + s_lag[k];
            if (s >= NST) s -= NST;
            pts_term<T, RY, UNIT>(acc, ring + s * PS + cell0 + s_off[k], W, LX, s_w[k],
                                  k == 0);
          }
#pragma unroll
          for (int r = 0; r < RY; ++r) {
            const int y = y0 + row0 + r;
            const bool row_on = ((rowmask >> r) & 1u) &&
                                (p.color < 0 || ((x0 + xl + y + z + p.color) & 1) == 0);
            if (row_on) {
#pragma unroll
              for (int j = 0; j < kPtsVX; ++j)
                if ((colmask >> j) & 1u) dst[r * p.row + LX * j] = acc[r][j];
            }
          }
        }
      }
      // plane z - rzl is done with; after the item's last step all its planes
      __syncwarp();
      const int freed = z + 1 < ze ? 1 : 1 + zext;
      for (int f = 0; f < freed; ++f) {
        if (lane == 0) mbar_arrive(&empty[cs]);
        if (++cs == NST) cs = 0;
      }
    }
  }
}

}  // namespace psg
