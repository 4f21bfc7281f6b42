// Point-list stencils and red/black sweeps on GB300 (sm_103a).
//
// Replaces the translator-generated run kernels of the reference
// (translator/cuda_runtime_builder.cc:1099-1228, red/black offsets
// 1206-1226; REF loops translator/reference_runtime_builder.cc:585-664) for
// stencils of the form
//     out(x,y,z) = w0*in(p0) + w1*in(p1) + ... + w(n-1)*in(p(n-1))
// evaluated left to right, p_i = (x+dx_i, y+dy_i, z+dz_i) mapped per axis by a
// boundary rule (none / periodic (i + n) % n, include/physis/physis_cuda.h:
// 247-269 / clamp to the grid).  With unit weights this is exactly the
// neighbour sums of the reference's system tests (27-point, 9-point 2D,
// 3-point 1D, asymmetric, hole, periodic variants, red/black).
//
// Design.  A tile is 128 cells wide in x and warps*RY rows high, or 64 or 32
// cells wide and two or four times as high (points_lanes); a lane owns RY rows
// of 16 bytes of consecutive cells (two such groups for 8-byte types) in the
// compiled form, RY rows of four lane-strided cells in the table form; work items are (z-chunk, tile) pairs in chunk-major order taken round-robin
// by a persistent grid, as in the 7-point kernels.
// * Each z-plane of the tile plus its x/y halo arrives in a ring of
//   shared-memory planes by one TMA 3D box load (mbarrier per stage, bounded
//   waits).  A box cannot wrap and fills cells outside the grid with zeros,
//   so on the edge tiles of periodic and clamped stencils those halo cells
//   that the offsets reach are then rewritten through the boundary map
//   (periodic cells from the opposite face, clamped ones from the face); the
//   compute loop is the same for every rule.
// * The ring holds rzl + rzh + 1 planes for the stencil's z extent plus one or
//   two planes in flight ahead of the newest one a step reads; loading runs on
//   into a CTA's next item.  A producer warp issues the boxes and rewrites the
//   halo cells (their values fetched a plane ahead); consumer warps release
//   stages one by one, so no step ends in a CTA barrier.
// Bound: issue slots where the stencil is wide (27 weighted points: 26 adds
// and, products being shared by a lane's cells, 7 multiplies of 48
// instructions a cell), HBM where it is narrow.  Measured, float, per sweep,
// against lane-strided cells, halos rewritten by all threads between two CTA
// barriers and no loading across items: 27 points periodic at 320 x 300 x 257
// 55 against 198 us, 9 points periodic at 4099 x 3001 18 against 41 us, one
// colour of the 7-point clamped stencil at 319 x 257 x 255 28 against 94 us.
// * The sweep body (points_body.cuh) is compiled two ways: here with the
//   point table (shared-memory offset, plane lag, weight) copied to shared
//   memory once per CTA and walked in order, and by jit.cpp with NVRTC per
//   stencil, the table baked in as constants.  The runtime uses the compiled
//   form when NVRTC is present (PS_POINTS_JIT=0 forces the table form).
// * Arithmetic is round-to-nearest without FMA contraction in the point
//   order, so results are bit-identical to the REF loops.
// * Red/black (color 0/1) writes only cells with (x + y + z + color) even --
//   the cells the REF loop start min + ((min & 1) ^ ((y + z + color) % 2))
//   visits -- in place.  The host admits only stencils whose non-centre
//   points all have odd parity, so a pass never reads a cell it writes
//   (other than each cell's own centre) and the parallel result equals the
//   sequential REF one.
#include <algorithm>
#include <array>
#include <cstdlib>
#include <cstring>
#include <map>
#include <type_traits>

#include "points_body.cuh"
#include "ps_device.cuh"
#include "ps_internal.h"

namespace psg {
namespace {

template <typename T, int RY, bool UNIT>
__global__ void __launch_bounds__(32 * 17, 1)
pts_kernel(const __grid_constant__ PtsParams<T> p, const __grid_constant__ PtsTmap tm) {
  extern __shared__ __align__(128) unsigned char smem[];
  pts_body<T, RY, UNIT, PtsTableSpec>(p, &tm, smem);
}

// Planes in flight ahead of the newest plane a step reads: two where four CTAs
// still fit an SM, else one (27 points periodic, float, 320 x 300 x 257: 57.9 us
// a sweep, against 59.8 with five CTAs and one plane and 59.9 with three CTAs
// and three; red/black 319 x 257 x 255 35.8, 37.2 and 37.9 us a colour).
size_t ring_bytes(const PointsArgs &a, const int lo[3], const int hi[3], int w, int h,
                  int *nstage) {
  const size_t stage = ((size_t)w * h * a.in.esz + 127) / 128 * 128;
  const int planes = hi[2] - lo[2] + 1;
  const size_t fixed = 128 + (size_t)kPtsRingOffset;
  *nstage = planes + (planes + 2 <= kPtsMaxStages && fixed + (planes + 2) * stage <= 56 * 1024 ? 2 : 1);
  return fixed + (size_t)*nstage * stage;
}

// Offsets' extent per axis: lo <= 0 <= hi.
void extents(const PointsArgs &a, int lo[3], int hi[3]) {
  for (int d = 0; d < 3; ++d) lo[d] = hi[d] = 0;
  for (int i = 0; i < a.n; ++i)
    for (int d = 0; d < 3; ++d) {
      lo[d] = a.d[i][d] < lo[d] ? a.d[i][d] : lo[d];
      hi[d] = a.d[i][d] > hi[d] ? a.d[i][d] : hi[d];
    }
}

// Fills everything but zlen / items (those need the occupancy).
template <typename T>
void fill_params(const PointsArgs &a, int warps, int ry, int lx, PtsParams<T> *pp) {
  constexpr int VEC = 16 / (int)sizeof(T);
  PtsParams<T> &p = *pp;
  memset(&p, 0, sizeof(p));
  p.in = static_cast<const T *>(a.in.ptr);
  p.out = static_cast<T *>(a.out.ptr);
  p.row = a.in.pitch / (long long)sizeof(T);
  p.plane = p.row * a.in.ny;
  p.nx = a.in.nx;
  p.ny = a.in.ny;
  p.nz = a.in.nz;
  p.dmin0 = a.dom.min[0];
  p.dmin1 = a.dom.min[1];
  p.dmin2 = a.dom.min[2];
  p.dmax0 = a.dom.max[0];
  p.dmax1 = a.dom.max[1];
  p.dmax2 = a.dom.max[2];
  p.boundary = a.boundary;
  p.color = a.color;
  p.n = a.n;
  int lo[3], hi[3];
  extents(a, lo, hi);
  p.rxl = -lo[0];
  p.rxh = hi[0];
  p.ryl = -lo[1];
  p.ryh = hi[1];
  p.rzl = -lo[2];
  p.rzh = hi[2];
  p.lp = (-lo[0] + VEC - 1) / VEC * VEC;
  const int rp = (hi[0] + VEC - 1) / VEC * VEC;
  const int TX = kPtsVX * lx, TY = warps * ry * (32 / lx);
  p.lx = lx;
  p.w = p.lp + TX + rp;
  p.rows_h = TY + p.ryl + hi[1];
  ring_bytes(a, lo, hi, p.w, p.rows_h, &p.nstage);
  p.plane_elems = p.rows_h * p.w;
  p.pstride = (int)(((size_t)p.plane_elems * sizeof(T) + 127) / 128 * 128 / sizeof(T));
  p.err = a.err;
  for (int i = 0; i < a.n; ++i) {
    p.off[i] = (p.ryl + a.d[i][1]) * p.w + p.lp + a.d[i][0];
    p.lag[i] = p.rzl + a.d[i][2];
    p.wt[i] = (T)a.w[i];
  }
  p.xbase = a.dom.min[0] / VEC * VEC;
  p.tiles_x = (a.dom.max[0] - p.xbase + TX - 1) / TX;
  const int tiles_y = (a.dom.max[1] - a.dom.min[1] + TY - 1) / TY;
  p.tiles = p.tiles_x * tiles_y;
}

// zlen, items and the grid size for `occ` resident CTAs per SM.
template <typename T>
int schedule(PtsParams<T> *p, int occ, int sm_count) {
  const int resident = sm_count * occ;
  const int nzd = p->dmax2 - p->dmin2;
  // chunks as short as fills every resident CTA: loading runs ahead into a CTA's
  // next item, so a short chunk's halo planes cost little (33 x 65 x 79, 27
  // points: 5.4 us a sweep against 7.7 with four planes)
  p->zlen = choose_zchunk_overhead(p->tiles, nzd, resident, p->rzl + p->rzh + 1, resident);
  // Wide enough double stencils are bound by the FP64 pipes, whose shares even out
  // best with one CTA per plane of a tile, handed to whichever SM is free (7
  // points 300 x 200 x 250: 364 us a sweep against 416); with fewer than 16 rounds
  // the round-robin is as good.
  const int planes = p->rzl + p->rzh + 1;
  const bool spread = std::is_same<T, double>::value && p->n >= 2 * planes &&
                      (long long)p->tiles * nzd >= 16LL * resident &&
                      (long long)p->tiles * nzd <= 0x7fffffff;
  if (spread) p->zlen = 1;
  const int chunks = (nzd + p->zlen - 1) / p->zlen;
  p->items = (long long)p->tiles * chunks;
  p->early = p->items >= resident;
  return (int)(p->items < resident || spread ? p->items : resident);
}

template <typename T>
size_t smem_for(const PtsParams<T> &p) {
  return 128 + (size_t)kPtsRingOffset + (size_t)p.nstage * p.pstride * sizeof(T);
}

bool jit_enabled() {
  const char *e = getenv("PS_POINTS_JIT");
  return !(e && e[0] == '0');
}

template <typename T, int RY, bool UNIT>
cudaError_t launch_t(const PointsArgs &a, int warps, int lx, int sm_count, cudaStream_t s) {
  PtsParams<T> p;
  fill_params<T>(a, warps, RY, lx, &p);
  const size_t smem = smem_for(p);
  PtsTmap tm;
  memset(&tm, 0, sizeof(tm));
  static_assert(sizeof(PtsTmap) == sizeof(CUtensorMap), "tensor map layout");
  memcpy(&tm, &a.tmap, sizeof(tm));
  if (jit_enabled()) {
    // The stencil compiled with its table as constants (cached per stencil,
    // type and tile shape); on any failure the table kernel below runs.
    PtsJitKey key;
    memset(&key, 0, sizeof(key));
    key.type = a.in.type;
    key.ry = RY;
    key.warps = warps;
    key.n = a.n;
    // Registers: four rows of four cells compile to 72 of 80 without spilling
    // (4-byte types, 7 to 27 points); 8-byte types need about 120.
    const int regs = a.in.esz == 4 ? 80 : 120;
    // Lists that come back late to what they have loaded hold more vectors than that
    // leaves room for: more than 28 of them (22 of 8-byte types) get the registers
    // of two CTAs to an SM (64 points within 2 of the cell, float, 256 x 250 x 120:
    // 56 us a sweep, 222 spilling at 72 registers; 25 points in a plane, double,
    // 2049 x 1500: 292 and 321).  Nor are registers saved for CTAs whose ring does
    // not fit.
    const int live = a.live[RY == 4 ? 2 : RY == 2 ? 1 : 0];
    int ctas = 65536 / (regs * 32 * (warps + 1));
    if (live > (a.in.esz == 4 ? 28 : 21)) ctas = std::min(ctas, 2);
    key.min_ctas = std::max(1, std::min(ctas, (int)(227 * 1024 / (smem + 1024))));
    key.unit = UNIT;
    key.lx = lx;
    key.w = p.w;
    key.nstage = p.nstage;
    key.pstride = p.pstride;
    key.planes = p.rzl + p.rzh + 1;
    key.centre = p.rzl;
    for (int i = 0; i < a.n; ++i) {
      key.dx[i] = a.d[i][0];
      key.dy[i] = a.d[i][1];
      key.lag[i] = p.lag[i];
      key.wt[i] = UNIT ? 1.0 : a.w[i];
    }
    int occ = 0;
    void *fn = jit_points_function(key, smem, &occ);
    if (fn && occ >= 1) {
      const int grid = schedule(&p, occ, sm_count);
      void *args[2] = {&p, &tm};
      return jit_launch_raw(fn, grid, dim3(32, warps + 1, 1), smem, a.overlap, s, args);
    }
  }
  auto kern = pts_kernel<T, RY, UNIT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * (warps + 1), smem);
  if (e != cudaSuccess) return e;
  if (occ < 1) return cudaErrorInvalidConfiguration;
  const int grid = schedule(&p, occ, sm_count);
  return launch_kernel(kern, (unsigned)grid, dim3(32, warps + 1, 1), smem, s, a.overlap, p, tm);
}

template <typename T>
cudaError_t launch_type(const PointsArgs &a, const MarchConfig &cfg, int sm_count,
                        cudaStream_t s) {
  const int warps = cfg.warps, lx = points_lanes(a, cfg);
  if (cfg.rows >= 4)
    return a.unit ? launch_t<T, 4, true>(a, warps, lx, sm_count, s)
                  : launch_t<T, 4, false>(a, warps, lx, sm_count, s);
  if (cfg.rows >= 2)
    return a.unit ? launch_t<T, 2, true>(a, warps, lx, sm_count, s)
                  : launch_t<T, 2, false>(a, warps, lx, sm_count, s);
  return a.unit ? launch_t<T, 1, true>(a, warps, lx, sm_count, s)
                : launch_t<T, 1, false>(a, warps, lx, sm_count, s);
}

}  // namespace

int points_rows(const MarchConfig &cfg) { return cfg.rows >= 4 ? 4 : (cfg.rows >= 2 ? 2 : 1); }

namespace {

// TMA box of one ring plane and shared memory with tiles of lx lanes in x.
void box_for(const PointsArgs &a, const MarchConfig &cfg, int lx, int *w, int *h) {
  const int vec = 16 / a.in.esz;
  int lo[3], hi[3];
  extents(a, lo, hi);
  *w = (-lo[0] + vec - 1) / vec * vec + kPtsVX * lx + (hi[0] + vec - 1) / vec * vec;
  *h = cfg.warps * points_rows(cfg) * (32 / lx) - lo[1] + hi[1];
}

size_t smem_bytes_for(const PointsArgs &a, const MarchConfig &cfg, int lx) {
  int lo[3], hi[3], w, h, nstage;
  extents(a, lo, hi);
  box_for(a, cfg, lx, &w, &h);
  return ring_bytes(a, lo, hi, w, h, &nstage);
}

}  // namespace

// Lanes side by side in x.  All three shapes hold the same cells, so the one
// that covers the domain with the fewest cells loaded (tiles x box) is taken,
// the wider one unless a narrower one saves 3 %.  Against 128-cell tiles, per
// sweep: 64-cell tiles, 27 points periodic 320 x 300 x 257 59.8 against 63 us,
// 27 points 60^3 4.3 against 4.9, 7 points 50 x 300 x 300 12.4 against 17.2;
// 32-cell tiles, double, 7 points 40 x 66 x 100 18 against 32 us.
static int best_lanes(const PointsArgs &a, const MarchConfig &cfg, double *cells) {
  const int vec = 16 / a.in.esz;
  const int nx = a.dom.max[0] - a.dom.min[0] / vec * vec, ny = a.dom.max[1] - a.dom.min[1];
  int best = 32;
  double cost = 0;
  for (int lx = 32; lx >= 8; lx /= 2) {
    const int tx = kPtsVX * lx, ty = cfg.warps * points_rows(cfg) * (32 / lx);
    int w, h;
    box_for(a, cfg, lx, &w, &h);
    if (lx < 32 && (h > 256 || smem_bytes_for(a, cfg, lx) > 220 * 1024)) continue;
    const double c = (double)((nx + tx - 1) / tx) * ((ny + ty - 1) / ty) * w * h;
    if (lx == 32 || c < 0.97 * cost) {
      best = lx;
      cost = c;
    }
  }
  *cells = cost;
  return best;
}

int points_lanes(const PointsArgs &a, const MarchConfig &cfg) {
  double cells;
  return best_lanes(a, cfg, &cells);
}

// Consumer warps of the default shape: three where the lower tiles load 3 % fewer
// cells than four warps' (red/black 319 x 257 x 255 28.8 us a colour against 33.0,
// tiles of 24 rows for 257; where neither saves, four are up to 2 % faster or slower).
int points_warps(const PointsArgs &a, const MarchConfig &cfg) {
  MarchConfig three = cfg;
  three.warps = 3;
  double c3, c4;
  best_lanes(a, three, &c3);
  best_lanes(a, cfg, &c4);
  return c3 < 0.97 * c4 ? 3 : cfg.warps;
}

int points_live(int n, const int (*d)[3], int esz, int rows) {
  const int vec = 16 / esz;
  // vectors of point k: plane, row and (column group, vector) of each of its cells
  std::map<std::array<int, 3>, std::pair<int, int>> use;
  for (int k = 0; k < n; ++k)
    for (int r = 0; r < rows; ++r)
      for (int c = 0; c < kPtsVX; ++c) {
        const int i = c % vec + d[k][0], v = (i + 8 * vec) / vec - 8;
        auto at = use.emplace(std::array<int, 3>{d[k][2], d[k][1] + r, c / vec * 64 + v},
                              std::make_pair(k, k));
        at.first->second.second = k;
      }
  int most = 0;
  for (int k = 0; k < n; ++k) {
    int live = 0;
    for (const auto &u : use) live += u.second.first <= k && k <= u.second.second;
    most = std::max(most, live);
  }
  return most;
}

void points_box(const PointsArgs &a, const MarchConfig &cfg, int *w, int *h) {
  box_for(a, cfg, points_lanes(a, cfg), w, h);
}

size_t points_smem_bytes(const PointsArgs &a, const MarchConfig &cfg) {
  return smem_bytes_for(a, cfg, points_lanes(a, cfg));
}

cudaError_t launch_points(const PointsArgs &a, const MarchConfig &cfg, int sm_count,
                          cudaStream_t s) {
  if (a.n < 1 || a.n > kMaxPoints || cfg.warps < 1 || cfg.warps > 16)
    return cudaErrorInvalidValue;
  if (a.dom.min[0] >= a.dom.max[0] || a.dom.min[1] >= a.dom.max[1] ||
      a.dom.min[2] >= a.dom.max[2])
    return cudaSuccess;
  switch (a.in.type) {
    case kFloat: return launch_type<float>(a, cfg, sm_count, s);
    case kDouble: return launch_type<double>(a, cfg, sm_count, s);
    case kInt: return launch_type<int>(a, cfg, sm_count, s);
    default: return launch_type<long long>(a, cfg, sm_count, s);
  }
}

}  // namespace psg
