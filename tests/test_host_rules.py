"""The host rules that cut a sweep into tiles and chunks, called in the built
objects themselves (a small C shim linked against them), with the kernels'
index arithmetic restated around them: every tile shape that a rule picks fits
shared memory and a TMA box, and the items write every cell of the domain
exactly once."""
import ctypes
import itertools
import os
import random
import subprocess

import pytest

from physis_gb300 import buildlib

SHIM = r"""
#include "ps_internal.h"
using namespace psg;
static Box box(const int *d) { return Box{{d[0], d[2], d[4]}, {d[1], d[3], d[5]}}; }
static MarchConfig cfg(const int *c) { return MarchConfig{c[0], c[1], c[2], 2, 0}; }
static PointsArgs points(const int *d, int type, int n, const int *offsets) {
  PointsArgs a{};
  a.in.type = type;
  a.in.esz = (type == kFloat || type == kInt) ? 4 : 8;
  a.dom = box(d);
  a.n = n;
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < 3; ++k) a.d[i][k] = offsets[3 * i + k];
  return a;
}
#define API extern "C" __attribute__((visibility("default")))
API int zchunk(int tiles, int nz, int resident, int overhead, int fill) {
  return choose_zchunk_overhead(tiles, nz, resident, overhead, fill);
}
API int s7(const int *d, int esz, int bound, const int *c, int *w, int *h) {
  const int lx = stencil7_lanes(box(d), esz, (S7Bound)bound, cfg(c));
  stencil7_box(esz, cfg(c), lx, w, h);
  return lx;
}
API int s7_bound(int type, int kernel, const int *d) {
  return (int)stencil7_bound(type, kernel, box(d));
}
API long long s7_smem(int esz, const int *c) { return (long long)stencil7_smem_bytes(esz, cfg(c)); }
API int himeno(const int *d, int warps, int *p, int *c) {
  const int lx = himeno19_lanes(box(d), warps);
  himeno19_boxes(lx, warps, p, c);
  return lx;
}
API int pts(const int *d, int type, int n, const int *offsets, const int *c, int *w, int *h,
            long long *smem) {
  const PointsArgs a = points(d, type, n, offsets);
  points_box(a, cfg(c), w, h);
  *smem = (long long)points_smem_bytes(a, cfg(c));
  return points_lanes(a, cfg(c));
}
API int resident(int nx, int ny, int nz, int esz, int sms, int *plan, long long *smem) {
  Resident7Plan q{};
  if (!choose_resident7(nx, ny, nz, esz, sms, &q)) return 0;
  plan[0] = q.by;
  plan[1] = q.bz;
  plan[2] = q.k;
  *smem = (long long)resident7_smem(q, nx, ny, nz, esz);
  return 1;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    buildlib.build()
    out = tmp_path_factory.mktemp("rules")
    src, lib = out / "shim.cu", out / "librules.so"
    src.write_text(SHIM)
    objs = [os.path.join(buildlib.BUILD, os.path.splitext(s)[0] + ".o") for s in buildlib.SOURCES]
    subprocess.run([buildlib.nvcc(), "-shared"] + buildlib.common_flags()
                   + ["-o", str(lib), str(src)] + objs + ["-ldl"], check=True)
    L = ctypes.CDLL(str(lib))
    L.s7_smem.restype = ctypes.c_longlong
    return L


def _ints(*v):
    return (ctypes.c_int * len(v))(*v)


def _domains(rnd, count, most=70000):
    """(x0, x1, y0, y1, z0, z1) of odd sizes, thin axes among them."""
    out = []
    while len(out) < count:
        n = [rnd.choice([1, 2, 3, 5, 8, 9, 16, 17, 31, 33, 50, 64, 66, 100, 129, 150, 257])
             for _ in range(3)]
        if n[0] * n[1] * n[2] > most:
            continue
        d = []
        for k in n:
            lo = rnd.choice([0, 0, 1, 3])
            d += [lo, lo + k]
        out.append(d)
    return out


def _covered(d, xbase, tx, ty, zlen, grid):
    """Every cell of the domain is written once by the items taken round-robin."""
    x0, x1, y0, y1, z0, z1 = d
    tiles_x = -(-(x1 - xbase) // tx)
    tiles = tiles_x * -(-(y1 - y0) // ty)
    items = tiles * -(-(z1 - z0) // zlen)
    seen = 0
    for b in range(min(grid, items)):
        for item in range(b, items, grid):
            chunk, tile = divmod(item, tiles)
            zs = z0 + chunk * zlen
            ze = min(zs + zlen, z1)
            assert z0 <= zs < ze
            x, y = xbase + tile % tiles_x * tx, y0 + tile // tiles_x * ty
            # tiles are disjoint by their origins: counting the clipped cells is enough
            seen += (min(x + tx, x1) - max(x, x0)) * (min(y + ty, y1) - y) * (ze - zs)
            assert max(x, x0) < min(x + tx, x1) and y < y1
    assert seen == (x1 - x0) * (y1 - y0) * (z1 - z0)


SHAPES7 = [(8, 2, 4), (4, 4, 4), (1, 1, 2), (16, 1, 4), (2, 8, 3), (16, 8, 2), (8, 4, 8)]


@pytest.mark.parametrize("esz,bound", [(4, 0), (8, 0), (8, 1), (4, 2)])  # S7Bound
def test_seven_point_tiles(rules, esz, bound):
    rnd, vec = random.Random(esz + bound), 16 // esz
    for d, shape in itertools.product(_domains(rnd, 25), SHAPES7):
        w, h = ctypes.c_int(), ctypes.c_int()
        lx = rules.s7(_ints(*d), esz, bound, _ints(*shape), ctypes.byref(w), ctypes.byref(h))
        assert lx in (8, 16, 32)
        tx, ty = lx * vec, shape[0] * shape[1] * (32 // lx)
        assert (w.value, h.value) == (tx + 2 * vec, ty + 2)
        stage = -(-w.value * h.value * esz // 128) * 128
        if lx < 32:  # the widest tile's limits are the shape's own
            assert h.value <= 256 and 256 + shape[2] * stage <= 200 * 1024
        xbase = d[0] // vec * vec
        tiles = -(-(d[1] - xbase) // tx) * -(-(d[3] - d[2]) // ty)
        for resident, fill in ((152, 152), (456, 152), (3, 1)):
            zlen = rules.zchunk(tiles, d[5] - d[4], resident, 1, fill)
            _covered(d, xbase, tx, ty, zlen, resident)
        _covered(d, xbase, tx, ty, 1, 10 ** 9)  # one CTA per plane of a tile


def test_seven_point_bounds(rules):
    # types kInt, kLong, kFloat, kDouble = 0..3; kernels DIFFUSION7, SUM7, COPY
    import physis_gb300 as ps
    small, large = _ints(0, 64, 0, 64, 0, 64), _ints(1, 599, 1, 599, 1, 599)
    for d in (small, large):
        assert rules.s7_bound(3, ps.PS_KERNEL_DIFFUSION7, d) == 1
        assert rules.s7_bound(3, ps.PS_KERNEL_SUM7, d) == 1
        assert all(rules.s7_bound(t, ps.PS_KERNEL_COPY, d) == 0 for t in range(4))
        assert rules.s7_bound(2, ps.PS_KERNEL_DIFFUSION7, d) == 0
        assert rules.s7_bound(1, ps.PS_KERNEL_SUM7, d) == 0
    assert rules.s7_bound(2, ps.PS_KERNEL_SUM7, small) == 0
    assert rules.s7_bound(2, ps.PS_KERNEL_SUM7, large) == 2

    def lanes(d, esz, bound):
        w, h = ctypes.c_int(), ctypes.c_int()
        return rules.s7(_ints(*d), esz, bound, _ints(8, 2, 4), ctypes.byref(w), ctypes.byref(h))

    # a double copy of a narrow grid loads fewest cells on the widest tiles
    assert lanes((0, 8, 0, 8, 0, 20000), 8, 0) == 32
    assert lanes((0, 8, 0, 8, 0, 20000), 8, 1) == 8
    # beyond L2 SUM7 gives up long rows for a large saving only
    assert lanes((1, 699, 1, 639, 1, 399), 4, 2) == 32
    assert lanes((1, 699, 1, 639, 1, 399), 4, 0) == 16
    assert lanes((0, 64, 0, 4000, 0, 900), 4, 2) == 16


@pytest.mark.parametrize("warps", [1, 3, 4, 8])
def test_himeno_tiles(rules, warps):
    for d in _domains(random.Random(warps), 40):
        p, c = _ints(0, 0), _ints(0, 0)
        lx = rules.himeno(_ints(*d), warps, p, c)
        tx, ty = 4 * lx, warps * (32 // lx)
        assert lx in (8, 16, 32) and list(c) == [tx, ty] and list(p) == [tx + 8, ty + 2]
        # a stage of p is sized for the widest tile, one of the coefficients for any
        assert p[0] * p[1] <= -(-136 * (warps + 2) * 4 // 128) * 32
        assert c[0] * c[1] == 128 * warps
        xbase = d[0] // 4 * 4
        tiles = -(-(d[1] - xbase) // tx) * -(-(d[3] - d[2]) // ty)
        _covered(d, xbase, tx, ty, rules.zchunk(tiles, d[5] - d[4], 456, 2, 0), 456)


LISTS = {"p7": [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)],
         "star4": [(k * s if a == 0 else 0, k * s if a == 1 else 0, k * s if a == 2 else 0)
                   for k in range(5) for a in range(3) for s in (1, -1)],
         "one_side": [(0, 0, 0), (4, 0, 0), (0, 3, 0), (0, 0, 4)], "plane": [(1, 1, 0), (-2, 0, 0)]}


@pytest.mark.parametrize("name", sorted(LISTS))
@pytest.mark.parametrize("type_", [0, 1, 2, 3])  # kInt, kLong, kFloat, kDouble in some order
def test_point_tiles(rules, name, type_):
    pts = LISTS[name]
    flat = _ints(*[v for p in pts for v in p])
    for d, shape in itertools.product(_domains(random.Random(7), 15), [(4, 4, 4), (3, 4, 4), (1, 1, 4),
                                                                     (16, 4, 4), (4, 2, 4)]):
        w, h, smem = ctypes.c_int(), ctypes.c_int(), ctypes.c_longlong()
        lx = rules.pts(_ints(*d), type_, len(pts), flat, _ints(*shape), ctypes.byref(w),
                       ctypes.byref(h), ctypes.byref(smem))
        assert lx in (8, 16, 32)
        ty = shape[0] * shape[1] * (32 // lx)
        lo = [min(0, min(p[i] for p in pts)) for i in range(3)]
        hi = [max(0, max(p[i] for p in pts)) for i in range(3)]
        assert h.value == ty + hi[1] - lo[1]
        vecs = [v for v in (2, 4) if w.value == (-(-(-lo[0]) // v) * v + 4 * lx + -(-hi[0] // v) * v)]
        assert vecs
        if lx < 32:
            assert h.value <= 256 and smem.value <= 220 * 1024
        xbase = d[0] // vecs[-1] * vecs[-1]
        tiles = -(-(d[1] - xbase) // (4 * lx)) * -(-(d[3] - d[2]) // ty)
        zlen = rules.zchunk(tiles, d[5] - d[4], 456, hi[2] - lo[2] + 1, 456)
        _covered(d, xbase, 4 * lx, ty, zlen, 456)


def test_resident_bricks(rules):
    rnd = random.Random(9)
    for _ in range(60):
        nx, ny, nz = [rnd.choice([8, 17, 33, 64, 90, 120, 128]) for _ in range(3)]
        for esz, sms in ((4, 152), (8, 152), (4, 30)):
            plan, smem = _ints(0, 0, 0), ctypes.c_longlong()
            if not rules.resident(nx, ny, nz, esz, sms, plan, ctypes.byref(smem)):
                continue
            by, bz, k = plan
            nby, nbz = -(-ny // by), -(-nz // bz)
            assert nby * nbz <= sms and smem.value <= 220 * 1024
            # the kernel's divisions by multiplication take numbers below 2^16
            assert smem.value // 32 < 1 << 16 and 1 <= k <= 4
