"""Performance cases of the stencil runtime: what they are, their inputs, one
pass of each through the public entry points, the work a pass cannot do
without, and its outputs in 64-bit arithmetic.

Every case is a dict with a "kind":
  diffusion    PS_KERNEL_DIFFUSION7 ping-pong runs (PSStencilRun); with
               "job" the whole program: copy-in, run, PSReduce, copy-out
  himeno       19-point sweeps, each with its residual (PSReduce's kernel form)
  batch        many uneven grids stepped together (PSBatchRun)
  reduce       PSReduce sum, max and min of one grid
  points       weighted point-list stencils, 3D or 2D, every boundary rule
  function     stencil functions compiled from their Physis source
  redblack     in-place red/black sweeps
  nn_layer     one layer of the warm-start network: forward, backward-data
               and weight gradient
  nn_train     a training step of the warm-start network
"""
import ctypes
import math

import numpy as np
import torch

import physis_gb300 as ps
from physis_gb300 import warmstart as ws

TORCH = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "i64": torch.int64}
NUMPY = {"f32": np.float32, "f64": np.float64, "i32": np.int32, "i64": np.int64}
SIZE = {"f32": 4, "f64": 8, "i32": 4, "i64": 8}
CTYPE = {"f32": ("Float", "float"), "f64": ("Double", "double")}

# The diffusion benchmark's coefficients in map order ce cw cn cs ct cb cc.
COEF = (0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.4)
# Its terms in expression order: centre, west, east, south, north, bottom, top.
P7 = ((0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, -1), (0, 0, 1))
P27 = tuple((x, y, z) for z in (-1, 0, 1) for (x, y) in
            ((0, 0), (1, 0), (-1, 0), (0, 1), (1, 1), (-1, 1), (0, -1), (1, -1), (-1, -1)))
P9 = ((0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (-1, -1, 0), (1, -1, 0),
      (-1, 1, 0), (1, 1, 0))
POINTS = {"p7": (P7, (0.4,) + (0.1,) * 6), "p27": (P27, (1.0 / 27.0,) * 27),
          "p9": (P9, (0.25,) + (0.125,) * 4 + (0.0625,) * 4)}
BOUNDARY = {"none": 0, "periodic": 1, "clamp": 2}
OMEGA = 0.8
LEARNING_RATE = 2e-3

FN_DIFFUSION = """
void diffusion(const int x, const int y, const int z, PSGrid3D@N g1, PSGrid3D@N g2,
               @T ce, @T cw, @T cn, @T cs, @T ct, @T cb, @T cc) {
  int nx = PSGridDim(g1, 0), ny = PSGridDim(g1, 1), nz = PSGridDim(g1, 2);
  @T c = PSGridGet(g1, x, y, z);
  @T w = (x == 0) ? c : PSGridGet(g1, x - 1, y, z);
  @T e = (x == nx - 1) ? c : PSGridGet(g1, x + 1, y, z);
  @T n = (y == 0) ? c : PSGridGet(g1, x, y - 1, z);
  @T s = (y == ny - 1) ? c : PSGridGet(g1, x, y + 1, z);
  @T b = (z == 0) ? c : PSGridGet(g1, x, y, z - 1);
  @T t = (z == nz - 1) ? c : PSGridGet(g1, x, y, z + 1);
  PSGridEmit(g2, cc * c + cw * w + ce * e + cs * s + cn * n + cb * b + ct * t);
}
"""

FN_MEAN27 = """
void mean27(const int x, const int y, const int z, PSGrid3D@N g1, PSGrid3D@N g2, @T scale) {
  const int dx[9] = {0, 1, -1, 0, 1, -1, 0, 1, -1};
  const int dy[9] = {0, 0, 0, 1, 1, 1, -1, -1, -1};
  @T v = PSGridGet(g1, x, y, z - 1);
  for (int dz = -1; dz <= 1; ++dz)
    for (int i = (dz == -1) ? 1 : 0; i < 9; ++i)
      v = v + PSGridGet(g1, x + dx[i], y + dy[i], z + dz);
  PSGridEmit(g2, v * scale);
}
"""

FN_REDBLACK = """
void relax(const int x, const int y, const int z, PSGrid3D@N g, @T cc, @T cn) {
  PSGridEmit(g, cc * PSGridGet(g, x, y, z) + cn * PSGridGet(g, x + 1, y, z)
      + cn * PSGridGet(g, x - 1, y, z) + cn * PSGridGet(g, x, y + 1, z)
      + cn * PSGridGet(g, x, y - 1, z) + cn * PSGridGet(g, x, y, z - 1)
      + cn * PSGridGet(g, x, y, z + 1));
}
"""


def listed():
    return [
        # The reference's own REF program: 100 steps on a small grid and a sum,
        # with the host copies around them.  Latency and launches.
        {"name": "diffusion_64_job", "kind": "diffusion", "nx": 64, "ny": 64, "nz": 64,
         "dtype": "f32", "iters": 50, "job": True},
        # The diffusion benchmark at its large size, a short run.
        {"name": "diffusion_512", "kind": "diffusion", "nx": 512, "ny": 512, "nz": 512,
         "dtype": "f32", "iters": 2, "job": False},
        # Himeno at the benchmark's M size, the residual read every sweep.
        {"name": "himeno_257x257x513", "kind": "himeno", "nx": 257, "ny": 257, "nz": 513,
         "sweeps": 2},
        # A parameter study: independent problems of uneven sizes, half
        # diffusion and half Himeno, stepped together.
        {"name": "batch_24_uneven", "kind": "batch", "count": 24, "dims_seed": 2, "xy_lo": 32,
         "xy_hi": 160, "z_lo": 32, "z_hi": 256, "iters": 20},
        # The global sums and extrema a solver prints, grid with ragged rows.
        {"name": "reduce_f32", "kind": "reduce", "nx": 509, "ny": 500, "nz": 301,
         "dtype": "f32"},
        # The 27-point periodic system test's stencil as a smoothing filter.
        {"name": "points27_periodic", "kind": "points", "stencil": "p27", "boundary": "periodic",
         "nx": 320, "ny": 300, "nz": 257, "dtype": "f32", "iters": 2},
        # A 9-point filter of a 2D grid (the 2D system tests' shape).
        {"name": "points9_2d", "kind": "points", "stencil": "p9", "boundary": "periodic",
         "nx": 4099, "ny": 3001, "nz": 1, "dtype": "f32", "iters": 4},
        # A user's own stencil: the diffusion benchmark's source compiled.
        {"name": "function_diffusion", "kind": "function", "stencil": "diffusion", "nx": 400,
         "ny": 384, "nz": 320, "dtype": "f32", "iters": 2},
        # A user's wide stencil in double precision, interior domain.
        {"name": "function_mean27_f64", "kind": "function", "stencil": "mean27", "nx": 258,
         "ny": 258, "nz": 200, "dtype": "f64", "iters": 2},
        # Gauss-Seidel style relaxation, odd sizes.
        {"name": "redblack_odd", "kind": "redblack", "form": "builtin", "nx": 319, "ny": 257,
         "nz": 255, "dtype": "f32", "iters": 2},
        # One hidden layer of the warm-start network over the coarse grids of
        # 1024 instances: forward (prediction), and both backward directions.
        {"name": "nn_layer_1024", "kind": "nn_layer", "batch": 1024, "nz": 17, "ny": 9, "nx": 9},
        # A training step of the network on the default minibatch.
        {"name": "nn_train_32", "kind": "nn_train", "batch": 32, "nz": 17, "ny": 9, "nx": 9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, most):
    """Three extents, log-uniform in [lo, hi], at most `most` cells."""
    while True:
        n = [_log(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= most:
            return {"nx": n[0], "ny": n[1], "nz": n[2]}


def _iters(cells):
    """Iterations of a run: long on small grids, where programs iterate long."""
    return 50 if cells <= 1 << 19 else (20 if cells <= 1 << 22 else 2)


def draw(rng):
    kind = rng.choice(["diffusion", "diffusion", "himeno", "batch", "reduce", "points", "points",
                       "points2d", "function", "function", "redblack", "nn_layer", "nn_train"])
    if kind == "diffusion":
        c = _box(rng, 32, 520, 1 << 26)
        cells = c["nx"] * c["ny"] * c["nz"]
        return {"kind": kind, **c, "dtype": rng.choice(["f32", "f32", "f64"]),
                "iters": _iters(cells), "job": cells <= 1 << 19 and rng.random() < 0.5}
    if kind == "himeno":
        return {"kind": kind, **_box(rng, 33, 300, 1 << 24), "sweeps": rng.choice([2, 4])}
    if kind == "batch":
        lo = rng.choice([16, 24, 32])
        return {"kind": kind, "count": rng.randrange(6, 28, 2), "dims_seed": rng.randrange(1 << 20),
                "xy_lo": lo, "xy_hi": lo * rng.choice([3, 4, 5]), "z_lo": lo,
                "z_hi": lo * rng.choice([3, 5, 8]), "iters": rng.choice([4, 20])}
    if kind == "reduce":
        return {"kind": kind, **_box(rng, 24, 520, 1 << 26),
                "dtype": rng.choice(["f32", "f32", "f64", "i32", "i64"])}
    if kind == "points":
        c = _box(rng, 32, 400, 1 << 25)
        return {"kind": kind, "stencil": rng.choice(["p7", "p27"]),
                "boundary": rng.choice(["none", "periodic", "clamp"]), **c,
                "dtype": rng.choice(["f32", "f32", "f64", "i32"]),
                "iters": min(20, _iters(c["nx"] * c["ny"] * c["nz"]))}
    if kind == "points2d":
        return {"kind": "points", "stencil": "p9", "nx": _log(rng, 64, 5000),
                "ny": _log(rng, 64, 5000), "nz": 1, "dtype": rng.choice(["f32", "f64", "i32"]),
                "boundary": rng.choice(["none", "periodic", "clamp"]), "iters": 4}
    if kind == "function":
        c = _box(rng, 32, 420, 1 << 25)
        return {"kind": kind, "stencil": rng.choice(["diffusion", "mean27"]), **c,
                "dtype": rng.choice(["f32", "f32", "f64"]),
                "iters": min(20, _iters(c["nx"] * c["ny"] * c["nz"]))}
    if kind == "redblack":
        c = _box(rng, 33, 400, 1 << 25)
        return {"kind": kind, "form": rng.choice(["builtin", "function"]), **c,
                "dtype": rng.choice(["f32", "f32", "f64"]),
                "iters": min(20, _iters(c["nx"] * c["ny"] * c["nz"]))}
    grid = rng.choice([(17, 9, 9), (9, 9, 17), (13, 11, 8), (16, 16, 16)])
    b = _log(rng, 16, 1024) if kind == "nn_layer" else _log(rng, 16, 64)
    return {"kind": kind, "batch": b, "nz": grid[0], "ny": grid[1], "nx": grid[2]}


# ---- grids ----------------------------------------------------------------------

class _Grid(ps.Grid):
    """A grid whose storage goes when nothing refers to it any more."""

    def __del__(self):
        self.free()


class _Alias:
    """A grid's device storage as __cuda_array_interface__ (keeps the grid)."""

    def __init__(self, grid):
        self.grid = grid
        e, (nz, ny, nx) = grid.dtype.itemsize, grid.shape
        p = grid.pitch
        self.__cuda_array_interface__ = {
            "shape": (nz, ny, nx), "strides": (p * ny, p, e), "typestr": grid.dtype.str,
            "data": (grid.dev_ptr, False), "version": 3}


def _view(grid):
    """The grid's present storage as a tensor (nz, ny, nx)."""
    key = grid.dev_ptr
    cached = getattr(grid, "_views", None)
    if cached is None:
        cached = grid._views = {}
    if key not in cached:
        # the alias holds a plain reference back to the grid: broken by State
        cached[key] = torch.as_tensor(_Alias(grid), device="cuda")
    return cached[key]


class State:
    """What a program keeps between calls; frees its batch and grids."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        if getattr(self, "batch", None) is not None:
            ps.batch_free(self.batch)
        for g in getattr(self, "grids", []):
            g._views = {}  # no cycle: a tensor given out keeps the grid alive


def _shape(c):
    return (c["nz"], c["ny"], c["nx"])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _field(shape, dtype, gen):
    """Uniform [0, 1) fields; integers uniform in [-1000, 1000)."""
    if dtype in ("i32", "i64"):
        return torch.randint(-1000, 1000, shape, generator=gen, device="cuda", dtype=TORCH[dtype])
    return torch.rand(shape, generator=gen, device="cuda", dtype=TORCH[dtype])


def _put(grid, tensor):
    _view(grid).copy_(tensor)


def _grid_of(tensor, dtype):
    g = _Grid(tuple(tensor.shape), NUMPY[dtype])
    _put(g, tensor)
    return g


def _batch_dims(c):
    """(nx, ny, nz) of each problem, X, Y and Z uniform in their ranges."""
    r = np.random.default_rng(c["dims_seed"])
    return [(int(r.integers(c["xy_lo"], c["xy_hi"] + 1)), int(r.integers(c["xy_lo"], c["xy_hi"] + 1)),
             int(r.integers(c["z_lo"], c["z_hi"] + 1))) for _ in range(c["count"])]


def _himeno_fields(shape, gen):
    """p and the 12 coefficient/source fields of a diagonally dominant
    19-point problem: a, c in [0.5, 2], small cross terms, a3 the inverse
    diagonal, bnd 1 inside and 0 on the faces."""
    def u(lo, hi):
        return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo
    p = u(0.0, 1.0)
    a = [u(0.5, 2.0) for _ in range(3)]
    a3 = 1.0 / (2.0 * (a[0] + a[1] + a[2]))
    b = [u(-0.05, 0.05) for _ in range(3)]
    bnd = torch.zeros(shape, device="cuda")
    bnd[1:-1, 1:-1, 1:-1] = 1.0
    w = u(-0.1, 0.1)
    return p, a + [a3] + b + a + [bnd, w]


def _inner(shape):
    nz, ny, nx = shape
    return ps.domain(1, nx - 1, 1, ny - 1, 1, nz - 1)


def _points_domain(c):
    if c["boundary"] != "none":
        return ps.full_domain(_shape(c)), (0, 0, 0)
    h = (1, 1, 1 if c["nz"] > 1 else 0)
    return ps.domain(h[0], c["nx"] - h[0], h[1], c["ny"] - h[1], h[2], c["nz"] - h[2]), h


def _source(text, dtype):
    return text.replace("@N", CTYPE[dtype][0]).replace("@T", CTYPE[dtype][1])


def _bf16(shape, gen, scale=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(torch.bfloat16)


def _nn_inputs(c, seed):
    """A layer's activations (about half of them zero, as ReLU leaves them),
    weights, bias and the gradient coming back."""
    g = _gen(seed)
    shape = (c["batch"], c["nz"], c["ny"], c["nx"], ws.C)
    x = torch.relu(_bf16(shape, g))
    w = torch.randn((27, ws.C, ws.C), generator=g, device="cuda") * math.sqrt(2.0 / (27 * ws.C))
    b = torch.randn(ws.C, generator=g, device="cuda") * 0.1
    return x, w, b, _bf16(shape, g, 1e-3)


def _train_inputs(c, seed):
    g = _gen(seed)
    dims = (c["batch"], c["nz"], c["ny"], c["nx"])
    x = torch.zeros(dims + (ws.C,), device="cuda", dtype=torch.bfloat16)
    x[..., :ws.CIN] = _bf16(dims + (ws.CIN,), g)
    return x, torch.randn(dims, generator=g, device="cuda")


def prepare(case, seed):
    c = case
    ps.init()
    kind = c["kind"]
    if kind == "nn_layer":
        x, w, b, dy = _nn_inputs(c, seed)
        bf = lambda: torch.empty(27 * ws.C * ws.C, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        nsplit = 64
        s = State(case=c, x=x, b=b, dy=dy, wf=bf(), wb=bf(), nsplit=nsplit,
                  work=torch.empty(nsplit * (27 * ws.C * ws.C + ws.C), device="cuda"),
                  y=torch.empty_like(x), dx=torch.empty_like(x), dw=torch.empty_like(w),
                  db=torch.empty_like(b))
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        if ps.lib().PSWarmStartPrepareWeights(_ptr(w), _ptr(s.wf), _ptr(s.wb), st) != ps.PS_OK:
            ps.check()
        torch.cuda.synchronize()
        return s
    if kind == "nn_train":
        x, t = _train_inputs(c, seed)
        n = t.numel()
        s = State(case=c, x=x.reshape(-1), t=t.reshape(-1), net=ws.Net(seed),
                  work=torch.empty(64 * (27 * ws.C * ws.C + ws.C), device="cuda"),
                  work64=torch.empty((n + 255) // 256, dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
        return s
    g = _gen(seed)
    if kind == "batch":
        runs, grids, out = [], [], []
        for i, (nx, ny, nz) in enumerate(_batch_dims(c)):
            shape = (nz, ny, nx)
            if i % 2 == 0:
                gs = [_grid_of(_field(shape, "f32", g), "f32"), _Grid(shape, np.float32)]
                k, dom, sc = ps.PS_KERNEL_DIFFUSION7, ps.full_domain(shape), COEF
            else:
                p, co = _himeno_fields(shape, g)
                gs = [_grid_of(t, "f32") for t in [p, p] + co]
                k, dom, sc = ps.PS_KERNEL_HIMENO19, _inner(shape), [OMEGA]
            runs.append([ps.stencil_map(k, dom, gs, sc),
                         ps.stencil_map(k, dom, [gs[1], gs[0]] + gs[2:], sc)])
            grids += gs
            out.append(gs[0])
        torch.cuda.synchronize()
        return State(case=c, grids=grids, out=out, batch=ps.batch_create(runs))
    shape = _shape(c)
    if kind == "himeno":
        p, co = _himeno_fields(shape, g)
        gs = [_grid_of(t, "f32") for t in [p, p] + co]
        torch.cuda.synchronize()
        return State(case=c, grids=gs, dom=_inner(shape))
    if kind == "diffusion" and c["job"]:
        host = _field(shape, c["dtype"], g).cpu().numpy()
        gs = [_Grid(shape, NUMPY[c["dtype"]]) for _ in range(2)]
        s = State(case=c, grids=gs, host=host, result=np.empty_like(host))
    else:
        init = _field(shape, c["dtype"], g)
        gs = [_grid_of(init, c["dtype"])]
        if kind not in ("reduce", "redblack"):
            gs.append(_grid_of(init, c["dtype"]))
        s = State(case=c, grids=gs)
    torch.cuda.synchronize()
    if kind == "diffusion":
        dom = ps.full_domain(shape)
        s.maps = [ps.stencil_map(ps.PS_KERNEL_DIFFUSION7, dom, p, COEF) for p in (gs, gs[::-1])]
    elif kind == "points":
        pts, wt = POINTS[c["stencil"]]
        wt = None if c["dtype"] in ("i32", "i64") else wt
        k = ps.point_stencil(pts, wt, BOUNDARY[c["boundary"]])
        dom = _points_domain(c)[0]
        s.maps = [ps.stencil_map(k, dom, p) for p in (gs, gs[::-1])]
    elif kind == "function":
        if c["stencil"] == "diffusion":
            k, dom, sc = (ps.stencil_function(_source(FN_DIFFUSION, c["dtype"]), "diffusion"),
                          ps.full_domain(shape), COEF)
        else:
            k, dom, sc = (ps.stencil_function(_source(FN_MEAN27, c["dtype"]), "mean27"),
                          _inner(shape), [1.0 / 27.0])
        s.maps = [ps.stencil_map(k, dom, p, sc) for p in (gs, gs[::-1])]
    elif kind == "redblack":
        if c["form"] == "builtin":
            k, dom, sc = ps.PS_KERNEL_DIFFUSION7, ps.full_domain(shape), COEF
        else:
            k, dom, sc = (ps.stencil_function(_source(FN_REDBLACK, c["dtype"]), "relax"),
                          _inner(shape), [0.4, 0.1])
        s.maps = [ps.stencil_map_color(k, ps.COLOR_REDBLACK, dom, gs, sc)]
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    s, c = state, state.case
    kind = c["kind"]
    if kind == "nn_layer":
        dims = (c["batch"], c["nz"], c["ny"], c["nx"])
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        L = ps.lib()
        if (L.PSWarmStartConv(_ptr(s.x), _ptr(s.wf), _ptr(s.b), None, 1, _ptr(s.y), None, *dims, st)
                or L.PSWarmStartWeightGrad(_ptr(s.x), _ptr(s.dy), _ptr(s.work), s.nsplit,
                                           _ptr(s.dw), _ptr(s.db), *dims, st)
                or L.PSWarmStartConv(_ptr(s.dy), _ptr(s.wb), None, _ptr(s.x), 0, _ptr(s.dx), None,
                                     *dims, st)):
            ps.check()
        return {"y": s.y, "dx": s.dx, "dw": s.dw, "db": s.db}
    if kind == "nn_train":
        dims = (c["batch"], c["nz"], c["ny"], c["nx"])
        pred = s.net.forward(s.x, dims)
        loss, dy = ws.loss_grad(pred, s.t, s.work64)
        s.net.backward(dy, dims, s.work)
        s.net.adam(LEARNING_RATE)
        return {"loss": loss, "pred": pred, "grads": s.net.grads, "params": s.net.params}
    if kind == "batch":
        ps.batch_run(s.batch, c["iters"])
        return [_view(g) for g in s.out]
    if kind == "himeno":
        gs, gosa = s.grids, []
        for i in range(c["sweeps"]):
            p = [gs[i % 2], gs[1 - i % 2]]
            gosa.append(float(ps.reduce_kernel(ps.PS_SUM, ps.PS_KERNEL_HIMENO19_GOSA, s.dom,
                                               p + gs[2:], [OMEGA])))
        return {"gosa": gosa, "p": [_view(gs[0]), _view(gs[1])]}
    if kind == "reduce":
        return [ps.reduce(s.grids[0], op) for op in (ps.PS_SUM, ps.PS_MAX, ps.PS_MIN)]
    if kind == "diffusion" and c["job"]:
        s.grids[0].copyin(s.host)
        ps.stencil_run(s.maps, c["iters"])
        total = ps.reduce(s.grids[0], ps.PS_SUM)
        return {"field": s.grids[0].copyout(s.result), "sum": total}
    ps.stencil_run(s.maps, c["iters"])
    return [_view(g) for g in s.grids]


# ---- the work a pass cannot do without ----------------------------------------------

def work(case):
    """Per sweep each grid read once and each written once (the sweeps of a
    run depend on one another); a red/black map's two colours are one pass
    over the grid each."""
    c = case
    kind = c["kind"]
    if kind in ("nn_layer", "nn_train"):
        n = c["batch"] * c["nz"] * c["ny"] * c["nx"]
        conv = 2.0 * 27 * ws.C * ws.C * n
        if kind == "nn_layer":  # x, dy read; y, dx written
            return {"bytes": n * ws.C * 2 * 4.0, "flops": 3 * conv}
        layers = ws.LAYERS  # activations written and read back once
        return {"bytes": n * ws.C * 2 * (2.0 * layers) + n * 8.0, "flops": (3 * layers - 1) * conv}
    if kind == "batch":
        b = f = 0.0
        for i, (nx, ny, nz) in enumerate(_batch_dims(c)):
            cells = float(nx) * ny * nz if i % 2 == 0 else float(nx - 2) * (ny - 2) * (nz - 2)
            b += cells * (8 if i % 2 == 0 else 56) * 2 * c["iters"]
            f += cells * (13 if i % 2 == 0 else 34) * 2 * c["iters"]
        return {"bytes": b, "flops": f}
    cells = float(c["nx"]) * c["ny"] * c["nz"]
    if kind == "himeno":
        cells = float(c["nx"] - 2) * (c["ny"] - 2) * (c["nz"] - 2)
        return {"bytes": 56 * cells * c["sweeps"], "flops": 34 * cells * c["sweeps"]}
    e = SIZE[c["dtype"]]
    if kind == "reduce":  # the three reductions are three calls
        return {"bytes": 3 * e * cells, "flops": 3 * cells}
    terms = {"p7": 7, "p27": 27, "p9": 9, "diffusion": 7, "mean27": 27}.get(c.get("stencil"), 7)
    sweeps = 2 * c["iters"]  # both maps of a pair, or both colours
    flops = (2 * terms - 1) * cells * sweeps
    return {"bytes": 2 * e * cells * sweeps, "flops": flops / 2 if kind == "redblack" else flops}


# ---- the same in 64 bits ---------------------------------------------------------------

def _shift(u, d, boundary):
    """u at (x + d0, y + d1, z + d2), neighbours outside wrapped or clamped."""
    for axis, k in ((2, d[0]), (1, d[1]), (0, d[2])):
        if not k:
            continue
        n = u.shape[axis]
        i = torch.arange(n, device=u.device) + k
        i = i % n if boundary == "periodic" else i.clamp(0, n - 1)
        u = u.index_select(axis, i)
    return u


def _sum64(u, pts, wt, boundary):
    v = torch.zeros_like(u)
    for d, w in zip(pts, wt):
        v += w * _shift(u, d, boundary)
    return v


def _keep_outside(new, old, h):
    """`new` inside the domain [h, n - h), `old` outside it."""
    nz, ny, nx = new.shape
    out = old.clone()
    sl = (slice(h[2], nz - h[2]), slice(h[1], ny - h[1]), slice(h[0], nx - h[0]))
    out[sl] = new[sl]
    return out


def _round(values, dtype):
    return [float(np.float32(v)) for v in values] if dtype == "f32" else [float(v) for v in values]


def _himeno64(p, co):
    """(new p, sum of ss^2) of one sweep over the interior."""
    a0, a1, a2, a3, b0, b1, b2, c0, c1, c2, bnd, w = co

    def at(x, y, z):
        return _shift(p, (x, y, z), "clamp")
    s0 = a0 * at(0, 0, 1) + a1 * at(0, 1, 0) + a2 * at(1, 0, 0)
    s0 += b0 * (at(0, 1, 1) - at(0, -1, 1) - at(0, 1, -1) + at(0, -1, -1))
    s0 += b1 * (at(1, 1, 0) - at(1, -1, 0) - at(-1, 1, 0) + at(-1, -1, 0))
    s0 += b2 * (at(1, 0, 1) - at(1, 0, -1) - at(-1, 0, 1) + at(-1, 0, -1))
    s0 += c0 * at(0, 0, -1) + c1 * at(0, -1, 0) + c2 * at(-1, 0, 0) + w
    ss = (s0 * a3 - p) * bnd
    om = float(np.float32(OMEGA))
    inner = ss[1:-1, 1:-1, 1:-1]
    return _keep_outside(p + om * ss, p, (1, 1, 1)), float((inner * inner).sum())


def _conv64(x, w):
    """3x3x3 convolution, channels last, zeros outside; w is [27][in][out]."""
    b, nz, ny, nx, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = None
    for t in range(27):
        z, yy, xx = t // 9, (t // 3) % 3, t % 3
        v = xp[:, z:z + nz, yy:yy + ny, xx:xx + nx, :] @ w[t]
        y = v if y is None else y + v
    return y


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "nn_layer":
        x, w, b, dy = _nn_inputs(c, seed)
        x, dy = x.double(), dy.double()
        w = w.to(torch.bfloat16).double()
        y = torch.relu(_conv64(x, w) + b.double())
        back = w.flip(0).transpose(1, 2)
        dx = _conv64(dy, back) * (x > 0)
        xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        _, nz, ny, nx, _ = x.shape
        d2 = dy.reshape(-1, ws.C)
        dw = torch.stack([xp[:, t // 9:t // 9 + nz, (t // 3) % 3:(t // 3) % 3 + ny,
                             t % 3:t % 3 + nx, :].reshape(-1, ws.C).T @ d2 for t in range(27)])
        return {"y": y, "dx": dx, "dw": dw, "db": d2.sum(0)}
    if kind == "nn_train":
        x, t = _train_inputs(c, seed)
        net = ws.Net(seed)  # the seeded initial weights
        params = [p.double().requires_grad_() for p in net.params]
        h = x.double()
        for i in range(ws.LAYERS):
            h = _conv64(h, params[i]) + params[ws.LAYERS + i]
            if i < ws.LAYERS - 1:
                h = torch.relu(h)
        pred = h[..., 0]
        loss = ((pred - t.double()) ** 2).mean()
        grads = torch.autograd.grad(loss, params)
        # the first Adam step: bias-corrected moments are g and g^2
        new = [p.detach() - LEARNING_RATE * g / (g.abs() + 1e-8) for p, g in zip(params, grads)]
        return {"loss": float(loss), "pred": pred.detach().reshape(-1), "grads": list(grads),
                "params": new}
    g = _gen(seed)
    if kind == "batch":
        out = []
        for i, (nx, ny, nz) in enumerate(_batch_dims(c)):
            if i % 2 == 0:
                u = _field((nz, ny, nx), "f32", g).double()
                k = _round(COEF, "f32")
                wt = (k[6], k[1], k[0], k[3], k[2], k[5], k[4])
                for _ in range(2 * c["iters"]):
                    u = _sum64(u, P7, wt, "clamp")
            else:
                p, co = _himeno_fields((nz, ny, nx), g)
                u, co = p.double(), [f.double() for f in co]
                for _ in range(2 * c["iters"]):
                    u = _himeno64(u, co)[0]
            out.append(u)
        return out
    if kind == "himeno":
        p, co = _himeno_fields(_shape(c), g)
        co = [f.double() for f in co]
        pair, gosa = [p.double(), p.double()], []
        for i in range(c["sweeps"]):
            pair[1 - i % 2], v = _himeno64(pair[i % 2], co)
            gosa.append(v)
        return {"gosa": gosa, "p": pair}
    u = _field(_shape(c), c["dtype"], g)
    if not u.is_floating_point():
        return None
    u = u.double()
    if kind == "reduce":
        return [u.sum(), u.max(), u.min()]
    if kind == "diffusion":
        k = _round(COEF, c["dtype"])
        wt, prev = (k[6], k[1], k[0], k[3], k[2], k[5], k[4]), u
        for _ in range(2 * c["iters"]):
            prev, u = u, _sum64(u, P7, wt, "clamp")
        return {"field": u, "sum": u.sum()} if c["job"] else [u, prev]
    if kind == "points":
        pts, wt = POINTS[c["stencil"]]
        wt, h, bc = _round(wt, c["dtype"]), _points_domain(c)[1], c["boundary"]
        pair = [u, u]
        for i in range(2 * c["iters"]):
            pair[1 - i % 2] = _keep_outside(_sum64(pair[i % 2], pts, wt, bc), pair[1 - i % 2], h)
        return pair
    if kind == "function":
        pair = [u, u]
        for i in range(2 * c["iters"]):
            src, dst = pair[i % 2], pair[1 - i % 2]
            if c["stencil"] == "diffusion":
                k = _round(COEF, c["dtype"])
                new = _sum64(src, P7, (k[6], k[1], k[0], k[3], k[2], k[5], k[4]), "clamp")
            else:
                scale = _round([1.0 / 27.0], c["dtype"])[0]
                new = _keep_outside(_sum64(src, P27, (scale,) * 27, "clamp"), dst, (1, 1, 1))
            pair[1 - i % 2] = new
        return pair
    nz, ny, nx = u.shape
    par = (torch.arange(nz, device="cuda")[:, None, None]
           + torch.arange(ny, device="cuda")[None, :, None]
           + torch.arange(nx, device="cuda")[None, None, :]) % 2
    k = _round(COEF, c["dtype"])
    h = (0, 0, 0) if c["form"] == "builtin" else (1, 1, 1)
    wt = (k[6],) + (k[0],) * 6
    for _ in range(c["iters"]):
        for color in (0, 1):
            new = _keep_outside(_sum64(u, P7, wt, "clamp"), u, h)
            u = torch.where((par + color) % 2 == 0, new, u)
    return [u]
