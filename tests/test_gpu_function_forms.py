"""The forms of the tiled entry of stencil functions: eight rows a thread or
four, grids staged for reads at the cell itself, grids left unstaged.  Each must
give the plain entry's bits at sizes around a tile's (64 x 16)."""
import numpy as np
import pytest

import physis_gb300 as ps

pytestmark = pytest.mark.gpu

SIX = " + ".join(f"PSGridGet({{0}}, {c})" for c in
                 ("x + 1, y, z", "x - 1, y, z", "x, y + 1, z", "x, y - 1, z", "x, y, z + 1",
                  "x, y, z - 1"))
AT = "PSGridGet({0}, x, y, z)"
HEAD = "void f(const int x, const int y, const int z, {grids}, PSGrid3D@N out, @T c) {{ {body} }}"


def _source(grids, body):
    return HEAD.format(grids=", ".join("PSGrid3D@N " + g for g in grids), body=body)


# name: (grids before the output, source, halo, element types)
FORMS = {
    "one coefficient": ("uk", _source("uk", f"PSGridEmit(out, {AT.format('u')} + c * {AT.format('k')} * ({SIX.format('u')}));")),
    "four coefficients": ("uabde", _source("uabde", f"PSGridEmit(out, {AT.format('a')} * {AT.format('u')} + {AT.format('b')} * ({SIX.format('u')}) + c * {AT.format('d')} - {AT.format('e')});")),
    "centre periodic": ("uk", _source("uk", f"PSGridEmit(out, PSGridGetPeriodic(k, x, y, z) * (PSGridGetPeriodic(u, x + 1, y, z) + PSGridGetPeriodic(u, x, y - 1, z) + PSGridGetPeriodic(u, x, y, z + 1)) * c);")),
    "four halos": ("uabd", _source("uabd", f"PSGridEmit(out, c * ({SIX.format('u')}) + ({SIX.format('a')}) * {AT.format('u')} + ({SIX.format('b')}) - ({SIX.format('d')}));")),
    "two halos": ("ua", _source("ua", f"PSGridEmit(out, c * ({SIX.format('u')}) - ({SIX.format('a')}) * {AT.format('u')});")),
    "reads the output": ("u", _source("u", f"PSGridEmit(out, 2 * {AT.format('u')} - {AT.format('out')} + c * ({SIX.format('u')}));")),
    "radius 3": ("u", _source("u", f"PSGridEmit(out, c * ({SIX.format('u')} + PSGridGet(u, x + 3, y, z) + PSGridGet(u, x, y - 3, z) + PSGridGet(u, x, y, z + 3) + PSGridGet(u, x, y, z - 2)));")),
    "nine grids": ("uabdeghij", _source("uabdeghij", f"PSGridEmit(out, {SIX.format('u')} + c * ({' + '.join(AT.format(g) for g in 'abdeghij')}));")),
    "early return": ("uk", _source("uk", f"if (x % 3 == 1) return; PSGridEmit(out, {AT.format('k')} * ({SIX.format('u')}) * c);")),
}
TYPES = {"f32": (np.float32, "Float", "float"), "f64": (np.float64, "Double", "double"),
         "i32": (np.int32, "Int", "int"), "i64": (np.int64, "Long", "long")}


@pytest.fixture(scope="module")
def rt():
    ps.build()
    ps.init()
    yield ps
    ps.clear_error()


@pytest.mark.parametrize("name", sorted(FORMS))
@pytest.mark.parametrize("dtype", sorted(TYPES))
def test_tiled_form_gives_the_plain_bits(rt, monkeypatch, name, dtype):
    np_type, suffix, ctype = TYPES[dtype]
    names, text = FORMS[name]
    k = ps.stencil_function(text.replace("@N", suffix).replace("@T", ctype), "f")
    h = 0 if name == "centre periodic" else 3 if name == "radius 3" else 1
    rng = np.random.default_rng(7)
    for shape in ((9, 18, 67), (8, 35, 132), (12, 16, 64), (7, 50, 9), (40, 9, 70)):
        nz, ny, nx = shape
        values = [(rng.integers(-50, 50, shape) if np.issubdtype(np_type, np.integer)
                   else rng.uniform(-1, 1, shape)).astype(np_type) for _ in range(len(names) + 1)]
        grids = [ps.Grid(shape, np_type) for _ in values]
        got = []
        for env in ("0", "1", None):
            if env is None:
                monkeypatch.delenv("PS_FUNCTION_TILED", raising=False)
            else:
                monkeypatch.setenv("PS_FUNCTION_TILED", env)
            for g, v in zip(grids, values):
                g.copyin(v)
            dom = ps.domain(h, nx - h, h, ny - h, h, nz - h)
            m = ps.stencil_map(k, dom, grids, [3.0])
            ps.stencil_run([m], 2)
            got.append(grids[-1].copyout())
        for g in grids:
            g.free()
        for other in got[1:]:
            assert np.array_equal(got[0].view(np.uint8), other.view(np.uint8)), shape


def test_read_after_an_emit_in_a_helper(rt, monkeypatch):
    # k is read at the cell only and emitted under another name: its second read
    # sees what was emitted, on both entries
    k = ps.stencil_function("""
void put(PSGrid3DFloat g, float v) { PSGridEmit(g, v); }
void f(const int x, const int y, const int z, PSGrid3DFloat u, PSGrid3DFloat k,
       PSGrid3DFloat out) {
  float a = PSGridGet(k, x, y, z) + PSGridGet(u, x + 1, y, z) + PSGridGet(u, x, y, z - 1);
  put(k, a);
  PSGridEmit(out, 2.0f * PSGridGet(k, x, y, z));
}
""", "f")
    shape = (9, 18, 67)
    nz, ny, nx = shape
    rng = np.random.default_rng(9)
    u, v = (rng.random(shape, dtype=np.float32) for _ in range(2))
    a = (v[1:-1, 1:-1, 1:-1] + u[1:-1, 1:-1, 2:]) + u[:-2, 1:-1, 1:-1]
    for env in ("0", "1"):
        monkeypatch.setenv("PS_FUNCTION_TILED", env)
        grids = [ps.Grid(shape) for _ in range(3)]
        for g, w in zip(grids, (u, v, np.zeros_like(u))):
            g.copyin(w)
        ps.stencil_run([ps.stencil_map(k, ps.domain(1, nx - 1, 1, ny - 1, 1, nz - 1), grids)])
        assert np.array_equal(grids[2].copyout()[1:-1, 1:-1, 1:-1], np.float32(2) * a)
        assert np.array_equal(grids[1].copyout()[1:-1, 1:-1, 1:-1], a)
        for g in grids:
            g.free()


@pytest.mark.parametrize("name", ["four coefficients", "nine grids"])
def test_large_domains_choose_for_themselves(rt, monkeypatch, name):
    # 4.5 M cells: past the line under which these run the plain entry
    names, text = FORMS[name]
    k = ps.stencil_function(text.replace("@N", "Float").replace("@T", "float"), "f")
    shape = (70, 250, 257)
    rng = np.random.default_rng(8)
    values = [rng.random(shape, dtype=np.float32) for _ in range(len(names) + 1)]
    grids = [ps.Grid(shape) for _ in values]
    got = []
    for env in ("0", None):
        if env is None:
            monkeypatch.delenv("PS_FUNCTION_TILED", raising=False)
        else:
            monkeypatch.setenv("PS_FUNCTION_TILED", env)
        for g, v in zip(grids, values):
            g.copyin(v)
        nz, ny, nx = shape
        ps.stencil_run([ps.stencil_map(k, ps.domain(1, nx - 1, 1, ny - 1, 1, nz - 1), grids, [0.5])])
        got.append(grids[-1].copyout())
    for g in grids:
        g.free()
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
