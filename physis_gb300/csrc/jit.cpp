// Stencil functions compiled at run time (NVRTC) -- the translator-free
// front end.
//
// The reference turns a user stencil function such as
//     void kernel(const int x, const int y, const int z,
//                 PSGrid3DFloat g1, PSGrid3DFloat g2, float c) {
//       float v = PSGridGet(g1, x, y, z) + ... ;
//       PSGridEmit(g2, v * c);
//     }
// into a CUDA kernel with its source-to-source translator (physisc;
// translator/cuda_runtime_builder.cc:1099-1228 generates the run kernel, one
// thread per (x, y) and a loop over z; include/physis/physis_cuda.h:237-269
// the index arithmetic).  Here the function's own source text is compiled at
// run time: a short device prelude gives PSGridGet / PSGridGetPeriodic /
// PSGridEmit / PSGridDim and the PSGrid* types their device meaning, every
// unannotated function is a device function (-default-device), and a
// generated __global__ entry walks the domain and calls the function at each
// point.  Options --fmad=false and IEEE division/square root keep every
// float expression exactly as the C source writes it, so results match the
// REF target (the same source built by gcc with -ffp-contract=off) bit for
// bit.  NVRTC is loaded with dlopen; without it the entry points report
// PS_ERR_UNSUPPORTED.  The compiled image is loaded with the driver API into
// the runtime's context and never inspected.
#include <cuda.h>
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <regex>
#include <string>
#include <vector>

#include "ps_internal.h"
// kEmbedArith, kEmbedPointsBody: ps_arith.cuh and points_body.cuh as text
// (written into the build directory by buildlib.py).
#include "embedded_headers.inc"

#include <map>

namespace psg {
namespace {

// ---- NVRTC, resolved at run time -----------------------------------------
typedef int nvrtcResult_t;
typedef struct _nvrtcProgram *nvrtcProgram_t;
struct Nvrtc {
  bool tried = false, ok = false;
  nvrtcResult_t (*create)(nvrtcProgram_t *, const char *, const char *, int,
                          const char *const *, const char *const *) = nullptr;
  nvrtcResult_t (*compile)(nvrtcProgram_t, int, const char *const *) = nullptr;
  nvrtcResult_t (*log_size)(nvrtcProgram_t, size_t *) = nullptr;
  nvrtcResult_t (*log)(nvrtcProgram_t, char *) = nullptr;
  nvrtcResult_t (*cubin_size)(nvrtcProgram_t, size_t *) = nullptr;
  nvrtcResult_t (*cubin)(nvrtcProgram_t, char *) = nullptr;
  nvrtcResult_t (*destroy)(nvrtcProgram_t *) = nullptr;
};
Nvrtc g_nvrtc;

bool load_nvrtc(std::string *err) {
  if (g_nvrtc.tried) {
    if (!g_nvrtc.ok) *err = "NVRTC (libnvrtc.so) is not available";
    return g_nvrtc.ok;
  }
  g_nvrtc.tried = true;
  const char *names[] = {"libnvrtc.so.13", "libnvrtc.so", "/usr/local/cuda/lib64/libnvrtc.so.13",
                         "/usr/local/cuda/lib64/libnvrtc.so"};
  void *h = nullptr;
  for (const char *n : names)
    if ((h = dlopen(n, RTLD_NOW | RTLD_LOCAL))) break;
  if (!h) {
    *err = "NVRTC (libnvrtc.so) is not available";
    return false;
  }
#define PS_NVRTC_SYM(field, sym) \
  g_nvrtc.field = reinterpret_cast<decltype(g_nvrtc.field)>(dlsym(h, sym))
  PS_NVRTC_SYM(create, "nvrtcCreateProgram");
  PS_NVRTC_SYM(compile, "nvrtcCompileProgram");
  PS_NVRTC_SYM(log_size, "nvrtcGetProgramLogSize");
  PS_NVRTC_SYM(log, "nvrtcGetProgramLog");
  PS_NVRTC_SYM(cubin_size, "nvrtcGetCUBINSize");
  PS_NVRTC_SYM(cubin, "nvrtcGetCUBIN");
  PS_NVRTC_SYM(destroy, "nvrtcDestroyProgram");
#undef PS_NVRTC_SYM
  g_nvrtc.ok = g_nvrtc.create && g_nvrtc.compile && g_nvrtc.log_size && g_nvrtc.log &&
               g_nvrtc.cubin_size && g_nvrtc.cubin && g_nvrtc.destroy;
  if (!g_nvrtc.ok) *err = "libnvrtc.so lacks the expected entry points";
  return g_nvrtc.ok;
}

// ---- driver API, resolved through the runtime ------------------------------
struct Driver {
  bool tried = false, ok = false;
  CUresult (*load)(CUmodule *, const void *) = nullptr;
  CUresult (*get)(CUfunction *, CUmodule, const char *) = nullptr;
  CUresult (*launch)(const CUlaunchConfig *, CUfunction, void **, void **) = nullptr;
  CUresult (*unload)(CUmodule) = nullptr;
  CUresult (*set_attr)(CUfunction, CUfunction_attribute, int) = nullptr;
  CUresult (*occupancy)(int *, CUfunction, int, size_t) = nullptr;
  CUresult (*global)(CUdeviceptr *, size_t *, CUmodule, const char *) = nullptr;
};
Driver g_drv;

bool load_driver(std::string *err) {
  if (g_drv.tried) {
    if (!g_drv.ok) *err = "driver entry points for module loading are unavailable";
    return g_drv.ok;
  }
  g_drv.tried = true;
  auto sym = [](const char *name) -> void * {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion(name, &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return fn;
  };
  g_drv.load = reinterpret_cast<decltype(g_drv.load)>(sym("cuModuleLoadData"));
  g_drv.get = reinterpret_cast<decltype(g_drv.get)>(sym("cuModuleGetFunction"));
  g_drv.launch = reinterpret_cast<decltype(g_drv.launch)>(sym("cuLaunchKernelEx"));
  g_drv.unload = reinterpret_cast<decltype(g_drv.unload)>(sym("cuModuleUnload"));
  g_drv.set_attr = reinterpret_cast<decltype(g_drv.set_attr)>(sym("cuFuncSetAttribute"));
  g_drv.occupancy = reinterpret_cast<decltype(g_drv.occupancy)>(
      sym("cuOccupancyMaxActiveBlocksPerMultiprocessor"));
  g_drv.global = reinterpret_cast<decltype(g_drv.global)>(sym("cuModuleGetGlobal"));
  g_drv.ok = g_drv.load && g_drv.get && g_drv.launch && g_drv.unload && g_drv.set_attr &&
             g_drv.occupancy && g_drv.global;
  if (!g_drv.ok) {
    cudaGetLastError();
    *err = "driver entry points for module loading are unavailable";
  }
  return g_drv.ok;
}

// ---- the device prelude -----------------------------------------------------
// PSGrid{1,2,3}D{Float,Double,Int,Long} are one device struct per element
// type; `e` is the element the map's current point emits to.  Index
// arithmetic as the reference's (physis_cuda.h:237-269): x fastest, periodic
// reads wrap with (i + n) % n.
const char *kPrelude = R"PSJIT(
#include "ps_arith.cuh"
typedef int PSIndex;
// Kernel parameter (host layout: GridArg in jit.cpp).
template <typename T> struct __PSGridArg {
  T *p; long long row; long long plane; int nx; int ny; int nz; int rank;
};
// What the stencil function sees.  For a grid the tiled entry staged in
// shared memory (staged == 1) the entry also records the cell being computed
// (cx, cy, cz) and, for each plane offset d within rz, a pointer c[d + 4] to
// that cell's position in the staged plane z + d; a read at (cx + dx, cy +
// dy, cz + dz) with |dx| <= rx, |dy| <= ry, |dz| <= rz is then
// c[dz + 4][dy * sw + dx].  With the function inlined, reads written as x +
// const make every test and index a constant; any other read is tested at
// run time and falls back to global memory outside the window.
template <typename T> struct __PSGridDev {
  T *p; long long row; long long plane; int nx; int ny; int nz; int rank; T *e;
  int staged, rx, ry, rz, sw, cx, cy, cz;
  const T *c[9];
};
template <typename T> __device__ __forceinline__ __PSGridDev<T> __ps_dev(const __PSGridArg<T> &a) {
  __PSGridDev<T> g;
  g.p = a.p; g.row = a.row; g.plane = a.plane; g.nx = a.nx; g.ny = a.ny; g.nz = a.nz;
  g.rank = a.rank; g.e = nullptr; g.staged = 0;
  return g;
}
#define __PS_GRID_TYPES(N, T) \
  typedef __PSGridDev<T> PSGrid1D##N; typedef __PSGridDev<T> PSGrid2D##N; \
  typedef __PSGridDev<T> PSGrid3D##N;
__PS_GRID_TYPES(Float, float)
__PS_GRID_TYPES(Double, double)
__PS_GRID_TYPES(Int, int)
__PS_GRID_TYPES(Long, long long)
template <typename T>
__device__ __forceinline__ bool __ps_in_stage(const __PSGridDev<T> &g, int x, int y, int z) {
  const int dx = x - g.cx, dy = y - g.cy, dz = z - g.cz;
  return g.staged && dx >= -g.rx && dx <= g.rx && dy >= -g.ry && dy <= g.ry && dz >= -g.rz &&
         dz <= g.rz;
}
template <typename T>
__device__ __forceinline__ T __ps_staged(const __PSGridDev<T> &g, int x, int y, int z) {
  return g.c[z - g.cz + 4][(y - g.cy) * g.sw + (x - g.cx)];
}
template <typename T> __device__ __forceinline__ T __ps_get(const __PSGridDev<T> &g, int x) {
  return g.p[x];
}
template <typename T> __device__ __forceinline__ T __ps_get(const __PSGridDev<T> &g, int x, int y) {
  return g.p[(long long)y * g.row + x];
}
template <typename T>
__device__ __forceinline__ T __ps_get(const __PSGridDev<T> &g, int x, int y, int z) {
  if (__ps_in_stage(g, x, y, z)) return __ps_staged(g, x, y, z);
  return g.p[(long long)z * g.plane + (long long)y * g.row + x];
}
template <typename T> __device__ __forceinline__ T __ps_getp(const __PSGridDev<T> &g, int x) {
  return g.p[(x + g.nx) % g.nx];
}
template <typename T>
__device__ __forceinline__ T __ps_getp(const __PSGridDev<T> &g, int x, int y) {
  return g.p[(long long)((y + g.ny) % g.ny) * g.row + (x + g.nx) % g.nx];
}
// Staged windows of periodic grids hold the wrapped values at the unwrapped
// coordinates, so the window is looked up before wrapping.
template <typename T>
__device__ __forceinline__ T __ps_getp(const __PSGridDev<T> &g, int x, int y, int z) {
  if (__ps_in_stage(g, x, y, z)) return __ps_staged(g, x, y, z);
  return g.p[(long long)((z + g.nz) % g.nz) * g.plane + (long long)((y + g.ny) % g.ny) * g.row +
             (x + g.nx) % g.nx];
}
template <typename T> __device__ __forceinline__ int __ps_dim(const __PSGridDev<T> &g, int d) {
  return d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
}
// Grids of a user-defined element type: the source's own struct definition
// and DeclareGrid line; PSGridEmitUtype(g.m, v) reaches __PS_EMITU as
// __PS_EMITU((g).e[0].m, v) (the front end rewrites the call), i.e. a
// store to member m of the point being computed.
#define DeclareGrid1D(N, T) typedef __PSGridDev<T> PSGrid1D##N
#define DeclareGrid2D(N, T) typedef __PSGridDev<T> PSGrid2D##N
#define DeclareGrid3D(N, T) typedef __PSGridDev<T> PSGrid3D##N
#define __PS_EMITU(lhs, v) ((void)((lhs) = (v)))
#define PSGridGet(g, ...) __ps_get((g), __VA_ARGS__)
#define PSGridGetPeriodic(g, ...) __ps_getp((g), __VA_ARGS__)
#define PSGridEmit(g, v) ((void)((g).e[0] = (v)))
#define PSGridDim(g, d) __ps_dim((g), (d))

// ---- staging for the tiled entry ----
// Opaque TMA descriptor (the layout of CUtensorMap: 128 bytes, 64-aligned).
struct alignas(64) __PSTmap { unsigned long long opaque[16]; };
template <bool PER> __device__ __forceinline__ int __ps_fit(int v, int n) {
  if (PER) {
    if ((unsigned)v >= (unsigned)n) {
      v %= n;
      if (v < 0) v += n;
    }
    return v;
  }
  return min(max(v, 0), n - 1);
}
// Whether the W x H window at (xs, ys) has cells outside an nx x ny plane.
__device__ __forceinline__ bool __ps_crosses(int xs, int ys, int w, int h, int nx, int ny) {
  return xs < 0 || ys < 0 || xs + w > nx || ys + h > ny;
}
// One plane of a staged window (W x H cells at (xs, ys), TMA-filled with zeros
// outside the grid): the warp rewrites the outside cells that a halo of RX x
// RY can reach with the wrapped (PER, fetched from the grid's plane zg) or
// nearest (copied within the window) values.
template <typename T, int W, int H, int RX, int RY, bool PER>
__device__ __forceinline__ void __ps_edges(T *box, const __PSGridArg<T> &a, int xs, int ys,
                                           int zg, int lane) {
  const int c0 = max(0, -RX - xs), c1 = min(W, a.nx + RX - xs);
  const int r0 = max(0, -RY - ys), r1 = min(H, a.ny + RY - ys);
  const int rin0 = max(r0, -ys), rin1 = min(r1, a.ny - ys);
  const int cl = max(c0, -xs), cr = min(c1, a.nx - xs);
  const T *plane = a.p + (long long)zg * a.plane;
  for (int r = r0; r < r1; ++r) {
    if (r >= rin0 && r < rin1) continue;
    const int y = __ps_fit<PER>(ys + r, a.ny);
    for (int c = c0 + lane; c < c1; c += 32) {
      const int x = __ps_fit<PER>(xs + c, a.nx);
      box[r * W + c] = PER ? plane[(long long)y * a.row + x] : box[(y - ys) * W + (x - xs)];
    }
  }
  const int nc = (cl - c0) + (c1 - cr);
  if (nc <= 0) return;
  for (int r = rin0 + lane; r < rin1; r += 32)
    for (int k = 0; k < nc; ++k) {
      const int c = k < cl - c0 ? c0 + k : cr + (k - (cl - c0));
      const int x = __ps_fit<PER>(xs + c, a.nx);
      box[r * W + c] = PER ? plane[(long long)(ys + r) * a.row + x] : box[r * W + (x - xs)];
    }
}
)PSJIT";

// Host mirror of __PSGridDev<T> (same layout for every T: one pointer).
struct GridArg {
  void *p;
  long long row, plane;
  int nx, ny, nz, rank;
};

std::string trim(const std::string &s) {
  size_t a = s.find_first_not_of(" \t\r\n"), b = s.find_last_not_of(" \t\r\n");
  return a == std::string::npos ? std::string() : s.substr(a, b - a + 1);
}

// User grid types the source declares: "PSGrid3DPoint" -> (3, "struct Point").
typedef std::map<std::string, std::pair<int, std::string>> UserGrids;

UserGrids declared_grids(const std::string &src) {
  UserGrids out;
  static const std::regex re("\\bDeclareGrid([123])D\\s*\\(\\s*(\\w+)\\s*,\\s*([^)]*?)\\s*\\)");
  for (auto it = std::sregex_iterator(src.begin(), src.end(), re); it != std::sregex_iterator();
       ++it) {
    const int rank = (*it)[1].str()[0] - '0';
    out["PSGrid" + (*it)[1].str() + "D" + (*it)[2].str()] = {rank, trim((*it)[3].str())};
  }
  return out;
}

// Parses one parameter declaration ("const int x", "PSGrid3DFloat g1",
// "float c") into p; false if its type is not one the front end knows.
bool parse_param(const std::string &decl, JitParam *p, std::string *err,
                 const UserGrids &user = UserGrids()) {
  static const std::regex grid_re("^PSGrid([123])D(Float|Double|Int|Long)$");
  std::string d = " " + trim(decl) + " ";
  for (const char *q : {" const ", " register ", " volatile "}) {
    size_t at;
    while ((at = d.find(q)) != std::string::npos) d.replace(at, strlen(q) - 1, "");
  }
  d = trim(d);
  const size_t cut = d.find_last_of(" \t*&");
  if (cut == std::string::npos) {
    *err = "parameter '" + trim(decl) + "' has no name";
    return false;
  }
  std::string type = trim(d.substr(0, cut));
  std::string t;  // type with single spaces
  for (char c : type)
    if (!(c == ' ' && (t.empty() || t.back() == ' '))) t += (c == '\t' ? ' ' : c);
  type = trim(t);
  p->decl_type = type;
  p->name = trim(d.substr(cut + 1));
  std::smatch m;
  const auto u = user.find(type);
  if (u != user.end()) {
    p->grid = true;
    p->rank = u->second.first;
    p->type = kUser;
    p->utype = u->second.second;
    return true;
  }
  if (std::regex_match(type, m, grid_re)) {
    p->grid = true;
    p->rank = m[1].str()[0] - '0';
    const std::string e = m[2].str();
    p->type = e == "Float" ? kFloat : e == "Double" ? kDouble : e == "Int" ? kInt : kLong;
    return true;
  }
  p->grid = false;
  p->rank = 0;
  if (type == "int" || type == "PSIndex" || type == "signed int") p->type = kInt;
  else if (type == "long" || type == "long int" || type == "long long" ||
           type == "long long int")
    p->type = kLong;
  else if (type == "float") p->type = kFloat;
  else if (type == "double") p->type = kDouble;
  else {
    *err = "parameter type '" + type + "' is not supported (grids PSGrid{1,2,3}D{Float,"
           "Double,Int,Long}, scalars int/long/float/double)";
    return false;
  }
  return true;
}

// Finds `void name(...)` in src and parses its parameters.
bool parse_signature(const std::string &src, const std::string &name, JitKernel *k,
                     std::string *err) {
  const std::regex head("\\bvoid\\s+" + name + "\\s*\\(");
  std::smatch m;
  if (!std::regex_search(src, m, head)) {
    *err = "no definition 'void " + name + "(...)' in the stencil source";
    return false;
  }
  size_t i = m.position(0) + m.length(0);
  int depth = 1;
  std::string cur;
  std::vector<std::string> decls;
  for (; i < src.size() && depth > 0; ++i) {
    const char c = src[i];
    if (c == '(') ++depth;
    if (c == ')' && --depth == 0) break;
    if (c == ',' && depth == 1) {
      decls.push_back(cur);
      cur.clear();
    } else {
      cur += c;
    }
  }
  if (depth != 0) {
    *err = "unbalanced parameter list of " + name;
    return false;
  }
  if (!trim(cur).empty()) decls.push_back(cur);
  k->params.clear();
  k->nd = 0;
  bool seen_grid = false;
  const UserGrids user = declared_grids(src);
  for (const std::string &d : decls) {
    JitParam p;
    if (!parse_param(d, &p, err, user)) return false;
    if (!p.grid && !seen_grid && p.type == kInt && k->params.empty() && k->nd < 3) {
      k->idx[k->nd++] = p.name;  // a leading index parameter
      continue;
    }
    if (p.grid) seen_grid = true;
    if (!p.grid && !seen_grid) {
      *err = "stencil " + name + ": index parameters must come first, then the grids";
      return false;
    }
    k->params.push_back(p);
  }
  if (k->nd < 1) {
    *err = "stencil " + name + " has no index parameters (const int x[, y[, z]])";
    return false;
  }
  k->ngrids = k->nscalars = 0;
  for (const JitParam &p : k->params) (p.grid ? k->ngrids : k->nscalars)++;
  if (k->ngrids < 1) {
    *err = "stencil " + name + " takes no grid";
    return false;
  }
  return true;
}

std::string scalar_ctype(int type) {
  switch (type) {
    case kInt: return "int";
    case kLong: return "long long";
    case kFloat: return "float";
    default: return "double";
  }
}

// A grid parameter's element type in generated code.
std::string elem_ctype(const JitParam &p) {
  return p.type == kUser ? p.utype : scalar_ctype(p.type);
}

// Source expression of the grid argument arg in an entry: the device view
// g<i> the entry built from kernel parameter a<i>.
std::string cur_expr(const JitParam &p, const std::string &g) {
  return p.rank == 1 ? std::string("x")
         : p.rank == 2 ? "(long long)y * " + g + ".row + x"
                       : "(long long)z * " + g + ".plane + (long long)y * " + g + ".row + x";
}

std::string entry_params(const JitKernel &k) {
  std::string s;
  for (size_t i = 0; i < k.params.size(); ++i) {
    const JitParam &p = k.params[i];
    s += ", " + (p.grid ? "__PSGridArg<" + elem_ctype(p) + ">" : scalar_ctype(p.type)) +
         " a" + std::to_string(i);
  }
  return s;
}

std::string call_source(const JitKernel &k) {
  std::string s = k.name + "(x";
  if (k.nd >= 2) s += ", y";
  if (k.nd >= 3) s += ", z";
  for (size_t i = 0; i < k.params.size(); ++i)
    s += (k.params[i].grid ? ", g" : ", a") + std::to_string(i);
  return s + ");\n";
}

// The generated entry: one thread per (x, y), a z-chunk per block row in z;
// red/black maps visit every other x from the REF start
// min + ((min & 1) ^ ((y + z + color) % 2))
// (translator/reference_runtime_builder.cc:585-600).
std::string entry_source(const JitKernel &k) {
  std::string s =
      "\nextern \"C\" __global__ void __launch_bounds__(256) __ps_entry(int dmin0, int dmax0, "
      "int dmin1, int dmax1, int dmin2, int dmax2, int color, int zlen, int early" +
      entry_params(k) + ") {\n";
  for (size_t i = 0; i < k.params.size(); ++i)
    if (k.params[i].grid)
      s += "  auto g" + std::to_string(i) + " = __ps_dev(a" + std::to_string(i) + ");\n";
  s += "  if (early) psg::launch_dependents();\n  psg::wait_for_predecessors();\n"
       "  const int tx = blockIdx.x * blockDim.x + threadIdx.x;\n"
       "  const int y = dmin1 + blockIdx.y * blockDim.y + threadIdx.y;\n"
       "  if (y >= dmax1) return;\n"
       "  const int zs = dmin2 + blockIdx.z * zlen;\n"
       "  const int ze = min(zs + zlen, dmax2);\n"
       "  for (int z = zs; z < ze; ++z) {\n"
       "    const int x = color < 0 ? dmin0 + tx\n"
       "        : dmin0 + ((dmin0 & 1) ^ ((y + z + color) % 2)) + 2 * tx;\n"
       "    if (x >= dmax0) continue;\n";
  for (size_t i = 0; i < k.params.size(); ++i) {
    if (!k.params[i].grid) continue;
    const std::string g = "g" + std::to_string(i);
    s += "    " + g + ".e = " + g + ".p + (" + cur_expr(k.params[i], g) + ");\n";
  }
  s += "    " + call_source(k) + "  }\n}\n";
  return s;
}

// ---- the tiled entry ---------------------------------------------------------
// A CTA of four warps and a producer warp owns a 64 x 16 (x, y) tile and a
// chunk of z; a thread computes eight consecutive rows of one column (or eight warps
// and four rows, see choose_form).  Grids
// the stencil reads at neighbour offsets (and never emits to) are staged: a
// ring of shared-memory planes of the tile plus halo, one TMA box per plane,
// loaded a step ahead of the compute by the producer warp, which on edge tiles
// also gives the cells outside the grid their values.  The function's reads
// inside the window come from there.  The reads themselves are unchanged, so
// every result is bit-identical to the plain entry's.
//
// Issue slots are what such a kernel is short of, so:
// * a thread's rows share their loads (the window positions of a thread's cells
//   differ by constants, so equal reads are one load to the compiler) and a
//   step's fixed work;
// * warps whose cells all lie at least one cell inside the domain's grids and
//   inside the domain run a copy of the function that may assume so: the
//   comparisons of a function that treats the faces itself fold away;
// * boxes arrive by TMA, where cp.async took a quarter of the instructions.
// Measured, one sweep against the cp.async entry (256 threads, two by two cells
// each, CTA barriers): clamped 7-point function at 400 x 384 x 320 float 87
// against 154 us (52 instructions a cell against 92, 66 % of the HBM rate),
// 27-point function at 258 x 258 x 200 double 673 against 727 us (the FP64
// pipe's time is 556).
constexpr int kTileX = 64, kTileY = 16;
int tile_warps(int rows) { return kTileX / 32 * kTileY / rows; }  // rows: per thread, 8 or 4
int tile_threads(int rows) { return 32 * (tile_warps(rows) + 1); }
constexpr size_t kStageBudget = 80 * 1024;                // two or more CTAs per SM
constexpr size_t kStageHead = 128;                        // mbarriers in front of the rings

// Ring planes of a grid staged with z halo rz: the 2 rz + 1 planes a step
// reads and the next one.
int ring_planes(int rz) { return 2 * rz + 2; }
// Bytes of one of them (TMA destinations are 128-byte aligned).
size_t plane_bytes(const JitStage &st) {
  return ((size_t)st.w * (kTileY + 2 * st.ry) * st.esz + 127) / 128 * 128;
}

// Splits the argument list of the call whose '(' is at src[open] into its
// top-level arguments; npos-safe (returns false if unbalanced).
bool call_args(const std::string &src, size_t open, std::vector<std::string> *args,
               size_t *close) {
  int depth = 0;
  std::string cur;
  for (size_t i = open; i < src.size(); ++i) {
    const char c = src[i];
    if (c == '(' || c == '[' || c == '{') {
      if (depth++ > 0) cur += c;
      continue;
    }
    if (c == ')' || c == ']' || c == '}') {
      if (--depth == 0) {
        args->push_back(cur);
        *close = i;
        return true;
      }
      cur += c;
      continue;
    }
    if (c == ',' && depth == 1) {
      args->push_back(cur);
      cur.clear();
      continue;
    }
    cur += c;
  }
  return false;
}

// How the source text reads a grid parameter of the stencil.
struct GridUse {
  int reads = 0;                 // PSGridGet / PSGridGetPeriodic of it
  bool emitted = false;          // a PSGridEmit anywhere in the source names it
  bool off_centre = false, periodic = false;
  int r[3] = {0, 0, 0};          // halo widths
};

// One per parameter; *elsewhere: some PSGridEmit names what is no grid parameter (a
// helper function's own), so any of them may be emitted.
std::vector<GridUse> grid_uses(const JitKernel &k, bool *elsewhere) {
  std::vector<GridUse> uses(k.params.size());
  *elsewhere = false;
  const std::string &src = k.source;
  const std::regex emit_re("\\bPSGridEmit(?:Utype)?\\s*\\(\\s*(\\w+)");
  for (auto it = std::sregex_iterator(src.begin(), src.end(), emit_re);
       it != std::sregex_iterator(); ++it) {
    bool ours = false;
    for (size_t pi = 0; pi < uses.size(); ++pi)
      if (k.params[pi].grid && k.params[pi].name == (*it)[1].str()) uses[pi].emitted = ours = true;
    *elsewhere |= !ours;
  }
  const std::regex get_re("\\bPSGridGet(Periodic)?\\s*\\(");
  for (auto it = std::sregex_iterator(src.begin(), src.end(), get_re);
       it != std::sregex_iterator(); ++it) {
    const size_t open = it->position(0) + it->length(0) - 1;
    std::vector<std::string> args;
    size_t close = 0;
    if (!call_args(src, open, &args, &close) || args.size() != 4) continue;
    for (size_t pi = 0; pi < uses.size(); ++pi) {
      if (!k.params[pi].grid || k.params[pi].rank != 3 || trim(args[0]) != k.params[pi].name)
        continue;
      GridUse &u = uses[pi];
      ++u.reads;
      if ((*it)[1].matched) u.periodic = true;
      for (int d = 0; d < 3; ++d) {
        std::smatch m;
        const std::string a = trim(args[d + 1]);
        static const std::regex lit_re("^(\\w+)\\s*(?:([+-])\\s*([0-9]+))?$");
        if (std::regex_match(a, m, lit_re) && m[1].str() == k.idx[d]) {
          const int c = m[3].matched ? std::atoi(m[3].str().c_str()) : 0;
          if (c) u.off_centre = true;
          u.r[d] = std::max(u.r[d], std::min(c, 4));
        } else {
          u.off_centre = true;
          u.r[d] = std::max(u.r[d], 1);
        }
      }
    }
  }
  return uses;
}

// Stages parameter pi if it can be and the budget lasts.
bool add_stage(JitKernel *k, size_t pi, const GridUse &u) {
  const JitParam &p = k->params[pi];
  if (!p.grid || p.rank != 3 || p.type == kUser || u.emitted) return false;
  JitStage st;
  st.param = (int)pi;
  st.rx = u.r[0];
  st.ry = u.r[1];
  st.rz = u.r[2];
  st.periodic = u.periodic;
  st.esz = (p.type == kFloat || p.type == kInt) ? 4 : 8;
  // the window starts on 16 bytes, up to v - 1 cells left of the halo
  const int v = 16 / st.esz;
  st.w = (kTileX + 2 * st.rx + 2 * (v - 1)) / v * v;
  st.bytes = (size_t)ring_planes(st.rz) * plane_bytes(st);
  if (k->stage_smem + st.bytes > kStageBudget) return false;
  st.off = k->stage_smem;
  k->stage_smem += st.bytes;
  k->stages.push_back(st);
  return true;
}

void no_stages(JitKernel *k) {
  k->stages.clear();
  k->stage_smem = 0;
}

// The form of the tiled entry, or none.  Its threads make up for few warps with
// rows whose loads do not wait for one another; a read from global memory does wait
// (for the row before it to be stored: the compiler cannot tell that the two do not
// overlap), so a stencil that leaves grids unstaged takes another form.  Times of
// four sweeps, in us, 256 x 256 x 128 and 400 x 384 x 320:
// * 4-byte grids read at the cell only are staged as well, where that leaves none
//   (two coefficient grids 136 and 562; unstaged in eight rows 355 and 1905, in
//   four 193 and 1081, plain entry 201 and 1301);
// * where one with a halo is left: four rows, eight warps (four inputs 328 and
//   1575; eight rows 419 and 2181, plain 510 and 3175);
// * else (an emitted grid that is read; many grids, whose rows would each hold a
//   register per grid) the plain entry (Himeno's 14 grids 472 and 3038; eight rows
//   2728 and 15732);
// * 8-byte grids, whose bound is the FP64 pipe: four rows on eight warps for a few
//   unstaged reads (three coefficients 670 and 3929; eight rows 742 and 4384, plain
//   689 and 4347), the plain entry for more or for two staged grids, whose rings
//   leave few CTAs to an SM (1171 and 7240; 1231 and 7372).
// Under 4 M cells (2^22) there are too few planes for a CTA to be worth the ring's
// start: plain (two coefficients 300 x 20 x 400 50, staged 79), also for one grid
// read three or more planes away (a star of radius 4, 61 and 160; 187 and 704
// above, 299 and 2041 plain).
void choose_form(JitKernel *k, const std::vector<GridUse> &uses, bool emits_elsewhere) {
  int grids = 0, left = 0, rz = 0;
  bool wide = false, left_off = false;
  for (size_t pi = 0; pi < uses.size(); ++pi) {
    if (!uses[pi].reads) continue;
    const JitParam &p = k->params[pi];
    ++grids;
    wide |= p.type == kDouble || p.type == kLong;
    bool staged = false;
    for (const JitStage &st : k->stages) staged |= st.param == (int)pi;
    if (staged) {
      rz = std::max(rz, uses[pi].r[2]);
    } else {
      left += uses[pi].reads;
      left_off |= uses[pi].off_centre;
    }
  }
  if (!left) {
    if (wide && k->stages.size() > 1) return no_stages(k);
    if (rz >= 3) {
      k->min_ctas = 3;
      k->plain_below = 1 << 22;
    }
    return;
  }
  if (grids > 8 || (wide && left > 6)) return no_stages(k);
  k->plain_below = 1 << 22;
  if (wide) {
    k->rows = 4;
    k->min_ctas = 4;
    return;
  }
  if (left_off) {
    k->rows = 4;
    k->min_ctas = 3;
    return;
  }
  // a cell that is read after it was emitted has to show what was emitted
  if (emits_elsewhere) return no_stages(k);
  for (size_t pi = 0; pi < uses.size(); ++pi) {
    bool staged = false;
    for (const JitStage &st : k->stages) staged |= st.param == (int)pi;
    if (uses[pi].reads && !staged && !add_stage(k, pi, uses[pi])) return no_stages(k);
  }
  if (k->stages.size() > 2) k->min_ctas = 3;
}

// Chooses the staged grids of a 3D stencil from its source text.  A grid is
// staged when some PSGridGet / PSGridGetPeriodic of it reads off the centre
// and no PSGridEmit anywhere in the source names it.  A coordinate written
// as `x`, `x + c` or `x - c` (x the index parameter of that axis, c a
// literal) widens the halo to c; any other coordinate expression widens it to
// at least 1.  Halos are capped at 4: the window test in the accessors sends
// any read outside the staged window to global memory, so the choice affects
// speed only, never results.
void choose_stages(JitKernel *k) {
  no_stages(k);
  if (k->nd != 3) return;
  bool elsewhere = false;
  const std::vector<GridUse> uses = grid_uses(*k, &elsewhere);
  for (size_t pi = 0; pi < uses.size(); ++pi)
    if (uses[pi].off_centre) add_stage(k, pi, uses[pi]);
  if (!k->stages.empty()) choose_form(k, uses, elsewhere);
}

std::string tiled_entry_source(const JitKernel &k) {
  const auto N = [](long long v) { return std::to_string(v); };
  std::string s = "\nextern \"C\" __global__ void __launch_bounds__(" + N(tile_threads(k.rows)) +
                  (k.min_ctas ? ", " + N(k.min_ctas) : std::string()) + ") __ps_entry_t(int dmin0, int dmax0, int dmin1, int dmax1, int dmin2, "
                  "int dmax2, int ntx, int zlen, int early, int *err";
  for (size_t j = 0; j < k.stages.size(); ++j)
    s += ", const __grid_constant__ __PSTmap tm" + N(j);
  s += entry_params(k) + ") {\n"
       "  extern __shared__ __align__(128) unsigned char __ps_raw[];\n"
       "  unsigned char *__ps_sm = __ps_raw + ((128u - (psg::smem_u32(__ps_raw) & 127u)) & 127u);\n"
       // barriers: group loaded (full), box landed (raw), step done (empty), two each
       "  unsigned long long *full = reinterpret_cast<unsigned long long *>(__ps_sm), *raw = full + 2,"
       " *empty = full + 4;\n"
       "  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;\n"
       "  const int x0 = dmin0 + (int)(blockIdx.x % (unsigned)ntx) * " + N(kTileX) + ";\n"
       "  const int y0 = dmin1 + (int)(blockIdx.x / (unsigned)ntx) * " + N(kTileY) + ";\n"
       "  const int zs = dmin2 + (int)blockIdx.y * zlen;\n"
       "  const int n = min(zs + zlen, dmax2) - zs;\n"
       "  if (n <= 0) return;\n"
       "  if (threadIdx.x == 0) {\n"
       "    for (int i = 0; i < 2; ++i) {\n"
       "      psg::mbar_init(&full[i], 1);\n      psg::mbar_init(&raw[i], 1);\n"
       "      psg::mbar_init(&empty[i], " + N(tile_warps(k.rows)) + ");\n    }\n"
       "    psg::fence_barrier_init();\n  }\n"
       "  __syncthreads();\n"
       "  if (early) psg::launch_dependents();\n  psg::wait_for_predecessors();\n";
  // the staged grids' rings and windows
  std::string edge, init, step, fixi, fixs;
  size_t bytes0 = 0, bytes1 = 0;
  for (size_t j = 0; j < k.stages.size(); ++j) {
    const JitStage &st = k.stages[j];
    const std::string i = N(st.param), sj = N(j);
    const std::string T = scalar_ctype(k.params[st.param].type);
    const int W = st.w, H = kTileY + 2 * st.ry, S = ring_planes(st.rz);
    const size_t pe = plane_bytes(st) / st.esz;
    const std::string fit = std::string("__ps_fit<") + (st.periodic ? "true" : "false") + ">";
    s += "  " + T + " *s" + sj + " = reinterpret_cast<" + T + " *>(__ps_sm + " +
         N(kStageHead + st.off) + ");\n";
    s += "  const int xs" + sj + " = (x0 - " + N(st.rx) + ") & ~" + N(16 / st.esz - 1) + ", ys" + sj +
         " = y0 - " + N(st.ry) + ";\n";
    edge += (j ? " || " : "") + ("__ps_crosses(xs" + sj + ", ys" + sj + ", " + N(W) + ", " + N(H) +
            ", a" + i + ".nx, a" + i + ".ny)");
    bytes0 += (size_t)(2 * st.rz + 1) * W * H * st.esz;
    bytes1 += (size_t)W * H * st.esz;
    const std::string load = "psg::tma_load_3d(s" + sj + " + ", at = ", &tm" + sj + ", xs" + sj +
                             ", ys" + sj + ", " + fit + "(";
    const std::string fix = "__ps_edges<" + T + ", " + N(W) + ", " + N(H) + ", " + N(st.rx) + ", " +
                            N(st.ry) + ", " + (st.periodic ? "true" : "false") + ">(s" + sj + " + ";
    // group 0: planes zs - rz .. zs + rz in slots 0 .. 2 rz; group i: plane
    // zs + i + rz in slot (i + 2 rz) % S
    init += "        for (int d = 0; d <= " + N(2 * st.rz) + "; ++d) " + load + "d * " + N(pe) + at +
            "zs - " + N(st.rz) + " + d, a" + i + ".nz), bar);\n";
    step += "        " + load + "(i + " + N(2 * st.rz) + ") % " + N(S) + " * " + N(pe) + at + "zs + i + " +
            N(st.rz) + ", a" + i + ".nz), bar);\n";
    fixi += "        for (int d = 0; d <= " + N(2 * st.rz) + "; ++d) " + fix + "d * " + N(pe) + ", a" + i +
            ", xs" + sj + ", ys" + sj + ", " + fit + "(zs - " + N(st.rz) + " + d, a" + i + ".nz), lane);\n";
    fixs += "        " + fix + "(i + " + N(2 * st.rz) + ") % " + N(S) + " * " + N(pe) + ", a" + i + ", xs" +
            sj + ", ys" + sj + ", " + fit + "(zs + i + " + N(st.rz) + ", a" + i + ".nz), lane);\n";
  }
  s += "  if (warp == " + N(tile_warps(k.rows)) + ") {\n"
       "    const bool edge = " + edge + ";\n"
       "    for (int i = 0; i < n; ++i) {\n"
       "      // group i replaces the plane that step i - 2 read last\n"
       "      if (i >= 2 && !__all_sync(0xffffffffu, psg::mbar_wait(&empty[i & 1], ((i - 2) >> 1) & 1, err)))"
       " return;\n"
       "      unsigned long long *bar = edge ? &raw[i & 1] : &full[i & 1];\n"
       "      if (lane == 0) {\n"
       "        psg::mbar_arrive_expect_tx(bar, i ? " + N(bytes1) + "u : " + N(bytes0) + "u);\n"
       "        if (i == 0) {\n" + init + "        } else {\n" + step + "        }\n      }\n"
       "      if (!edge) continue;\n"
       "      if (!__all_sync(0xffffffffu, psg::mbar_wait(bar, (i >> 1) & 1, err))) return;\n"
       "      if (i == 0) {\n" + fixi + "      } else {\n" + fixs + "      }\n"
       "      asm volatile(\"fence.proxy.async.shared::cta;\" ::: \"memory\");\n"
       "      __syncwarp();\n"
       "      if (lane == 0) psg::mbar_arrive(&full[i & 1]);\n    }\n"
       "    // the last copies land before the CTA may end\n"
       "    for (int i = max(0, n - 2); i < n; ++i)\n"
       "      psg::mbar_wait(&full[i & 1], (i >> 1) & 1, nullptr, 1u << 16);\n"
       "    return;\n  }\n";
  // consumers
  s += "  const int x = x0 + lane + 32 * (warp % " + N(kTileX / 32) + ");\n"
       "  const int yb = y0 + " + N(k.rows) + " * (warp / " + N(kTileX / 32) + ");\n";
  std::string inner = "__all_sync(0xffffffffu, x >= dmin0 && x < dmax0 && yb + " +
                      N(k.rows) + " <= dmax1", zin, assume;
  for (size_t i = 0; i < k.params.size(); ++i) {
    if (!k.params[i].grid) continue;
    const JitParam &p = k.params[i];
    const std::string si = N(i), g = "g" + si, a = "a" + si;
    s += "  auto " + g + " = __ps_dev(" + a + ");\n";
    // the element of the thread's first row, advanced by a plane per step
    s += "  auto *e" + si + " = " + a + ".p + (" +
         (p.rank == 1 ? std::string("x")
          : p.rank == 2 ? "(long long)yb * " + a + ".row + x"
                        : "(long long)zs * " + a + ".plane + (long long)yb * " + a + ".row + x") + ");\n";
    if (p.rank != 3) continue;
    inner += " && x >= 1 && x < " + a + ".nx - 1 && yb >= 1 && yb + " + N(k.rows) + " <= " + a +
             ".ny - 1";
    zin += " && z < " + a + ".nz - 1";
    for (const char *d : {"x", "y", "z"}) {
      const std::string dim = g + ".n" + d;
      assume += std::string("__builtin_assume(") + d + " < " + dim + " - 1); __builtin_assume(" + d +
                " + 1 < " + dim + "); ";
    }
  }
  s += "  const bool inner = " + inner + ");\n";
  for (size_t j = 0; j < k.stages.size(); ++j) {
    const JitStage &st = k.stages[j];
    const std::string g = "g" + N(st.param);
    s += "  " + g + ".staged = 1; " + g + ".rx = " + N(st.rx) + "; " + g + ".ry = " + N(st.ry) + "; " + g +
         ".rz = " + N(st.rz) + "; " + g + ".sw = " + N(st.w) + ";\n";
    s += "  const int w" + N(j) + " = (yb - ys" + N(j) + ") * " + N(st.w) + " + (x - xs" +
         N(j) + ");\n";
  }
  s += "  bool ok = true;\n"
       "  for (int i = 0; i < n; ++i) {\n"
       "    const int z = zs + i;\n"
       "    if (ok) ok = __all_sync(0xffffffffu, psg::mbar_wait(&full[i & 1], (i >> 1) & 1, err));\n"
       "    if (ok) {\n";
  std::string cell, advance;
  for (size_t j = 0; j < k.stages.size(); ++j) {
    const JitStage &st = k.stages[j];
    const std::string g = "g" + N(st.param), sj = N(j);
    const int S = ring_planes(st.rz);
    s += "      const " + scalar_ctype(k.params[st.param].type) + " *pl" + sj + "[" + N(2 * st.rz + 1) + "];\n"
         "#pragma unroll\n"
         "      for (int d = 0; d <= " + N(2 * st.rz) + "; ++d) pl" + sj + "[d] = s" + sj +
         " + (i + d) % " + N(S) + " * " + N(plane_bytes(st) / st.esz) + " + w" + sj + ";\n";
    cell += "          " + g + ".cx = x; " + g + ".cy = y; " + g + ".cz = z;\n"
            "          for (int d = 0; d <= " + N(2 * st.rz) + "; ++d) " + g + ".c[d + " + N(4 - st.rz) +
            "] = pl" + sj + "[d] + r * " + N(st.w) + ";\n";
  }
  for (size_t i = 0; i < k.params.size(); ++i) {
    if (!k.params[i].grid) continue;
    const JitParam &p = k.params[i];
    const std::string si = N(i);
    cell += "          g" + si + ".e = e" + si + (p.rank == 1 ? "" : " + r * a" + si + ".row") + ";\n";
    if (p.rank == 3) advance += "    e" + si + " += a" + si + ".plane;\n";
  }
  const std::string rows = "#pragma unroll\n        for (int r = 0; r < " + N(k.rows) + "; ++r) {\n"
                           "          const int y = yb + r;\n";
  s += "      if (inner && z > 0" + zin + ") {\n" + rows +
       "          __builtin_assume(x > 0); __builtin_assume(y > 0); __builtin_assume(z > 0); " + assume +
       "\n" + cell + "          " + call_source(k) + "        }\n      } else {\n" + rows +
       "          if (x < dmin0 || x >= dmax0 || y >= dmax1) continue;\n" + cell + "          " +
       call_source(k) + "        }\n      }\n    }\n"
       "    __syncwarp();\n"
       "    if (lane == 0) psg::mbar_arrive(&empty[i & 1]);\n" + advance + "  }\n}\n";
  return s;
}

}  // namespace

namespace {

// PSGridEmitUtype(g.member, v) -> __PS_EMITU((g).e[0].member, v): the
// member expression is applied to the point being computed.
std::string rewrite_emit_utype(const std::string &src) {
  static const std::regex re("\\bPSGridEmitUtype\\s*\\(\\s*([A-Za-z_]\\w*)");
  return std::regex_replace(src, re, "__PS_EMITU(($1).e[0]");
}

// One device global per user-type grid parameter holding its element size,
// read back after loading to check the grids a map passes.
std::string utype_sizes_source(const JitKernel &k) {
  std::string s;
  for (size_t i = 0; i < k.params.size(); ++i)
    if (k.params[i].grid && k.params[i].type == kUser)
      s += "extern \"C\" __device__ const int __ps_esz" + std::to_string(i) +
           " = (int)sizeof(" + k.params[i].utype + ");\n";
  return s;
}

// Compiles one program text for sm_103a (headers: ps_arith.cuh).
bool nvrtc_compile(const std::string &program, std::vector<char> *image, std::string *log) {
  nvrtcProgram_t prog = nullptr;
  const char *hdr_src[] = {kEmbedArith};
  const char *hdr_name[] = {"ps_arith.cuh"};
  if (g_nvrtc.create(&prog, program.c_str(), "stencil.cu", 1, hdr_src, hdr_name) != 0) {
    *log = "nvrtcCreateProgram failed";
    return false;
  }
  const char *opts[] = {"--gpu-architecture=sm_103a", "--std=c++17", "--fmad=false",
                        "--prec-div=true", "--prec-sqrt=true", "--ftz=false",
                        "--device-as-default-execution-space", "-DPS_JIT=1"};
  const int rc = g_nvrtc.compile(prog, (int)(sizeof(opts) / sizeof(opts[0])), opts);
  if (rc != 0) {
    size_t n = 0;
    g_nvrtc.log_size(prog, &n);
    log->assign(n, '\0');
    if (n) g_nvrtc.log(prog, &(*log)[0]);
    g_nvrtc.destroy(&prog);
    return false;
  }
  size_t n = 0;
  g_nvrtc.cubin_size(prog, &n);
  image->resize(n);
  g_nvrtc.cubin(prog, image->data());
  g_nvrtc.destroy(&prog);
  return true;
}

}  // namespace

bool jit_build(const char *source, const char *name, JitKernel *k, std::vector<char> *image,
               std::string *err) {
  if (!load_nvrtc(err)) return false;
  k->name = name;
  k->source = source;
  if (!parse_signature(k->source, k->name, k, err)) return false;
  choose_stages(k);
  const std::string base = std::string(kPrelude) + "#line 1 \"stencil\"\n" +
                           rewrite_emit_utype(k->source) + "\n" + entry_source(*k) +
                           utype_sizes_source(*k);
  std::string log;
  // PS_JIT_DUMP=<dir> writes the generated program to <dir>/<name>.cu (for
  // building it offline with nvcc to read its resource usage).
  if (const char *dir = getenv("PS_JIT_DUMP")) {
    const std::string path = std::string(dir) + "/" + k->name + ".cu";
    if (FILE *f = fopen(path.c_str(), "w")) {
      const std::string text = base + (k->stages.empty() ? "" : tiled_entry_source(*k));
      fwrite(text.data(), 1, text.size(), f);
      fclose(f);
    }
  }
  // Both entries in one program; should the tiled one not compile, the plain
  // entry alone (the stencil then runs untiled).
  if (!k->stages.empty() && nvrtc_compile(base + tiled_entry_source(*k), image, &log))
    return true;
  k->stages.clear();
  k->stage_smem = 0;
  if (nvrtc_compile(base, image, &log)) return true;
  *err = "stencil " + k->name + " does not compile: " + log.substr(0, 600);
  return false;
}

// Dynamic shared memory of the tiled entry (with slack to align its base).
static size_t stage_dynamic(const JitKernel &k) { return 128 + kStageHead + k.stage_smem; }

bool jit_compile(const char *source, const char *name, JitKernel *k, std::string *err) {
  std::vector<char> image;
  if (!jit_build(source, name, k, &image, err) || !load_driver(err)) return false;
  CUmodule mod = nullptr;
  CUfunction fn = nullptr, fn_t = nullptr;
  if (g_drv.load(&mod, image.data()) != CUDA_SUCCESS) {
    *err = "loading the compiled stencil failed";
    return false;
  }
  if (g_drv.get(&fn, mod, "__ps_entry") != CUDA_SUCCESS) {
    g_drv.unload(mod);
    *err = "compiled stencil has no entry";
    return false;
  }
  if (!k->stages.empty()) {
    if (g_drv.get(&fn_t, mod, "__ps_entry_t") != CUDA_SUCCESS ||
        g_drv.set_attr(fn_t, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES,
                       (int)stage_dynamic(*k)) != CUDA_SUCCESS) {
      fn_t = nullptr;
      k->stages.clear();
      k->stage_smem = 0;
    }
  }
  k->tiled_occ = 0;
  if (fn_t && (g_drv.occupancy(&k->tiled_occ, fn_t, tile_threads(k->rows), stage_dynamic(*k)) !=
                   CUDA_SUCCESS ||
               k->tiled_occ < 1)) {
    k->tiled_occ = 0;
    fn_t = nullptr;
  }
  // element sizes of the user-type grid parameters, as the compiler laid
  // the structs out
  for (size_t i = 0; i < k->params.size(); ++i) {
    JitParam &p = k->params[i];
    if (!p.grid || p.type != kUser) continue;
    CUdeviceptr dptr = 0;
    size_t bytes = 0;
    int esz = 0;
    const std::string sym = "__ps_esz" + std::to_string(i);
    if (g_drv.global(&dptr, &bytes, mod, sym.c_str()) != CUDA_SUCCESS || bytes != sizeof(int) ||
        cudaMemcpy(&esz, reinterpret_cast<void *>(dptr), sizeof(int), cudaMemcpyDeviceToHost) !=
            cudaSuccess) {
      cudaGetLastError();
      g_drv.unload(mod);
      *err = "cannot read the element size of " + p.utype;
      return false;
    }
    p.esz = esz;
  }
  k->module = mod;
  k->func = fn;
  k->func_tiled = fn_t;
  return true;
}

void jit_unload(JitKernel *k) {
  if (k->module && g_drv.unload) g_drv.unload(static_cast<CUmodule>(k->module));
  k->module = k->func = k->func_tiled = nullptr;
}

namespace {

// PS_FUNCTION_TILED=0 runs every map on the plain entry, =1 every map on the tiled
// one that it can run, however small (read per launch).
bool tiled_wanted(const JitKernel &k, long long cells) {
  const char *e = getenv("PS_FUNCTION_TILED");
  if (e && e[0] == '0') return false;
  return (e && e[0] == '1') || cells >= k.plain_below;
}

}  // namespace

// A launch of a compiled kernel; with `overlap` it may start before the stream's
// previous kernel ends.
static CUresult launch_function(void *fn, dim3 grid, dim3 block, size_t smem, bool overlap,
                                cudaStream_t s, void **args) {
  CUlaunchAttribute at = {};
  at.id = CU_LAUNCH_ATTRIBUTE_PROGRAMMATIC_STREAM_SERIALIZATION;
  at.value.programmaticStreamSerializationAllowed = 1;
  CUlaunchConfig c = {};
  c.gridDimX = grid.x;
  c.gridDimY = grid.y;
  c.gridDimZ = grid.z;
  c.blockDimX = block.x;
  c.blockDimY = block.y;
  c.blockDimZ = block.z;
  c.sharedMemBytes = (unsigned)smem;
  c.hStream = static_cast<CUstream>(s);
  c.attrs = &at;
  c.numAttrs = overlap ? 1 : 0;
  return g_drv.launch(&c, static_cast<CUfunction>(fn), args, nullptr);
}

// The tiled entry runs every-point maps of stencils with staged grids when
// no staged grid shares its memory with another grid argument (a staged copy
// of a grid that the same launch writes would be stale) and TMA can describe
// each of them; red/black maps and everything else run the plain entry.
cudaError_t jit_launch(const JitKernel &k, const Box &dom, int color, const GridView *grids,
                       const double *scalars, int sm_count, int *dev_err, bool overlap,
                       cudaStream_t s) {
  const int nxd = dom.max[0] - dom.min[0], nyd = dom.max[1] - dom.min[1],
            nzd = dom.max[2] - dom.min[2];
  if (nxd <= 0 || nyd <= 0 || nzd <= 0) return cudaSuccess;
  bool tiled = k.func_tiled && color < 0 && k.tiled_occ > 0 &&
               tiled_wanted(k, (long long)nxd * nyd * nzd);
  std::vector<CUtensorMap> maps(tiled ? k.stages.size() : 0);
  for (size_t t = 0; t < maps.size() && tiled; ++t) {
    const JitStage &st = k.stages[t];
    int gi = 0, sgi = -1;
    for (size_t i = 0; i < k.params.size(); ++i)
      if (k.params[i].grid) {
        if ((int)i == st.param) sgi = gi;
        ++gi;
      }
    for (int j = 0; j < gi && tiled; ++j)
      if (j != sgi && grids[j].ptr == grids[sgi].ptr) tiled = false;
    if (tiled) tiled = make_tmap_3d(&maps[t], grids[sgi], st.w, kTileY + 2 * st.ry);
  }
  unsigned gx, gy, gz, bx, by;
  int head[9];
  if (tiled) {
    const long long ntx = (nxd + kTileX - 1) / kTileX, nty = (nyd + kTileY - 1) / kTileY;
    const long long tiles = ntx * nty;
    // z chunks: one wave of resident CTAs while chunks are short, else chunks
    // of five planes (times the stencil's z radius): many small CTAs even out
    // edge tiles and tails, and neighbouring chunks' halo planes come from L2
    // (400 x 384 x 320, 7 points: 88 us a sweep with 5 planes, 98 with 2, 129 with
    // 1, 91 with 12).  Double functions are bound by the SMs' FP64 pipes, which
    // chunks of one plane (or the radius) share out best: 27 points 281 x 194 x 51
    // 152 us with 1 plane, 157 with 2, 195 with 3, 164 with 5; 258 x 258 x 200 674,
    // 676, 677 and 684; 7 points 200 x 150 x 180 163, 167, 174 and 180.
    const long long want = std::max(1LL, (long long)k.tiled_occ * sm_count);
    int rz = 1;
    bool fp64 = false;
    for (const JitStage &st : k.stages) {
      rz = std::max(rz, st.rz);
      fp64 |= k.params[st.param].type == kDouble;
    }
    const int zlen = (int)std::max({1LL, std::min((long long)nzd * tiles / want, (fp64 ? 1LL : 5LL) * rz),
                                    (nzd + 65534LL) / 65535});
    const long long chunks = (nzd + zlen - 1) / zlen;
    if (tiles > 0x7fffffffLL || chunks > 65535) return cudaErrorInvalidConfiguration;
    gx = (unsigned)tiles;
    gy = (unsigned)chunks;
    gz = 1;
    bx = (unsigned)tile_threads(k.rows);
    by = 1;
    const int h[9] = {dom.min[0], dom.max[0], dom.min[1], dom.max[1], dom.min[2], dom.max[2],
                      (int)ntx,   zlen,       tiles * chunks >= want};
    memcpy(head, h, sizeof(h));
  } else {
    bx = 64;
    by = 4;
    const int xs = color < 0 ? nxd : (nxd + 1) / 2;
    gx = (unsigned)((xs + bx - 1) / bx);
    gy = (unsigned)((nyd + by - 1) / by);
    long long want = 8LL * sm_count;  // blocks in flight: a few per SM
    long long nz = (want + (long long)gx * gy - 1) / ((long long)gx * gy);
    if (nz < 1) nz = 1;
    if (nz > nzd) nz = nzd;
    const int zlen = (int)((nzd + nz - 1) / nz);
    nz = (nzd + zlen - 1) / zlen;
    if (gy > 65535 || nz > 65535) return cudaErrorInvalidConfiguration;
    gz = (unsigned)nz;
    // The next sweep's CTAs may take places while this one runs if it fills the GPU,
    // but not among CTAs of one plane (1D, 2D and wide flat grids): these end at once,
    // and opening the gate to the next launch is then most of their time (per sweep of
    // floats, us, open and shut: 5 M cells in 1D 79 and 40, 3000 x 4000 49 and 40).
    const bool early = zlen > 1 && gx * gy * nz >= want;
    const int h[9] = {dom.min[0], dom.max[0], dom.min[1], dom.max[1], dom.min[2],
                      dom.max[2], color,      zlen,       early};
    memcpy(head, h, sizeof(h));
  }

  // argument storage: 9 ints, then each parameter at its alignment
  std::vector<unsigned char> buf(64 + 64 * k.params.size() + 16);
  std::vector<void *> args;
  size_t off = 0;
  auto put = [&](const void *v, size_t n, size_t align) {
    off = (off + align - 1) / align * align;
    memcpy(buf.data() + off, v, n);
    args.push_back(buf.data() + off);
    off += n;
  };
  for (int v : head) put(&v, 4, 4);
  if (tiled) {
    put(&dev_err, 8, 8);
    for (CUtensorMap &m : maps) args.push_back(&m);
  }
  int gi = 0, si = 0;
  for (const JitParam &p : k.params) {
    if (p.grid) {
      const GridView &g = grids[gi++];
      GridArg a;
      a.p = g.ptr;
      a.row = g.pitch / g.esz;
      a.plane = a.row * g.ny;
      a.nx = g.nx;
      a.ny = g.ny;
      a.nz = g.nz;
      a.rank = p.rank;
      put(&a, sizeof(a), 8);
    } else {
      const double v = scalars[si++];
      switch (p.type) {
        case kInt: { const int t = (int)v; put(&t, 4, 4); break; }
        case kLong: { const long long t = (long long)v; put(&t, 8, 8); break; }
        case kFloat: { const float t = (float)v; put(&t, 4, 4); break; }
        default: put(&v, 8, 8); break;
      }
    }
  }
  const CUresult r = launch_function(tiled ? k.func_tiled : k.func, dim3(gx, gy, gz), dim3(bx, by),
                                     tiled ? stage_dynamic(k) : 0, overlap, s, args.data());
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorLaunchFailure;
}

namespace {

const char *type_name(int type) {
  switch (type) {
    case kFloat: return "float";
    case kDouble: return "double";
    case kInt: return "int";
    default: return "long long";
  }
}

std::string points_source(const PtsJitKey &k) {
  std::string s = "#include \"points_body.cuh\"\nstruct GenSpec {\n"
                  "  static constexpr bool kStatic = true;\n";
  char buf[96];
  snprintf(buf, sizeof(buf), "  static constexpr int kN = %d;\n", k.n);
  s += buf;
  s += "  static constexpr int kW = " + std::to_string(k.w) + ", kPlanes = " +
       std::to_string(k.planes) + ", kCentre = " + std::to_string(k.centre) +
       ", kLX = " + std::to_string(k.lx) + ";\n";
  // several loads in flight per lane take registers that narrow halos do not repay
  // (9 points periodic, 4099 x 3001: 158 us a run with them, 152 without)
  int reach = 0;
  for (int i = 0; i < k.n; ++i) reach = std::max({reach, std::abs(k.dx[i]), std::abs(k.dy[i])});
  s += std::string("  static constexpr bool kWideHalo = ") + (reach >= 3 ? "true" : "false") + ";\n";
  s += "  static constexpr int kDx[kN] = {";
  for (int i = 0; i < k.n; ++i) s += (i ? ", " : "") + std::to_string(k.dx[i]);
  s += "};\n  static constexpr int kDy[kN] = {";
  for (int i = 0; i < k.n; ++i) s += (i ? ", " : "") + std::to_string(k.dy[i]);
  s += "};\n  static constexpr int kLag[kN] = {";
  for (int i = 0; i < k.n; ++i) s += (i ? ", " : "") + std::to_string(k.lag[i]);
  s += "};\n  static constexpr double kWt[kN] = {";
  for (int i = 0; i < k.n; ++i) {
    snprintf(buf, sizeof(buf), "%s%a", i ? ", " : "", k.wt[i]);
    s += buf;
  }
  s += "};\n";
  snprintf(buf, sizeof(buf), "%d", k.w);
  s += "  template <typename T> static __device__ __forceinline__ int lx("
       "const psg::PtsParams<T> &) { return kLX; }\n";
  s += "  template <typename T> static __device__ __forceinline__ int w(const psg::PtsParams<T> &)"
       " { return " + std::string(buf) + "; }\n";
  s += "  template <typename T> static __device__ __forceinline__ int nstage("
       "const psg::PtsParams<T> &) { return " + std::to_string(k.nstage) + "; }\n";
  s += "  template <typename T> static __device__ __forceinline__ int pstride("
       "const psg::PtsParams<T> &) { return " + std::to_string(k.pstride) + "; }\n};\n";
  const std::string T = type_name(k.type);
  s += "extern \"C\" __global__ void __launch_bounds__(" + std::to_string(32 * (k.warps + 1)) +
       ", " + std::to_string(k.min_ctas) + ") __ps_points(const __grid_constant__ psg::PtsParams<" + T + "> p, "
       "const __grid_constant__ psg::PtsTmap tm) {\n"
       "  extern __shared__ __align__(128) unsigned char smem[];\n"
       "  psg::pts_body<" + T + ", " + std::to_string(k.ry) + ", " +
       (k.unit ? "true" : "false") + ", GenSpec>(p, &tm, smem);\n}\n";
  return s;
}

struct PointsJit {
  void *fn = nullptr;  // CUfunction (nullptr: failed)
  int occ = 0;
};
std::map<std::string, PointsJit> g_points_jit;  // by the key's bytes and smem

}  // namespace

void *jit_points_function(const PtsJitKey &k, size_t smem, int *occ) {
  std::string key(reinterpret_cast<const char *>(&k), sizeof(k));
  key.append(reinterpret_cast<const char *>(&smem), sizeof(smem));
  auto hit = g_points_jit.find(key);
  if (hit != g_points_jit.end()) {
    *occ = hit->second.occ;
    return hit->second.fn;
  }
  std::string err;
  void *fn = nullptr;
  if (load_nvrtc(&err) && load_driver(&err)) {
    const std::string program = points_source(k);
    const char *hdr_src[] = {kEmbedArith, kEmbedPointsBody};
    const char *hdr_name[] = {"ps_arith.cuh", "points_body.cuh"};
    nvrtcProgram_t prog = nullptr;
    if (g_nvrtc.create(&prog, program.c_str(), "points.cu", 2, hdr_src, hdr_name) == 0) {
      const char *opts[] = {"--gpu-architecture=sm_103a", "--std=c++17", "--fmad=false"};
      const int rc = g_nvrtc.compile(prog, 3, opts);
      if (rc != 0 && getenv("PS_JIT_LOG")) {
        size_t n = 0;
        g_nvrtc.log_size(prog, &n);
        std::string log(n, '\0');
        if (n) g_nvrtc.log(prog, &log[0]);
        fprintf(stderr, "%s\n", log.c_str());
      }
      if (rc == 0) {
        size_t n = 0;
        g_nvrtc.cubin_size(prog, &n);
        std::vector<char> image(n);
        g_nvrtc.cubin(prog, image.data());
        CUmodule mod = nullptr;
        CUfunction f = nullptr;
        if (g_drv.load(&mod, image.data()) == CUDA_SUCCESS) {
          if (g_drv.get(&f, mod, "__ps_points") == CUDA_SUCCESS) fn = f;
          else g_drv.unload(mod);
        }
      }
      g_nvrtc.destroy(&prog);
    }
  }
  PointsJit e;
  e.fn = fn;
  CUfunction f = static_cast<CUfunction>(fn);
  if (fn && (g_drv.set_attr(f, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)smem) !=
                 CUDA_SUCCESS ||
             g_drv.occupancy(&e.occ, f, 32 * (k.warps + 1), smem) != CUDA_SUCCESS))
    e.occ = 0;
  g_points_jit[key] = e;
  *occ = e.occ;
  return fn;
}

cudaError_t jit_launch_raw(void *fn, int grid, dim3 block, size_t smem, bool overlap,
                           cudaStream_t s, void **args) {
  const CUresult r = launch_function(fn, dim3(grid), block, smem, overlap, s, args);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorLaunchFailure;
}

}  // namespace psg
