// Runs the grid walk and the fast triangle test of
// form_factors_b200/csrc/ffb_grid.cuh as plain C++ against the brute-force scan
// (ray_caster/naive_cpu.cpp:65-97): binning, test records, empty-space distances
// and the traversal are the header's own functions, the CUDA names below stand
// in for what the compiler gives device code.  Every cell record the walk reads
// is checked against the table's bounds.  Usage:
//   tracer_check
// Prints the rays and the mismatches; exit status 1 on any.
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_runtime.h>

// ---- stand-ins for device code (the kernels of the header are never run) ----
using std::isfinite;
using std::max;
using std::min;
static dim3 threadIdx, blockIdx, blockDim, gridDim;
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static float __fadd_rd(float a, float b)
{
  volatile float x = a, y = b;
  const int mode = std::fegetround();
  std::fesetround(FE_DOWNWARD);
  volatile float s = x + y;
  std::fesetround(mode);
  return s;
}
template <class To, class From>
static To bits_as(From x)
{
  To y;
  memcpy(&y, &x, sizeof y);
  return y;
}
static inline int __float_as_int(float x) { return bits_as<int>(x); }
static inline uint32_t __float_as_uint(float x) { return bits_as<uint32_t>(x); }
static inline float __int_as_float(int x) { return bits_as<float>(x); }
static inline float __uint_as_float(uint32_t x) { return bits_as<float>(x); }
static uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s)
{
  const uint64_t v = (uint64_t)y << 32 | x;
  uint32_t r = 0;
  for (int k = 0; k < 4; ++k)
    r |= (uint32_t)((v >> (8 * ((s >> (4 * k)) & 7u))) & 0xFFu) << (8 * k);
  return r;
}
static const uint2 *g_table, *g_table_end;
static long g_outside = 0;
static uint2 __ldg(const uint2* p)
{
  if (p >= g_table && p < g_table_end)
    return *p;
  ++g_outside;
  return make_uint2(0x01010101u, 0x81010101u);
}
static float __ldg(const float* p) { return *p; }
static uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static int __clz(unsigned x) { return x ? __builtin_clz(x) : 32; }
template <class T> static T __shfl_xor_sync(unsigned, T v, int) { return v; }
template <class T> static T __shfl_up_sync(unsigned, T v, int) { return v; }
static unsigned __ballot_sync(unsigned, int x) { return x ? 1u : 0u; }
#ifndef __launch_bounds__
#define __launch_bounds__(...)
#endif
static void __syncthreads() {}
static void __syncwarp() {}
template <class T> static T atomicAdd(T* p, T v) { const T o = *p; *p += v; return o; }
template <class T> static T atomicMin(T* p, T v) { const T o = *p; *p = min(o, v); return o; }
template <class T> static T atomicMax(T* p, T v) { const T o = *p; *p = max(o, v); return o; }

// A float's conversion to int as the GPU does it: saturating, not a number to 0.
struct Floor {
  float v;
  explicit operator int() const
  {
    return v != v ? 0 : v >= 2147483648.f ? INT32_MAX : v < -2147483648.f ? INT32_MIN : (int)v;
  }
};
static Floor floor_gpu(float x) { return {std::floor(x)}; }
#define floorf floor_gpu
#include "ffb_grid.cuh"
#undef floorf

using namespace ffb;

namespace {

long g_binned = 0, g_walks = 0, g_rays = 0, g_bad = 0, g_hits = 0;

struct Scene {
  std::vector<float> faces9;
  std::vector<TriRec> tri;
  std::vector<float4> box_lo, box_hi;
  int n = 0;
};

struct Grid {
  GridView view;
  std::vector<uint2> cells;
  std::vector<TestRec> refs;
};

Scene make_scene(const std::vector<float>& faces9)
{
  Scene s;
  s.faces9 = faces9;
  s.n = (int)faces9.size() / 9;
  s.tri.resize(s.n);
  s.box_lo.resize(s.n);
  s.box_hi.resize(s.n);
  std::vector<uint32_t> ord(6);
  blockDim = dim3(1, 1, 1);
  threadIdx = dim3(0, 0, 0);
  for (int f = 0; f < s.n; ++f) {
    blockIdx = dim3(f, 0, 0);
    k_face_prepare(s.faces9.data(), s.n, s.tri.data(), s.box_lo.data(), s.box_hi.data(), ord.data());
  }
  return s;
}

// The grid of ffb_grid_build for nx x ny x nz cells.
Grid make_grid(const Scene& s, int nx, int ny, int nz, bool skip)
{
  float smin[3] = {INFINITY, INFINITY, INFINITY}, smax[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int f = 0; f < s.n; ++f) {
    if (s.box_lo[f].x > s.box_hi[f].x)
      continue;
    const float lo[3] = {s.box_lo[f].x, s.box_lo[f].y, s.box_lo[f].z};
    const float hi[3] = {s.box_hi[f].x, s.box_hi[f].y, s.box_hi[f].z};
    for (int a = 0; a < 3; ++a) {
      smin[a] = min(smin[a], lo[a]);
      smax[a] = max(smax[a], hi[a]);
    }
  }
  float max_ext = 0.f, max_abs = 0.f;
  for (int a = 0; a < 3; ++a) {
    max_ext = max(max_ext, smax[a] - smin[a]);
    max_abs = max(max_abs, max(std::fabs(smin[a]), std::fabs(smax[a])));
  }
  const float margin = max_ext * 0x1p-12f + max_abs * 0x1p-17f + 1e-30f;
  const int dims[3] = {nx, ny, nz};
  float lo[3], hi[3], cell[3];
  TestGeom t{};
  double d2 = 0.0;
  for (int a = 0; a < 3; ++a) {
    lo[a] = smin[a] - 2.f * margin;
    hi[a] = smax[a] + 2.f * margin;
    cell[a] = (float)(((double)hi[a] - (double)lo[a]) / dims[a]);
    while (lo[a] + (float)dims[a] * cell[a] < hi[a])
      cell[a] = std::nextafter(cell[a], INFINITY);
    hi[a] = lo[a] + (float)dims[a] * cell[a];
    t.lo[a] = lo[a];
    t.cs[a] = 1.0 / (double)(1.f / cell[a]);
    const double e = (double)hi[a] - (double)lo[a];
    d2 += e * e;
    t.reach = max(t.reach, max(std::fabs((double)lo[a]), std::fabs((double)hi[a])));
  }
  t.size = std::sqrt(d2);
  Grid G;
  GridView& g = G.view;
  memset(&g, 0, sizeof g);
  const auto corner = [](float x) { return isfinite(x) ? x : 0.f; };
  g.lo = f3(corner(lo[0]), corner(lo[1]), corner(lo[2]));
  g.inv_cs = f3(1.f / cell[0], 1.f / cell[1], 1.f / cell[2]);
  g.nf = f3((float)nx, (float)ny, (float)nz);
  const auto bias = [&](float ics) {
    const float e = 0.25f * margin * ics;
    return e < 0.25f ? e : 0.25f;
  };
  g.eps = f3(bias(g.inv_cs.x), bias(g.inv_cs.y), bias(g.inv_cs.z));
  g.nx = nx;
  g.nxy = nx * ny;
  g.nxm = nx - 1;
  g.nym = (ny - 1) * nx;
  g.nzm = (nz - 1) * nx * ny;
  g.slack = 2.5f * margin;
  g.tie = 3.5f * margin;
  g.near_err = 0.25f * margin;
  g.inv_size = (float)(1.25 / t.size);
  g.tri = s.tri.data();
  BinGeom bg;
  bg.lo = f3(lo[0], lo[1], lo[2]);
  bg.cs = f3(cell[0], cell[1], cell[2]);
  bg.inv_cs = g.inv_cs;
  bg.nx = nx;
  bg.ny = ny;
  bg.nz = nz;
  bg.margin = margin;
  const int n_cells = nx * ny * nz;
  std::vector<std::vector<int>> list((size_t)n_cells);
  for (int f = 0; f < s.n; ++f)
    for_each_cell(bg, s.faces9.data(), f, s.box_lo[f], s.box_hi[f], 0, 1, [&](int c) { list[(size_t)c].push_back(f); });
  // the cells of a face dealt over the lanes of a group: each once
  std::vector<int> seen((size_t)n_cells, 0);
  for (int lanes = 2; lanes <= 32; lanes *= 4)
    for (int f = 0; f < s.n; ++f) {
      for (int lane = 0; lane < lanes; ++lane)
        for_each_cell(bg, s.faces9.data(), f, s.box_lo[f], s.box_hi[f], lane, lanes, [&](int c) { ++seen[(size_t)c]; });
      for_each_cell(bg, s.faces9.data(), f, s.box_lo[f], s.box_hi[f], 0, 1, [&](int c) { --seen[(size_t)c]; });
    }
  for (int n : seen)
    g_binned += n != 0;
  std::vector<uint32_t> start((size_t)n_cells + 1, 0);
  for (int c = 0; c < n_cells; ++c) {
    start[(size_t)c + 1] = start[(size_t)c] + (uint32_t)list[(size_t)c].size();
    for (int f : list[(size_t)c])
      G.refs.push_back(make_testrec(s.tri[f], f, t));
  }
  // empty-space distance of each octant, by its recurrence over the seven
  // neighbours of a cell's corner
  std::vector<uint8_t> dist;
  if (skip) {
    dist.assign((size_t)kOctants * n_cells, 0);
    for (int o = 0; o < kOctants; ++o) {
      const int d[3] = {o & 1 ? -1 : 1, o & 2 ? -1 : 1, o & 4 ? -1 : 1};
      const auto at = [&](int i, int j, int k) -> int {
        if (i < 0 || i >= nx || j < 0 || j >= ny || k < 0 || k >= nz)
          return kEmptyCap;
        return dist[(size_t)o * n_cells + (k * ny + j) * nx + i];
      };
      for (int kk = 0; kk < nz; ++kk)
        for (int jj = 0; jj < ny; ++jj)
          for (int ii = 0; ii < nx; ++ii) {
            const int i = d[0] < 0 ? ii : nx - 1 - ii, j = d[1] < 0 ? jj : ny - 1 - jj, k = d[2] < 0 ? kk : nz - 1 - kk;
            const int c = (k * ny + j) * nx + i;
            int v = 0;
            if (list[(size_t)c].empty()) {
              v = kEmptyCap;
              for (int m = 1; m < 8; ++m)
                v = min(v, at(i + (m & 1 ? d[0] : 0), j + (m & 2 ? d[1] : 0), k + (m & 4 ? d[2] : 0)) + 1);
              v = min(v, kEmptyCap);
            }
            dist[(size_t)o * n_cells + c] = (uint8_t)v;
          }
    }
  }
  const long long pad = cell_pad(nx, ny);
  G.cells.resize((size_t)(n_cells + 2 * pad));
  blockIdx = threadIdx = dim3(0, 0, 0);
  blockDim = gridDim = dim3(1, 1, 1);
  k_cell_rec(start.data(), skip ? dist.data() : nullptr, n_cells, pad, G.cells.data());
  g.cell_rec = G.cells.data() + pad;
  g.ref_rec = G.refs.data();
  return G;
}

int brute(const Scene& s, float3 o, float3 dir)
{
  float best = 3.40282347e+38f;
  int at = -1;
  for (int f = 0; f < s.n; ++f) {
    float3 p;
    if (tri_hit(reinterpret_cast<const float4*>(&s.tri[f]), o, dir, p)) {
      const float d = dist2(p, o);
      if (d < best) {
        best = d;
        at = f;
      }
    }
  }
  return at;
}

// The loop of the trace kernels for one ray.
template <bool kFar>
int walk(const Grid& G, float3 o, float3 dir)
{
  const GridView& g = G.view;
  g_table = G.cells.data();
  g_table_end = g_table + G.cells.size();
  Tracer T;
  float t0;
  uint32_t n = 0, moves = 0, jumps = 0;
  if (!tracer_begin<kFar>(T, g, o, dir, &t0, n))
    return -1;
  for (;;) {
    while (T.i < T.en) {
      if (T.en > G.refs.size()) {
        ++g_outside;
        return -2;
      }
      const int open = tracer_test<kFar, false>(T, g, n);
      if (open >= 0)
        tracer_exact(T, g, open, o, dir, t0);
    }
    if (!tracer_advance(T, g, moves, jumps))
      return T.face;
    if (moves > 1024) {  // at most nx + ny + nz are needed
      printf("endless walk\n");
      exit(1);
    }
  }
}

// One ray given by origin and end point, as casts get it.
void check(const char* what, const Scene& s, const Grid& G, const float* o, const float* e)
{
  const float3 org = f3(o[0], o[1], o[2]), dir = sub3(f3(e[0], e[1], e[2]), org);
  const int want = brute(s, org, dir);
  const int got[2] = {walk<true>(G, org, dir), walk<false>(G, org, dir)};
  ++g_rays;
  g_hits += want >= 0;
  for (int k = 0; k < 2; ++k)
    if (got[k] != want) {
      if (g_bad++ < 12)
        printf("%s: o (%a %a %a) e (%a %a %a): got %d want %d (far %d, grid %g x %g x %g)\n", what, o[0], o[1], o[2],
               e[0], e[1], e[2], got[k], want, k == 0, G.view.nf.x, G.view.nf.y, G.view.nf.z);
    }
}

std::vector<float> closed_box(float size, int cells, const float* at)
{
  std::vector<float> f;
  for (int a = 0; a < 3; ++a)
    for (int side = 0; side < 2; ++side)
      for (int i = 0; i < cells; ++i)
        for (int j = 0; j < cells; ++j)
          for (int h = 0; h < 2; ++h) {
            const float q[3][2] = {{(float)i, (float)j}, {(float)(i + 1), (float)(j + (h ? 1 : 0))},
                                   {(float)(i + (h ? 0 : 1)), (float)(j + 1)}};
            for (int v = 0; v < 3; ++v) {
              float p[3];
              p[a] = side ? size : 0.f;
              p[(a + 1) % 3] = q[v][0] * (size / (float)cells);
              p[(a + 2) % 3] = q[v][1] * (size / (float)cells);
              for (int b = 0; b < 3; ++b)
                f.push_back(at[b] + p[b]);
            }
          }
  return f;
}

// Rays whose direction has components far below the others: from 2^-60 to the
// smallest float, on each axis and sign, one or two of them small, aimed from
// inside the box and from in front of it.
void small_components()
{
  std::mt19937 rng(11);
  std::uniform_real_distribution<float> u(0.05f, 0.95f);
  for (const float scale : {0.02f, 1.f, 1000.f}) {  // below 0.01 every face is degenerate (dot(n, n) < 1e-8)
    const float low[3] = {-0.53f * scale, -0.41f * scale, -0.47f * scale};
    std::vector<float> faces = closed_box(scale, scale < 1.f ? 1 : 3, low);
    const auto inside = [&](int a) { return low[a] + u(rng) * scale; };
    for (int k = 0; k < 60; ++k) {  // occluders
      const float c[3] = {inside(0), inside(1), inside(2)};
      for (int v = 0; v < 3; ++v)
        for (int a = 0; a < 3; ++a)
          faces.push_back(c[a] + (u(rng) - 0.5f) * 0.2f * scale);
    }
    const Scene s = make_scene(faces);
    const int dims[][3] = {{1, 1, 1}, {24, 24, 24}, {256, 5, 3}, {2, 90, 7}};
    for (const auto& d : dims)
      for (const bool skip : {false, true}) {
        const Grid G = make_grid(s, d[0], d[1], d[2], skip);
        for (int axis = 0; axis < 3; ++axis)
          for (int sign = 0; sign < 2; ++sign)
            for (int p = 60; p <= 149; ++p)
              for (int kind = 0; kind < 4; ++kind) {
                // the small components need origins of 0 to survive the
                // subtraction of the end point
                float o[3] = {0.f, 0.f, 0.f}, e[3] = {0.f, 0.f, 0.f};
                const int main = (axis + 1) % 3, third = (axis + 2) % 3;
                const float tiny = std::ldexp(sign ? -1.f : 1.f, -p);
                e[axis] = tiny;
                if (kind == 1)
                  e[third] = tiny;
                else
                  o[third] = e[third] = inside(third);
                if (kind == 2)
                  e[third] += (u(rng) - 0.5f) * scale;
                o[main] = kind == 3 ? -2.f * scale : inside(main);
                e[main] = o[main] + (kind == 3 || (p & 1) ? 1.f : -1.f) * (p % 3 ? scale : 1.f);
                check("small components", s, G, o, e);
              }
      }
  }
}

// Rays given by end points from half a scene to a billionth of it away, whose
// error bounds widen with the inverse of the length: from inside and outside, at
// faces, vertices and along edges.
void short_rays()
{
  std::mt19937 rng(13);
  std::uniform_real_distribution<float> u(0.05f, 0.95f);
  std::normal_distribution<float> gauss;
  for (const float scale : {0.2f, 1.f, 300.f}) {
    const float low[3] = {-0.53f * scale, -0.41f * scale, -0.47f * scale};
    std::vector<float> faces = closed_box(scale, scale < 1.f ? 2 : 5, low);
    for (int k = 0; k < 150; ++k) {
      float c[3];
      for (int a = 0; a < 3; ++a)
        c[a] = low[a] + u(rng) * scale;
      const float thin = k % 3 ? 0.25f : 0.01f;  // every third a needle
      for (int v = 0; v < 3; ++v)
        for (int a = 0; a < 3; ++a)
          faces.push_back(c[a] + (u(rng) - 0.5f) * scale * (v == 2 ? 0.25f : thin));
    }
    const Scene s = make_scene(faces);
    const int dims[][3] = {{1, 1, 1}, {20, 20, 20}, {256, 5, 3}};
    for (const auto& d : dims) {
      const Grid G = make_grid(s, d[0], d[1], d[2], d[0] > 1);
      for (int n = 0; n < 12000; ++n) {
        float o[3], e[3], dir[3], len = 0.f;
        const float* f = s.faces9.data() + 9 * (rng() % (unsigned)s.n);
        for (int a = 0; a < 3; ++a) {
          o[a] = low[a] + u(rng) * scale + (n % 7 == 0 ? 2.f * scale * gauss(rng) : 0.f);
          const float at = n % 4 == 0 ? f[a] : n % 4 == 1 ? 0.5f * (f[a] + f[3 + a]) : n % 4 == 2
                           ? (f[a] + f[3 + a] + f[6 + a]) / 3.f : o[a] + gauss(rng);
          dir[a] = at - o[a];
          if (n % 11 == 0) {  // along an edge
            o[a] = 0.5f * (f[a] + f[3 + a]);
            dir[a] = f[3 + a] - f[a];
          }
          len += dir[a] * dir[a];
        }
        const float k = scale * std::ldexp(1.f, -1 - (int)(rng() % 30)) / std::sqrt(len);
        if (n % 5 == 0)  // an origin of 0 keeps the direction's bits
          o[0] = o[1] = o[2] = 0.f;
        for (int a = 0; a < 3; ++a)
          e[a] = o[a] + k * dir[a];
        check("short rays", s, G, o, e);
      }
    }
  }
}

// Scenes from the smallest to the largest floats, and two whose extent overflows
// in some axes or all: no read outside the table and an end to every walk, whatever
// the reference's own arithmetic makes of them.
void extreme_scales()
{
  std::mt19937 rng(12);
  std::uniform_real_distribution<float> u(0.05f, 0.95f);
  std::vector<int> exponents;
  for (int e2 = -140; e2 <= 126; e2 += 7)
    exponents.push_back(e2);
  exponents.insert(exponents.end(), {127, 1000, 1001});
  for (const int e2 : exponents) {
    const float scale = e2 < 1000 ? std::ldexp(1.f, e2) : 1.f;
    const float low[3] = {-0.53f * scale, -0.41f * scale, -0.47f * scale};
    std::vector<float> faces = closed_box(scale, 2, low);
    if (e2 >= 1000)  // a box beside a face too wide for floats
      for (const float x : {-3e38f, 1.f, 2.f, 3e38f, 2.f, 1.f, 0.f, 3e38f, 3.f})
        faces.push_back(e2 == 1000 ? x : x > 1e30f || x < -1e30f ? x : -3e38f);
    const Scene s = make_scene(faces);
    const int dims[][3] = {{1, 1, 1}, {16, 16, 16}, {8, 8, 8}, {256, 2, 3}};
    for (const auto& d : dims) {
      const Grid G = make_grid(s, d[0], d[1], d[2], true);
      for (int n = 0; n < 1500; ++n) {
        float o[3], dir[3];
        for (int a = 0; a < 3; ++a) {
          o[a] = low[a] + u(rng) * scale * (n % 5 == 0 ? 3.f : 1.f);
          dir[a] = std::ldexp(u(rng) - 0.5f, n % 3 == 0 ? (int)(rng() % 150) - 149 : 0);
        }
        const float k = n % 2 ? scale : 1.f;
        const float3 org = f3(o[0], o[1], o[2]), v = f3(dir[0] * k, dir[1] * k, dir[2] * k);
        walk<true>(G, org, v);
        walk<false>(G, org, v);
        ++g_walks;
        if (e2 >= 1000) {
          const float e[3] = {o[0] + dir[0], o[1] + dir[1], o[2] + dir[2]};
          check("overflowing extent", s, G, o, e);
        }
      }
    }
  }
}

}  // namespace

int main()
{
  small_components();
  short_rays();
  extreme_scales();
  printf("cells binned otherwise %ld, walks %ld, rays %ld, hits %ld, reads outside the table %ld, mismatches %ld\n",
         g_binned, g_walks, g_rays, g_hits, g_outside, g_bad);
  return g_binned || g_bad || g_outside || g_hits * 2 < g_rays;
}
