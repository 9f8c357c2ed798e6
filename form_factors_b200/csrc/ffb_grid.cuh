// ffb_grid.cuh -- uniform 3-D grid over the scene: device build (counting
// sort of triangle references into cells) and 3-D DDA nearest-hit traversal.
//
// The reference accelerates the same query with a 2-D grid over X/Y and
// infinite Z columns (math/grid.cpp, ray_caster/zgrid_cpu.cpp:57-132).  This
// grid is a different structure with the same answer: hit index and hit point
// equal to the brute-force definition (ray_caster/naive_cpu.cpp:65-97) for
// every ray.  Four rules make that hold:
//  1. Binning is conservative.  A triangle goes into every cell that its
//     bounding box, grown by a margin, overlaps and whose box its plane (grown
//     by the same margin) crosses.  The margin covers the rounding of a
//     computed hit point, including the extra error of sliver triangles.
//  2. A reference is first tested with fused multiply-adds on precomputed rows
//     (tracer_test).  The test knows the bounds of its own error and of the
//     reference's float test, and decides only what lies outside both; the
//     rest takes the reference's test operation by operation.
//  3. Hits are merged as a lexicographic minimum of (squared distance, index),
//     which equals a strict '<' scan in index order.  Two hits nearer to each
//     other than their errors are compared by the reference's own values.
//  4. Traversal stops only when the best distance is below the distance at
//     which the ray leaves the current cell (or the empty cube it jumps
//     across) by more than the margins; nothing in an unvisited cell can then
//     compute a smaller one.
#pragma once

#include "ffb_device.cuh"

namespace ffb {

// Conservative test record of a face in the grid's coordinates (cells from
// the box's low corner): the plane n.x = c, scaled so that 1 / |n.d| is the
// bound on the error of the barycentric coordinates for a ray of unit (world)
// direction d, and the two barycentric coordinates as affine functions of the
// point.  h turns that bound into the bound on the error of the distance.
// 64 bytes, read as two 256-bit loads.
struct alignas(32) TestRec {
  float nx, ny, nz, c;
  float sx, sy, sz, s0;
  float tx, ty, tz, t0;
  int32_t face;
  float h;
  float pad[2];
};

// The order of the members decides which constants the compiler keeps in
// registers and so what the trace kernels spill: in this one of 15 tried the
// shapes without direction order spill nothing with the warp histogram and 4
// bytes a thread without it, as in every order; in the others up to 44 bytes (28 in
// shape 12 cost 6 % on 19 M rays between 1104 meshes).
struct GridView {
  const uint2* __restrict__ cell_rec;       // per cell: {start, end} of its references, or octant distances
  float3 lo;            // grid box, low corner
  float near_err;       // margin / 4: the largest distance error of a hit accepted without the exact test
  float tie;            // slack + margin
  float inv_size;       // 1.25 / box diagonal
  const TriRec* __restrict__ tri;           // exact triangle record per face
  float3 eps;           // landing bias, cells: a quarter of the margin (at most a quarter of a cell)
  int nx, nxy;          // cell strides along y and z
  const TestRec* __restrict__ ref_rec;      // test record per reference (a copy of its face's)
  int nxm, nym, nzm;    // index offset of the last cell per axis: (n - 1) * stride
  float3 nf;            // cells per axis
  float3 inv_cs;        // 1 / cell size
  float slack;          // 2.5 margins, world units
};

// Packed cell record: an occupied cell holds {first reference, end}; an
// empty one {0, kCellEmpty | d} with d its empty-space distance (1 when the
// grid has no distance map).  One 8-byte load replaces the distance byte and
// the two offsets.
constexpr uint32_t kCellEmpty = 0x80000000u;

// Ordered-integer image of a float for atomicMin/atomicMax reductions.
__device__ __forceinline__ uint32_t f2ord(float f)
{
  uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__host__ __device__ inline float ord2f(uint32_t u)
{
  uint32_t b = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

__device__ __forceinline__ bool finite3(float3 p)
{
  return isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
}

// ---------------------------------------------------------------------------
// Per-face preparation: triangle record, binning box and the scene box.
// A face that can never be hit (degenerate: n = 0; or non-finite vertices,
// whose test always yields NaN) is marked with an empty box and not binned.
// ---------------------------------------------------------------------------
__global__ void k_face_prepare(const float* __restrict__ faces9, int n_faces, TriRec* __restrict__ tri,
                               float4* __restrict__ box_lo, float4* __restrict__ box_hi,
                               uint32_t* __restrict__ scene_ord /* 6: min xyz, max xyz (ordered) */)
{
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  float3 mn = f3(INFINITY, INFINITY, INFINITY), mx = f3(-INFINITY, -INFINITY, -INFINITY);
  if (f < n_faces) {
    const float* p = faces9 + 9 * (size_t)f;
    float3 p0 = f3(p[0], p[1], p[2]), p1 = f3(p[3], p[4], p[5]), p2 = f3(p[6], p[7], p[8]);
    TriRec t = make_trirec(p0, p1, p2);
    tri[f] = t;
    bool live = finite3(p0) && finite3(p1) && finite3(p2) && !(t.q1.x == 0.f && t.q1.y == 0.f && t.q1.z == 0.f);
    // Sliver factor kappa = uu*vv/|D| = 1/sin^2(angle at p0): bounds how far
    // a computed hit point can stray from the triangle in its plane.
    float kappa = 0.f;
    float diam = 0.f;
    if (live) {
      mn = f3(fminf(fminf(p0.x, p1.x), p2.x), fminf(fminf(p0.y, p1.y), p2.y), fminf(fminf(p0.z, p1.z), p2.z));
      mx = f3(fmaxf(fmaxf(p0.x, p1.x), p2.x), fmaxf(fmaxf(p0.y, p1.y), p2.y), fmaxf(fmaxf(p0.z, p1.z), p2.z));
      float3 w = sub3(p2, p1);
      diam = sqrtf(fmaxf(fmaxf(t.q0.w, t.q2.w), dot3(w, w)));
      float D = t.q3.w;
      kappa = (D < 0.f) ? (t.q0.w * t.q2.w) / (-D) : INFINITY;
      if (!(kappa < 1e5f))
        kappa = -1.f;  // ill-conditioned: widen by the full diameter
    }
    // .w carries the face's own extra margin (world units) beyond the grid
    // margin; a negative box (lo > hi) marks a face that is never binned.
    float extra = kappa < 0.f ? diam : 16.f * 1.1920929e-07f * kappa * diam;
    if (live) {
      box_lo[f] = make_float4(mn.x, mn.y, mn.z, extra);
      box_hi[f] = make_float4(mx.x, mx.y, mx.z, 0.f);
    } else {
      box_lo[f] = make_float4(1.f, 1.f, 1.f, 0.f);
      box_hi[f] = make_float4(-1.f, -1.f, -1.f, 0.f);
    }
  }
  // block reduction of the scene box (dead faces contribute +-inf)
  __shared__ float red[6][32];
  float v[6] = {mn.x, mn.y, mn.z, -mx.x, -mx.y, -mx.z};
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    float x = v[k];
    for (int o = 16; o > 0; o >>= 1)
      x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
    if ((threadIdx.x & 31) == 0)
      red[k][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      float x = threadIdx.x < nw ? red[k][threadIdx.x] : INFINITY;
      for (int o = 16; o > 0; o >>= 1)
        x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
      if (threadIdx.x == 0 && x < INFINITY) {
        if (k < 3)
          atomicMin(scene_ord + k, f2ord(x));
        else
          atomicMax(scene_ord + k, f2ord(-x));
      }
    }
  }
}

// Emission frame per face (see emit_ray): p0, e1, e2 and the rotation of +z
// towards the face normal, normalised unless ref_normal is set.
__global__ void k_face_frames(const float* __restrict__ faces9, int n_faces, int ref_normal,
                              float* __restrict__ frames /* 20 per face */)
{
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces)
    return;
  const float* p = faces9 + 9 * (size_t)f;
  float3 p0 = f3(p[0], p[1], p[2]), p1 = f3(p[3], p[4], p[5]), p2 = f3(p[6], p[7], p[8]);
  float3 e1 = sub3(p1, p0), e2 = sub3(p2, p0);
  float3 n = cross3(e1, e2);
  if (!ref_normal) {
    float len = sqrtf(dot3(n, n));
    if (len > 0.f)
      n = f3(n.x / len, n.y / len, n.z / len);
  }
  float* out = frames + 20 * (size_t)f;
  out[0] = p0.x; out[1] = p0.y; out[2] = p0.z;
  out[3] = e1.x; out[4] = e1.y; out[5] = e1.z;
  out[6] = e2.x; out[7] = e2.y; out[8] = e2.z;
  rotate_towards(f3(0.f, 0.f, 1.f), n, out + 9);
  out[18] = 0.f;
  out[19] = 0.f;
}

struct BinGeom {
  float3 lo, cs, inv_cs;
  int nx, ny, nz;
  float margin;
};

// Calls fn(cell) for every cell a face is binned into.  The cells of its box
// are dealt over the `lanes` lanes of a group, `lane` among them.
template <class Fn>
__device__ __forceinline__ void for_each_cell(const BinGeom& g, const float* __restrict__ faces9, int f, float4 blo,
                                              float4 bhi, int lane, int lanes, Fn fn)
{
  if (blo.x > bhi.x)
    return;
  float m = g.margin + blo.w;
  int i0 = max(0, (int)floorf((blo.x - m - g.lo.x) * g.inv_cs.x));
  int j0 = max(0, (int)floorf((blo.y - m - g.lo.y) * g.inv_cs.y));
  int k0 = max(0, (int)floorf((blo.z - m - g.lo.z) * g.inv_cs.z));
  int i1 = min(g.nx - 1, (int)floorf((bhi.x + m - g.lo.x) * g.inv_cs.x));
  int j1 = min(g.ny - 1, (int)floorf((bhi.y + m - g.lo.y) * g.inv_cs.y));
  int k1 = min(g.nz - 1, (int)floorf((bhi.z + m - g.lo.z) * g.inv_cs.z));
  const float* p = faces9 + 9 * (size_t)f;
  float3 p0 = f3(p[0], p[1], p[2]);
  float3 n = cross3(sub3(f3(p[3], p[4], p[5]), p0), sub3(f3(p[6], p[7], p[8]), p0));
  float nl = sqrtf(dot3(n, n));
  n = f3(n.x / nl, n.y / nl, n.z / nl);
  // plane-box test: |n.(c - p0)| <= sum |n_a| h_a + margin, checked with a
  // little extra slack for the rounding of this float test itself
  float3 h = mul3(g.cs, 0.5f);
  float reach = fabsf(n.x) * h.x + fabsf(n.y) * h.y + fabsf(n.z) * h.z + m * 1.5f;
  bool flat = (i1 - i0 + 1) * (j1 - j0 + 1) * (k1 - k0 + 1) <= 2;
  // Edge axes of the separating-axis test: edge x unit axis, for the three
  // edges.  Each axis is an exact float vector (a permutation of an edge's
  // components), so only the projections round.  The cell grown by the
  // margin on every axis, as the box range above grows it, reaches
  // r = sum (h_a + m) |A_a| along axis A; a further 0.5 m per axis covers
  // the rounding of the projections (coordinates relative to p0).  An axis
  // that separates the triangle from the grown cell proves that no hit point
  // computed on the triangle can land in the cell.
  const float3 ed[3] = {sub3(f3(p[3], p[4], p[5]), p0), sub3(f3(p[6], p[7], p[8]), f3(p[3], p[4], p[5])),
                        sub3(p0, f3(p[6], p[7], p[8]))};
  const float3 q1 = ed[0], q2 = sub3(f3(p[6], p[7], p[8]), p0);  // vertices relative to p0 (q0 = 0)
  const float3 hm = f3(h.x + 1.5f * m, h.y + 1.5f * m, h.z + 1.5f * m);
  float ax_lo[9], ax_hi[9], ax_r[9];
#pragma unroll
  for (int e = 0; e < 3; ++e) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float3 A = a == 0 ? f3(0.f, ed[e].z, -ed[e].y) : (a == 1 ? f3(-ed[e].z, 0.f, ed[e].x)
                                                                     : f3(ed[e].y, -ed[e].x, 0.f));
      const float v1 = dot3(q1, A), v2 = dot3(q2, A);
      ax_lo[3 * e + a] = fminf(0.f, fminf(v1, v2));
      ax_hi[3 * e + a] = fmaxf(0.f, fmaxf(v1, v2));
      ax_r[3 * e + a] = fabsf(A.x) * hm.x + fabsf(A.y) * hm.y + fabsf(A.z) * hm.z;
    }
  }
  const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, count = ni * nj * (k1 - k0 + 1);
  if (ni <= 0 || nj <= 0)
    return;
  const int row = lane / ni;
  int i = i0 + lane - row * ni, j = j0 + row % nj, k = k0 + row / nj;
  const auto step = [&] {  // `lanes` cells further; carries instead of divisions
    for (i += lanes; i > i1; i -= ni)
      if (++j > j1) {
        j = j0;
        ++k;
      }
  };
  for (int at = lane; at < count; at += lanes, step()) {
    if (!flat) {
      float3 c = f3(g.lo.x + ((float)i + 0.5f) * g.cs.x, g.lo.y + ((float)j + 0.5f) * g.cs.y,
                    g.lo.z + ((float)k + 0.5f) * g.cs.z);
      const float3 dc = sub3(c, p0);
      float d = fabsf(dot3(n, dc));
      if (d > reach)
        continue;
      bool sep = false;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float3 A = a == 0 ? f3(0.f, ed[e].z, -ed[e].y) : (a == 1 ? f3(-ed[e].z, 0.f, ed[e].x)
                                                                         : f3(ed[e].y, -ed[e].x, 0.f));
          const float pc = dot3(dc, A);
          sep |= (ax_lo[3 * e + a] > pc + ax_r[3 * e + a]) | (ax_hi[3 * e + a] < pc - ax_r[3 * e + a]);
        }
      }
      if (sep)
        continue;
    }
    fn((k * g.ny + j) * g.nx + i);
  }
}

// Lanes per face (a power of two up to 32) of the binning kernels: the boxes
// of a face's cells are walked by as many lanes as keep the GPU busy.
struct FaceLane {
  int face, lane, lanes;
};
__device__ __forceinline__ FaceLane face_lane(int lanes_log2)
{
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  return FaceLane{(int)(t >> lanes_log2), (int)(t & ((1 << lanes_log2) - 1)), 1 << lanes_log2};
}

__global__ void k_grid_count(BinGeom g, const float* __restrict__ faces9, const float4* __restrict__ box_lo,
                             const float4* __restrict__ box_hi, int n_faces, int lanes_log2,
                             uint32_t* __restrict__ cell_count)
{
  const FaceLane l = face_lane(lanes_log2);
  const int f = l.face;
  if (f >= n_faces)
    return;
  for_each_cell(g, faces9, f, box_lo[f], box_hi[f], l.lane, l.lanes, [&](int c) { atomicAdd(cell_count + c, 1u); });
}

__global__ void k_grid_fill(BinGeom g, const float* __restrict__ faces9, const float4* __restrict__ box_lo,
                            const float4* __restrict__ box_hi, int n_faces, int lanes_log2,
                            const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ cell_fill,
                            int32_t* __restrict__ ref_tri)
{
  const FaceLane l = face_lane(lanes_log2);
  const int f = l.face;
  if (f >= n_faces)
    return;
  for_each_cell(g, faces9, f, box_lo[f], box_hi[f], l.lane, l.lanes, [&](int c) {
    uint32_t pos = atomicAdd(cell_fill + c, 1u);
    ref_tri[cell_start[c] + pos] = f;
  });
}

// Sorts each cell's references by triangle index (insertion sort, one thread
// per cell): the grid is then a deterministic function of the scene.
__global__ void k_cell_sort(const uint32_t* __restrict__ cell_start, int n_cells, int32_t* __restrict__ ref_tri)
{
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cells)
    return;
  uint32_t b = cell_start[c], e = cell_start[c + 1];
  for (uint32_t i = b + 1; i < e; ++i) {
    int32_t x = ref_tri[i];
    uint32_t j = i;
    while (j > b && ref_tri[j - 1] > x) {
      ref_tri[j] = ref_tri[j - 1];
      --j;
    }
    ref_tri[j] = x;
  }
}

// Geometry the test records are computed from: the grid's coordinates and the
// sizes the error bounds grow with.
struct TestGeom {
  double lo[3], cs[3];  // box corner and cell size (1 / the float inverse the rays use)
  double size;          // box diagonal
  double reach;         // largest coordinate magnitude of the box
};

// Test record of face f (TestRec).  The exact test (tri_hit_regs) evaluates,
// in float, the plane parameter r = n.(p0 - o) / n.dir and the barycentric
// coordinates s, t of o + r dir with the record's n, u, v, uu, uv, vv, D.  The
// rows here are the same functions of the same float constants, formed in
// double: the ideal values both evaluations approximate.
//
// First-order forward errors, with e = 2^-24, L the box diagonal (no origin,
// vertex or hit is further apart), M the largest coordinate and cos the
// cosine between ray and normal:
//   exact test: plane parameter, as a distance: 4eL/cos (numerator) +
//     3eL/cos (denominator) + eL; hit point: that + e(2L + M); s and t:
//     kappa (2 x the point's error + 10eL), kappa = 1 / (shorter of |u|, |v|
//     * sin^2 of their angle) = kappa e (30L + 2M) / cos;
//   fast test: grid coordinates 2eL, direction 2eL, row rounding and three
//     fused operations per product 10eL, reciprocal and product 3eL: distance
//     19eL / cos, s and t kappa e 32L / cos.
// Twice the sum for s + t is kappa e (124L + 4M) / cos; rays moved to the box
// add 2e(M + ..) to the point.  K below rounds it up, and is at least the
// value that makes the exact test's |n.dir| >= 1e-8 certain for an accepted
// hit (|dir| >= 1/16).  The distance error is e(48L + 2M) / cos.
__device__ inline TestRec make_testrec(const TriRec& r, int face, const TestGeom& g)
{
  const double u2 = 1.0 / 16777216.0;
  const double n[3] = {r.q1.x, r.q1.y, r.q1.z}, p0[3] = {r.q0.x, r.q0.y, r.q0.z};
  const double u[3] = {r.q2.x, r.q2.y, r.q2.z}, v[3] = {r.q3.x, r.q3.y, r.q3.z};
  const double uu = r.q0.w, uv = r.q1.w, vv = r.q2.w, D = r.q3.w;
  const double nl = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  const double kappa = uu * vv / (fabs(D) * sqrt(fmin(uu, vv)));
  const double K = fmax(1.05 * u2 * kappa * (128.0 * g.size + 8.0 * g.reach), 1.6e-7 / nl);
  const double E0 = 1.05 * u2 * (48.0 * g.size + 2.0 * g.reach);
  double c = 0, s0 = 0, t0 = 0, N[3], S[3], T[3];
  for (int a = 0; a < 3; ++a) {
    const double q = p0[a] - g.lo[a];
    const double sa = (uv * v[a] - vv * u[a]) / D, ta = (uv * u[a] - uu * v[a]) / D;
    const double na = n[a] / (nl * K);
    c += na * q;
    s0 -= sa * q;
    t0 -= ta * q;
    N[a] = na * g.cs[a];
    S[a] = sa * g.cs[a];
    T[a] = ta * g.cs[a];
  }
  TestRec o;
  o.nx = (float)N[0]; o.ny = (float)N[1]; o.nz = (float)N[2]; o.c = (float)c;
  o.sx = (float)S[0]; o.sy = (float)S[1]; o.sz = (float)S[2]; o.s0 = (float)s0;
  o.tx = (float)T[0]; o.ty = (float)T[1]; o.tz = (float)T[2]; o.t0 = (float)t0;
  o.face = face;
  o.h = (float)(E0 / K);
  o.pad[0] = o.pad[1] = 0.f;
  // Outside the range the bounds are derived for (or not finite): a NaN plane
  // sends every ray to the exact test.
  const float sum = fabsf(o.nx) + fabsf(o.ny) + fabsf(o.nz) + fabsf(o.sx) + fabsf(o.sy) + fabsf(o.sz) + fabsf(o.tx) +
                    fabsf(o.ty) + fabsf(o.tz) + fabsf(o.c) + fabsf(o.s0) + fabsf(o.t0) + o.h;
  const bool sane = D < 0.0 && K < 1.0 && nl < 1e15 && uu < 1e15 && vv < 1e15 && g.size < 1e12 && g.reach < 1e12 &&
                    isfinite(sum);
  if (!sane)
    o.c = __int_as_float(0x7FC00000);
  return o;
}

// Counts the faces with a non-empty binning box (the grid's live faces): one
// atomic per warp; and writes the live faces' test records.
__global__ void k_face_test(const float4* __restrict__ box_lo, const float4* __restrict__ box_hi,
                            const TriRec* __restrict__ tri, int n_faces, const __grid_constant__ TestGeom geom,
                            TestRec* __restrict__ rec, uint32_t* __restrict__ live)
{
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = f < n_faces && box_lo[f].x <= box_hi[f].x;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, ok);
  if ((threadIdx.x & 31) == 0 && m)
    atomicAdd(live, (uint32_t)__popc(m));
  if (ok)
    rec[f] = make_testrec(tri[f], f, geom);
}

// Per-reference copy of the test records: a cell's candidates are contiguous
// and a test needs no index load before its record.  Four threads per record.
__global__ void k_ref_gather(const int32_t* __restrict__ ref_tri, uint32_t n_refs, const TestRec* __restrict__ rec,
                             TestRec* __restrict__ ref_rec)
{
  const uint4* src = reinterpret_cast<const uint4*>(rec);
  uint4* dst = reinterpret_cast<uint4*>(ref_rec);
  const unsigned long long n = 4ull * n_refs;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x)
    dst[i] = src[4 * (size_t)ref_tri[i >> 2] + (i & 3)];
}

// ---------------------------------------------------------------------------
// Exclusive scan of uint32 counts (n + 1 outputs, out[n] = total) in three
// passes: per-block sums, a single-block scan of the sums, per-block scan.
// ---------------------------------------------------------------------------
constexpr int kScanBlock = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t x, uint32_t* total)
{
  __shared__ uint32_t warp_sums[kScanBlock / 32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t v = x;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o)
      v += y;
  }
  if (lane == 31)
    warp_sums[w] = v;
  __syncthreads();
  if (w == 0) {
    uint32_t s = lane < kScanBlock / 32 ? warp_sums[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o)
        s += y;
    }
    if (lane < kScanBlock / 32)
      warp_sums[lane] = s;
  }
  __syncthreads();
  uint32_t before = (w > 0 ? warp_sums[w - 1] : 0u) + v - x;
  *total = warp_sums[kScanBlock / 32 - 1];
  __syncthreads();
  return before;
}

__global__ void k_scan_reduce(const uint32_t* __restrict__ in, int n, uint32_t* __restrict__ block_sums)
{
  size_t base = (size_t)blockIdx.x * kScanTile;
  uint32_t s = 0;
  for (int k = 0; k < kScanItems; ++k) {
    size_t i = base + (size_t)k * kScanBlock + threadIdx.x;
    if (i < (size_t)n)
      s += in[i];
  }
  uint32_t total;
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0)
    block_sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(uint32_t* __restrict__ block_sums, int n_blocks)
{
  // one block; exclusive scan in place, looping over tiles of kScanBlock
  uint32_t carry = 0;
  for (int base = 0; base < n_blocks; base += kScanBlock) {
    int i = base + threadIdx.x;
    uint32_t x = i < n_blocks ? block_sums[i] : 0u;
    uint32_t total;
    uint32_t ex = block_exclusive_scan(x, &total);
    if (i < n_blocks)
      block_sums[i] = carry + ex;
    carry += total;
  }
}

__global__ void k_scan_apply(const uint32_t* __restrict__ in, int n, const uint32_t* __restrict__ block_offsets,
                             uint32_t* __restrict__ out)
{
  __shared__ uint32_t tile[kScanTile];
  size_t base = (size_t)blockIdx.x * kScanTile;
  for (int k = 0; k < kScanItems; ++k) {
    size_t i = base + (size_t)k * kScanBlock + threadIdx.x;
    tile[k * kScanBlock + threadIdx.x] = i < (size_t)n ? in[i] : 0u;
  }
  __syncthreads();
  // each thread owns kScanItems consecutive items
  uint32_t local[kScanItems];
  uint32_t s = 0;
  for (int k = 0; k < kScanItems; ++k) {
    local[k] = tile[threadIdx.x * kScanItems + k];
    s += local[k];
  }
  uint32_t total;
  uint32_t ex = block_exclusive_scan(s, &total) + block_offsets[blockIdx.x];
  for (int k = 0; k < kScanItems; ++k) {
    size_t i = base + (size_t)threadIdx.x * kScanItems + k;
    if (i < (size_t)n)
      out[i] = ex;
    ex += local[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanBlock - 1)
    out[n] = ex;  // grand total: the last thread's running sum covers the tail
}

// ---------------------------------------------------------------------------
// Empty-space distance per octant.  For each empty cell and each of the 8
// octants of ray directions, the largest k such that the cube of k x k x k
// cells with the cell at its corner, extending from it in the octant's
// directions, holds no reference: the L-infinity distance to the nearest
// occupied cell lying in that octant of the cell.  A ray whose direction
// lies in the octant leaves the cube only through its far faces, so it jumps
// to them (tracer_advance); occupied cells behind the ray do not shorten the
// jump.  The transform is separable: pass a computes, along axis a and in
// each direction, new[i] = min_{r >= 0} max(r, old[i + r*s]), starting from
// 0 (occupied) / kEmptyCap (empty), in one scan per line.  Octant o has bit a
// set when it points down axis a.  A saturated value under-states the distance, which only
// shortens a jump.
// ---------------------------------------------------------------------------
#ifndef FFB_EMPTY_CAP
#define FFB_EMPTY_CAP 127
#endif
constexpr int kEmptyCap = FFB_EMPTY_CAP;  // at most 127: 7 bits per octant in the cell record
static_assert(kEmptyCap >= 1 && kEmptyCap <= 127, "octant distances are 7-bit fields");
constexpr int kOctants = 8;
constexpr int kMaxDim = 256;

// First pass, along x: both directions of every cell from the occupancy
// itself, slot 0 the positive and slot 1 the negative one (slots are n_cells
// bytes apart).  One warp per line of cells: a ballot per 32 cells, then the
// next set bit ahead and behind.
constexpr int kEmptyThreads = 128;
__global__ void __launch_bounds__(kEmptyThreads) k_empty_x(const uint32_t* __restrict__ cell_start, long long n_cells,
                                                           int nx, int n_lines, uint8_t* __restrict__ d)
{
  constexpr int kWords = kMaxDim / 32;
  __shared__ uint32_t s_occ[kEmptyThreads / 32][kWords];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* occ = s_occ[warp];
  const int line = blockIdx.x * (kEmptyThreads / 32) + warp;
  if (line >= n_lines)
    return;
  const uint32_t* start = cell_start + (size_t)line * nx;
  const int words = (nx + 31) >> 5;
  for (int w = 0; w < words; ++w) {
    const int i = 32 * w + lane;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, i < nx && start[i + 1] > start[i]);
    if (lane == 0)
      occ[w] = m;
  }
  __syncwarp();
  for (int w = 0; w < words; ++w) {
    const int i = 32 * w + lane;
    if (i >= nx)
      continue;
    int ahead = kEmptyCap, behind = kEmptyCap;
    uint32_t m = occ[w] >> lane;
    for (int v = w, base = 0;;) {
      if (m) {
        ahead = min(kEmptyCap, base + __ffs(m) - 1);
        break;
      }
      base = 32 * (++v) - i;
      if (v == words || base >= kEmptyCap)
        break;
      m = occ[v];
    }
    m = occ[w] << (31 - lane);
    for (int v = w, base = 0;;) {
      if (m) {
        behind = min(kEmptyCap, base + __clz(m));
        break;
      }
      base = i - (32 * v - 1);
      if (--v < 0 || base >= kEmptyCap)
        break;
      m = occ[v];
    }
    d[(size_t)line * nx + i] = (uint8_t)ahead;
    d[(size_t)n_cells + (size_t)line * nx + i] = (uint8_t)behind;
  }
}

// The passes along y (axis 1) and z (axis 2): octant slot blockIdx.y (< 2^axis,
// the octants of the axes before) holds the input; the negative direction is
// written to slot blockIdx.y | 2^axis and the positive one back in place.  One
// thread per line of cells, neighbouring threads on neighbouring x.
//
// Linear scan against the direction.  With G the value one step ahead, the new
// value is min(w, G) when a position within G steps ahead holds G, else min(w,
// G + 1): the positions within G steps all hold at least G.  last[v] is the
// scan index of the nearest position seen holding v; the second scan's indices
// start further than any distance past the first one's, so that the table
// needs no clearing in between.
//
// A serial chain per line, so its latency counts: the line is fetched to
// shared memory first (many loads in flight), and the table is there too.  In
// local memory, which shares L1 with everything else, the three passes took
// 62 us at 51^3 cells and 322 us at 147^3; now 24 and 87 us.
constexpr int kLineThreads = 64;
__global__ void __launch_bounds__(kLineThreads) k_empty_pass(uint8_t* __restrict__ d, long long n_cells, int nx, int ny,
                                                             int nz, int axis)
{
  __shared__ __align__(16) uint16_t s_last[(kEmptyCap + 1) * kLineThreads];
  __shared__ uint8_t s_in[kMaxDim * kLineThreads];
  {
    uint4* z = reinterpret_cast<uint4*>(s_last);
    for (int i = threadIdx.x; i < (int)(sizeof s_last / sizeof(uint4)); i += kLineThreads)
      z[i] = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  uint16_t* last = s_last + threadIdx.x;  // value v at last[v * kLineThreads]
  uint8_t* line = s_in + threadIdx.x;     // cell i at line[i * kLineThreads]
  const int t = blockIdx.x * kLineThreads + threadIdx.x;
  const int other = axis == 1 ? nz : ny, n_len = axis == 1 ? ny : nz;
  if (t >= nx * other)
    return;
  const size_t stride = axis == 1 ? (size_t)nx : (size_t)nx * ny;
  const size_t base = axis == 1 ? (size_t)(t / nx) * nx * ny + t % nx : (size_t)t;
  uint8_t* in = d + (size_t)blockIdx.y * n_cells + base;
  uint8_t* neg = d + (size_t)(blockIdx.y | (1u << axis)) * n_cells + base;
#pragma unroll 16
  for (int i = 0; i < n_len; ++i)
    line[i * kLineThreads] = in[i * stride];
#pragma unroll 1
  for (int dir = 1; dir >= 0; --dir) {
    uint8_t* out = dir ? neg : in;
    const int k0 = dir ? kEmptyCap + 1 : n_len + 2 * (kEmptyCap + 1);
    int G = kEmptyCap;  // no position holds it yet: the first step keeps its own value
#pragma unroll 4
    for (int k = 0; k < n_len; ++k) {
      const int i = dir ? k : n_len - 1 - k;
      const int w = line[i * kLineThreads];
      const int h = k + k0 - (int)last[G * kLineThreads] <= G ? G : min(G + 1, kEmptyCap);
      G = min(w, h);
      last[w * kLineThreads] = (uint16_t)(k + k0);
      out[i * stride] = (uint8_t)G;
    }
  }
}

// Packs the cell records: occupied {start, end}; empty {octants 0-3, flag |
// octants 4-7}, one byte per octant (octant o in byte o & 3).  Without a
// distance map every octant distance is 1 (single DDA steps).  `pad` records
// before and after the table are empty cells with distance 1.
__global__ void k_cell_rec(const uint32_t* __restrict__ cell_start, const uint8_t* __restrict__ empty_dist,
                           long long n_cells, long long pad, uint2* __restrict__ rec)
{
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_cells + 2 * pad;
       i += (long long)gridDim.x * blockDim.x) {
    const long long c = i - pad;
    uint32_t w[2] = {0x01010101u, 0x01010101u};
    if (c >= 0 && c < n_cells) {
      const uint32_t b = cell_start[c], e = cell_start[c + 1];
      if (e > b) {
        rec[i] = make_uint2(b, e);
        continue;
      }
      if (empty_dist) {
        w[0] = w[1] = 0;
#pragma unroll
        for (int o = 0; o < kOctants; ++o)
          w[o >> 2] |= (uint32_t)empty_dist[(size_t)o * n_cells + c] << (8 * (o & 3));
      }
    }
    rec[i] = make_uint2(w[0], kCellEmpty | w[1]);
  }
}

// ---------------------------------------------------------------------------
// Nearest hit through the grid as a per-lane state machine.  A lane tests the
// references of its current cell and, when they are exhausted, stops or moves
// to the next cell (or jumps over empty space).  Lanes of a warp stay in step
// whatever the cell occupancy, and a lane whose ray finishes can start another
// ray at once (persistent refill).
//
// Everything here works in grid coordinates (cells) and in world distance
// along the ray, with fused multiply-adds: the walk only has to visit the
// cells whose references may hold the nearest hit (the binning margin is far
// above its rounding), and the fast test only has to decide within the bounds
// of make_testrec.  What they leave open goes to the exact test of the
// reference (tri_hit_regs), so the face found is the reference's.
//
// The walk uses mirrored coordinates (an axis the ray descends is counted from
// the far side), so that every ray moves up on every axis and steps and jumps
// need no sign.  A cell is held as the float 1.5 * 2^23 + cell (kBias): adding
// a distance or rounding a position down to its cell is one float addition,
// and the low mantissa bits are the integer index.  No conversion
// instructions, no selects on the direction: about 35 instructions per move
// and per test, where the exact test in every reference and a walk with
// conversions and signs took about 90 and 120.  The trace issues fewer
// instructions and, with the record in two 256-bit loads instead of four of
// 128 bits, fewer L1 wavefronts: 22 080 faces, 22.08 M rays, 162^3 cells:
// 9.69 -> 5.50 ms; 400 faces, 40 M rays, 16^3 cells: 8.81 -> 5.38 ms.
//
// Stopping rule: after a cell, stop when the best distance, plus 2.5 margins,
// is below the distance at which the ray leaves that cell (or the empty cube
// it is about to cross); any triangle not yet tested lies in unvisited cells
// and cannot compute a smaller distance.
// ---------------------------------------------------------------------------
constexpr float kBias = 12582912.f;           // 1.5 * 2^23: one unit in the last place is 1
constexpr uint32_t kBiasBits = 0x4B400000u;   // its bit pattern; kBias + c has kBiasBits + c

struct Tracer {
  float3 og, dg;     // origin and direction (per world unit), grid coordinates; a NaN origin makes every test exact
  float3 po, pd;     // mirrored: origin + landing bias, |direction|
  float3 iv, io;     // 1 / |direction| and -(mirrored origin) / |direction|: a plane e is reached at e * iv + io
  float bx, by, bz;  // current cell, biased
  float jump;        // empty-space distance of the cell - kBias
  float t_stop;      // the walk ends here: the box exit, or the best hit + slack
  float far;         // kFar: error factor of a ray from outside the box, negative for a short one
  uint32_t i, en;    // pending references of the current cell
  int face;          // best hit, -1 if none
  int sx, sy, sz;    // signed cell strides
  uint32_t base;     // cell index offset
  uint32_t oct;      // octant of the direction
};

// Built as plain C++ (a check of the walk on the CPU) the functions with GPU
// instructions take a few lines of C++ instead.
__device__ __forceinline__ float rcp_approx(float x)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return fabsf(x) < 0x1p-126f ? copysignf(INFINITY, x) : 1.f / x;
#endif
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return fabsf(x) < 0x1p-126f ? copysignf(INFINITY, x) : 1.f / sqrtf(x);
#endif
}

// 256-bit read-only load (32-byte aligned).  With kStream the line does not
// enter the L1 cache.
//
// Scenes whose test records are larger than the L1 cache hit there seldom (7 %
// in a closed room of 22 080 faces), and filling and evicting lines costs more
// than the hits save: with 0.26 to 28 MB of records 60 of 60 grids traced 2 to
// 22 % faster without (the room at 162^3 cells 4.80 -> 4.63 ms, plates of
// 10 000 faces 1.32 -> 1.10 ms).  Smaller tables are found in L1, and need it:
// 0.05 to 0.2 MB of records up to 1.6 times slower without.  So do launches
// whose rays start at few faces (stream_records).
template <bool kStream>
__device__ __forceinline__ void ldg8(const void* p, float* v)
{
#ifndef __CUDA_ARCH__
  memcpy(v, p, 8 * sizeof(float));
#else
  if constexpr (kStream)
    asm("ld.global.nc.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
  else
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
#endif
}

// Reads the record of the current cell: its references, or its empty-space
// distance in the octant of the ray.  A position within rounding of the box's
// far side can land one cell beyond it: the table has a border of empty cells
// (cell_pad) below and above, and nothing lies within two margins of the box.
__device__ __forceinline__ void tracer_enter(Tracer& T, const GridView& g)
{
  // modulo 2^32: the products of the bias overflow and cancel against the base
  const uint32_t cell = T.base + __float_as_uint(T.bx) * (uint32_t)T.sx + __float_as_uint(T.by) * (uint32_t)T.sy +
                        __float_as_uint(T.bz) * (uint32_t)T.sz;
  const uint2 r = __ldg(g.cell_rec + (int)cell);
  const bool empty = (int)r.y < 0;
  const uint32_t d = (__byte_perm(r.x, r.y, T.oct) & 0x7Fu) | 0x4B000000u;  // the octant's byte as 2^23 + d
  T.jump = (empty ? __uint_as_float(d) : 8388609.f) - (8388608.f + kBias);
  T.i = r.x;
  T.en = empty ? 0u : r.y;
}

// Cells of padding before and after the cell table: one index step beyond
// either end of each axis.
__host__ __device__ inline long long cell_pad(int nx, int ny) { return 1ll + nx + (long long)nx * ny; }

// Speed of the walk along an axis, cells per world unit; one so small that a
// plane's distance (up to 256 cells and a jump of 127 over the speed) might
// overflow counts as zero, whose reciprocal is infinite: the axis is then never
// stepped and drops out of the minima as a NaN.  Over the diagonal of a box of
// 2^64, past which squared edges overflow in the reference's test, the ray
// moves 2^-53 cells along it, far below the landing bias.  Times 2^-9 with
// flushing, and back: a comparison and a selection for each axis cost k_cast 3 %
// (2.4 M rays 0.91 -> 0.93 ms).
__device__ __forceinline__ float walk_speed(float d)
{
#ifdef __CUDA_ARCH__
  float a;
  asm("mul.ftz.f32 %0, %1, 0f3B000000;" : "=f"(a) : "f"(fabsf(d)));
  return a * 512.f;
#else
  return fabsf(d) >= 0x1p-117f ? fabsf(d) : 0.f;
#endif
}

// Sets up the ray o + t dir; false when it misses the grid box (no hit
// possible).  *t0 gets the distance from o to the point the walk starts at (0
// inside the box).  kFar: rays may start far outside the box, and their tests
// widen the error bounds in proportion, or be given by an end point very near,
// and then only rejections are left to the fast test; otherwise such a ray takes
// the exact test for every reference.  2 M rays cast in the closed room of 22 080
// faces as segments of 1/32 and 1e-5: 0.89 and 1.12 ms, 1.42 and 1.62 with exact
// tests alone; whole rays 0.80.
template <bool kFar>
__device__ __forceinline__ bool tracer_begin(Tracer& T, const GridView& g, float3 o, float3 dir, float* t0,
                                             uint32_t& n_cells)
{
  *t0 = 0.f;
  const float dd = __fmaf_rn(dir.x, dir.x, __fmaf_rn(dir.y, dir.y, dir.z * dir.z));
  bool exact = false;
  float rd = rsqrt_approx(dd);
  T.far = 1.f;
  if (kFar && dd >= 0x1p-100f && dd < 0.00390625f) {
    // shorter than 1/16: the exact test's |n.dir| >= 1e-8 is not certain, so it
    // decides what the fast test does not reject
    T.far = -1.f;
  } else if (!(dd >= 0.00390625f && dd < 1e30f)) {
    // the fast test's bounds do not hold: every test is exact.  Zero or not
    // finite: hits nothing
    const float m = fmaxf(fmaxf(fabsf(dir.x), fabsf(dir.y)), fabsf(dir.z));
    if (!(m > 0.f && m < INFINITY) || !(dd == dd))
      return false;
    const float e = 1.f / m;
    const float3 q = e < INFINITY ? mul3(dir, e) : mul3(mul3(dir, 0x1p60f), 1.f / (m * 0x1p60f));
    dir = q;
    rd = rsqrt_approx(dot3(q, q));
    exact = true;
  }
  T.og = f3((o.x - g.lo.x) * g.inv_cs.x, (o.y - g.lo.y) * g.inv_cs.y, (o.z - g.lo.z) * g.inv_cs.z);
  T.dg = f3((dir.x * rd) * g.inv_cs.x, (dir.y * rd) * g.inv_cs.y, (dir.z * rd) * g.inv_cs.z);
  const bool mx = T.dg.x < 0.f, my = T.dg.y < 0.f, mz = T.dg.z < 0.f;
  float3 om = f3(mx ? g.nf.x - T.og.x : T.og.x, my ? g.nf.y - T.og.y : T.og.y, mz ? g.nf.z - T.og.z : T.og.z);
  if (!(om.x <= g.nf.x && om.y <= g.nf.y && om.z <= g.nf.z))
    return false;  // beyond the far side of an axis (or not a number)
  T.pd = f3(walk_speed(T.dg.x), walk_speed(T.dg.y), walk_speed(T.dg.z));
  T.iv = f3(rcp_approx(T.pd.x), rcp_approx(T.pd.y), rcp_approx(T.pd.z));
  T.io = f3(-om.x * T.iv.x, -om.y * T.iv.y, -om.z * T.iv.z);
  if (om.x < 0.f || om.y < 0.f || om.z < 0.f) {
    // outside: the walk starts where the ray enters the box
    const float te = fmaxf(fmaxf(T.io.x, T.io.y), T.io.z);
    if (!(te < INFINITY))
      return false;
    T.og = f3(__fmaf_rn(te, T.dg.x, T.og.x), __fmaf_rn(te, T.dg.y, T.og.y), __fmaf_rn(te, T.dg.z, T.og.z));
    om = f3(mx ? g.nf.x - T.og.x : T.og.x, my ? g.nf.y - T.og.y : T.og.y, mz ? g.nf.z - T.og.z : T.og.z);
    if (!(om.x <= g.nf.x && om.y <= g.nf.y && om.z <= g.nf.z))
      return false;  // passes beside the box (whose outer two margins are empty)
    om = f3(fminf(fmaxf(om.x, 0.f), g.nf.x), fminf(fmaxf(om.y, 0.f), g.nf.y), fminf(fmaxf(om.z, 0.f), g.nf.z));
    T.io = f3(-om.x * T.iv.x, -om.y * T.iv.y, -om.z * T.iv.z);
    *t0 = te;
    if (kFar)
      T.far *= __fmaf_rn(te, g.inv_size, 1.f);
    else
      exact = true;
  }
  T.po = f3(om.x + g.eps.x, om.y + g.eps.y, om.z + g.eps.z);
  T.t_stop = fminf(fminf(__fmaf_rn(g.nf.x, T.iv.x, T.io.x), __fmaf_rn(g.nf.y, T.iv.y, T.io.y)),
                   __fmaf_rn(g.nf.z, T.iv.z, T.io.z));
  if (exact)
    T.og.x = __int_as_float(0x7FC00000);
  T.sx = mx ? -1 : 1;
  T.sy = my ? -g.nx : g.nx;
  T.sz = mz ? -g.nxy : g.nxy;
  T.base = (uint32_t)((mx ? g.nxm : 0) + (my ? g.nym : 0) + (mz ? g.nzm : 0)) -
           kBiasBits * (uint32_t)(T.sx + T.sy + T.sz);
  T.oct = (mx ? 1u : 0u) | (my ? 2u : 0u) | (mz ? 4u : 0u);
  T.bx = __fadd_rd(T.po.x, kBias);
  T.by = __fadd_rd(T.po.y, kBias);
  T.bz = __fadd_rd(T.po.z, kBias);
  T.face = -1;
  ++n_cells;
  tracer_enter(T, g);
  return true;
}

// The current cell is exhausted: stop, or move to the next cell.  Returns
// false when the ray is finished.
//
// Every move leaves the empty cube of `jump` cells per side that extends from
// the cell in the octant of the ray's direction (the cell itself when jump is
// 1: an occupied cell, or a plain DDA step).  The ray starts inside the cube
// and moves monotonically, so it leaves through a far face, at tj, and lands
// in the cell where it crosses that face.  Landing positions are biased
// forward by eps (a quarter of the margin, over a hundred times their
// rounding), so the exit axis always advances to the cube's far side -- a ray
// leaves the grid after at most nx + ny + nz moves -- and a cell the ray only
// touches within eps of its boundary may be skipped: its triangles there are
// within the margin of the landing cell, which lists them too.
__device__ __forceinline__ bool tracer_advance(Tracer& T, const GridView& g, uint32_t& n_cells, uint32_t& n_jumps)
{
  const float ex = __fmaf_rn(T.bx + T.jump, T.iv.x, T.io.x);
  const float ey = __fmaf_rn(T.by + T.jump, T.iv.y, T.io.y);
  const float ez = __fmaf_rn(T.bz + T.jump, T.iv.z, T.io.z);
  const float tj = fminf(fminf(ex, ey), ez);
  if (!(tj < T.t_stop))
    return false;
  n_jumps += T.jump >= 2.f - kBias;
  T.bx = __fadd_rd(__fmaf_rn(tj, T.pd.x, T.po.x), kBias);
  T.by = __fadd_rd(__fmaf_rn(tj, T.pd.y, T.po.y), kBias);
  T.bz = __fadd_rd(__fmaf_rn(tj, T.pd.z, T.po.z), kBias);
  ++n_cells;
  tracer_enter(T, g);
  return true;
}

// Fast test of the next pending reference of the current cell.  Returns the
// face when only the exact test can decide it (tracer_exact), else -1: the
// face is missed for certain, or no nearer than the best hit, or it is hit for
// certain and nearer by more than the errors of both (then it is the best).
// The comparisons are written so that a NaN goes to the exact test.
template <bool kFar, bool kStream>
__device__ __forceinline__ int tracer_test(Tracer& T, const GridView& g, uint32_t& n_tests)
{
  float q[16];
  const TestRec* rec = g.ref_rec + T.i;
  ldg8<kStream>(rec, q);
  ldg8<kStream>(reinterpret_cast<const float*>(rec) + 8, q + 8);
  ++T.i;
  ++n_tests;
  const float b = __fmaf_rn(q[2], T.dg.z, __fmaf_rn(q[1], T.dg.y, q[0] * T.dg.x));
  const float a = __fmaf_rn(-q[2], T.og.z, __fmaf_rn(-q[1], T.og.y, __fmaf_rn(-q[0], T.og.x, q[3])));
  const float ib = rcp_approx(b);
  const float t = a * ib;
  const float x = __fmaf_rn(t, T.dg.x, T.og.x), y = __fmaf_rn(t, T.dg.y, T.og.y), z = __fmaf_rn(t, T.dg.z, T.og.z);
  const float s = __fmaf_rn(q[6], z, __fmaf_rn(q[5], y, __fmaf_rn(q[4], x, q[7])));
  const float r = __fmaf_rn(q[10], z, __fmaf_rn(q[9], y, __fmaf_rn(q[8], x, q[11])));
  const float m = fminf(fminf(s, r), (1.f - s) - r);
  const float e = kFar ? fabsf(ib * T.far) : fabsf(ib);
  const float t_lo = __fmaf_rn(-q[13], e, t), t_hi = __fmaf_rn(q[13], e, t);
  if ((m < -e) | (t_hi < 0.f) | (t_lo > T.t_stop))
    return -1;
  const int f = __float_as_int(q[12]);
  if (f == T.face)
    return -1;
  const bool inside = m > e && (!kFar || T.far > 0.f);
  if (inside && t_lo > 0.f && t_hi - t < g.near_err && (T.face < 0 || t_hi < T.t_stop - g.tie)) {
    T.face = f;
    T.t_stop = fminf(T.t_stop, t + g.slack);
    return -1;
  }
  return f;
}

// The exact test of face f for the ray (o, dir, start distance t0), merged
// into the best hit: the smallest squared distance wins and, among equal
// distances, the lowest face index, which equals the reference's strict '<'
// scan in index order from FLT_MAX.  Where the best hit's distance is not
// clear of this one's, both are computed exactly.
__device__ __forceinline__ void tracer_exact(Tracer& T, const GridView& g, int f, float3 o, float3 dir, float t0)
{
  float3 pt;
  if (!tri_hit(reinterpret_cast<const float4*>(g.tri + f), o, dir, pt))
    return;
  const float d = dist2(pt, o);
  if (!(d < 3.40282347e+38f))
    return;
  const float t = sqrtf(d) - t0;
  if (T.face >= 0 && !(t < T.t_stop - g.tie)) {
    float3 pb;
    if (tri_hit(reinterpret_cast<const float4*>(g.tri + T.face), o, dir, pb)) {
      const float db = dist2(pb, o);
      if (!(d < db || (d == db && f < T.face)))
        return;
    }
  }
  T.face = f;
  T.t_stop = fminf(T.t_stop, t + g.slack);
}

}  // namespace ffb
