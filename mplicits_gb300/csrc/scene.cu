// Triangle scene and the tubular-neighbourhood deltas (calc_deltas).
//
// experiment_scripts/utils.py:46-89 bisects, for every vertex v with unit
// normal n, the radius delta of the largest ball q = v + delta * n that still
// touches the mesh only near v: each iteration asks the unsigned distance D
// from q to the mesh (an open3d RaycastingScene, built at
// experiment_scripts/train_sdf_on_neighborhood.py:145-146) and halves the step
// and steps back when |delta - D| > eps, else steps forward, while
// max(delta) < max_delta.
//
// Scene: a uniform grid of cubic cells over the mesh's bounding box (one cell
// of margin on every side).  Each cell lists the triangles whose bounding box,
// grown by a relative 1e-5, overlaps it; the lists are stored in cell order as
// the triangles' corner coordinates (three float4 per entry) beside one
// bounding sphere per entry (a separate float4 array, read first), so a query
// reads a cell's triangles as one contiguous run and computes the exact
// distance only for entries whose sphere comes near enough.  Built on the
// device by a count pass, an exclusive scan and a fill pass.
//
// Distance: the closest point of each triangle by the Voronoi-region method
// of C. Ericson, "Real-Time Collision Detection" (2005), section 5.1.5, in
// float32 with every rounding explicit (__f*_rn, fmaf where written), so the
// CPU oracle that writes the same operations gets the same bits.  A query
// visits the cells within a radius R of q in shells of growing Chebyshev
// distance from q's cell, skipping cells whose box is farther than R.
//
// Decision of one bisection step (shrink_step_warp): |delta - D| > eps for the
// minimum D is rewritten as "some triangle nearer than delta - eps, or none
// within delta + eps" (exact in float32, see shrink_step_warp), so the search
// stops at the first near triangle and, once one triangle within delta + eps
// is found, ignores everything beyond delta - eps.  The result equals the
// brute-force minimum's comparison bit for bit.  calc_deltas searches once per
// certified stretch of a vertex's ray instead of once per step (see below).
//
// One launch per iteration for small meshes, three (decide, search by warps, search
// by blocks) for others: the stopping rule max(delta) < max_delta couples all
// vertices, so iteration i reads the maximum left by iteration i - 1 (a float per
// iteration, reduced with one atomic per block) and returns at once when it is
// reached, passing the value on; no host round trip.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cstring>

#include "common.cuh"

struct MplScene {
  int device;
  float lo[3];
  float h;
  int32_t dim[3];
  int64_t n_faces;
  int64_t n_refs;
  uint32_t* start;  // [cells + 1] offsets into tris (in entries)
  float4* tris;     // [n_refs * 3] corners a, b, c (a.w: the first entry of the
                    // same triangle, as bits)
  float4* bound;    // [n_refs] bounding sphere: centre, radius
  uint2* plane;     // [n_refs] unit normal, 3 x 10 bits (kNoPlane: degenerate);
                    // cell of the triangle's first entry, 3 x 10 bits (bit 31:
                    // this is that entry)
};

namespace mpl {
namespace scene {

constexpr int kThreads = 256;
constexpr int64_t kMaxDim = 1024;
constexpr int64_t kMaxCells = int64_t(1) << 25;
constexpr int64_t kMaxRefs = int64_t(1) << 31;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kThreads * kScanItems;
// calc_deltas: triangles a vertex keeps between iterations
constexpr int kList = 16;
// resident blocks per SM of its search kernels (four spill: 48.3 against 45.3 ms
// on the 523,266-vertex sphere mesh; two 43.1 against 37.4, a torus of 240,000
// vertices 10.9 against 9.3)
constexpr int kSearchBlocks = 3;
// Warps that share a heavy search, and the listed vertices up to which they take
// every search (the others would leave warps idle).  4096 / 8192 / 16384 / 32768
// listed: sheets of 32,768 vertices 2.57 / 2.58 / 2.91 / 3.77 ms, the sphere mesh of
// 32,514 4.37 / 4.37 / 4.38 / 5.54 and of 523,266 37.9 / 37.5 / 37.4 / 37.7.
constexpr int kHeavyWarps = 4;
constexpr uint32_t kFewSearches = 8192;
// Vertices up to which a step is one launch (deltas_fused), and its blocks per SM.
// Below, three dependent launches a step and a thread per vertex cost more than the
// searches.  100 steps of a sphere-like mesh, a torus and two parallel sheets, by one
// launch and by three: 482 / 384 / 512 vertices 0.78 / 0.74 / 0.74 and 1.70 / 1.38 /
// 1.57 ms, 16,022 / 16,224 / 16,200 vertices 2.4 / 2.3 / 2.0 and 3.7 / 2.9 / 2.8;
// 32,514 / 24,576 / 32,768 4.6 / 3.1 / 3.4 and 4.4 / 2.4 / 2.9.  (Six blocks per SM:
// 4514 vertices 1.32 instead of 1.15 ms; ten spill, 1.26.)
constexpr int64_t kFusedVertices = 16384;
constexpr int kFusedBlocks = 8;
// entries in a search's ball from which a block takes it instead of a warp (2048 and
// 8192: within 1% on the same meshes, but 38.0 and 37.8 ms on the largest)
constexpr uint32_t kHeavy = 4096;

struct View {
  float lo[3];
  float h;
  int32_t dim[3];
  const uint32_t* __restrict__ start;
  const float4* __restrict__ tris;
  const float4* __restrict__ bound;
  const uint2* __restrict__ plane;
};

// ---- the exact float32 point-triangle distance -----------------------------
struct V3 {
  float x, y, z;
};
__device__ __forceinline__ V3 sub(V3 a, V3 b) {
  return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
__device__ __forceinline__ float dot(V3 u, V3 v) {
  return __fmaf_rn(u.z, v.z, __fmaf_rn(u.y, v.y, __fmul_rn(u.x, v.x)));
}
// p - (s * u + o), per component
__device__ __forceinline__ V3 off_axpy(V3 p, float s, V3 u, V3 o) {
  return {__fsub_rn(p.x, __fmaf_rn(s, u.x, o.x)), __fsub_rn(p.y, __fmaf_rn(s, u.y, o.y)),
          __fsub_rn(p.z, __fmaf_rn(s, u.z, o.z))};
}

// p minus its closest point on the triangle; the distance is its length
__device__ __forceinline__ V3 tri_closest(V3 p, V3 a, V3 b, V3 c) {
  const V3 ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
  const float d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0.f && d2 <= 0.f) return ap;
  const V3 bp = sub(p, b);
  const float d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0.f && d4 <= d3) return bp;
  const float vc = __fmaf_rn(d1, d4, -__fmul_rn(d3, d2));
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    return off_axpy(p, __fdiv_rn(d1, __fsub_rn(d1, d3)), ab, a);
  }
  const V3 cp = sub(p, c);
  const float d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0.f && d5 <= d6) return cp;
  const float vb = __fmaf_rn(d5, d2, -__fmul_rn(d1, d6));
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    return off_axpy(p, __fdiv_rn(d2, __fsub_rn(d2, d6)), ac, a);
  }
  const float va = __fmaf_rn(d3, d6, -__fmul_rn(d5, d4));
  const float e43 = __fsub_rn(d4, d3), e56 = __fsub_rn(d5, d6);
  if (va <= 0.f && e43 >= 0.f && e56 >= 0.f) {
    return off_axpy(p, __fdiv_rn(e43, __fadd_rn(e43, e56)), sub(c, b), b);
  }
  const float denom = __fdiv_rn(1.0f, __fadd_rn(__fadd_rn(va, vb), vc));
  const float v = __fmul_rn(vb, denom), w = __fmul_rn(vc, denom);
  return {__fsub_rn(p.x, __fmaf_rn(ac.x, w, __fmaf_rn(ab.x, v, a.x))),
          __fsub_rn(p.y, __fmaf_rn(ac.y, w, __fmaf_rn(ab.y, v, a.y))),
          __fsub_rn(p.z, __fmaf_rn(ac.z, w, __fmaf_rn(ab.z, v, a.z)))};
}

__device__ __forceinline__ int cell_of(float x, float lo, float h, int dim) {
  const float f = floorf(__fdiv_rn(__fsub_rn(x, lo), h));
  if (!(f >= 0.f)) return 0;
  if (f >= (float)(dim - 1)) return dim - 1;
  return (int)f;
}

__device__ __forceinline__ bool finite3(V3 q) {
  return isfinite(q.x) && isfinite(q.y) && isfinite(q.z);
}

// squared distance from q to the box of cell (x, y, z)
__device__ __forceinline__ float cell_box_d2(const View& S, V3 q, int x, int y, int z) {
  auto gap = [&](float v, float lo, int i) {
    const float a = lo + S.h * (float)i, b = lo + S.h * (float)(i + 1);
    return v < a ? a - v : (v > b ? v - b : 0.f);
  };
  const float gx = gap(q.x, S.lo[0], x), gy = gap(q.y, S.lo[1], y), gz = gap(q.z, S.lo[2], z);
  return gx * gx + gy * gy + gz * gz;
}

// Visits the cells within R of q in shells of growing Chebyshev distance from
// q's cell (clamped to the grid); visit(cell, box_d2) returns true to stop.
template <class Visit>
__device__ __forceinline__ void walk_cells(const View& S, V3 q, float R, Visit&& visit) {
  int lo[3], hi[3], c[3];
  const float qa[3] = {q.x, q.y, q.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = cell_of(qa[k] - R, S.lo[k], S.h, S.dim[k]);
    hi[k] = cell_of(qa[k] + R, S.lo[k], S.h, S.dim[k]);
    c[k] = cell_of(qa[k], S.lo[k], S.h, S.dim[k]);
  }
  int rmax = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) rmax = max(rmax, max(c[k] - lo[k], hi[k] - c[k]));
  for (int r = 0; r <= rmax; ++r) {
    const int z0 = max(lo[2], c[2] - r), z1 = min(hi[2], c[2] + r);
    const int y0 = max(lo[1], c[1] - r), y1 = min(hi[1], c[1] + r);
    for (int z = z0; z <= z1; ++z) {
      const bool zs = (z == c[2] - r) || (z == c[2] + r);
      for (int y = y0; y <= y1; ++y) {
        const bool full = zs || (y == c[1] - r) || (y == c[1] + r);
        // a full row of the shell, or only its two end cells
        const int xs = full ? max(lo[0], c[0] - r) : c[0] - r;
        const int xe = full ? min(hi[0], c[0] + r) : c[0] + r;
        const int xstep = full ? 1 : max(2 * r, 1);
        for (int x = xs; x <= xe; x += xstep) {
          if (x < lo[0] || x > hi[0]) continue;
          const int64_t cell = ((int64_t)z * S.dim[1] + y) * S.dim[0] + x;
          if (visit(cell, cell_box_d2(S, q, x, y, z))) return;
        }
      }
    }
  }
}

__device__ __forceinline__ float entry_dist(const View& S, V3 q, uint32_t e) {
  const float4 A = S.tris[3 * (int64_t)e], B = S.tris[3 * (int64_t)e + 1],
               C = S.tris[3 * (int64_t)e + 2];
  const V3 v = tri_closest(q, {A.x, A.y, A.z}, {B.x, B.y, B.z}, {C.x, C.y, C.z});
  return __fsqrt_rn(dot(v, v));
}

constexpr uint32_t kNoPlane = 0xffffffffu;
// a stored normal's error: half a step of 1 / 511 per component
constexpr float kPlaneErr = 1.8e-3f;

// the triangle's unit normal, or kNoPlane
__device__ __forceinline__ uint32_t pack_plane(const float4 (&c)[3]) {
  const double ux = (double)c[1].x - c[0].x, uy = (double)c[1].y - c[0].y,
               uz = (double)c[1].z - c[0].z;
  const double vx = (double)c[2].x - c[0].x, vy = (double)c[2].y - c[0].y,
               vz = (double)c[2].z - c[0].z;
  const double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
  const double n2 = nx * nx + ny * ny + nz * nz;
  const double l2 = (ux * ux + uy * uy + uz * uz) * (vx * vx + vy * vy + vz * vz);
  if (!(n2 > 1e-16 * l2) || !(l2 < 1e300)) return kNoPlane;
  const float k = (float)(511.0 / sqrt(n2));
  auto q = [&](double v) { return (uint32_t)(__float2int_rn((float)v * k) + 512) & 1023u; };
  return q(nx) | q(ny) << 10 | q(nz) << 20;
}

// The triangle lies in the disc of its bounding sphere across its normal, so
// seen along the unit vector w it reaches at most r |w x n| past the centre
// (linear in the stored normal's error).  A lower bound of its distance from
// the point at offset v = q - centre of length l.
__device__ __forceinline__ float disc_distance(V3 v, float l, float r, uint32_t plane) {
  const V3 n = {(float)(int)(plane & 1023u) * (1.f / 511.f) - 512.f / 511.f,
                (float)(int)(plane >> 10 & 1023u) * (1.f / 511.f) - 512.f / 511.f,
                (float)(int)(plane >> 20 & 1023u) * (1.f / 511.f) - 512.f / 511.f};
  const float x = v.y * n.z - v.z * n.y, y = v.z * n.x - v.x * n.z, z = v.x * n.y - v.y * n.x;
  const float s = l > 0.f ? sqrtf(x * x + y * y + z * z) / l + kPlaneErr : 1.f;
  return l - r * fminf(plane == kNoPlane ? 1.f : s, 1.f);
}

// entry_dist as a call: kernels that evaluate in several places and run few
// warps wait on instruction fetches when each place has its own copy
__device__ __noinline__ float entry_dist_call(const float4* tris, V3 q, uint32_t e) {
  View S;
  S.tris = tris;
  return entry_dist(S, q, e);
}

// squared distance from q to an entry's bounding-sphere centre
__device__ __forceinline__ float centre_d2(V3 q, float4 b) {
  const float dx = q.x - b.x, dy = q.y - b.y, dz = q.z - b.z;
  return dx * dx + dy * dy + dz * dz;
}

// margin added to a search radius: far above the rounding of the cell, box
// and sphere arithmetic at the coordinates' magnitude
__device__ __forceinline__ float margin(V3 q, float h) {
  return 1e-5f * (fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))) + h);
}

// Minimum distance from q over the triangles within R of q (INFINITY when
// none).  An entry whose bounding sphere lies farther than the best so far
// cannot lower it and is skipped; the minimum is the same.
__device__ float nearest(const View& S, V3 q, float R) {
  const float m = margin(q, S.h);
  float best = INFINITY;
  walk_cells(S, q, R, [&](int64_t cell, float box_d2) {
    const float lim = fminf(best * 1.0001f + m, R);
    if (box_d2 > lim * lim) return false;
    const uint32_t e0 = S.start[cell], e1 = S.start[cell + 1];
    for (uint32_t e = e0; e < e1; ++e) {
      const float4 b = S.bound[e];
      const float l = (fminf(best * 1.0001f + m, R) + b.w) * 1.00002f;
      if (centre_d2(q, b) > l * l) continue;
      const float d = entry_dist(S, q, e);
      if (d < best) best = d;
    }
    return false;
  });
  return best;
}

// (A call: it is the rare path, for normals not of unit length.)
// One bisection decision, |delta - D| > eps for D the minimum distance over
// all triangles, in float32.  With d_t each triangle's distance and the
// rounded differences monotone in d_t, it equals
//   (some t has delta - d_t > eps)  or  (no t has d_t - delta <= eps):
// the first ("close") ends the search; the second needs one witness
// ("touch").  Triangles farther than delta + eps can be neither; once a
// witness is found, only triangles nearer than delta - eps still matter.
// Both radii carry a margin, so the skips (cells by box, entries by bounding
// sphere) never drop a triangle that could change the answer.
//
// One query per warp; the close/touch flags are combined with __any_sync
// (they do not depend on the visiting order).
__device__ __noinline__ bool shrink_step_warp(const View& S, V3 q, float delta, float eps, int lane) {
  const float m = margin(q, S.h);
  const float r_touch = (delta + eps) * 1.0001f + m;
  const float r_close = fmaxf(delta - eps, 0.f) * 1.0001f + m;
  const int y0 = cell_of(q.y - r_touch, S.lo[1], S.h, S.dim[1]);
  const int z0 = cell_of(q.z - r_touch, S.lo[2], S.h, S.dim[2]);
  const int ny = cell_of(q.y + r_touch, S.lo[1], S.h, S.dim[1]) - y0 + 1;
  const int nz = cell_of(q.z + r_touch, S.lo[2], S.h, S.dim[2]) - z0 + 1;
  const int rows = ny * nz;
  const float inv_ny = 1.f / (float)ny;
  bool touch = false;
  // Rows of cells (y, z) are contiguous in the entry lists, so the entries of
  // the x-segment a row shares with the ball are one range: each lane takes a
  // row, and a warp prefix sum over the ranges hands the entries out one per
  // lane.
  for (int base = 0; base < rows; base += 32) {
    const float lim = touch ? r_close : r_touch;
    const int k = base + lane;
    uint32_t e0 = 0, cnt = 0;
    if (k < rows) {
      // k -> (y, z): a float quotient and exact integer corrections
      int zq = (int)((float)k * inv_ny);
      int yr = k - zq * ny;
      while (yr < 0) --zq, yr += ny;
      while (yr >= ny) ++zq, yr -= ny;
      const int y = y0 + yr, z = z0 + zq;
      const float ya = S.lo[1] + S.h * (float)y, yb = ya + S.h;
      const float za = S.lo[2] + S.h * (float)z, zb = za + S.h;
      const float gy = q.y < ya ? ya - q.y : (q.y > yb ? q.y - yb : 0.f);
      const float gz = q.z < za ? za - q.z : (q.z > zb ? q.z - zb : 0.f);
      const float w2 = lim * lim - gy * gy - gz * gz;
      if (w2 >= 0.f) {
        const float w = sqrtf(w2);
        const int xa = cell_of(q.x - w, S.lo[0], S.h, S.dim[0]);
        const int xb = cell_of(q.x + w, S.lo[0], S.h, S.dim[0]);
        const int64_t row = ((int64_t)z * S.dim[1] + y) * S.dim[0];
        e0 = S.start[row + xa];
        cnt = S.start[row + xb + 1] - e0;
      }
    }
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t T = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t j0 = 0; j0 < T; j0 += 32) {
      const uint32_t j = j0 + lane;
      // the owning row's lane: the first lane whose inclusive count exceeds j
      int L = 0;
#pragma unroll
      for (int st = 16; st; st >>= 1)
        if (__shfl_sync(0xffffffffu, incl, L + st - 1) <= j) L += st;
      const uint32_t oi = __shfl_sync(0xffffffffu, incl, L & 31);
      const uint32_t oc = __shfl_sync(0xffffffffu, cnt, L & 31);
      const uint32_t oe = __shfl_sync(0xffffffffu, e0, L & 31);
      bool c_close = false, c_touch = false;
      if (j < T) {
        const uint32_t e = oe + (j - (oi - oc));
        const float4 b = S.bound[e];
        const float l = ((touch ? r_close : r_touch) + b.w) * 1.00002f;
        if (centre_d2(q, b) <= l * l) {
          const float d = entry_dist(S, q, e);
          c_close = __fsub_rn(delta, d) > eps;
          c_touch = __fsub_rn(d, delta) <= eps;
        }
      }
      if (__any_sync(0xffffffffu, c_close)) return true;
      touch = touch || __any_sync(0xffffffffu, c_touch);
    }
  }
  return !touch;
}

// ---- scene build -----------------------------------------------------------
__device__ __forceinline__ uint32_t ord(float f) {  // order-preserving float key
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float unord(uint32_t k) {
#ifdef __CUDA_ARCH__
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
#else
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}

// stats: [0..2] min keys, [3..5] max keys, [6..7] sum of edge lengths (double)
__global__ void bounds_kernel(const float* __restrict__ pos, int64_t nv,
                              const int32_t* __restrict__ faces, int64_t nf, uint32_t* keys,
                              double* edge_sum, int* bad_index) {
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  double es = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nf; i += stride) {
    int32_t f[3] = {faces[3 * i], faces[3 * i + 1], faces[3 * i + 2]};
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 3; ++j) ok &= f[j] >= 0 && f[j] < nv;
    if (!ok) {
      atomicExch(bad_index, 1);
      continue;
    }
    float p[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k) p[j][k] = pos[3 * (int64_t)f[j] + k];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        mn[k] = fminf(mn[k], p[j][k]);
        mx[k] = fmaxf(mx[k], p[j][k]);
      }
      const int j1 = (j + 1) % 3;
      const float dx = p[j1][0] - p[j][0], dy = p[j1][1] - p[j][1], dz = p[j1][2] - p[j][2];
      es += sqrt((double)dx * dx + (double)dy * dy + (double)dz * dz);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
    }
  }
  for (int o = 16; o; o >>= 1) es += __shfl_xor_sync(0xffffffffu, es, o);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (mn[k] <= mx[k]) {
        atomicMin(&keys[k], ord(mn[k]));
        atomicMax(&keys[3 + k], ord(mx[k]));
      }
    }
    atomicAdd(edge_sum, es);
  }
}

__device__ __forceinline__ void tri_cells(const View& S, const float* __restrict__ pos,
                                          const int32_t* __restrict__ faces, int64_t t,
                                          int (&a)[3], int (&b)[3], float4 (&corner)[3]) {
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int64_t v = faces[3 * t + j];
    const float x = pos[3 * v], y = pos[3 * v + 1], z = pos[3 * v + 2];
    corner[j] = make_float4(x, y, z, 0.f);
    mn[0] = fminf(mn[0], x), mn[1] = fminf(mn[1], y), mn[2] = fminf(mn[2], z);
    mx[0] = fmaxf(mx[0], x), mx[1] = fmaxf(mx[1], y), mx[2] = fmaxf(mx[2], z);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float m = 1e-5f * (fabsf(mn[k]) + fabsf(mx[k]) + S.h);
    a[k] = cell_of(mn[k] - m, S.lo[k], S.h, S.dim[k]);
    b[k] = cell_of(mx[k] + m, S.lo[k], S.h, S.dim[k]);
  }
}

__global__ void count_kernel(View S, const float* __restrict__ pos,
                             const int32_t* __restrict__ faces, int64_t nf, uint32_t* counts,
                             unsigned long long* total) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long n = 0;
  if (t < nf) {
    int a[3], b[3];
    float4 cr[3];
    tri_cells(S, pos, faces, t, a, b, cr);
    for (int z = a[2]; z <= b[2]; ++z)
      for (int y = a[1]; y <= b[1]; ++y)
        for (int x = a[0]; x <= b[0]; ++x)
          atomicAdd(&counts[((int64_t)z * S.dim[1] + y) * S.dim[0] + x], 1u);
    n = (unsigned long long)(b[0] - a[0] + 1) * (b[1] - a[1] + 1) * (b[2] - a[2] + 1);
  }
  for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(total, n);
}

// exclusive scan of n uint32 counts in three passes (blocks of kScanBlock)
__global__ void scan_blocks(const uint32_t* __restrict__ in, uint32_t* out, int64_t n,
                            uint32_t* block_sums) {
  __shared__ uint32_t warp_tot[kThreads / 32];
  const int64_t base = (int64_t)blockIdx.x * kScanBlock + (int64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems], s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    v[j] = base + j < n ? in[base + j] : 0u;
    s += v[j];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = s;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t woff = 0;
  for (int w = 0; w < warp; ++w) woff += warp_tot[w];
  uint32_t run = woff + incl - s;
#pragma unroll
  for (int j = 0; j < kScanItems; ++j) {
    if (base + j < n) out[base + j] = run;
    run += v[j];
  }
  if (threadIdx.x == kThreads - 1) block_sums[blockIdx.x] = run;
}

__global__ void scan_top(uint32_t* block_sums, int64_t nb) {
  // one block: a sequential chunk per thread, then a scan of the chunk sums
  __shared__ uint32_t tot[kThreads];
  const int64_t per = (nb + kThreads - 1) / kThreads;
  const int64_t b0 = threadIdx.x * per, b1 = min(nb, b0 + per);
  uint32_t s = 0;
  for (int64_t b = b0; b < b1; ++b) s += block_sums[b];
  tot[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
    for (int i = 0; i < kThreads; ++i) {
      const uint32_t t = tot[i];
      tot[i] = run;
      run += t;
    }
  }
  __syncthreads();
  uint32_t run = tot[threadIdx.x];
  for (int64_t b = b0; b < b1; ++b) {
    const uint32_t t = block_sums[b];
    block_sums[b] = run;
    run += t;
  }
}

__global__ void scan_add(uint32_t* out, int64_t n, const uint32_t* __restrict__ block_sums,
                         uint32_t total) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += block_sums[i / kScanBlock];
  if (i == n) out[n] = total;
}

__global__ void fill_kernel(View S, const float* __restrict__ pos,
                            const int32_t* __restrict__ faces, int64_t nf, uint32_t* cursor,
                            float4* tris, float4* bound, uint2* plane) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nf) return;
  int a[3], b[3];
  float4 cr[3];
  tri_cells(S, pos, faces, t, a, b, cr);
  // bounding sphere about the centroid, grown past its own rounding
  const float cx = (cr[0].x + cr[1].x + cr[2].x) / 3.f, cy = (cr[0].y + cr[1].y + cr[2].y) / 3.f,
              cz = (cr[0].z + cr[1].z + cr[2].z) / 3.f;
  float r2 = 0.f;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float dx = cr[j].x - cx, dy = cr[j].y - cy, dz = cr[j].z - cz;
    r2 = fmaxf(r2, dx * dx + dy * dy + dz * dz);
  }
  const float rad = sqrtf(r2) * 1.0001f +
                    1e-5f * (fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + S.h);
  const float4 sphere = make_float4(cx, cy, cz, rad);
  const uint32_t normal = pack_plane(cr);
  const uint32_t home = (uint32_t)a[0] | (uint32_t)a[1] << 10 | (uint32_t)a[2] << 20;
  uint32_t first = 0xffffffffu;
  for (int z = a[2]; z <= b[2]; ++z)
    for (int y = a[1]; y <= b[1]; ++y)
      for (int x = a[0]; x <= b[0]; ++x) {
        const uint32_t e = atomicAdd(&cursor[((int64_t)z * S.dim[1] + y) * S.dim[0] + x], 1u);
        if (first == 0xffffffffu) {
          first = e;
          cr[0].w = __uint_as_float(e);
        }
        tris[3 * (int64_t)e] = cr[0];
        tris[3 * (int64_t)e + 1] = cr[1];
        tris[3 * (int64_t)e + 2] = cr[2];
        bound[e] = sphere;
        plane[e] = make_uint2(normal, home | (e == first ? 0x80000000u : 0u));
      }
}

// ---- queries ----------------------------------------------------------------
__global__ void distance_kernel(View S, const float* __restrict__ pts, int64_t n,
                                float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V3 q = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
  if (!finite3(q)) {
    out[i] = __int_as_float(0x7fc00000);
    return;
  }
  // grow the radius until the nearest triangle found lies inside it (no
  // unvisited triangle can then be nearer), or it reaches every cell: rmax
  // is the distance to the grid's farthest corner
  const float qa[3] = {q.x, q.y, q.z};
  float far2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float a = fabsf(qa[k] - S.lo[k]), b = fabsf(qa[k] - (S.lo[k] + S.h * S.dim[k]));
    far2 += fmaxf(a, b) * fmaxf(a, b);
  }
  const float rmax = sqrtf(far2) * 1.001f + S.h;
  float r = S.h;
  float best;
  for (;;) {
    best = nearest(S, q, r * 1.0001f + margin(q, S.h));
    if (best <= r || r >= rmax) break;
    r = fminf(r * 4.f, rmax);
  }
  out[i] = best;
}

// ---- calc_deltas -------------------------------------------------------------
// The bisection walks delta along one ray q(delta) = v + delta n, and with a
// unit normal the balls B(q(delta), delta - eps) grow inside one another: a
// triangle that is not "close" at delta_t is not close at any smaller delta.
// So a search does not only answer one step, it also certifies a stretch of
// the ray (clear_until), and later steps inside that stretch need no search:
//
//   clear     below it, only the listed triangles can be close;
//   key/ent   up to kList listed triangles, ascending: triangle i cannot be
//             close below key[i], so a step evaluates those with key <= delta;
//   touch     a triangle that was within eps of delta: evaluated every step;
//   close     the last triangle found close (tried before a new search).
//
// Every decision is still the exact float32 predicate of the brute-force
// minimum: a triangle is left out only where the certificate proves its
// predicate false.  A step whose result no longer changes delta ends the
// vertex (q, and with it every later decision, stays what it is).
// Bound: gathers of grid entries that hit L2, in the searches.  On the
// 523,266-vertex sphere mesh (99 iterations) a search per vertex and step took
// 204.7 ms (51.8 M searches); with certified stretches 38 ms (about 2 M
// searches).
struct Bisect {
  const float* __restrict__ v;
  int64_t M;
  int C;
  float max_delta, eps;
  float* __restrict__ out;
  float4* __restrict__ state;  // step, clear, upper, flags (int bits)
  uint2* __restrict__ wit;     // touch and close entries (kNone: none)
  float* __restrict__ key;     // [kList][M], with one launch a step [M][kList]
  uint32_t* __restrict__ ent;  // as key
  uint32_t* __restrict__ todo;  // [M] vertices of this step that need a search
  uint32_t* __restrict__ heavy;  // [M] of these, the ones for a whole block
};
// a step's work lists: lengths and how many were taken (zeroed by the call)
struct StepCount {
  uint32_t listed, taken, heavy, heavy_taken;
};
constexpr uint32_t kNone = 0xffffffffu;
constexpr int kCountMask = 0xff;  // flags: listed triangles
constexpr int kDone = 0x100;      // delta no longer changes
constexpr int kShort = 0x400;     // the last list overflowed: certify less at once
constexpr int kPlain = 0x200;     // normal not of unit length: search every step

// calc_deltas: normalise normals, copy the rows, append delta = step0
__global__ void deltas_init(Bisect B, float step0, float* maxd) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) maxd[0] = step0;
  if (i >= B.M) return;
  const float* r = B.v + i * B.C;
  float* o = B.out + i * (B.C + 1);
  for (int k = 0; k < B.C; ++k) o[k] = r[k];
  const float len = __fsqrt_rn(
      __fadd_rn(__fadd_rn(__fmul_rn(r[3], r[3]), __fmul_rn(r[4], r[4])), __fmul_rn(r[5], r[5])));
  const float n0 = __fdiv_rn(r[3], len), n1 = __fdiv_rn(r[4], len), n2 = __fdiv_rn(r[5], len);
  o[3] = n0;
  o[4] = n1;
  o[5] = n2;
  o[B.C] = step0;
  // subnormal squares can leave a "unit" normal far from length 1
  const bool unit = fabsf(n0 * n0 + n1 * n1 + n2 * n2 - 1.f) <= 4e-6f;
  B.state[i] = make_float4(step0, -INFINITY, INFINITY, __int_as_float(unit ? 0 : kPlain));
  B.wit[i] = make_uint2(kNone, kNone);
}

// A delta below which the triangle (a, b, c), whose computed offset from
// q = q(delta) is e of length d, cannot satisfy  t - d_t > eps  for any t (t on
// the ray, d_t the computed distance from q(t)).  For any unit vector w the
// triangle lies beyond its nearest corner along w, so its distance from q(t)
// is at least  min_x w.(q - x) + (t - delta) w.n,  whatever e's own error (a
// sliver's closest point may be far off); with w = e / d the bound is the
// distance itself up to that error.  t - d_t then grows at most at the rate
// 1 - w.n, and for t < delta it is smaller, the balls being nested.  The
// computed closest point lies on the triangle, so the computed distance is
// not below the true one by more than the rounding in m.
__device__ __forceinline__ float clear_until(float delta, float eps, V3 q, V3 a, V3 b, V3 c, V3 e,
                                             float d, V3 n, float m) {
  float lb = 0.f, wn = -1.f;
  if (d > 0.f) {
    const float i = 1.f / d;
    const V3 w = {e.x * i, e.y * i, e.z * i};
    lb = fminf(dot(w, sub(q, a)), fminf(dot(w, sub(q, b)), dot(w, sub(q, c))));
    wn = dot(w, n);
  }
  const float gap = eps - (delta - lb) - (2.f * m + 1e-5f * delta);
  if (!(gap > 0.f)) return -INFINITY;
  return delta + 0.9999f * gap / (fmaxf(1.f - wn, 0.f) + 2e-5f);
}

__device__ __forceinline__ uint64_t sort_word(float key, uint32_t e) {
  const uint32_t u = __float_as_uint(key);
  return ((uint64_t)((u & 0x80000000u) ? ~u : (u | 0x80000000u)) << 32) | e;
}
__device__ __forceinline__ float word_key(uint64_t w) {
  const uint32_t k = (uint32_t)(w >> 32);
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// one compare-exchange stage over the warp
__device__ __forceinline__ uint64_t exchange(uint64_t x, int j, bool up, int lane) {
  const uint64_t y = __shfl_xor_sync(0xffffffffu, x, j);
  const bool low = ((lane & j) == 0) == up;
  return low == (y < x) ? y : x;
}
__device__ __noinline__ uint64_t sort32(uint64_t x, int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j; j >>= 1) x = exchange(x, j, (lane & k) == 0, lane);
  return x;
}
// the 32 smallest of two ascending sequences, ascending
__device__ __noinline__ uint64_t merge32(uint64_t a, uint64_t b, int lane) {
  const uint64_t r = __shfl_sync(0xffffffffu, b, 31 - lane);
  uint64_t x = a < r ? a : r;
#pragma unroll
  for (int j = 16; j; j >>= 1) x = exchange(x, j, true, lane);
  return x;
}

struct Search {
  bool shrink;
  bool heavy;             // given up (kWarps = 1): more entries than kHeavy
  uint32_t touch, close;  // witnesses (kNone: none found)
  bool certified;         // list and clear are valid (not close)
  uint64_t list;          // lane i: i-th smallest (key, entry)
  float clear;            // listed keys lie below it, no other key does
};

constexpr int kUnroll = 2;                // entries a thread tests at a time
constexpr int kQueue = 32 * (kUnroll + 1);  // per warp: a batch and what they add
// shared memory of a search by kWarps warps
template <int kWarps>
struct SearchShared {
  uint32_t incl[kWarps * 64];  // inclusive entry counts of the chunk's rows
  uint32_t from[kWarps * 64];  // first entry minus the exclusive count
  uint32_t near[kWarps][kQueue];   // entries whose sphere comes near enough
  uint32_t queue[kWarps][64];      // of these, the ones to evaluate
  uint32_t warp_sum[kWarps];
  uint64_t cand[kWarps][64];   // candidates of the list: key, entry
  uint64_t touch[kWarps];
  float tau[kWarps];
  uint32_t close;
};

// One vertex per group of kWarps warps (a warp, or the whole block): the exact
// decision at delta, and the certificate up to delta_t >= delta.  `touched`:
// the caller has a touching triangle.  The result is the same in every thread
// for kWarps = 1 and in warp 0 else (shrink and close in every thread).
template <int kWarps>
__device__ Search search(const View& S, V3 q, V3 qt, V3 n, float delta, float delta_t, float eps,
                         bool touched, SearchShared<kWarps>& sm) {
  constexpr int G = kWarps * 32;
  const int lane = threadIdx.x & 31, warp = kWarps > 1 ? threadIdx.x >> 5 : 0;
  const int tid = warp * 32 + lane;
  auto sync = [] {
    if (kWarps > 1)
      __syncthreads();
    else
      __syncwarp();
  };
  uint32_t *queue = sm.queue[warp], *nearq = sm.near[warp];
  Search r;
  r.shrink = true;
  r.heavy = false;
  r.touch = r.close = kNone;
  r.certified = false;
  r.list = ~uint64_t(0);
  const float m = margin(q, S.h), mt = margin(qt, S.h);
  const float r_touch = (delta + eps) * 1.0001f + m;
  const float r_close = fmaxf(delta_t - eps, 0.f) * 1.0001f + mt;
  // the ball of delta_t holds every smaller delta's
  const float lim = touched ? r_close : (delta_t + eps) * 1.0001f + mt;
  const int y0 = cell_of(qt.y - lim, S.lo[1], S.h, S.dim[1]);
  const int z0 = cell_of(qt.z - lim, S.lo[2], S.h, S.dim[2]);
  const int ny = cell_of(qt.y + lim, S.lo[1], S.h, S.dim[1]) - y0 + 1;
  const int nz = cell_of(qt.z + lim, S.lo[2], S.h, S.dim[2]) - z0 + 1;
  const int rows = ny * nz;
  const float inv_ny = 1.f / (float)ny;
  float tau = delta_t;  // keys from here on are not listed
  float td = INFINITY;  // this lane's nearest touching triangle
  uint32_t te = kNone;
  int nn = 0, qn = 0, cn = 0;
  uint32_t seen = 0;
  uint64_t* cand = sm.cand[warp];
  if (kWarps > 1 && threadIdx.x == 0) sm.close = kNone;

  // evaluates the queue's last cnt entries, one per lane; true: a close one
  auto evaluate = [&](int cnt) {
    qn -= cnt;
    bool c_close = false;
    uint32_t e = kNone;
    uint64_t w = ~uint64_t(0);
    if (lane < cnt) {
      e = queue[qn + lane];
      const float4 A = S.tris[3 * (int64_t)e], Bv = S.tris[3 * (int64_t)e + 1],
                   Cv = S.tris[3 * (int64_t)e + 2];
      const V3 a = {A.x, A.y, A.z}, b = {Bv.x, Bv.y, Bv.z}, c = {Cv.x, Cv.y, Cv.z};
      const V3 v = tri_closest(q, a, b, c);
      const float d = __fsqrt_rn(dot(v, v));
      e = __float_as_uint(A.w);
      c_close = __fsub_rn(delta, d) > eps;
      if (__fsub_rn(d, delta) <= eps && d < td) td = d, te = e;
      const float k = clear_until(delta, eps, q, a, b, c, v, d, n, m);
      if (k < tau) w = sort_word(k, e);
    }
    const unsigned cm = __ballot_sync(0xffffffffu, c_close);
    if (cm) {
      r.close = __shfl_sync(0xffffffffu, e, __ffs(cm) - 1);
      return true;
    }
    const unsigned wm = __ballot_sync(0xffffffffu, ~w != 0);
    if (wm) {
      if (~w != 0) cand[cn + __popc(wm & ((1u << lane) - 1u))] = w;
      cn += __popc(wm);
      __syncwarp();
      if (cn > 32) {
        // the 32 smallest stay (entries of one triangle carry the same word:
        // once); no key from the last one's on is listed
        const uint64_t hi = 32 + lane < cn ? cand[32 + lane] : ~uint64_t(0);
        const uint64_t x = merge32(sort32(cand[lane], lane), sort32(hi, lane), lane);
        tau = fminf(tau, word_key(__shfl_sync(0xffffffffu, x, 31)));
        const uint64_t prev = __shfl_up_sync(0xffffffffu, x, 1);
        const bool own = word_key(x) < tau && !(lane > 0 && prev == x);
        const unsigned om = __ballot_sync(0xffffffffu, own);
        __syncwarp();
        if (own) cand[__popc(om & ((1u << lane) - 1u))] = x;
        cn = __popc(om);
        __syncwarp();
      }
    }
    return false;
  };

  // the cells of row (y, z) within lim of qt
  auto row_cells = [&](int y, int z, int& xa, int& xb) {
    const float ya = S.lo[1] + S.h * (float)y, yb = ya + S.h;
    const float za = S.lo[2] + S.h * (float)z, zb = za + S.h;
    const float gy = qt.y < ya ? ya - qt.y : (qt.y > yb ? qt.y - yb : 0.f);
    const float gz = qt.z < za ? za - qt.z : (qt.z > zb ? qt.z - zb : 0.f);
    const float w2 = lim * lim - gy * gy - gz * gz;
    if (!(w2 >= 0.f)) return false;
    const float w = sqrtf(w2);
    xa = cell_of(qt.x - w, S.lo[0], S.h, S.dim[0]);
    xb = cell_of(qt.x + w, S.lo[0], S.h, S.dim[0]);
    return true;
  };
  // whether the search also visits the first of a triangle's entries, from the
  // word of a later one
  auto visits_first = [&](uint32_t home) {
    const int y = (int)(home >> 10 & 1023u) - y0, z = (int)(home >> 20 & 1023u) - z0;
    int xa, xb;
    return y >= 0 && y < ny && z >= 0 && z < nz && row_cells(y + y0, z + z0, xa, xb) &&
           (int)(home & 1023u) >= xa && (int)(home & 1023u) <= xb;
  };

  // Rows of cells (y, z) are contiguous in the entry lists, so the entries of
  // the x-segment a row shares with the ball are one range: each thread takes
  // two rows, and a prefix sum over the ranges hands the entries out one per
  // thread, kUnroll at a time so that their loads overlap.
  // One round more than the rows need empties the queues.
  bool found = false;
  for (int base = 0;; base += 2 * G) {
    const bool last = base >= rows;
    uint32_t e0[2] = {0, 0}, cnt[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = base + 2 * tid + h;
      if (k < rows) {
        // k -> (y, z): a float quotient and exact integer corrections
        int zq = (int)((float)k * inv_ny);
        int yr = k - zq * ny;
        while (yr < 0) --zq, yr += ny;
        while (yr >= ny) ++zq, yr -= ny;
        const int y = y0 + yr, z = z0 + zq;
        int xa, xb;
        if (row_cells(y, z, xa, xb)) {
          const int64_t row = ((int64_t)z * S.dim[1] + y) * S.dim[0];
          e0[h] = S.start[row + xa];
          cnt[h] = S.start[row + xb + 1] - e0[h];
        }
      }
    }
    const uint32_t own = cnt[0] + cnt[1];
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (kWarps > 1) {
      if (lane == 31) sm.warp_sum[warp] = incl;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < kWarps; ++w) incl += w < warp ? sm.warp_sum[w] : 0u;
    }
    const uint32_t x0 = incl - own, x1 = x0 + cnt[0];
    sm.incl[2 * tid] = x1;
    sm.incl[2 * tid + 1] = incl;
    sm.from[2 * tid] = e0[0] - x0;
    sm.from[2 * tid + 1] = e0[1] - x1;
    sync();
    const uint32_t T = sm.incl[2 * G - 1];
    if (kWarps == 1) {
      seen += T;
      if (seen > kHeavy) {
        r.heavy = true;
        return r;
      }
    }
    uint32_t j0 = 0;
    do {
      uint32_t e[kUnroll];
      float4 b[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const uint32_t j = j0 + u * G + tid;
        e[u] = kNone;
        if (j < T) {
          // the owning row: the first whose inclusive count exceeds j
          int L = 0;
#pragma unroll
          for (int st = G; st; st >>= 1)
            if (sm.incl[L + st - 1] <= j) L += st;
          e[u] = sm.from[L] + j;
          b[u] = S.bound[e[u]];
        }
      }
      // sphere in the ball of delta_t, or (without a touching triangle) in the
      // touch shell of delta
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        bool keep = false;
        if (e[u] != kNone) {
          const float l = (r_close + b[u].w) * 1.00002f, l2 = (r_touch + b[u].w) * 1.00002f;
          keep = centre_d2(qt, b[u]) <= l * l || (!touched && centre_d2(q, b[u]) <= l2 * l2);
        }
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) nearq[nn + __popc(km & ((1u << lane) - 1u))] = e[u];
        nn += __popc(km);
      }
      __syncwarp();
      while (!found && (nn >= 32 || (last && (nn > 0 || qn > 0)))) {
        // the tighter disc, and one entry per triangle
        const int c = min(nn, 32);
        nn -= c;
        bool keep = false;
        uint32_t f = kNone;
        if (lane < c) {
          f = nearq[nn + lane];
          const float4 bd = S.bound[f];
          const uint2 pl = S.plane[f];
          const V3 v = {qt.x - bd.x, qt.y - bd.y, qt.z - bd.z};
          keep = disc_distance(v, sqrtf(centre_d2(qt, bd)), bd.w, pl.x) <= r_close;
          if (!touched && !keep) {
            const float l = (r_touch + bd.w) * 1.00002f;
            keep = centre_d2(q, bd) <= l * l;
          }
          if (keep && !(pl.y & 0x80000000u)) keep = !visits_first(pl.y);
        }
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) queue[qn + __popc(km & ((1u << lane) - 1u))] = f;
        qn += __popc(km);
        __syncwarp();
        if (qn >= 32 || (last && nn == 0 && qn > 0)) found = evaluate(min(qn, 32));
        __syncwarp();
      }
      if (kWarps > 1) {
        if (found && lane == 0) sm.close = r.close;
        found = found || *(volatile uint32_t*)&sm.close != kNone;
      }
      j0 += kUnroll * G;
    } while (j0 < T && !found);
    if (kWarps == 1) {
      if (found) return r;
      __syncwarp();
    } else {
      // block-uniform: the rows' arrays are free, and a close triangle ends it
      __syncthreads();
      if (sm.close != kNone) {
        r.close = sm.close;
        return r;
      }
    }
    if (last) break;
  }
  r.list = sort32(lane < cn ? cand[lane] : ~uint64_t(0), lane);
  // the nearest touching triangle of all lanes
  uint64_t tw = te == kNone ? ~uint64_t(0) : ((uint64_t)__float_as_uint(td) << 32) | te;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const uint64_t y = __shfl_xor_sync(0xffffffffu, tw, o);
    tw = y < tw ? y : tw;
  }
  if (kWarps > 1) {
    __syncwarp();
    cand[lane] = r.list;
    if (lane == 0) {
      sm.touch[warp] = tw;
      sm.tau[warp] = tau;
    }
    __syncthreads();
#pragma unroll 1
    for (int w = 0; w < kWarps; ++w) {
      tw = sm.touch[w] < tw ? sm.touch[w] : tw;
      tau = fminf(tau, sm.tau[w]);
      if (warp == 0 && w > 0) {
        // a full list may have lost keys, each at least the last one kept
        r.list = merge32(r.list, sm.cand[w][lane], lane);
        const uint64_t last = __shfl_sync(0xffffffffu, r.list, 31);
        if (~last != 0) tau = fminf(tau, word_key(last));
      }
    }
  }
  if (~tw != 0) r.touch = (uint32_t)tw;
  r.shrink = !touched && ~tw == 0;
  r.certified = true;
  r.clear = tau;
  return r;
}

// the update of one step; flags of the vertex's next state
__device__ __forceinline__ float advance(bool shrink, float delta, float& s, int& flags) {
  if (shrink) s = __fmul_rn(s, 0.5f);
  const float nd = shrink ? __fsub_rn(delta, s) : __fadd_rn(delta, s);
  if (nd == delta) flags |= kDone;
  return nd;
}

// the ray's point at delta
__device__ __forceinline__ V3 ray_point(const Bisect& B, int64_t i, float delta, V3 n) {
  const float* r = B.v + i * B.C;
  return {__fadd_rn(r[0], __fmul_rn(delta, n.x)), __fadd_rn(r[1], __fmul_rn(delta, n.y)),
          __fadd_rn(r[2], __fmul_rn(delta, n.z))};
}

// the block's maximum delta into maxd_next (deltas are positive whenever the
// loop runs, so the float bits order as integers; one atomic per block)
__device__ __forceinline__ void block_max(float wmax, float* maxd_next) {
  __shared__ float wmax_s[kThreads / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
  if ((threadIdx.x & 31) == 0) wmax_s[threadIdx.x >> 5] = wmax;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b = fmaxf(b, wmax_s[w]);
    if (b > 0.f) atomicMax((int*)maxd_next, __float_as_int(b));
  }
}

// One bisection step, first half: every thread decides its own vertex from its
// listed triangles where the certificate reaches, and lists the others for the
// search kernel.  maxd[it] is the maximum delta before the step, maxd[it + 1]
// collects the maximum after it.
__global__ void __launch_bounds__(kThreads) deltas_step(View S, Bisect B, float* maxd,
                                                        StepCount* count, int it) {
  const float before = maxd[it];
  if (!(before < B.max_delta)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) maxd[it + 1] = before;
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const float eps = B.eps;
  float wmax = 0.f;
  bool search = false;
  if (i < B.M) {
    float* o = B.out + i * (B.C + 1);
    const float delta = o[B.C];
    float4 st = B.state[i];
    int flags = __float_as_int(st.w);
    if (flags & kDone) {
      wmax = delta;
    } else {
      const V3 n = {o[3], o[4], o[5]};
      const V3 q = ray_point(B, i, delta, n);
      bool shrink = false;
      if (finite3(q)) {
        const uint2 wit = B.wit[i];
        search = true;
        if (!(flags & kPlain) && wit.x != kNone &&
            __fsub_rn(entry_dist_call(S.tris, q, wit.x), delta) <= eps) {
          if (delta < st.y) {
            search = false;
            const int cnt = flags & kCountMask;
            for (int k = 0; k < cnt && !shrink; ++k) {
              if (B.key[(int64_t)k * B.M + i] > delta) break;
              const uint32_t e = B.ent[(int64_t)k * B.M + i];
              if (__fsub_rn(delta, entry_dist_call(S.tris, q, e)) > eps) {
                shrink = true;
                B.wit[i].y = e;
              }
            }
          } else if (wit.y != kNone && __fsub_rn(delta, entry_dist_call(S.tris, q, wit.y)) > eps) {
            search = false;
            shrink = true;
          }
        }
      }
      if (!search) {
        if (shrink) st.z = fminf(st.z, delta);
        const float nd = advance(shrink, delta, st.x, flags);
        st.w = __int_as_float(flags);
        B.state[i] = st;
        o[B.C] = nd;
        wmax = nd;
      }
    }
  }
  const unsigned sm = __ballot_sync(0xffffffffu, search);
  uint32_t at = 0;
  if (lane == 0 && sm) at = atomicAdd(&count[it].listed, (uint32_t)__popc(sm));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (search) B.todo[at + __popc(sm & ((1u << lane) - 1u))] = (uint32_t)i;
  block_max(wmax, maxd + it + 1);
}

// One vertex's step by a search, by a warp (kWarps = 1, which lists a heavy one for
// the blocks and gives it up) or a block.  kFused: its lists are laid out by vertex.
template <int kWarps, bool kFused>
__device__ __forceinline__ void search_vertex(const View& S, const Bisect& B, int64_t i,
                                              SearchShared<kWarps>& sm, float& wmax,
                                              StepCount* ct) {
  constexpr bool kBlock = kWarps > 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool lead = kBlock ? threadIdx.x == 0 : lane == 0;  // writes the state
  const float eps = B.eps;
  float* o = B.out + i * (B.C + 1);
  const float delta = o[B.C];
  const V3 n = {o[3], o[4], o[5]};
  const V3 q = ray_point(B, i, delta, n);
  float4 st = B.state[i];
  int flags = __float_as_int(st.w);
  uint2 wit = B.wit[i];
  bool shrink;
  // the stretch to certify: half as far again as delta (at least eight
  // steps; a far ball costs more entries than the searches it saves: to four
  // times delta 45.3 ms on the sphere mesh, twice 38.2, half again 38.5, a
  // quarter 41.0), no farther than a delta known to be close or the end of
  // the loop
  float delta_t = delta + ((flags & kShort) ? 4.f * fabsf(st.x)
                                            : fmaxf(0.5f * delta, 8.f * fabsf(st.x)));
  delta_t = fminf(delta_t, B.max_delta + 2.f * fabsf(st.x));
  delta_t = fmaxf(fminf(delta_t, st.z), delta * 1.00001f);
  const V3 qt = ray_point(B, i, delta_t, n);
  if ((flags & kPlain) || !(delta > 0.f) || !finite3(qt)) {
    shrink = shrink_step_warp(S, q, delta, eps, lane);
  } else {
    const bool touched = wit.x != kNone && __fsub_rn(entry_dist_call(S.tris, q, wit.x), delta) <= eps;
    const Search r = search<kWarps>(S, q, qt, n, delta, delta_t, eps, touched, sm);
    if (kWarps == 1 && r.heavy) {
      if (lane == 0) B.heavy[atomicAdd(&ct->heavy, 1u)] = (uint32_t)i;
      __syncwarp();
      return;
    }
    shrink = r.shrink;
    if (r.touch != kNone) wit.x = r.touch;
    if (r.close != kNone) wit.y = r.close;
    if (r.certified && (!kBlock || warp == 0)) {
      // keep the kList nearest triangles (entries of one triangle carry the
      // same word); the next one ends the certified stretch
      const uint64_t prev = __shfl_up_sync(0xffffffffu, r.list, 1);
      const bool own = word_key(r.list) < r.clear && !(lane > 0 && prev == r.list);
      const unsigned om = __ballot_sync(0xffffffffu, own);
      const int rank = __popc(om & ((1u << lane) - 1u));
      if (own && rank < kList) {
        const int64_t at = kFused ? i * kList + rank : (int64_t)rank * B.M + i;
        B.key[at] = word_key(r.list);
        B.ent[at] = (uint32_t)r.list;
      }
      float clear = r.clear;
      const unsigned nm = __ballot_sync(0xffffffffu, own && rank == kList);
      if (nm) clear = fminf(clear, word_key(__shfl_sync(0xffffffffu, r.list, __ffs(nm) - 1)));
      st.y = clear;
      flags = (flags & ~(kCountMask | kShort)) | min(__popc(om), kList);
      if (clear < delta_t) flags |= kShort;
    }
  }
  if (shrink) st.z = fminf(st.z, delta);
  const float nd = advance(shrink, delta, st.x, flags);
  st.w = __int_as_float(flags);
  // every warp has read the vertex's state before it changes
  if (kBlock)
    __syncthreads();
  else
    __syncwarp();
  if (lead) {
    B.state[i] = st;
    B.wit[i] = wit;
    o[B.C] = nd;
    wmax = fmaxf(wmax, nd);
  }
  __syncwarp();
}

// Second half: the listed vertices, one per warp (kWarps = 1) or one per block
// of kWarps warps at a time, handed out by a counter: a search's cost varies by
// a hundred between the mesh's sparse and dense parts, which lie together in
// the vertex order.  A warp gives up a search of more than kHeavy entries and
// lists it for the block kernel, and up to kFewSearches listed vertices all go
// to blocks: there a step lasts as long as its longest search (a warp alone
// took 0.2 ms of each step for a few thousand searches).  Both kernels were
// bound by instruction fetches when the evaluation, the sorts and the list
// tests were inlined several times (58% of warp stalls; 67 ms in all), so each
// stands once in the code.
template <int kWarps>
__global__ void __launch_bounds__(kWarps > 1 ? kWarps * 32 : kThreads,
                                  kWarps > 1 ? kSearchBlocks * 8 / kWarps : kSearchBlocks)
    deltas_search(View S, Bisect B, float* maxd, StepCount* count, int it) {
  if (!(maxd[it] < B.max_delta)) return;
  constexpr bool kBlock = kWarps > 1;
  __shared__ SearchShared<kWarps> shared[kBlock ? 1 : kThreads / 32];
  __shared__ uint32_t next_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  SearchShared<kWarps>& sm = shared[kBlock ? 0 : warp];
  StepCount& ct = count[it];
  const bool few = ct.listed <= kFewSearches;
  const uint32_t total = kBlock ? (few ? ct.listed : ct.heavy) : (few ? 0u : ct.listed);
  const uint32_t* todo = kBlock && !few ? B.heavy : B.todo;
  float wmax = 0.f;
  for (;;) {
    uint32_t t = 0;
    if (kBlock) {
      __syncthreads();  // the last search's shared memory and next_s are read
      if (threadIdx.x == 0) next_s = atomicAdd(&ct.heavy_taken, 1u);
      __syncthreads();
      t = next_s;
    } else {
      if (lane == 0) t = atomicAdd(&ct.taken, 1u);
      t = __shfl_sync(0xffffffffu, t, 0);
    }
    if (t >= total) break;
    search_vertex<kWarps, false>(S, B, todo[t], sm, wmax, &ct);
  }
  block_max(wmax, maxd + it + 1);
}

// The same step by a warp: a lane per listed triangle, one for the touching one and
// one for the last close one.  True: decided (and the state written).
__device__ __forceinline__ bool decide_by_warp(const View& S, const Bisect& B, int64_t i, int lane,
                                               float& wmax) {
  float* o = B.out + i * (B.C + 1);
  const float delta = o[B.C];
  float4 st = B.state[i];
  int flags = __float_as_int(st.w);
  if (flags & kDone) {
    wmax = fmaxf(wmax, delta);
    return true;
  }
  const V3 q = ray_point(B, i, delta, {o[3], o[4], o[5]});
  bool shrink = false;
  if (finite3(q)) {
    if (flags & kPlain) return false;
    const uint2 wit = B.wit[i];
    const bool inside = delta < st.y;  // of the certified stretch
    uint32_t e = lane == 0 ? wit.x : (lane == 1 && !inside ? wit.y : kNone);
    if (inside && lane >= 2 && lane - 2 < (flags & kCountMask)) {
      const int64_t at = i * kList + lane - 2;
      if (!(B.key[at] > delta)) e = B.ent[at];
    }
    const float d = e != kNone ? entry_dist(S, q, e) : 0.f;
    const bool hit = e != kNone && (lane == 0 ? __fsub_rn(d, delta) <= B.eps
                                              : __fsub_rn(delta, d) > B.eps);
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    shrink = m > 1u;
    if (!(m & 1u) || (!inside && !shrink)) return false;
    if (inside && shrink && lane == __ffs(m & ~1u) - 1) B.wit[i].y = e;
  }
  if (shrink) st.z = fminf(st.z, delta);
  const float nd = advance(shrink, delta, st.x, flags);
  st.w = __int_as_float(flags);
  __syncwarp();  // every lane has read the state
  if (lane == 0) {
    B.state[i] = st;
    o[B.C] = nd;
  }
  wmax = fmaxf(wmax, nd);
  return true;
}

// A step in one launch, for meshes of up to kFusedVertices: a block of kHeavyWarps
// warps takes `per` vertices at a time, a warp decides each from its lists, and the
// block searches together for those that are left.
__global__ void __launch_bounds__(kHeavyWarps * 32, kFusedBlocks)
    deltas_fused(View S, Bisect B, float* maxd, int it, int per) {
  const float before = maxd[it];
  if (!(before < B.max_delta)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) maxd[it + 1] = before;
    return;
  }
  __shared__ SearchShared<kHeavyWarps> sm;
  __shared__ bool left[kHeavyWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float wmax = 0.f;
  for (int64_t i0 = (int64_t)blockIdx.x * per; i0 < B.M; i0 += (int64_t)gridDim.x * per) {
    const bool own = warp < per && i0 + warp < B.M;
    const bool decided = !own || decide_by_warp(S, B, i0 + warp, lane, wmax);
    if (lane == 0) left[warp] = !decided;
    __syncthreads();
#pragma unroll 1
    for (int w = 0; w < per; ++w) {
      if (left[w]) {
        search_vertex<kHeavyWarps, true>(S, B, i0 + w, sm, wmax, nullptr);
        __syncthreads();  // its shared memory is read
      }
    }
    __syncthreads();  // `left` is read
  }
  block_max(wmax, maxd + it + 1);
}

__global__ void deltas_count(const float* __restrict__ maxd, int n_iters, float max_delta,
                             int32_t* iterations) {
  int n = 0;
  for (int i = 0; i < n_iters; ++i) n += maxd[i] < max_delta ? 1 : 0;
  *iterations = n;
}

inline View view(const MplScene* s) {
  View v;
  for (int k = 0; k < 3; ++k) v.lo[k] = s->lo[k], v.dim[k] = s->dim[k];
  v.h = s->h;
  v.start = s->start;
  v.tris = s->tris;
  v.bound = s->bound;
  v.plane = s->plane;
  return v;
}

inline unsigned blocks(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// queries run on the device that holds the scene's grid
inline int check_device(const MplScene* s) {
  int dev = -1;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_last_cuda_error(e);
    return MPL_ERR_CUDA;
  }
  return dev == s->device ? MPL_OK : MPL_ERR_INVALID_ARG;
}

}  // namespace scene
}  // namespace mpl

using namespace mpl;
using namespace mpl::scene;

extern "C" int mpl_scene_create(const float* positions_dev, int64_t n_positions,
                                const int32_t* faces_dev, int64_t n_faces, float cell,
                                MplScene** out, void* stream) {
  if (!out) return MPL_ERR_INVALID_ARG;
  *out = nullptr;
  if (!positions_dev || !faces_dev || n_positions < 3 || n_faces < 1 || !(cell >= 0.f))
    return MPL_ERR_INVALID_ARG;
  if (n_faces >= kMaxRefs) return MPL_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0;
  MPL_CUDA_TRY(cudaGetDevice(&dev));

  // bounds, mean edge length, face-index check
  struct Stats {
    uint32_t keys[6];
    int bad;
    int pad;
    double edge_sum;
  };
  Stats* st = nullptr;
  MPL_CUDA_TRY(cudaMalloc(&st, sizeof(Stats)));
  Stats init;
  for (int k = 0; k < 3; ++k) init.keys[k] = 0xffffffffu, init.keys[3 + k] = 0u;
  init.bad = 0;
  init.pad = 0;
  init.edge_sum = 0.0;
  Stats host;
  cudaError_t e = cudaMemcpyAsync(st, &init, sizeof(Stats), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    const int64_t nb_want = blocks(n_faces), nb_cap = (int64_t)sm_count() * 8;
    const unsigned nb = (unsigned)(nb_want < nb_cap ? nb_want : nb_cap);
    bounds_kernel<<<nb, kThreads, 0, s>>>(positions_dev, n_positions, faces_dev, n_faces,
                                          st->keys, &st->edge_sum, &st->bad);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&host, st, sizeof(Stats), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(st);
  if (e != cudaSuccess) {
    set_last_cuda_error(e);
    return MPL_ERR_CUDA;
  }
  if (host.bad) return MPL_ERR_INVALID_ARG;
  float lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = unord(host.keys[k]);
    hi[k] = unord(host.keys[3 + k]);
    if (!isfinite(lo[k]) || !isfinite(hi[k])) return MPL_ERR_INVALID_ARG;
  }
  float h = cell;
  if (h <= 0.f) h = (float)(2.0 * host.edge_sum / (3.0 * (double)n_faces));
  float ext = 0.f;
  for (int k = 0; k < 3; ++k) ext = fmaxf(ext, hi[k] - lo[k]);
  if (!(h > 0.f)) h = ext > 0.f ? ext : 1.f;
  // bound the cell count: each dimension <= kMaxDim (an entry's home cell has 10 bits
  // for each), the product <= kMaxCells.  1.25^1000 spans all of float's range.
  int64_t dim[3], cells = 0;
  bool fits = false;
  for (int guard = 0; guard < 1000 && !fits; ++guard) {
    cells = 1;
    fits = true;
    for (int k = 0; k < 3 && fits; ++k) {
      const float n = (hi[k] - lo[k]) / h;
      fits = n < (float)kMaxDim;  // false for an infinite extent too
      dim[k] = fits ? (int64_t)n + 3 : 0;
      fits = fits && dim[k] <= kMaxDim;
      cells *= dim[k];
    }
    fits = fits && cells <= kMaxCells;
    if (!fits) h *= 1.25f;
  }
  if (!fits) return MPL_ERR_UNSUPPORTED;

  MplScene* sc = new MplScene();
  sc->device = dev;
  sc->h = h;
  for (int k = 0; k < 3; ++k) sc->lo[k] = lo[k] - h, sc->dim[k] = (int32_t)dim[k];
  sc->n_faces = n_faces;
  const int64_t nb = (cells + kScanBlock - 1) / kScanBlock;
  uint32_t *counts = nullptr, *bsum = nullptr;
  unsigned long long* total = nullptr;
  unsigned long long total_h = 0;
  auto fail = [&](cudaError_t err) {
    set_last_cuda_error(err);
    cudaFree(counts);
    cudaFree(bsum);
    cudaFree(total);
    cudaFree(sc->start);
    cudaFree(sc->tris);
    cudaFree(sc->bound);
    cudaFree(sc->plane);
    delete sc;
    return MPL_ERR_CUDA;
  };
  if ((e = cudaMalloc(&counts, sizeof(uint32_t) * cells)) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&sc->start, sizeof(uint32_t) * (cells + 1))) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&bsum, sizeof(uint32_t) * nb)) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&total, sizeof(unsigned long long))) != cudaSuccess) return fail(e);
  if ((e = cudaMemsetAsync(counts, 0, sizeof(uint32_t) * cells, s)) != cudaSuccess) return fail(e);
  if ((e = cudaMemsetAsync(total, 0, sizeof(unsigned long long), s)) != cudaSuccess)
    return fail(e);
  View v = view(sc);
  count_kernel<<<blocks(n_faces), kThreads, 0, s>>>(v, positions_dev, faces_dev, n_faces, counts,
                                                    total);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
  if ((e = cudaMemcpyAsync(&total_h, total, sizeof(total_h), cudaMemcpyDeviceToHost, s)) !=
      cudaSuccess)
    return fail(e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(e);
  if (total_h >= (unsigned long long)kMaxRefs) {
    fail(cudaSuccess);
    return MPL_ERR_UNSUPPORTED;
  }
  sc->n_refs = (int64_t)total_h;
  scan_blocks<<<(unsigned)nb, kThreads, 0, s>>>(counts, sc->start, cells, bsum);
  scan_top<<<1, kThreads, 0, s>>>(bsum, nb);
  scan_add<<<blocks(cells + 1), kThreads, 0, s>>>(sc->start, cells, bsum, (uint32_t)total_h);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&sc->tris, sizeof(float4) * 3 * (total_h > 0 ? total_h : 1))) !=
      cudaSuccess)
    return fail(e);
  if ((e = cudaMalloc(&sc->bound, sizeof(float4) * (total_h > 0 ? total_h : 1))) != cudaSuccess)
    return fail(e);
  if ((e = cudaMalloc(&sc->plane, sizeof(uint2) * (total_h > 0 ? total_h : 1))) != cudaSuccess)
    return fail(e);
  // counts becomes the fill cursor
  if ((e = cudaMemcpyAsync(counts, sc->start, sizeof(uint32_t) * cells, cudaMemcpyDeviceToDevice,
                           s)) != cudaSuccess)
    return fail(e);
  v = view(sc);
  fill_kernel<<<blocks(n_faces), kThreads, 0, s>>>(v, positions_dev, faces_dev, n_faces, counts,
                                                   sc->tris, sc->bound, sc->plane);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(e);
  cudaFree(counts);
  cudaFree(bsum);
  cudaFree(total);
  *out = sc;
  return MPL_OK;
}

extern "C" int mpl_scene_destroy(MplScene* scene) {
  if (!scene) return MPL_OK;
  // queries still queued on any stream read the grid: let them finish
  const cudaError_t e = cudaDeviceSynchronize();
  cudaFree(scene->start);
  cudaFree(scene->tris);
  cudaFree(scene->bound);
  cudaFree(scene->plane);
  delete scene;
  if (e != cudaSuccess) {
    set_last_cuda_error(e);
    return MPL_ERR_CUDA;
  }
  return MPL_OK;
}

extern "C" int mpl_scene_info(const MplScene* scene, float* lo3, float* cell, int32_t* dims3,
                              int64_t* n_refs) {
  if (!scene) return MPL_ERR_INVALID_ARG;
  for (int k = 0; k < 3; ++k) {
    if (lo3) lo3[k] = scene->lo[k];
    if (dims3) dims3[k] = scene->dim[k];
  }
  if (cell) *cell = scene->h;
  if (n_refs) *n_refs = scene->n_refs;
  return MPL_OK;
}

extern "C" int mpl_scene_compute_distance(const MplScene* scene, const float* points_dev,
                                          int64_t n, float* out_dev, void* stream) {
  if (!scene || n < 0 || (n > 0 && (!points_dev || !out_dev))) return MPL_ERR_INVALID_ARG;
  if (n == 0) return MPL_OK;
  const int dst = check_device(scene);
  if (dst != MPL_OK) return dst;
  const View v = view(scene);
  distance_kernel<<<blocks(n), kThreads, 0, (cudaStream_t)stream>>>(v, points_dev, n, out_dev);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}

namespace {
// scratch of one calc_deltas call: the per-iteration maxima and search counts
// (zeroed by the call), then the vertices' state in arrays of their own
struct ScratchLayout {
  int64_t count, state, wit, key, ent, todo, heavy, total;
};
ScratchLayout scratch_layout(int64_t M, int32_t n_iters) {
  auto up = [](int64_t x) { return (x + 255) & ~int64_t(255); };
  ScratchLayout l;
  l.count = up((n_iters + 1) * (int64_t)sizeof(float));
  l.state = l.count + up(n_iters * (int64_t)sizeof(StepCount));
  l.wit = l.state + up(M * (int64_t)sizeof(float4));
  l.key = l.wit + up(M * (int64_t)sizeof(uint2));
  l.ent = l.key + up(M * (int64_t)sizeof(float) * kList);
  l.todo = l.ent + up(M * (int64_t)sizeof(uint32_t) * kList);
  l.heavy = l.todo + up(M * (int64_t)sizeof(uint32_t));
  l.total = l.heavy + up(M * (int64_t)sizeof(uint32_t));
  return l;
}
}  // namespace

extern "C" int mpl_calc_deltas_scratch_bytes(int64_t n_vertices, int32_t n_iters,
                                             int64_t* bytes) {
  if (!bytes || n_vertices < 1 || n_iters < 1) return MPL_ERR_INVALID_ARG;
  *bytes = scratch_layout(n_vertices, n_iters).total;
  return MPL_OK;
}

extern "C" int mpl_calc_deltas(const MplScene* scene, const float* vertices_dev,
                               int64_t n_vertices, int32_t cols, float max_delta, float step0,
                               int32_t n_iters, float eps, void* scratch_dev, float* out_dev,
                               int32_t* iterations_dev, void* stream) {
  if (!scene || !vertices_dev || !out_dev || !scratch_dev || n_vertices < 1 || cols < 6 ||
      n_iters < 1 || !isfinite(max_delta) || !isfinite(step0) || !(eps >= 0.f))
    return MPL_ERR_INVALID_ARG;
  if (((uintptr_t)scratch_dev & 255) != 0) return MPL_ERR_INVALID_ARG;
  const int dst = check_device(scene);
  if (dst != MPL_OK) return dst;
  cudaStream_t s = (cudaStream_t)stream;
  const ScratchLayout lay = scratch_layout(n_vertices, n_iters);
  char* base = (char*)scratch_dev;
  float* maxd = (float*)base;
  Bisect B;
  B.v = vertices_dev;
  B.M = n_vertices;
  B.C = cols;
  B.max_delta = max_delta;
  B.eps = eps;
  B.out = out_dev;
  B.state = (float4*)(base + lay.state);
  B.wit = (uint2*)(base + lay.wit);
  B.key = (float*)(base + lay.key);
  B.ent = (uint32_t*)(base + lay.ent);
  B.todo = (uint32_t*)(base + lay.todo);
  B.heavy = (uint32_t*)(base + lay.heavy);
  StepCount* count = (StepCount*)(base + lay.count);
  MPL_CUDA_TRY(cudaMemsetAsync(base, 0, lay.state, s));  // the maxima and counts
  deltas_init<<<blocks(n_vertices), kThreads, 0, s>>>(B, step0, maxd);
  MPL_LAUNCH_CHECK();
  const View v = view(scene);
  // searches: as many blocks as are resident, each warp taking the next vertex
  const int64_t want = (n_vertices + kThreads / 32 - 1) / (kThreads / 32);
  const int64_t cap = (int64_t)sm_count() * kSearchBlocks;
  const unsigned nsearch = (unsigned)(want < cap ? want : cap);
  const int64_t hcap = cap * 8 / kHeavyWarps;
  const unsigned nheavy = (unsigned)(n_vertices < hcap ? n_vertices : hcap);
  const int64_t resident = (int64_t)sm_count() * kFusedBlocks;
  const int64_t share = (n_vertices + resident - 1) / resident;
  const int per = share < kHeavyWarps ? (int)share : kHeavyWarps;
  const int64_t groups = (n_vertices + per - 1) / per;
  const unsigned nfused = (unsigned)(groups < resident ? groups : resident);
  for (int it = 0; it < n_iters; ++it) {
    if (n_vertices <= kFusedVertices) {
      deltas_fused<<<nfused, kHeavyWarps * 32, 0, s>>>(v, B, maxd, it, per);
      MPL_LAUNCH_CHECK();
      continue;
    }
    deltas_step<<<blocks(n_vertices), kThreads, 0, s>>>(v, B, maxd, count, it);
    MPL_LAUNCH_CHECK();
    deltas_search<1><<<nsearch, kThreads, 0, s>>>(v, B, maxd, count, it);
    MPL_LAUNCH_CHECK();
    deltas_search<kHeavyWarps><<<nheavy, kHeavyWarps * 32, 0, s>>>(v, B, maxd, count, it);
    MPL_LAUNCH_CHECK();
  }
  if (iterations_dev) {
    deltas_count<<<1, 1, 0, s>>>(maxd, n_iters, max_delta, iterations_dev);
    MPL_LAUNCH_CHECK();
  }
  return MPL_OK;
}
