// Marching cubes on the GPU, replacing the CPU call to scikit-image's
// marching_cubes in convert_sdf_samples_to_ply (i3d/meshing.py:291-313)
// and the 512 MiB device->host copy before it (i3d/meshing.py:242).
//
// The volume is C-order [N][N][N]; a *row* is the N points (i, j, 0..N-1).
//   count:  one warp per four rows classifies their points (crossing edges
//           owned by each point) and cells (case -> triangle count) and writes
//           the row totals;
//   scan:   exclusive prefix sums of the row totals (int64);
//   emit:   one CTA per non-empty row rebuilds the in-row vertex prefixes of
//           the four rows a cell touches with warp scans, writes the row's
//           vertices and its triangles.
// Output order is canonical (see mplicits.h) and matches the CPU restatement
// in oracle/mc.c bit for bit: all arithmetic is float32 with explicit
// round-to-nearest intrinsics and no contraction.
#include <atomic>
#include <mutex>

#include "common.cuh"
#include "mc_tables.h"

namespace mpl {

namespace {

__constant__ unsigned char c_tri_count[256];
__constant__ signed char c_tri_edges[256][MPL_MC_MAX_TRIS * 3];
__constant__ signed char c_edge[12][7];

struct McWork {
  int32_t* row_v;   // [N*N]
  int32_t* row_t;   // [N*N]
  int64_t* pre_v;   // [N*N]
  int64_t* pre_t;   // [N*N]
  int64_t* blk;     // [2 * nblk]
  int64_t* totals;  // [2]
};

constexpr int kScanChunk = 2048;  // rows per scan block

__host__ __device__ inline int64_t mc_nblk(int64_t N) {
  return (N * N + kScanChunk - 1) / kScanChunk;
}

__host__ __device__ inline McWork mc_work(void* base, int64_t N) {
  McWork w;
  char* p = (char*)base;
  const int64_t R = N * N;
  w.row_v = (int32_t*)p;
  p += align256(R * 4);
  w.row_t = (int32_t*)p;
  p += align256(R * 4);
  w.pre_v = (int64_t*)p;
  p += align256(R * 8);
  w.pre_t = (int64_t*)p;
  p += align256(R * 8);
  w.blk = (int64_t*)p;
  p += align256(2 * mc_nblk(N) * 8);
  w.totals = (int64_t*)p;
  return w;
}

__host__ inline int64_t mc_work_bytes(int64_t N) {
  const int64_t R = N * N;
  return align256(R * 4) * 2 + align256(R * 8) * 2 + align256(2 * mc_nblk(N) * 8) + 256;
}

// Sign bits (S < iso) of the four values of a line at k (a multiple of 4), bits
// 0..3: one 16-byte load when the grid size is a multiple of 4 (kVec: every
// line then starts 16-byte aligned and ends at a multiple of 4), otherwise
// scalar loads; 0 past N.  Indices are 32-bit (N <= 1024): in 64 bits their
// arithmetic bounded the counting kernel.
template <bool kVec>
__device__ __forceinline__ uint32_t sign4(const float* __restrict__ line, int k, int N,
                                          float iso) {
  uint32_t b = 0;
  if (kVec) {
    if (k < N) {
      const float4 f = *reinterpret_cast<const float4*>(line + k);
      b = (f.x < iso ? 1u : 0u) | (f.y < iso ? 2u : 0u) | (f.z < iso ? 4u : 0u) |
          (f.w < iso ? 8u : 0u);
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) b |= (k + e < N && line[k + e] < iso ? 1u : 0u) << e;
  }
  return b;
}

// Sign of the value after a warp's 128 (lane 31's fifth bit; 0 past the line).
__device__ __forceinline__ uint32_t sign_after(const float* __restrict__ line, int k, int N,
                                               float iso, int lane) {
  return lane == 31 && k + 4 < N && line[k + 4] < iso ? 1u : 0u;
}

// Bits e of a lane with k + e < N, e = 0..4.
__device__ __forceinline__ uint32_t in_line5(int k, int N) {
  const int left = N - k;
  return left >= 5 ? 31u : (left <= 0 ? 0u : (1u << left) - 1u);
}

// One warp per strip of kCountRows rows (i, j..), 128 points per step (4 per
// lane): crossing edges owned by each point (along i, j, k, in that order of
// the mask bits) and the triangle count of each cell (i, j, k) -> (i+1, j+1,
// k+1).
// Bound: L2 and issue.  A strip reads each of its 2 x 5 lines once (a warp per
// row reads every line four times), all of a step's loads are issued before
// the first is used, the fifth sign of a lane comes from its neighbour, and
// the case look-ups are left out where a lane's cells have one sign: with the
// scans, 512 -> 191 us at 512^3 (eight rows 197), 75 -> 41 us at 256^3.
constexpr int kCountRows = 4;

template <bool kVec>
__global__ void __launch_bounds__(256) mc_count_kernel(const float* __restrict__ S, int N,
                                                       float iso, McWork w) {
  constexpr int kLines = kCountRows + 1;
  const int lane = threadIdx.x & 31;
  const int g = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int strips = (N + kCountRows - 1) / kCountRows;
  const int i = g / strips, j0 = (g % strips) * kCountRows;
  if (i >= N) return;
  const bool has_i = i + 1 < N;
  const float* L0 = S + (int64_t)(i * N + j0) * N;
  uint32_t tot[kCountRows] = {};  // vertices | triangles << 16 (at most 3 N and 5 N)
  for (int k0 = 0; k0 < N; k0 += 128) {
    const int k = k0 + 4 * lane;
    uint32_t a[2][kLines];
    uint32_t first = 0, after = 0;  // bit 2 q + p: the lines' first and following signs
#pragma unroll
    for (int q = 0; q < kLines; ++q)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const bool in = j0 + q < N && (p == 0 || has_i);
        const float* line = L0 + p * N * N + q * N;
        a[p][q] = in ? sign4<kVec>(line, k, N, iso) : 0u;
        after |= (in ? sign_after(line, k, N, iso, lane) : 0u) << (2 * q + p);
      }
#pragma unroll
    for (int q = 0; q < kLines; ++q)
#pragma unroll
      for (int p = 0; p < 2; ++p) first |= (a[p][q] & 1u) << (2 * q + p);
    const uint32_t next = __shfl_down_sync(0xffffffffu, first, 1);
    if (lane < 31) after = next;
    const uint32_t in5 = in_line5(k, N);
#pragma unroll
    for (int q = 0; q < kLines; ++q)
#pragma unroll
      for (int p = 0; p < 2; ++p) a[p][q] |= ((after >> (2 * q + p)) & 1u) << 4;
#pragma unroll
    for (int q = 0; q < kCountRows; ++q) {
      const bool has_j = j0 + q + 1 < N;
      if (j0 + q >= N) break;
      const uint32_t s = a[0][q], b = has_i ? a[1][q] : s, c = has_j ? a[0][q + 1] : s;
      const uint32_t d = has_i && has_j ? a[1][q + 1] : s;
      if (((s | b | c | d) == 0u) || ((s & b & c & d) == in5)) continue;  // one sign
      const uint32_t pts = in5 & 15u, cells = in5 >> 1;  // points, points with a successor
      uint32_t v = __popc((s ^ b) & pts) + __popc((s ^ c) & pts) + __popc((s ^ (s >> 1)) & cells);
      if (has_i && has_j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (!((cells >> e) & 1u)) continue;
          // corner: (i + (x & 1), j + ((x >> 1) & 1), k + e + (x >> 2))
          const uint32_t cs = ((s >> e) & 1u) | (((b >> e) & 1u) << 1) | (((c >> e) & 1u) << 2) |
                              (((d >> e) & 1u) << 3) | (((s >> (e + 1)) & 1u) << 4) |
                              (((b >> (e + 1)) & 1u) << 5) | (((c >> (e + 1)) & 1u) << 6) |
                              (((d >> (e + 1)) & 1u) << 7);
          v += (uint32_t)c_tri_count[cs] << 16;
        }
      }
      tot[q] += v;
    }
  }
#pragma unroll
  for (int q = 0; q < kCountRows; ++q) {
    const uint32_t t = __reduce_add_sync(0xffffffffu, tot[q]);
    if (lane == 0 && j0 + q < N) {
      w.row_v[i * N + j0 + q] = (int32_t)(t & 0xffffu);
      w.row_t[i * N + j0 + q] = (int32_t)(t >> 16);
    }
  }
}

int launch_count(const float* S, int64_t N, float iso, const McWork& w, cudaStream_t s) {
  const int64_t warps = N * ((N + kCountRows - 1) / kCountRows);
  const unsigned grid = (unsigned)((warps + 7) / 8);
  if ((N & 3) == 0)
    mc_count_kernel<true><<<grid, 256, 0, s>>>(S, (int)N, iso, w);
  else
    mc_count_kernel<false><<<grid, 256, 0, s>>>(S, (int)N, iso, w);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}

// block-wide exclusive scan of one int64 per thread (blockDim.x a multiple
// of 32, at most 256)
__device__ int64_t block_exclusive_scan(int64_t v, int64_t* total) {
  __shared__ int64_t warp_sums[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  int64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int64_t s = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) warp_sums[lane] = s;
  }
  __syncthreads();
  const int64_t before = wid > 0 ? warp_sums[wid - 1] : 0;
  if (total) *total = warp_sums[nw - 1];
  __syncthreads();
  return before + x - v;
}

// phase 1: per-block exclusive scan of kScanChunk rows (256 threads x 8)
__global__ void mc_scan_blocks(int64_t N, McWork w) {
  const int64_t R = N * N;
  const int64_t base = (int64_t)blockIdx.x * kScanChunk + threadIdx.x * 8;
  int64_t lv[8], lt[8], sv = 0, st = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int64_t r = base + q;
    lv[q] = r < R ? w.row_v[r] : 0;
    lt[q] = r < R ? w.row_t[r] : 0;
    sv += lv[q];
    st += lt[q];
  }
  int64_t tv, tt;
  int64_t ov = block_exclusive_scan(sv, &tv);
  int64_t ot = block_exclusive_scan(st, &tt);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int64_t r = base + q;
    if (r < R) {
      w.pre_v[r] = ov;
      w.pre_t[r] = ot;
    }
    ov += lv[q];
    ot += lt[q];
  }
  if (threadIdx.x == 0) {
    w.blk[2 * blockIdx.x] = tv;
    w.blk[2 * blockIdx.x + 1] = tt;
  }
}

// phase 2: one CTA scans the block totals in place, writes the grand totals
__global__ void mc_scan_top(int64_t nblk, McWork w, int64_t* counts_out) {
  int64_t carry_v = 0, carry_t = 0;
  for (int64_t b0 = 0; b0 < nblk; b0 += blockDim.x) {
    const int64_t b = b0 + threadIdx.x;
    const int64_t v = b < nblk ? w.blk[2 * b] : 0;
    const int64_t t = b < nblk ? w.blk[2 * b + 1] : 0;
    int64_t tv, tt;
    const int64_t ev = block_exclusive_scan(v, &tv);
    const int64_t et = block_exclusive_scan(t, &tt);
    if (b < nblk) {
      w.blk[2 * b] = carry_v + ev;
      w.blk[2 * b + 1] = carry_t + et;
    }
    carry_v += tv;
    carry_t += tt;
  }
  if (threadIdx.x == 0) {
    w.totals[0] = carry_v;
    w.totals[1] = carry_t;
    if (counts_out) {
      counts_out[0] = carry_v;
      counts_out[1] = carry_t;
    }
  }
}

// phase 3: add block offsets
__global__ void mc_scan_add(int64_t N, McWork w) {
  const int64_t R = N * N;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= R) return;
  const int64_t b = r / kScanChunk;
  w.pre_v[r] += w.blk[2 * b];
  w.pre_t[r] += w.blk[2 * b + 1];
}

// Central difference at point p along the axis of the given stride, one-sided at
// the first and last of the N points (x: the point's index on the axis).
__device__ __forceinline__ float grad_axis(const float* __restrict__ S, int N, int p, int x,
                                           int stride) {
  const int lo = x > 0 ? 1 : 0, hi = x + 1 < N ? 1 : 0;
  const float d = __fsub_rn(S[p + hi * stride], S[p - lo * stride]);
  return __fdiv_rn(d, (float)(hi + lo));
}

constexpr int kEmitThreads = 128;
constexpr int kMaxN = 1024;

// One warp: the crossing-edge masks (with the point's sign in bit 3) and the
// in-line vertex prefix of line (ri, rj), kSteps x 128 points at a time, and
// (list given) the line's vertices as 4 k + axis.  Returns their number.
template <int kSteps, bool kVec>
__device__ __forceinline__ int emit_line(const float* __restrict__ S, int N, float iso, int ri,
                                         int rj, int lane, int16_t* pre, uint8_t* msk,
                                         uint16_t* list) {
  const bool has_i = ri + 1 < N, has_j = rj + 1 < N;
  const float* L = S + (ri * N + rj) * N;
  int carry = 0;
  for (int k0 = 0; k0 < N; k0 += 128 * kSteps) {
    uint32_t a[kSteps], b[kSteps], c[kSteps], after[kSteps];
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
      const int k = k0 + 128 * t + 4 * lane;
      a[t] = sign4<kVec>(L, k, N, iso);
      after[t] = sign_after(L, k, N, iso, lane);
      b[t] = has_i ? sign4<kVec>(L + N * N, k, N, iso) : a[t];
      c[t] = has_j ? sign4<kVec>(L + N, k, N, iso) : a[t];
    }
    uint64_t x = 0;  // vertices of the lane's points, 16 bits a step (at most 12)
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
      const int k = k0 + 128 * t + 4 * lane;
      const uint32_t next = __shfl_down_sync(0xffffffffu, a[t], 1);
      a[t] |= (lane < 31 ? next & 1u : after[t]) << 4;
      const uint32_t in5 = in_line5(k, N), pts = in5 & 15u, succ = in5 >> 1;
      b[t] = (a[t] ^ b[t]) & pts;           // from here on the crossings along i,
      c[t] = (a[t] ^ c[t]) & pts;           // along j
      after[t] = (a[t] ^ (a[t] >> 1)) & succ;  // and along k
      x |= (uint64_t)(__popc(b[t]) + __popc(c[t]) + __popc(after[t])) << (16 * t);
    }
    const uint64_t own = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const uint64_t total = __shfl_sync(0xffffffffu, x, 31);
    x -= own;
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
      const int k = k0 + 128 * t + 4 * lane;
      int run = carry + (int)((x >> (16 * t)) & 0xffffu);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (k + e < N) {
          const uint32_t m = ((b[t] >> e) & 1u) | (((c[t] >> e) & 1u) << 1) |
                             (((after[t] >> e) & 1u) << 2);
          pre[k + e] = (int16_t)run;
          msk[k + e] = (uint8_t)(m | (((a[t] >> e) & 1u) << 3));
          if (list) {
#pragma unroll
            for (int ax = 0; ax < 3; ++ax)
              if ((m >> ax) & 1u) list[run + __popc(m & ((1u << ax) - 1u))] = (uint16_t)(4 * (k + e) + ax);
          }
          run += __popc(m);
        }
      }
      carry += (int)((total >> (16 * t)) & 0xffffu);
    }
  }
  return carry;
}

// One CTA (4 warps) per row r = (i, j); rows without vertices or triangles
// return at once.
//   1. warp w walks line (i + (w >> 1), j + (w & 1)), 512 points per step (128
//      where the line is no longer): the crossing-edge mask and sign bit of
//      each point and its in-line vertex prefix (warp scan), into shared
//      memory, and for line (i, j) the list of its vertices;
//   2. the vertices of line (i, j), one a thread (interpolation,
//      central-difference normals);
//   3. the triangles of the cells of row (i, j): each thread takes four
//      consecutive cells, the cases come from the sign bits of the four
//      lines, one block scan orders them.
// Bound: latency (a chain of loads, scans and barriers per row, ten CTAs
// per SM).  The loads of a step are all issued before the first is used, the
// four scans of a step are one, the vertices come from a list, indices are
// 32-bit: 1015 -> 593 us at 512^3 (459,208 vertices), 191 -> 130 us at 256^3.
// Ten CTAs per SM in the launch bounds: 9 646, 11 658, 12 657 us; several rows
// per CTA are no faster (2: 669, 8: 674 us with 12).
template <bool kVec>
__global__ void __launch_bounds__(kEmitThreads, 10) mc_emit_kernel(
    const float* __restrict__ S, int N, float iso, float vs, float o0, float o1, float o2,
    McWork w, float* __restrict__ verts, float* __restrict__ normals, float* __restrict__ values,
    int32_t* __restrict__ faces, int64_t max_verts, int64_t max_tris) {
  // in-line vertex prefix (< 3 kMaxN) and, per point, the crossing-edge mask
  // (bits 0-2: along i, j, k) with the point's sign S < iso in bit 3
  __shared__ int16_t pre[4][kMaxN];
  __shared__ __align__(4) uint8_t msk[4][kMaxN];
  __shared__ uint16_t list[3 * kMaxN];  // vertices of line (i, j): 4 k + axis
  __shared__ int64_t line_v[4];         // first vertex of the four lines
  __shared__ int line_n;                // vertices of line (i, j)
  const int r = blockIdx.x;
  const int i = r / N, j = r % N;
  if (w.row_v[r] == 0 && w.row_t[r] == 0) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const float org[3] = {o0, o1, o2};

  // 1. masks, prefixes and signs of the four lines
  {
    const int ri = i + (wid >> 1), rj = j + (wid & 1);
    if (ri < N && rj < N) {
      if (lane == 0) line_v[wid] = w.pre_v[ri * N + rj];
      uint16_t* own = wid == 0 ? list : nullptr;
      const int cnt = N <= 128
                          ? emit_line<1, kVec>(S, N, iso, ri, rj, lane, pre[wid], msk[wid], own)
                          : emit_line<4, kVec>(S, N, iso, ri, rj, lane, pre[wid], msk[wid], own);
      if (wid == 0 && lane == 0) line_n = cnt;
    }
  }
  __syncthreads();

  // 2. vertices of line (i, j)
  const int64_t vbase = line_v[0];
  const int nv = line_n;
  for (int q = threadIdx.x; q < nv; q += kEmitThreads) {
    const int64_t v = vbase + q;
    if (v >= max_verts) break;
    const int a = list[q] & 3;
    const int k = list[q] >> 2;
    const int idx0[3] = {i, j, k};
    const int stride[3] = {N * N, N, 1};
    const int p0 = r * N + k, p1 = p0 + (a == 0 ? N * N : (a == 1 ? N : 1));
    const float v0 = S[p0], v1 = S[p1];
    const float t = __fdiv_rn(__fsub_rn(iso, v0), __fsub_rn(v1, v0));
    float n[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      float c = (float)idx0[d];
      if (d == a) c = __fadd_rn(c, t);
      verts[3 * v + d] = __fadd_rn(__fmul_rn(c, vs), org[d]);
      const float g0 = grad_axis(S, N, p0, idx0[d], stride[d]);
      const float g1 = grad_axis(S, N, p1, idx0[d] + (d == a), stride[d]);
      n[d] = __fadd_rn(g0, __fmul_rn(t, __fsub_rn(g1, g0)));
    }
    float l2 = __fmul_rn(n[0], n[0]);
    l2 = __fadd_rn(l2, __fmul_rn(n[1], n[1]));
    l2 = __fadd_rn(l2, __fmul_rn(n[2], n[2]));
    const float len = __fsqrt_rn(l2);
#pragma unroll
    for (int d = 0; d < 3; ++d) normals[3 * v + d] = len > 0.0f ? __fdiv_rn(n[d], len) : 0.0f;
    if (values) values[v] = v0 > v1 ? v0 : v1;
  }

  // 3. triangles of the cells of row (i, j), four consecutive cells a thread
  if (i + 1 >= N || j + 1 >= N) return;
  int64_t tcarry = w.pre_t[r];
  for (int k0 = 0; k0 < N - 1; k0 += 4 * kEmitThreads) {
    const int kb = k0 + 4 * threadIdx.x;
    // signs of the four lines (line (di, dj) = di * 2 + dj) at kb .. kb + 4
    const uint32_t in5 = in_line5(kb, N);
    uint32_t sg[4] = {}, any = 0, all = 31;
    if (kb < N) {
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const uint32_t x = (*reinterpret_cast<const uint32_t*>(&msk[l][kb]) >> 3) & 0x01010101u;
        sg[l] = (x | (x >> 7) | (x >> 14) | (x >> 21)) & 15u;
        if (kb + 4 < N) sg[l] |= ((uint32_t)msk[l][kb + 4] >> 3 & 1u) << 4;
        sg[l] &= in5;
        any |= sg[l];
        all &= sg[l];
      }
    }
    int cs[4] = {}, nts[4] = {}, ntot = 0;
    if (any && all != in5) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // corner q: (i + (q & 1), j + ((q >> 1) & 1), k + (q >> 2))
        if (!((in5 >> (e + 1)) & 1u)) break;
        int c = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          c |= (int)((sg[((q & 1) << 1) | ((q >> 1) & 1)] >> (e + (q >> 2))) & 1u) << q;
        cs[e] = c;
        nts[e] = c_tri_count[c];
        ntot += nts[e];
      }
    }
    int64_t tot;
    int64_t t = tcarry + block_exclusive_scan(ntot, &tot);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = kb + e;
      for (int q = 0; q < nts[e]; ++q, ++t) {
        if (t >= max_tris) break;
#pragma unroll
        for (int sidx = 0; sidx < 3; ++sidx) {
          const int ed = c_tri_edges[cs[e]][3 * q + sidx];
          const int axis = c_edge[ed][0];
          const int row = c_edge[ed][1] * 2 + c_edge[ed][2];
          const int kk = k + c_edge[ed][3];
          const int64_t vid = line_v[row] + pre[row][kk] +
                              __popc((int)msk[row][kk] & ((1 << axis) - 1));
          faces[3 * t + sidx] = (int32_t)vid;
        }
      }
    }
    tcarry += tot;
  }
}

int launch_emit(const float* S, int64_t N, float iso, float vs, const float* origin,
                const McWork& w, float* verts, float* normals, float* values, int32_t* faces,
                int64_t max_verts, int64_t max_tris, cudaStream_t s) {
  auto* kernel = (N & 3) == 0 ? &mc_emit_kernel<true> : &mc_emit_kernel<false>;
  kernel<<<(unsigned)(N * N), kEmitThreads, 0, s>>>(S, (int)N, iso, vs, origin[0], origin[1],
                                                    origin[2], w, verts, normals, values, faces,
                                                    max_verts, max_tris);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}

// Per-device one-time set-up (case tables here, the no-allocation
// workspace's address below): the flags are read without a lock on the fast
// path; the first calls on a device, from any number of host threads,
// serialise on g_setup_mutex, so the upload happens once.
std::atomic<bool> g_tables_loaded[64];
std::mutex g_setup_mutex;

int ensure_tables() {
  int dev = 0;
  MPL_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return MPL_ERR_INVALID_ARG;
  if (g_tables_loaded[dev].load(std::memory_order_acquire)) return MPL_OK;
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (g_tables_loaded[dev].load(std::memory_order_relaxed)) return MPL_OK;
  MPL_CUDA_TRY(cudaMemcpyToSymbol(c_tri_count, MPL_MC_TRI_COUNT, sizeof(MPL_MC_TRI_COUNT)));
  MPL_CUDA_TRY(cudaMemcpyToSymbol(c_tri_edges, MPL_MC_TRI_EDGES, sizeof(MPL_MC_TRI_EDGES)));
  MPL_CUDA_TRY(cudaMemcpyToSymbol(c_edge, MPL_MC_EDGE, sizeof(MPL_MC_EDGE)));
  g_tables_loaded[dev].store(true, std::memory_order_release);
  return MPL_OK;
}

}  // namespace

}  // namespace mpl

using namespace mpl;

extern "C" int mpl_mc_workspace_bytes(int64_t N, int64_t* bytes) {
  if (!bytes || N < 2 || N > kMaxN) return N > kMaxN ? MPL_ERR_UNSUPPORTED : MPL_ERR_INVALID_ARG;
  *bytes = mc_work_bytes(N);
  return MPL_OK;
}

extern "C" int mpl_mc_count(const float* S, int64_t N, float iso, void* workspace,
                            int64_t* counts_dev, void* stream) {
  if (!S || !workspace || N < 2) return MPL_ERR_INVALID_ARG;
  if (N > kMaxN) return MPL_ERR_UNSUPPORTED;
  if (((uintptr_t)workspace & 255) != 0) return MPL_ERR_INVALID_ARG;
  int st = ensure_tables();
  if (st != MPL_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  McWork w = mc_work(workspace, N);
  const int64_t R = N * N;
  st = launch_count(S, N, iso, w, s);
  if (st != MPL_OK) return st;
  const int64_t nblk = mc_nblk(N);
  mc_scan_blocks<<<(unsigned)nblk, 256, 0, s>>>(N, w);
  MPL_LAUNCH_CHECK();
  mc_scan_top<<<1, 256, 0, s>>>(nblk, w, counts_dev);
  MPL_LAUNCH_CHECK();
  mc_scan_add<<<(unsigned)((R + 255) / 256), 256, 0, s>>>(N, w);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}

extern "C" int mpl_mc_emit(const float* S, int64_t N, float iso, float voxel_size,
                           const float* origin, const void* workspace, float* verts,
                           float* normals, float* values, int32_t* faces, int64_t max_verts,
                           int64_t max_tris, void* stream) {
  if (!S || !workspace || !origin || N < 2) return MPL_ERR_INVALID_ARG;
  if (N > kMaxN) return MPL_ERR_UNSUPPORTED;
  if ((max_verts > 0 && (!verts || !normals)) || (max_tris > 0 && !faces))
    return MPL_ERR_INVALID_ARG;
  int st = ensure_tables();
  if (st != MPL_OK) return st;
  cudaStream_t s = (cudaStream_t)stream;
  McWork w = mc_work(const_cast<void*>(workspace), N);
  return launch_emit(S, N, iso, voxel_size, origin, w, verts, normals, values, faces, max_verts,
                     max_tris, s);
}

// ---------------------------------------------------------------------------
// Marching cubes without any allocation, for callers that cannot allocate
// device memory.  A real-time frame loop cannot afford cudaMalloc/cudaFree,
// which synchronise the whole device, and a host that hands this library
// only buffers it registered itself (an engine plug-in, or a foreign-language
// binding without access to a CUDA allocator) has no way to provide the
// workspace mpl_mc_count/mpl_mc_emit need.  This entry point keeps that
// workspace in a fixed file-scope device array instead, sized for grids up
// to kStaticMaxN^3, which every GPU that loads the library holds until the
// process exits.
// ---------------------------------------------------------------------------
namespace mpl {

namespace {

constexpr int64_t kStaticMaxN = 256;

constexpr int64_t static_align256(int64_t x) { return (x + 255) & ~int64_t(255); }

constexpr int64_t static_ws_bytes(int64_t N) {
  return static_align256(N * N * 4) * 2 + static_align256(N * N * 8) * 2 +
         static_align256(2 * ((N * N + kScanChunk - 1) / kScanChunk) * 8) + 256;
}

// 1.5 MiB: the count/prefix workspace of a 256^3 grid.
__device__ __align__(256) unsigned char g_mc_static_ws[static_ws_bytes(kStaticMaxN)];

// Device address of g_mc_static_ws on the current device.  In host code the
// symbol itself is only a host-side stand-in, so the address is looked up
// once per device (with that device current) and cached.
int static_ws_address(void** out) {
  static std::atomic<void*> cached[64];
  int dev = 0;
  MPL_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return MPL_ERR_INVALID_ARG;
  void* p = cached[dev].load(std::memory_order_acquire);
  if (!p) {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    p = cached[dev].load(std::memory_order_relaxed);
    if (!p) {
      MPL_CUDA_TRY(cudaGetSymbolAddress(&p, g_mc_static_ws));
      cached[dev].store(p, std::memory_order_release);
    }
  }
  *out = p;
  return MPL_OK;
}

}  // namespace

}  // namespace mpl

extern "C" int mpl_mc_noalloc(const float* S, int64_t N, float iso, float voxel_size,
                              const float* origin, float* verts, float* normals, float* values,
                              int32_t* faces, int64_t max_verts, int64_t max_tris,
                              int64_t* counts_dev, void* stream) {
  if (!S || !origin || !counts_dev || N < 2) return MPL_ERR_INVALID_ARG;
  if (N > kStaticMaxN || mc_work_bytes(N) > (int64_t)sizeof(g_mc_static_ws))
    return MPL_ERR_CAPACITY;
  if (max_verts < 0 || max_tris < 0) return MPL_ERR_INVALID_ARG;
  if ((max_verts > 0 && (!verts || !normals)) || (max_tris > 0 && !faces))
    return MPL_ERR_INVALID_ARG;
  int st = ensure_tables();
  if (st != MPL_OK) return st;
  void* ws = nullptr;
  st = static_ws_address(&ws);
  if (st != MPL_OK) return st;
  // Every workspace entry the kernels read is written earlier in this same
  // call, so the previous call's leftovers need no clearing.
  cudaStream_t s = (cudaStream_t)stream;
  McWork w = mc_work(ws, N);
  const int64_t R = N * N;
  st = launch_count(S, N, iso, w, s);
  if (st != MPL_OK) return st;
  const int64_t nblk = mc_nblk(N);
  mc_scan_blocks<<<(unsigned)nblk, 256, 0, s>>>(N, w);
  MPL_LAUNCH_CHECK();
  mc_scan_top<<<1, 256, 0, s>>>(nblk, w, counts_dev);
  MPL_LAUNCH_CHECK();
  mc_scan_add<<<(unsigned)((R + 255) / 256), 256, 0, s>>>(N, w);
  MPL_LAUNCH_CHECK();
  return launch_emit(S, N, iso, voxel_size, origin, w, verts, normals, values, faces, max_verts,
                     max_tris, s);
}
