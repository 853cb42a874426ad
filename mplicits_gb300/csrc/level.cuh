// Arguments shared by the level-evaluation kernels.
#pragma once

#include "common.cuh"

namespace mpl {

struct LevelArgs {
  const char* packed;
  PackLayout lay;
  float omega[MPL_MAX_LAYERS];
  MplPoints pts;
  const int32_t* index;  // nullable
  const int32_t* n_dev;  // nullable
  int64_t n;
  float* S;
  int32_t store_mode;
  int32_t has_band;
  float band_delta;
  float band_lower;
  int32_t* band_out;
  int32_t* band_count;
  int64_t band_capacity;
  int* status;  // device status word
  int32_t grad;  // also compute df/dx (forward mode) into G
  float* G;      // [*, 3] gradients, indexed like S (nullable in grad mode)
  // training: pre-activations a_l of every layer and row, FP32 plain GRAD
  // kernel only: pre[((l * n + q) * 4 + row) * WP + j] (row 0 value with bias,
  // rows 1..3 the tangents d/dx, d/dy, d/dz without bias)
  float* pre;
};

__device__ __forceinline__ int64_t level_point_count(const LevelArgs& a) {
  int64_t n = a.n;
  if (a.n_dev) {
    int64_t m = (int64_t)(*a.n_dev);
    n = m < n ? m : n;
  }
  return n < 0 ? 0 : n;
}

// Coordinates of point p (grid index or row of the point list).
__device__ __forceinline__ void point_coords(const LevelArgs& a, int64_t p, float& x, float& y,
                                             float& z) {
  if (a.pts.kind == MPL_POINTS_GRID) {
    grid_point(p, a.pts.grid_n, a.pts.voxel_size, a.pts.offset[0], a.pts.offset[1],
               a.pts.offset[2], x, y, z);
  } else {
    x = a.pts.xyz[3 * p + 0];
    y = a.pts.xyz[3 * p + 1];
    z = a.pts.xyz[3 * p + 2];
  }
}

__device__ __forceinline__ void load_point(const LevelArgs& a, int64_t q, int64_t& p, float& x,
                                           float& y, float& z) {
  p = a.index ? (int64_t)a.index[q] : q;
  point_coords(a, p, x, y, z);
}

// Stores f into S[p] (or adds it) and appends p to the band list when
// |S[p]| < delta.  Called by every lane of a full warp; `valid` masks lanes
// without a point.
__device__ __forceinline__ void store_and_band(const LevelArgs& a, bool valid, int64_t p,
                                               float f);

// As store_and_band, with the value S[p] held before this level already read
// (MPL_ACCUMULATE; ignored in MPL_STORE), so that its load can be issued early.
__device__ __forceinline__ void store_and_band_old(const LevelArgs& a, bool valid, int64_t p,
                                                   float f, float old) {
  float s = f;
  if (valid) {
    if (a.store_mode == MPL_ACCUMULATE) s = __fadd_rn(old, f);
    a.S[p] = s;
  }
  if (a.has_band) {
    const bool keep = valid && fabsf(s) < a.band_delta && fabsf(s) >= a.band_lower;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(a.band_count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) {
      const int64_t pos = (int64_t)base + __popc(m & ((1u << lane) - 1u));
      if (pos < a.band_capacity) a.band_out[pos] = (int32_t)p;
    }
  }
}

__device__ __forceinline__ void store_and_band(const LevelArgs& a, bool valid, int64_t p,
                                               float f) {
  float s = f;
  if (valid) {
    if (a.store_mode == MPL_ACCUMULATE) s = __fadd_rn(a.S[p], f);
    a.S[p] = s;
  }
  if (a.has_band) {
    const bool keep = valid && fabsf(s) < a.band_delta && fabsf(s) >= a.band_lower;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(a.band_count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) {
      const int64_t pos = (int64_t)base + __popc(m & ((1u << lane) - 1u));
      if (pos < a.band_capacity) a.band_out[pos] = (int32_t)p;
    }
  }
}

int launch_level_fp32(const LevelArgs& a, cudaStream_t s);
// Thread layout of the FP32 kernels' register tiles: TX threads along the
// features, the rest along the rows, a warp being 8 x 4 of them (lane bits 0, 3
// and 4 along the features, so that the quarter of a warp that one 16-byte read
// serves at a time is 2 x 4).  With a row of 32 threads along the features, a
// warp's reads of a K row took 10 shared-memory cycles, its stores of the next
// operand 32; gradient of 14,592 points, 256 wide, 295 -> 272 us (lane bits
// 0, 1, 2 along the features 286, bits 0, 1, 3 275, bits 0, 2, 4 274).
template <int TX>
__device__ __forceinline__ void fp32_tile_thread(int tid, int& tx, int& ty) {
  constexpr int WX = TX / 8;  // warps along the features
  const int warp = tid >> 5, lane = tid & 31;
  tx = (warp % WX) * 8 + ((lane & 1) | ((lane >> 2) & 6));
  ty = (warp / WX) * 4 + ((lane >> 1) & 3);
}

// Whether the FP32 gradient and backward kernels run n points in half tiles
// (16 points, two CTAs per SM) instead of full ones (32 points, one CTA): not
// for the smaller width, whose half tiles lose 5-8% everywhere.  In units of a
// full tile's time a wave of pairs measured 1.02-1.06, a half tile with an SM
// to itself 0.61, and a last wave that fills at most half of the SMs 0.4-0.5
// (it starts while the slower half of each pair still runs; beyond that, two
// of its tiles can meet on one SM).  Gradient of n points, 256 wide, full and
// half: 500 99.6 / 60.5 us, 4864 100 / 106, 6000 197 / 149, 7000 197 / 206,
// 12,000 295 / 307, 30,000 683 / 657 (since then both forms are faster: half
// tiles 500 54.6, 6000 129, 30,000 574 us; full ones 4864 88.7, 7000 175).  At 128
// wide the line lies in the same places: 500 63.5 / 53.9 us, 4865 89.1 / 77.2, 7000
// 92.0 / 95.0, 11,000 120 / 104 (full ones taken), 14,592 123 / 125, 15,000 145 / 132.
inline bool half_tiles(int64_t n, int WP) {
  if (WP < 128) return false;
  const int64_t sms = sm_count(), full = (n + 31) / 32, half = (n + 15) / 16;
  if (half <= sms) return true;
  const int64_t rest = half % (2 * sms);
  const double t = 1.05 * (double)(half / (2 * sms)) +
                   (rest == 0 ? 0.0 : (2 * rest <= sms ? 0.5 : 1.05));
  return t < (double)((full + sms - 1) / sms);
}
int launch_level_split(const LevelArgs& a, cudaStream_t s);
int launch_level_bf16(const LevelArgs& a, cudaStream_t s);
int launch_level_f16(const LevelArgs& a, cudaStream_t s);

}  // namespace mpl
