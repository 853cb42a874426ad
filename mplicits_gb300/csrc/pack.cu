// Weight packing: nn.Linear tensors -> the device image the level kernels
// read.  Replaces the per-layer CUTLASS tensors of the reference renderer
// (renderer/cuda/gemms.cu:5-100, loaded by tools.cu:81-111).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <string.h>

#include "common.cuh"

namespace mpl {

int make_layout(const MplNet* net, PackLayout* lay) {
  if (!net || !lay) return MPL_ERR_INVALID_ARG;
  const int L = net->n_layers;
  if (L < 2 || L > MPL_MAX_LAYERS) return MPL_ERR_UNSUPPORTED;
  if (net->dims[0] != 3 || net->dims[L] != 1) return MPL_ERR_UNSUPPORTED;
  int wmax = 0;
  for (int l = 1; l < L; ++l) {
    if (net->dims[l] < 1 || net->dims[l] > 256) return MPL_ERR_UNSUPPORTED;
    wmax = net->dims[l] > wmax ? net->dims[l] : wmax;
  }
  const int WP = wmax <= 64 ? 64 : (wmax <= 128 ? 128 : 256);
  lay->L = L;
  lay->WP = WP;
  lay->nh = L - 2;
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    int64_t at = o;
    o = align256(o + bytes);
    return at;
  };
  lay->w0t = take(3 * WP * 4);
  lay->b0 = take(WP * 4);
  for (int l = 0; l < MPL_MAX_LAYERS; ++l) {
    lay->wht[l] = lay->bh[l] = lay->hb[l] = lay->hw[l] = lay->hwT[l] = lay->hbx[l] = -1;
    lay->hwh[l] = lay->hbxh[l] = lay->whn[l] = lay->hwTh[l] = -1;
    lay->ws[l] = lay->us[l] = lay->eq[l] = -1;
  }
  for (int l = 1; l <= L - 2; ++l) {
    lay->wht[l] = take((int64_t)WP * WP * 4);
    lay->bh[l] = take(WP * 4);
  }
  lay->wout = take(WP * 4);
  lay->bout = take(16);
  lay->w0f = take(WP * 16);
  for (int l = 1; l <= L - 2; ++l) {
    lay->hb[l] = take(WP * 4);
    lay->hw[l] = take((int64_t)WP * WP * 2);
    lay->hwT[l] = take((int64_t)WP * WP * 2);
    lay->hbx[l] = take((int64_t)WP * 16 * 2);
    lay->hwh[l] = take((int64_t)WP * WP * 2);
    lay->hbxh[l] = take((int64_t)WP * 16 * 2);
    lay->whn[l] = take((int64_t)WP * WP * 4);
    lay->hwTh[l] = take((int64_t)WP * WP * 2);
  }
  lay->w0u = take((4 * WP + 4) * 4);
  lay->ub = take(MPL_MAX_LAYERS * 16);
  for (int l = 1; l <= L - 2; ++l) {
    lay->ws[l] = take((int64_t)WP * WP * 4);
    lay->us[l] = take((int64_t)WP * 4);
    lay->eq[l] = take((int64_t)2 * WP * 4);
  }
  lay->total = o;
  return MPL_OK;
}

// offset (in elements) of (row n, col k) in the K-chunked core-matrix tiling
__device__ __forceinline__ int64_t umma_tile_offset(int n, int k, int WP) {
  const int c = k >> 6, kk = k & 63;
  return (int64_t)c * WP * 64 + ((int64_t)(n >> 3) * 8 + (kk >> 3)) * 64 + (n & 7) * 8 + (k & 7);
}

struct PackHidden {
  const float *W, *b;
  int out, in;
  float omega;
  double turns;  // omega / pi
  float *wt, *bh, *hb, *whn, *us, *ub, *eq;
  const float* eq_in;  // of the layer before; null for the first hidden one
  __nv_bfloat16 *hw, *hwT, *hbx;
  __half *hwh, *hwTh, *hbxh, *ws;
};
struct PackArgs {
  const float *W0, *b0, *Wl, *bl;  // first and output layer
  int out0, inl, WP;
  float omega0;
  double turns0;
  float *w0t, *b0p, *w0f, *w0u, *wout, *bout;
  PackHidden hid[MPL_MAX_LAYERS];
};

// maximum of non-negative v over the block (NaN ignored), to every thread
__device__ __forceinline__ float block_max(float v) {
  __shared__ float s[8];
#pragma unroll
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  v = s[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = fmaxf(v, s[w]);
  return v;
}

// e of the smallest 2^e that a magnitude does not exceed (up to rounding); 0 for
// 0, an infinity or a NaN; within the range whose powers are normal floats
__device__ __forceinline__ int magnitude_exponent(float m) {
  int e = 0;
  if (isfinite(m) && m > 0.f) frexpf(m, &e);
  return e < -110 ? -110 : e;
}

constexpr float kNormScale = 1073741824.f;

// Row bounds of a hidden layer (blockIdx.y; one block of WP threads per row):
// |phase| <= sum |w'| + |b'|, since activations are at most 1, and the power of
// two that brings a small activation up to 1: mostly about pi times the 2-norm of
// (w', b'), and by Cauchy-Schwarz never above 17 times that, which FP16 holds.
// (The bound itself is some 18 times the usual activation of a 256-wide row:
// scaled by it, phases of 2^-6 gave outputs five times as far from float64.)
__global__ void pack_rows(const PackArgs a) {
  const PackHidden& h = a.hid[blockIdx.y];
  const int n = blockIdx.x, k = threadIdx.x;
  float sum = 0.f;
  if (n < h.out && k < h.in) sum = fabsf((float)(h.turns * (double)h.W[(int64_t)n * h.in + k]));
  // squares of 2^30 times the values, so that those of 2^-60 are still normal (in
  // double the launch takes 7.0 us instead of 4.3: a training step packs each time)
  float sq = (sum * kNormScale) * (sum * kNormScale);
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  __shared__ float part[8];
  __shared__ float part2[8];
  if ((k & 31) == 0) part[k >> 5] = sum, part2[k >> 5] = sq;
  __syncthreads();
  if (k == 0) {
    const float bu = n < h.out ? (float)(h.turns * (double)h.b[n]) : 0.f;
    float t = fabsf(bu);
    sq = (bu * kNormScale) * (bu * kNormScale);
    for (int i = 0; i < a.WP / 32; ++i) t += part[i], sq += part2[i];
    h.us[n] = bu;
    // non-negative floats order as their bits, infinity and NaN last
    atomicMax(reinterpret_cast<unsigned int*>(h.ub), __float_as_uint(fabsf(t)));
    int p = -magnitude_exponent(sqrtf(sq) * (3.2f / kNormScale));
    p = p < 0 ? 0 : (p > 60 ? 60 : p);
    h.eq[n] = ldexpf(1.f, p);
    if (p) h.ub[2] = 1.f;
  }
}

// 2^e, |e| <= 1022
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// omega / pi W of one element, the column scaled as its activation is
__device__ __forceinline__ double split_weight(const PackHidden& h, float w, int k) {
  const double u = h.turns * (double)w;
  return h.eq_in ? u * (double)__frcp_rn(h.eq_in[k]) : u;  // a power of two: exact
}

// largest such magnitude of each hidden layer into its ub[1] (zeroed before);
// one block of WP threads per row
__global__ void pack_range(const PackArgs a) {
  const PackHidden& h = a.hid[blockIdx.y];
  const int n = blockIdx.x, k = threadIdx.x;
  float m = 0.f;
  if (n < h.out && k < h.in)
    m = fabsf((float)split_weight(h, h.W[(int64_t)n * h.in + k], k));
  m = block_max(m);
  if (k == 0) atomicMax(reinterpret_cast<unsigned int*>(h.ub + 1), __float_as_uint(m));
}

// Rows more powers of two than this below their layer's largest are packed at a
// scale of their own: at the layer's, the lo parts of a row at 2^-17 of it leave
// FP16's normal range (phase of such a row 3e-7 off at 2^-17, 6e-5 at 2^-25).
constexpr int kSplitRange = 14;

// One block of WP threads per row of a hidden layer (blockIdx.y - 1), and one
// (blockIdx.y = 0, x = 0) for the first and output layers: the whole image in
// one launch (a training step packs the level it has just updated).
__global__ void pack_level(const PackArgs a) {
  const int WP = a.WP, k = threadIdx.x;
  if (blockIdx.y == 0) {
    if (blockIdx.x != 0) return;
    const bool v = k < a.out0;
    float mag[4];
    for (int c = 0; c < 4; ++c) {
      const float w = !v ? 0.f : (c < 3 ? a.W0[k * 3 + c] : a.b0[k]);
      const float u = (float)(a.turns0 * (double)w);
      if (c < 3)
        a.w0t[c * WP + k] = w;
      else
        a.b0p[k] = w;
      a.w0f[c * WP + k] = a.omega0 * w;
      a.w0u[c * WP + k] = u;
      // a NaN weight makes the bound infinite: such phases need no fast path
      mag[c] = u == u ? fabsf(u) : INFINITY;
    }
    for (int c = 0; c < 4; ++c) {
      const float mx = block_max(mag[c]);
      if (k == 0) a.w0u[4 * WP + c] = mx;
    }
    a.wout[k] = k < a.inl ? a.Wl[k] : 0.f;
    if (k < 4) a.bout[k] = k == 0 ? a.bl[0] : 0.f;
    return;
  }
  const PackHidden& h = a.hid[blockIdx.y - 1];
  const int n = blockIdx.x;  // output row; k: input column
  const float w = (n < h.out && k < h.in) ? h.W[(int64_t)n * h.in + k] : 0.f;
  h.wt[(int64_t)k * WP + n] = w;
  h.whn[(int64_t)n * WP + k] = w;
  h.hw[umma_tile_offset(n, k, WP)] = __float2bfloat16_rn(h.omega * w);
  h.hwT[umma_tile_offset(k, n, WP)] = __float2bfloat16_rn(h.omega * w);
  h.hwh[umma_tile_offset(n, k, WP)] = __float2half_rn(h.omega * w);
  h.hwTh[umma_tile_offset(k, n, WP)] = __float2half_rn(h.omega * w);
  // bias tile of the MMA (PackLayout::hbx): row n, K columns 0 and 1 of 16
  const float bb = n < h.out ? h.b[n] : 0.f;
  const float v = h.omega * bb;
  if (k < 16) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __half hh = __float2half_rn(v);
    const int at = ((n >> 3) * 2 + (k >> 3)) * 64 + (n & 7) * 8 + (k & 7);
    h.hbx[at] = k == 0 ? hi
                       : (k == 1 ? __float2bfloat16_rn(v - __bfloat162float(hi))
                                 : __float2bfloat16_rn(0.f));
    h.hbxh[at] = k == 0 ? hh : (k == 1 ? __float2half_rn(v - __half2float(hh))
                                       : __float2half_rn(0.f));
  }
  if (k == 0) {
    h.bh[n] = bb;
    h.hb[n] = v;
  }
  // split parts: 2^k puts the layer's largest magnitude into [2^14, 2^15], or the
  // row's own where that is more than kSplitRange powers of two smaller; the
  // row's hi parts are multiples of 2^(e - 11), e its own largest exponent
  const double wu = split_weight(h, w, k);
  const float mx = block_max(fabsf((float)wu));
  const int el = magnitude_exponent(h.ub[1]), er = magnitude_exponent(mx);
  const bool own = mx > 0.f && isfinite(mx) && er < el - kSplitRange;
  const int k2 = 15 - (own ? er : el);
  if (k == 0) {
    h.eq[WP + n] = own ? (float)pow2(er - el) : 1.f;
    if (own) h.ub[0] = INFINITY;
    if (n == 0) h.ub[3] = (float)pow2(el - 15);
  }
  const double wn = wu * pow2(k2);
  const int eu = er + k2 - 11;
  const double hi = rint(wn * pow2(-eu)) * pow2(eu);
  const int kk = k % kSplitK;
  __half* dst = h.ws + (int64_t)(k / kSplitK) * 2 * WP * kSplitK +
                ((n >> 3) * (kSplitK / 8) + (kk >> 3)) * 64 + (n & 7) * 8 + (kk & 7);
  dst[0] = __float2half_rn((float)hi);
  dst[(int64_t)WP * kSplitK] = __float2half_rn((float)(wn - hi));
}

}  // namespace mpl

using namespace mpl;

extern "C" int mpl_net_packed_bytes(const MplNet* net, int64_t* bytes) {
  if (!bytes) return MPL_ERR_INVALID_ARG;
  PackLayout lay;
  int st = make_layout(net, &lay);
  if (st != MPL_OK) return st;
  *bytes = lay.total;
  return MPL_OK;
}

extern "C" int mpl_net_pack(const MplNet* net, const float* const* weights,
                            const float* const* biases, void* packed, void* stream) {
  PackLayout lay;
  int st = make_layout(net, &lay);
  if (st != MPL_OK) return st;
  if (!weights || !biases || !packed) return MPL_ERR_INVALID_ARG;
  if (((uintptr_t)packed & 255) != 0) return MPL_ERR_INVALID_ARG;
  for (int l = 0; l < lay.L; ++l)
    if (!weights[l] || !biases[l]) return MPL_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  char* base = (char*)packed;
  const int WP = lay.WP;
  PackArgs a;
  memset(&a, 0, sizeof(a));
  a.WP = WP;
  a.W0 = weights[0];
  a.b0 = biases[0];
  a.Wl = weights[lay.L - 1];
  a.bl = biases[lay.L - 1];
  a.out0 = net->dims[1];
  a.inl = net->dims[lay.L - 1];
  constexpr double kInvPi = 0.31830988618379067154;
  a.omega0 = net->omega[0];
  a.turns0 = (double)net->omega[0] * kInvPi;
  auto f32 = [&](int64_t off) { return (float*)(base + off); };
  a.w0t = f32(lay.w0t);
  a.b0p = f32(lay.b0);
  a.w0f = f32(lay.w0f);
  a.w0u = f32(lay.w0u);
  a.wout = f32(lay.wout);
  a.bout = f32(lay.bout);
  for (int l = 1; l <= lay.nh; ++l) {
    PackHidden& h = a.hid[l - 1];
    h.W = weights[l];
    h.b = biases[l];
    h.out = net->dims[l + 1];
    h.in = net->dims[l];
    h.omega = net->omega[l];
    h.turns = (double)net->omega[l] * kInvPi;
    h.wt = f32(lay.wht[l]);
    h.bh = f32(lay.bh[l]);
    h.hb = f32(lay.hb[l]);
    h.whn = f32(lay.whn[l]);
    h.us = f32(lay.us[l]);
    h.ub = f32(lay.ub) + 4 * l;
    h.eq = f32(lay.eq[l]);
    h.eq_in = l > 1 ? f32(lay.eq[l - 1]) : nullptr;
    h.hw = (__nv_bfloat16*)(base + lay.hw[l]);
    h.hwT = (__nv_bfloat16*)(base + lay.hwT[l]);
    h.hbx = (__nv_bfloat16*)(base + lay.hbx[l]);
    h.hwh = (__half*)(base + lay.hwh[l]);
    h.hwTh = (__half*)(base + lay.hwTh[l]);
    h.hbxh = (__half*)(base + lay.hbxh[l]);
    h.ws = (__half*)(base + lay.ws[l]);
  }
  MPL_CUDA_TRY(cudaMemsetAsync(base + lay.ub, 0, MPL_MAX_LAYERS * 16, s));  // maxima, flags
  const dim3 grid(lay.nh > 0 ? WP : 1, 1 + lay.nh);
  if (lay.nh > 0) {
    pack_rows<<<dim3(WP, lay.nh), WP, 0, s>>>(a);
    MPL_LAUNCH_CHECK();
    pack_range<<<dim3(WP, lay.nh), WP, 0, s>>>(a);
    MPL_LAUNCH_CHECK();
  }
  pack_level<<<grid, WP, 0, s>>>(a);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}
