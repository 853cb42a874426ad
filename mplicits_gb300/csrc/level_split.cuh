// FP32 level evaluator on the tensor cores (sm_103a): every hidden GEMM as
// three FP16 GEMMs of split operands, accumulated in FP32.
//
// A 24-bit product does not fit kind::f16, but the operands are bounded, so
// they split exactly where it matters:
//   activations  s in [-1, 1]:  hi = s rounded to a multiple of 2^-10 (exact
//                in FP16), lo = s - hi rounded to FP16 (error <= 2^-23);
//                hidden activations that are usually small are scaled up to 1
//                (PackLayout::eq) so that layers of small rows lose nothing;
//   weights      w' = w omega / pi times a power of two that puts the layer's
//                largest into FP16's top binade (PackLayout::ub), and a row far
//                below it into the same (PackLayout::eq); in a row n of largest
//                magnitude 2^e_n, hi is a multiple of 2^(e_n - 11), lo = FP16 of
//                the rest (error <= 2^(e_n - 24)).
// hi*hi products are multiples of 2^(e_n - 21), so their sum over K is exact in
// the FP32 accumulator up to 2^24 units (|sum| <= 2^(e_n + 3); larger sums lose
// their last bit, as an FP32 chain does at every step).  hi*lo and lo*hi go to a second
// accumulator, lo*lo (2^-23 relative) is left out.  The phase leaves in half
// turns u = z / pi, so the sine reduces exactly: r = u - rint(u), sin(pi r)
// by an odd polynomial of degree 9 (minimax, error 3.4e-9), sign by the
// parity of rint(u).
//
// Error of one trained 256-wide level against float64 (relative 2-norm):
// 2.0e-7 with this kernel, 2.5e-7 with the FP32 FMA kernel.  (One accumulator
// for all three products: 8.6e-7, the tensor cores truncate their sums.)
//
// One persistent CTA per SM walks 128-point tiles.  The two parts of A take
// 128 KB of shared memory at width 256 and the two accumulators all 512 TMEM
// columns, so one tile is in flight; what overlaps is inside the tile: the 16
// epilogue warps first read a finished accumulator into registers (64 phases
// a thread), which frees it, then take the sines and hand the next A operand
// over in 64-feature chunks while its GEMM already runs.  The first chunk of
// the next tile's first layer is computed into registers during the last GEMM
// and written as soon as that GEMM frees A; the other chunks and the last
// layer's sines and output dot run under the next tile's first GEMM.  Weights stream from L2 in K = 32 stages.
// Bound: the tensor pipe and the sines together (12.3k cycles of MMA and about
// 11k issue slots per scheduler in the 22k cycles of a tile at width 256).
// 262,144 points 1694 -> 173 us, a 256^3 grid 104.3 -> 10.2 ms against the FMA
// kernel.  On the way: MMAs issued by a lane in a branch of its own cost 200
// cycles a K step instead of 128 (tc.cuh, 15.4 -> 12.5 us per tile); 8 epilogue
// warps of twice the registers 13.5 us.
//
// Phases that could leave the range of the exact reduction (|u| up to 2^21, by
// a bound per point or per layer) are first wrapped to one turn, which changes
// no other value's bits: a point's result never depends on its neighbours.
// Every wait is bounded (the abort protocol of level_bf16.cuh).
#pragma once

#include "level_bf16.cuh"

namespace mpl {
namespace split {

using bf16::f2pack;
using bf16::f2unpack;
using bf16::ffma2;
using bf16::kM;
using bf16::kMaxNC;

constexpr int kU = 16;  // features of each 64-feature chunk per epilogue warp
constexpr int kQ = 64 / kU;
constexpr int kEpiWarps = 4 * kQ;
constexpr int kMmaWarp = kEpiWarps;
constexpr int kTmaWarp = kEpiWarps + 1;
constexpr int kThreads = (kEpiWarps + 4) * 32;
constexpr int kLaunchRegs = kQ == 4 ? 96 : 168;
constexpr int kEpiRegs = kQ == 4 ? 112 : 216, kRoleRegs = kQ == 4 ? 32 : 72;
static_assert(kEpiWarps * 32 * kEpiRegs + 128 * kRoleRegs <= kThreads * kLaunchRegs,
              "register split");
constexpr float kPhaseLimit = 65536.f;  // |u| that the reduction takes unwrapped

template <int WP, int STAGES>
struct Cfg {
  static constexpr int NC = WP / 64;                          // A chunks
  static constexpr int NK = WP / kSplitK;                     // weight stages per part
  static constexpr uint32_t kABytes = kM * WP * 2;            // one part of A
  static constexpr uint32_t kStageBytes = WP * kSplitK * 2;
  static constexpr uint32_t kTmemCols = WP == 64 ? 128 : (WP == 128 ? 256 : 512);
  static constexpr uint32_t oA = 0;                           // hi, lo
  static constexpr uint32_t oW = 2 * kABytes;
  static constexpr uint32_t oW0 = oW + STAGES * kStageBytes;  // float [4][WP] + bounds
  static constexpr uint32_t oWout = oW0 + (4 * WP + 4) * 4;
  static constexpr uint32_t oRed = oWout + WP * 4;            // float [2][kQ - 1][128]
  static constexpr uint32_t oBar = oRed + 2 * (kQ - 1) * kM * 4;
  // wfull/wempty [S], achunk [kMaxNC], dfull, dempty, redfull [2], final
  static constexpr uint32_t kNumBars = 2 * STAGES + kMaxNC + 5;
  static constexpr uint32_t oMisc = oBar + kNumBars * 8;
  static constexpr uint32_t oU = (oMisc + 16 + 15) & ~15u;    // float [nh][WP] biases
  static constexpr uint32_t kFixedBytes = oU;
  static size_t bytes(int nh) { return kFixedBytes + (size_t)nh * WP * 4; }
};

__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t both(float v) { return f2pack(v, v); }

// rint of two phases, |u| < 2^22: n, and t, whose low mantissa bits are the
// parities (adding 1.5 * 2^23 rounds to integers)
__device__ __forceinline__ uint64_t rint2(uint64_t u, uint64_t& t) {
  t = fadd2(u, both(12582912.f));
  return fadd2(t, both(-12582912.f));
}
// sin(pi (r + n)) of two rests r, |r| <= 0.51, parities in t; the odd polynomial of
// degree 9 of least absolute error on [0, 1/2] (six extrema of 3.34e-9; Lawson's
// iteratively reweighted least squares finds it).
__device__ __forceinline__ void sinpi2(uint64_t r, uint64_t t, float& s0, float& s1) {
  const uint64_t x = fmul2(r, r);
  uint64_t p = ffma2(x, both(0.0772201637866401f), both(-0.5980451913904322f));
  p = ffma2(p, x, both(2.550031380059994f));
  p = ffma2(p, x, both(-5.167706879085096f));
  p = ffma2(p, x, both(3.141592580046961f));
  const uint64_t s = fmul2(r, p);
  float t0, t1;
  f2unpack(t, t0, t1);
  f2unpack(s, s0, s1);
  s0 = __uint_as_float(__float_as_uint(s0) ^ (__float_as_uint(t0) << 31));
  s1 = __uint_as_float(__float_as_uint(s1) ^ (__float_as_uint(t1) << 31));
}

// the same phase within one turn, exactly (a rest of u by an even integer; NaN
// for an infinite one); phases that need no reduction keep their sine's bits
__device__ __forceinline__ uint64_t wrap2(uint64_t u) {
  float a, b;
  f2unpack(u, a, b);
  return f2pack(fmaf(-2.f, rintf(0.5f * a), a), fmaf(-2.f, rintf(0.5f * b), b));
}

// the two FP16 parts of a pair of sines
__device__ __forceinline__ void split2(float s0, float s1, uint32_t& hi, uint32_t& lo) {
  const uint64_t s = f2pack(s0, s1);
  const uint64_t h = fadd2(fadd2(s, both(12288.f)), both(-12288.f));
  const uint64_t l = ffma2(h, both(-1.f), s);
  float a, b;
  f2unpack(h, a, b);
  hi = bf16::Operand<__half>::pack(a, b);
  f2unpack(l, a, b);
  lo = bf16::Operand<__half>::pack(a, b);
}

// the same of scaled sines, up to 2^5: beyond 2, hi is rounded to FP16's 11 bits
__device__ __forceinline__ void split2_scaled(float s0, float s1, uint32_t& hi, uint32_t& lo) {
  const uint64_t s = f2pack(s0, s1);
  float a, b;
  f2unpack(fadd2(fadd2(s, both(12288.f)), both(-12288.f)), a, b);
  hi = bf16::Operand<__half>::pack(a, b);
  const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  f2unpack(ffma2(f2pack(h.x, h.y), both(-1.f), s), a, b);
  lo = bf16::Operand<__half>::pack(a, b);
}

// 8 features (packed pairs) of row m, feature group k8, into both parts of A
template <uint32_t kABytes>
__device__ __forceinline__ void store_a8(uint8_t* sA, int m, int k8, const uint32_t* hi,
                                         const uint32_t* lo) {
  const uint32_t off = (uint32_t)((k8 * 16 + (m >> 3)) * 128 + (m & 7) * 16);
  *reinterpret_cast<uint4*>(sA + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(sA + kABytes + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

template <int WP, int STAGES>
__global__ void __launch_bounds__(kThreads, 1) level_split_kernel(const LevelArgs a) {
  using C = Cfg<WP, STAGES>;
  constexpr int NC = C::NC, NK = C::NK, S = STAGES;
  constexpr uint32_t IDESC = tc::idesc_f16kind_f32(kM, WP, 0u);
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sA = smem + C::oA;
  uint8_t* sW = smem + C::oW;
  float* w0s = reinterpret_cast<float*>(smem + C::oW0);
  float* wout = reinterpret_cast<float*>(smem + C::oWout);
  float* red = reinterpret_cast<float*>(smem + C::oRed);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::oBar);
  uint64_t* wfull = bars;             // [S]  TMA -> MMA
  uint64_t* wempty = bars + S;        // [S]  MMA -> TMA
  uint64_t* achunk = bars + 2 * S;    // [NC] epilogue -> MMA, once per GEMM
  uint64_t* dfull = achunk + kMaxNC;  // MMA -> epilogue: accumulator done, A free
  uint64_t* dempty = dfull + 1;       // epilogue -> MMA: accumulator read
  uint64_t* redfull = dempty + 1;     // [2]  h > 0 warps -> h = 0 warps, by tile parity
  uint64_t* finalb = redfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::oMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::oMisc + 4);
  float* us = reinterpret_cast<float*>(smem + C::oU);  // [nh][WP]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nh = a.lay.nh;
  const int64_t n = level_point_count(a);
  const int64_t ntiles = (n + kM - 1) / kM;
  if ((int64_t)blockIdx.x >= ntiles) return;
  const int64_t G = gridDim.x;
  const int64_t nt = (ntiles - blockIdx.x + G - 1) / G;  // tiles of this CTA

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&wfull[s], 1);
      mbar_init(&wempty[s], 1);
    }
    for (int c = 0; c < kMaxNC; ++c) mbar_init(&achunk[c], kEpiWarps);
    mbar_init(dfull, 1);
    mbar_init(dempty, kEpiWarps);
    for (int b = 0; b < 2; ++b) mbar_init(&redfull[b], 4 * (kQ - 1));
    mbar_init(finalb, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) tc::tmem_alloc(tmem_slot, C::kTmemCols);
  const char* pk = a.packed;
  {
    const float* g0 = reinterpret_cast<const float*>(pk + a.lay.w0u);
    for (int i = threadIdx.x; i < 4 * WP + 4; i += kThreads) w0s[i] = g0[i];
    for (int i = threadIdx.x; i < WP; i += kThreads)
      wout[i] = reinterpret_cast<const float*>(pk + a.lay.wout)[i];
    for (int l = 1; l <= nh; ++l) {
      const float* gu = reinterpret_cast<const float*>(pk + a.lay.us[l]);
      for (int i = threadIdx.x; i < WP; i += kThreads) us[(l - 1) * WP + i] = gu[i];
    }
  }
  const float bout = reinterpret_cast<const float*>(pk + a.lay.bout)[0];
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp >= kEpiWarps) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRoleRegs));
  if (warp == kTmaWarp) {
    // ================= TMA: weight stages in the MMA's order ===============
    if (lane == 0) {
      // stage and phase kept as counters: a division by the ring size on each
      // stage sits on the refill's latency
      int64_t w = 0;
      int st = 0;
      uint32_t par = 1;  // of the wait for a free stage: the first pass is free
      bool ok = true;
      for (int64_t k = 0; k < nt && ok && !*abort_flag; ++k) {
        for (int l = 1; l <= nh && ok; ++l) {
          const char* src = pk + a.lay.ws[l];
#pragma unroll 1
          for (int c = 0; c < 2 * NK; ++c, ++w) {
            if (!bf16::mbar_wait_abort(&wempty[st], par, a.status, abort_flag)) {
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&wfull[st], C::kStageBytes);
            tma_bulk_g2s(sW + st * C::kStageBytes, src + (size_t)c * C::kStageBytes,
                         C::kStageBytes, &wfull[st]);
            if (++st == S) st = 0, par ^= 1u;
          }
        }
      }
      const int64_t first = w > S ? w - S : 0;
      for (int64_t v = first; v < w; ++v)
        mbar_wait(&wfull[v % S], (uint32_t)((v / S) & 1), a.status);
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA issuer (the whole warp, one lane issues) ========
    const uint32_t lead = tc::elect_lane();
    const uint64_t aHi = tc::smem_desc(smem_u32(sA), 2048u, 128u);
    const uint64_t aLo = aHi + (uint64_t)(C::kABytes >> 4);
    const uint64_t wDesc = tc::smem_desc(smem_u32(sW), 128u, kSplitK * 16u);
    uint32_t gemm = 0;
    int st = 0;
    uint32_t par = 0;
    bool ok = true;
    for (int64_t k = 0; k < nt && ok; ++k) {
      for (int l = 1; l <= nh && ok; ++l, ++gemm) {
        if (gemm > 0 && !bf16::warp_wait(dempty, (gemm - 1) & 1, a.status, abort_flag)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
#pragma unroll
        for (int kc = 0; kc < NK; ++kc) {  // K blocks of kSplitK
          if ((kc * kSplitK) % 64 == 0 && !bf16::warp_wait(&achunk[kc * kSplitK / 64], gemm & 1,
                                                           a.status, abort_flag)) {
            ok = false;
            break;
          }
          const uint64_t aOff = (uint64_t)((kc * (kSplitK / 8) * 2048) >> 4);
#pragma unroll
          for (int part = 0; part < 2; ++part) {  // of the weights
            if (!bf16::warp_wait(&wfull[st], par, a.status, abort_flag)) {
              ok = false;
              break;
            }
            tc::fence_after_sync();
            const uint64_t wC = wDesc + (uint64_t)((st * C::kStageBytes) >> 4);
#pragma unroll
            for (int ks = 0; ks < kSplitK / 16; ++ks) {
              const uint64_t aK = aOff + (uint64_t)((ks * 2 * 2048) >> 4);
              const uint64_t wK = wC + (uint64_t)((ks * 256) >> 4);
              if (part == 0) {
                tc::mma_lead(lead, tmem, aHi + aK, wK, IDESC, kc + ks > 0);
                tc::mma_lead(lead, tmem + WP, aLo + aK, wK, IDESC, kc + ks > 0);
              } else {
                tc::mma_lead(lead, tmem + WP, aHi + aK, wK, IDESC, true);
              }
            }
            tc::commit_lead(lead, &wempty[st]);
            if (++st == S) st = 0, par ^= 1u;
          }
          if (!ok) break;
        }
        if (ok) tc::commit_lead(lead, dfull);
      }
    }
    tc::commit_lead(lead, finalb);
    __syncwarp();
    mbar_wait(finalb, 0u, a.status);
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
    // ================= epilogue warps =====================================
    const int q = warp & 3, h = warp >> 2;  // rows 32 q .., features kU h .. of each chunk
    const int m = 32 * q + lane;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    int64_t gemm = 0;

    // The first layer has a mapping of its own: a warp takes 64 rows (two a
    // lane) and kL0 features of a chunk, which halves its reads of the weights
    // (shared memory feeds the tensor cores beside it).
    constexpr int kL0 = 2 * kU / 4;
    const int r0 = (warp & 1) * 64 + lane, g0 = (warp >> 1) * kL0;
    auto point_id = [&](int64_t k, int row) -> int64_t {
      const int64_t qi = ((int64_t)blockIdx.x + k * G) * kM + row;
      return k < nt && qi < n ? (a.index ? (int64_t)a.index[qi] : qi) : -1;
    };
    float px[2], py[2], pz[2];  // the next tile's two points
    bool near[2], all_near = true;
    auto load_next = [&](int64_t k) {
      // a bound of |u| over the layer's features (false for a NaN too)
      const float* b = w0s + 4 * WP;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int64_t p = point_id(k, r0 + 32 * r);
        px[r] = py[r] = pz[r] = 0.f;
        if (p >= 0) point_coords(a, p, px[r], py[r], pz[r]);
        near[r] = fmaf(fabsf(px[r]), b[0],
                       fmaf(fabsf(py[r]), b[1], fmaf(fabsf(pz[r]), b[2], b[3]))) <= kPhaseLimit;
      }
      all_near = __all_sync(0xffffffffu, near[0] && near[1]);
    };
    // Chunk c of the next tile's first layer, both parts.  The phase is rounded
    // at its full size only to find its integer part, which is then taken off
    // the bias before the dot product is summed again: the layer's error, which
    // every later layer amplifies, is that of a phase of less than a turn.
    auto first_layer = [&](int c, uint32_t (&hi)[2][kL0 / 2], uint32_t (&lo)[2][kL0 / 2]) {
      const float* w = w0s + c * 64 + g0;
#pragma unroll
      for (int j = 0; j < kL0; j += 4) {
        const ulonglong2 wx = *reinterpret_cast<const ulonglong2*>(w + j);
        const ulonglong2 wy = *reinterpret_cast<const ulonglong2*>(w + WP + j);
        const ulonglong2 wz = *reinterpret_cast<const ulonglong2*>(w + 2 * WP + j);
        const ulonglong2 wb = *reinterpret_cast<const ulonglong2*>(w + 3 * WP + j);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint64_t X = both(px[r]), Y = both(py[r]), Z = both(pz[r]);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint64_t vx = i ? wx.y : wx.x, vy = i ? wy.y : wy.x, vz = i ? wz.y : wz.x,
                           vb = i ? wb.y : wb.x;
            const uint64_t u = ffma2(X, vx, ffma2(Y, vy, ffma2(Z, vz, vb)));
            uint64_t t;
            const uint64_t n2 = rint2(u, t);
            uint64_t rest = ffma2(X, vx, ffma2(Y, vy, ffma2(Z, vz, ffma2(n2, both(-1.f), vb))));
            if (!all_near && !near[r]) {
              const uint64_t v = wrap2(u);
              rest = ffma2(rint2(v, t), both(-1.f), v);
            }
            float s0, s1;
            sinpi2(rest, t, s0, s1);
            split2(s0, s1, hi[r][j / 2 + i], lo[r][j / 2 + i]);
          }
        }
      }
    };
    auto hand_over = [&](int c) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&achunk[c]);
    };
    auto write_first = [&](int c, const uint32_t (&hi)[2][kL0 / 2], const uint32_t (&lo)[2][kL0 / 2]) {
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int g = 0; g < kL0 / 8; ++g)
          store_a8<C::kABytes>(sA, r0 + 32 * r, c * 8 + g0 / 8 + g, hi[r] + 4 * g, lo[r] + 4 * g);
      hand_over(c);
    };
    // the finished accumulator as phases: u = (hi + lo) * scale + bias, with the
    // layer's one scale
    uint64_t u[NC][kU / 2];
    auto read_phases = [&](int l) {
      const float* bias = us + (l - 1) * WP;
      const float* lay = reinterpret_cast<const float*>(pk + a.lay.ub) + 4 * l;
      const uint64_t scale = both(lay[3]);
      const bool far = !(lay[0] <= kPhaseLimit);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int j0 = c * 64 + h * kU;
        uint32_t hi[kU], lo[kU];
        tc::ld_32x32b<kU>(tl + (uint32_t)j0, hi);
        tc::ld_32x32b<kU>(tl + (uint32_t)(WP + j0), lo);
        tc::wait_ld();
#pragma unroll
        for (int j = 0; j < kU; j += 4) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bias + j0 + j);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int e = j + 2 * i;
            const uint64_t v = fadd2(f2pack(__uint_as_float(hi[e]), __uint_as_float(hi[e + 1])),
                                     f2pack(__uint_as_float(lo[e]), __uint_as_float(lo[e + 1])));
            u[c][e / 2] = ffma2(v, scale, i ? b.y : b.x);
          }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(dempty);
      if (far) {
        // rows at a scale of their own have 2^d_n (phase - bias) + bias
        const float* own = reinterpret_cast<const float*>(pk + a.lay.eq[l]) + WP;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < kU; j += 2) {
            const int at = c * 64 + h * kU + j;
            const float2 d = *reinterpret_cast<const float2*>(own + at);
            float x, y;
            f2unpack(u[c][j / 2], x, y);
            if (d.x != 1.f) x = fmaf(x - bias[at], d.x, bias[at]);
            if (d.y != 1.f) y = fmaf(y - bias[at + 1], d.y, bias[at + 1]);
            u[c][j / 2] = wrap2(f2pack(x, y));
          }
      }
    };
    auto sine = [&](uint64_t v, float& s0, float& s1) {
      uint64_t t;
      const uint64_t n2 = rint2(v, t);
      sinpi2(ffma2(n2, both(-1.f), v), t, s0, s1);
    };

    load_next(0);
#pragma unroll 1
    for (int c = 0; c < NC; ++c) {
      uint32_t hi[2][kL0 / 2], lo[2][kL0 / 2];
      first_layer(c, hi, lo);
      write_first(c, hi, lo);
    }
    bool ok = true;
#pragma unroll 1
    for (int64_t k = 0; k < nt && ok; ++k) {
#pragma unroll 1
      for (int l = 1; l < nh; ++l, ++gemm) {
        if (!bf16::warp_wait(dfull, (uint32_t)(gemm & 1), a.status, abort_flag)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        read_phases(l);
        // null unless some activation of the layer is always small
        const float* eq = reinterpret_cast<const float*>(pk + a.lay.ub)[4 * l + 2] != 0.f
                              ? reinterpret_cast<const float*>(pk + a.lay.eq[l])
                              : nullptr;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          uint32_t hi[kU / 2], lo[kU / 2];
#pragma unroll
          for (int j = 0; j < kU / 2; ++j) {
            float s0, s1;
            sine(u[c][j], s0, s1);
            if (eq) {
              const float2 e = *reinterpret_cast<const float2*>(eq + c * 64 + h * kU + 2 * j);
              split2_scaled(s0 * e.x, s1 * e.y, hi[j], lo[j]);
            } else {
              split2(s0, s1, hi[j], lo[j]);
            }
          }
#pragma unroll
          for (int g = 0; g < kU / 8; ++g)
            store_a8<C::kABytes>(sA, m, c * 8 + h * (kU / 8) + g, hi + 4 * g, lo + 4 * g);
          hand_over(c);
        }
      }
      if (!ok) break;
      // last GEMM: the first chunk of the next tile's first layer under it
      const bool more = k + 1 < nt;
      load_next(k + 1);
      uint32_t hi0[2][kL0 / 2], lo0[2][kL0 / 2];
      first_layer(0, hi0, lo0);
      const int64_t ps = h == 0 ? point_id(k, m) : -1;  // point of this row
      float sold = 0.f;
      if (h == 0 && ps >= 0 && a.store_mode == MPL_ACCUMULATE) sold = a.S[ps];
      if (!bf16::warp_wait(dfull, (uint32_t)(gemm & 1), a.status, abort_flag)) {
        ok = false;
        break;
      }
      ++gemm;
      tc::fence_after_sync();
      if (more) write_first(0, hi0, lo0);
      read_phases(nh);
      // the other chunks while that GEMM begins
      if (more) {
#pragma unroll 1
        for (int c = 1; c < NC; ++c) {
          uint32_t hi[2][kL0 / 2], lo[2][kL0 / 2];
          first_layer(c, hi, lo);
          write_first(c, hi, lo);
        }
      }
      uint64_t part[2] = {both(0.f), both(0.f)};
#pragma unroll
      for (int c = 0; c < NC; ++c) {
#pragma unroll
        for (int j = 0; j < kU / 2; j += 2) {
          const ulonglong2 wo =
              *reinterpret_cast<const ulonglong2*>(wout + c * 64 + h * kU + 2 * j);
          float s0, s1;
          sine(u[c][j], s0, s1);
          part[0] = ffma2(f2pack(s0, s1), wo.x, part[0]);
          sine(u[c][j + 1], s0, s1);
          part[1] = ffma2(f2pack(s0, s1), wo.y, part[1]);
        }
      }
      float p0, p1;
      f2unpack(fadd2(part[0], part[1]), p0, p1);
      const float sum = __fadd_rn(p0, p1);
      // a buffer's next tile but one needs this warp's first layer of that
      // tile, so it is free again without a barrier of its own
      float* rs = red + (k & 1) * (kQ - 1) * kM;
      uint64_t* rb = &redfull[k & 1];
      if (h > 0) {
        rs[(h - 1) * kM + m] = sum;
        __syncwarp();
        if (lane == 0) mbar_arrive(rb);
      } else {
        if (!bf16::warp_wait(rb, (uint32_t)((k >> 1) & 1), a.status, abort_flag)) {
          ok = false;
          break;
        }
        float f = sum;
#pragma unroll
        for (int i = 0; i < kQ - 1; ++i) f = __fadd_rn(f, rs[i * kM + m]);
        store_and_band_old(a, ps >= 0, ps, __fadd_rn(f, bout), sold);
      }
    }
  }

  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == kMmaWarp) tc::tmem_dealloc(tmem, C::kTmemCols);
}

template <int WP, int STAGES>
int launch_cfg(const LevelArgs& a, cudaStream_t s) {
  const size_t smem = Cfg<WP, STAGES>::bytes(a.lay.nh);
  MPL_CUDA_TRY(cudaFuncSetAttribute(level_split_kernel<WP, STAGES>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int64_t grid = sm_count();
  if (!a.n_dev) {
    const int64_t ntiles = (a.n + kM - 1) / kM;
    grid = ntiles < grid ? ntiles : grid;
  }
  if (grid <= 0) return MPL_OK;
  level_split_kernel<WP, STAGES><<<(unsigned)grid, kThreads, smem, s>>>(a);
  MPL_LAUNCH_CHECK();
  return MPL_OK;
}

// five weight stages: the deepest ring that fits at every depth
template <int WP>
int launch_wp(const LevelArgs& a, cudaStream_t s) {
  static_assert(Cfg<WP, 5>::kFixedBytes + (MPL_MAX_LAYERS - 2) * WP * 4 <= 227 * 1024,
                "shared memory");
  return launch_cfg<WP, 5>(a, s);
}

}  // namespace split
}  // namespace mpl
