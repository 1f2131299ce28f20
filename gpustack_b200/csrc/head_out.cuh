// A recurrent mixer's closing step per (token, head): the head's fp32 output over its root mean square, times a weight, times the
// gate's activation, rounded once.  A head of dv = 4 LPH values is held by LPH lanes as one 16-byte piece each, one head per group of
// lanes.  Of many rows (MORE) a group goes through the heads of one number (its weight stays in registers, a step is an addition per
// pointer), the next head's loads in flight.  Bound: launch and latency up to 1000 rows, then instructions.  8 heads of 128, bf16 gates,
// 8192 rows: a head per group, its place divided out, 20.7 us (205 instructions a thread), 18.4 of many (155 a head).
#pragma once
#include "common.cuh"
#include "runtime.h"

namespace b200 {

constexpr int kHoThreads = 256, kHoCtas = 5;           // CTAs per SM

__device__ __forceinline__ float4 ho_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ho_ld4(const bf16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
}
__device__ __forceinline__ void ho_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void ho_st4(bf16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }

template <typename TA, int LPH, bool MORE>
__global__ void __launch_bounds__(kHoThreads, MORE ? kHoCtas : 0)
head_out_kernel(const float* __restrict__ o, const TA* __restrict__ proj, int64_t ld, int gate_col, const bf16* __restrict__ w, int w_head,
                TA* out, int64_t ldo, int items, int H, int step, int silu, float eps) {
  constexpr int DV = 4 * LPH;
  const int lane = threadIdx.x & 31, d = (lane % LPH) * 4;
  const int first = (blockIdx.x * (kHoThreads / 32) + (threadIdx.x >> 5)) * (32 / LPH), i0 = first + lane / LPH;
  if (first >= step) return;                           // (step: a multiple of H)
  const int t0 = i0 / H, h = i0 - t0 * H, rows = MORE ? step / H : 0;
  const bool mine = i0 < step;
  const float* op = o + (size_t)i0 * DV + d;
  const TA* gp = gate_col >= 0 ? proj + (size_t)t0 * ld + gate_col + h * DV + d : nullptr;
  TA* to = out + (size_t)t0 * ldo + h * DV + d;
  float4 ww = make_float4(1.f, 1.f, 1.f, 1.f);
  if (mine && w != nullptr) ww = ho_ld4(w + h * w_head + d);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 x = zero, g = zero;
  if (mine && i0 < items) {
    x = ho_ld4(op);
    if (gate_col >= 0) g = ho_ld4(gp);
  }
  for (int at = first, i = i0; at < items; at += step, i += step) {
    const bool live = mine && i < items;
    float4 xn = zero, gn = zero;
    if constexpr (MORE) {
      op += (size_t)step * DV;
      if (mine && i < items - step) {
        xn = ho_ld4(op);
        if (gate_col >= 0) gn = ho_ld4(gp += (size_t)rows * ld);
      }
    }
    float ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
#pragma unroll
    for (int off = LPH / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float mul = inv_sqrt(ss * (1.0f / DV) + eps);
    float v[4] = {x.x * mul, x.y * mul, x.z * mul, x.w * mul};
    v[0] *= ww.x; v[1] *= ww.y; v[2] *= ww.z; v[3] *= ww.w;
    if (gate_col >= 0) {
      const float gv[4] = {g.x, g.y, g.z, g.w};
      float sg[4];
      logistic_all<false>(gv, sg);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] *= silu ? gv[e] * sg[e] : sg[e];
    }
    if (live) ho_st4(to, make_float4(v[0], v[1], v[2], v[3]));
    if constexpr (!MORE) break;
    to += (size_t)rows * ldo;
    x = xn;
    g = gn;
  }
}

// Heads of 32, 64 or 128 values with aligned 4-value pieces on every side; false: the caller's general kernel.
template <typename TA>
bool head_out_launch(const float* o, const void* proj, int64_t ld, int gate_col, const void* w, int w_head, void* out, int64_t ldo, int T,
                     int H, int dv, int silu, float eps, cudaStream_t s) {
  const uintptr_t al = 4 * sizeof(TA) - 1;
  if (!(dv == 32 || dv == 64 || dv == 128) || ((uintptr_t)o & 15) || ((uintptr_t)out & al) || ldo % 4 != 0 || ((uintptr_t)w & 7) ||
      (int64_t)T * H > INT32_MAX / 2)
    return false;
  if (gate_col >= 0 && (ld % 4 != 0 || gate_col % 4 != 0 || ((uintptr_t)proj & al))) return false;
  const int items = T * H, per = kHoThreads / 32 * (128 / dv);      // groups per CTA
  // groups in whole multiples of the heads; no more CTAs than are resident.  Fewer registers and more CTAs serve less than five rounds
  // better: 16 heads of 64 in bf16, a head per group and resident CTAs, 1000 rows 4.5 and 5.0 us, 2048 6.7 and 7.3, 3000 8.7 and 9.0,
  // 4100 10.7 and 10.9; 32 heads of 32, 4100 rows, 10.8 and 10.4
  constexpr int kRounds = 5;
  const int resident = kHoCtas * sm_count() * per;
  int step = items;
  if (items > kRounds * resident && H <= resident) step = resident / H * H;
  const int grid = (step + per - 1) / per;
#define B200_HO(L)                                                                                                                 \
  do {                                                                                                                             \
    if (step < items)                                                                                                              \
      head_out_kernel<TA, L, true><<<grid, kHoThreads, 0, s>>>(o, (const TA*)proj, ld, gate_col, (const bf16*)w, w_head, (TA*)out, ldo, \
                                                               items, H, step, silu, eps);                                         \
    else                                                                                                                           \
      head_out_kernel<TA, L, false><<<grid, kHoThreads, 0, s>>>(o, (const TA*)proj, ld, gate_col, (const bf16*)w, w_head, (TA*)out, ldo, \
                                                                items, H, step, silu, eps);                                        \
  } while (0)
  if (dv == 32) B200_HO(8);
  else if (dv == 64) B200_HO(16);
  else B200_HO(32);
#undef B200_HO
  return true;
}

}  // namespace b200
