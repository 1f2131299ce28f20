// A recurrent mixer's closing step per (token, head): the head's fp32 output over its root mean square, times a weight, times the
// gate's activation, rounded once.  A head of dv = 4 LPH values is held by LPH lanes as one 16-byte piece each, one head per group of
// lanes: many small warps keep the bytes in flight.  Bound: launch and latency up to 1000 rows, then instructions (3.1 per clock and SM,
// 8192 rows at 4.1 TB/s).  8 heads of 128, bf16 gates, warm: 1.8 us for one row, 5.4 for 2048, 16.3 for 8192 (with four heads in flight per lane
// 4.5, 7.0 and 19.5; a CTA or a warp per head, looping, 2.6, 7.4 and 22.9).
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int kHoThreads = 256;

__device__ __forceinline__ float4 ho_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ho_ld4(const bf16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
}
__device__ __forceinline__ void ho_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void ho_st4(bf16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }

template <typename TA, int LPH>
__global__ void __launch_bounds__(kHoThreads)
head_out_kernel(const float* __restrict__ o, const TA* __restrict__ proj, int64_t ld, int gate_col, const bf16* __restrict__ w, int w_head,
                TA* out, int64_t ldo, int items, int H, int silu, float eps) {
  constexpr int DV = 4 * LPH;
  const int lane = threadIdx.x & 31, i = (blockIdx.x * (kHoThreads / 32) + (threadIdx.x >> 5)) * (32 / LPH) + lane / LPH, d = (lane % LPH) * 4;
  const int t = i / H, h = i - t * H;
  const bool live = i < items;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), g = x;
  if (live) {
    x = ho_ld4(o + (size_t)i * DV + d);
    if (gate_col >= 0) g = ho_ld4(proj + (size_t)t * ld + gate_col + h * DV + d);
  }
  float ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
#pragma unroll
  for (int off = LPH / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if (!live) return;
  const float mul = 1.0f / sqrtf(ss / (float)DV + eps);
  float v[4] = {x.x * mul, x.y * mul, x.z * mul, x.w * mul};
  if (w != nullptr) {
    const float4 ww = ho_ld4(w + h * w_head + d);
    v[0] *= ww.x; v[1] *= ww.y; v[2] *= ww.z; v[3] *= ww.w;
  }
  if (gate_col >= 0) {
    const float gv[4] = {g.x, g.y, g.z, g.w};
    float sg[4];
    logistic_all<false>(gv, sg);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] *= silu ? gv[e] * sg[e] : sg[e];
  }
  ho_st4(out + (size_t)t * ldo + h * DV + d, make_float4(v[0], v[1], v[2], v[3]));
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
  const int items = T * H, per = kHoThreads / 32 * (128 / dv), grid = (items + per - 1) / per;
#define B200_HO(L)                                                                                                                 \
  head_out_kernel<TA, L><<<grid, kHoThreads, 0, s>>>(o, (const TA*)proj, ld, gate_col, (const bf16*)w, w_head, (TA*)out, ldo, items, H, \
                                                     silu, eps)
  if (dv == 32) B200_HO(8);
  else if (dv == 64) B200_HO(16);
  else B200_HO(32);
#undef B200_HO
  return true;
}

}  // namespace b200
