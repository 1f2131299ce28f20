// Preparation steps of latent attention (keys and values expanded from one small latent per token).
//
//   rms_rows:     out[t, :] = x[t, :] / sqrt(mean(x[t, :]^2) + eps) * w over a column slice of a wider row
//                 (the query latent between its two projections).  fp32 statistics.
//   latent_prep:  one pass over a token's fused projection row  [ ... | latent: R | key part: dr ]  and its
//                 query rows  [H][dn unrotated | dr rotated]:
//                   * the latent is RMS-normed (weight, eps) and written to the token's cache row [0, R),
//                   * the key part is rotated at the token's position and written to cache row [R, R + dr),
//                   * every head's rotated query part is rotated and written to qa[t][h][R, R + dr) -- the tail
//                     of the absorbed query, whose first R entries  W_uk[h]^T q_unrotated  a batched linear fills.
//                 Rotation: the first `dims` entries of a part, pairs (2i, 2i+1) ("interleaved") or
//                 (i, i + dims/2) ("half"), angle = position * freq[i] formed and reduced to [-pi, pi] in fp64 (once
//                 per token and pair, shared by the key part and all heads), cos and sin multiplied by one factor
//                 (frequency-scaled variants); the rest of the part passes unchanged.
// Cache layout: [blocks][page][R + dr]: one row per token shared by all heads.
#include "common.cuh"
#include "runtime.h"
#include "../../include/b200.h"

namespace b200 {

__device__ __forceinline__ float lt_f32(float v) { return v; }
__device__ __forceinline__ float lt_f32(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void lt_out(float* p, float v) { *p = v; }
__device__ __forceinline__ void lt_out(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

constexpr int kLtWarps = 4;
constexpr int kLtPrepMaxWarps = 16;

template <typename TA>
__global__ void __launch_bounds__(kLtWarps * 32)
rms_rows_kernel(const TA* __restrict__ x, int64_t ldx, const bf16* __restrict__ w, TA* out, int64_t ldo, int T, int n,
                float eps) {
  const int t = blockIdx.x * kLtWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const TA* xr = x + (size_t)t * ldx;
  float ss = 0.f;
  for (int d = lane; d < n; d += 32) {
    const float v = lt_f32(xr[d]);
    ss = fmaf(v, v, ss);
  }
  const float mul = 1.0f / sqrtf(warp_sum(ss) / (float)n + eps);
  for (int d = lane; d < n; d += 32) lt_out(out + (size_t)t * ldo + d, lt_f32(xr[d]) * mul * __bfloat162float(w[d]));
}

constexpr int kLtMaxPairs = 256;   // rotated pairs per part (dims <= 512)

// src / dst: a part of `width` entries; entries [0, dims) are rotated by the token's angles (cs / sn, one per pair).
template <typename TA>
__device__ __forceinline__ void rotate_part(const TA* src, TA* dst, int width, int dims, int half_layout,
                                            const float* cs, const float* sn, int lane) {
  const int half = dims >> 1;
  for (int i = lane; i < half; i += 32) {
    const int a = half_layout ? i : 2 * i, b = half_layout ? i + half : 2 * i + 1;
    const float c = cs[i], s = sn[i];
    const float u = lt_f32(src[a]), v = lt_f32(src[b]);
    lt_out(dst + a, u * c - v * s);
    lt_out(dst + b, v * c + u * s);
  }
  for (int d = dims + lane; d < width; d += 32) lt_out(dst + d, lt_f32(src[d]));
}

// One CTA per token.  The token's cos / sin (angle formed and reduced in fp64, one evaluation per pair for all heads)
// go to shared memory first; then the warps take the tasks in turn: task 0 = the latent and the key part, task 1 + h =
// head h's rotated query part.
template <typename TA>
__global__ void __launch_bounds__(kLtPrepMaxWarps * 32)
latent_prep_kernel(const TA* __restrict__ proj, int64_t ld, int kv_col, const TA* __restrict__ q, int64_t ldq,
                   const bf16* __restrict__ kv_norm_w, const int32_t* __restrict__ positions,
                   const int32_t* __restrict__ slots, TA* cache, TA* qa, int64_t ldqa, int H, int dn, int dr, int R,
                   int dims, int half_layout, const double* __restrict__ freq, float mag, float eps) {
  __shared__ float cs[kLtMaxPairs], sn[kLtMaxPairs];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = positions[t];
  for (int i = threadIdx.x; i < (dims >> 1); i += blockDim.x) {
    // the angle and its reduction to [-pi, pi] in fp64 (a handful of operations), cos / sin of the remainder in fp32
    const double ang = (double)pos * freq[i];
    const double turns = rint(ang * 0.15915494309189535);
    const float rem = (float)fma(-turns, 6.283185307179586, ang);
    float s_, c_;
    sincosf(rem, &s_, &c_);
    cs[i] = c_ * mag;
    sn[i] = s_ * mag;
  }
  __syncthreads();
  for (int task = warp; task <= H; task += (int)(blockDim.x >> 5)) {
    if (task == 0) {
      const int slot = slots[t];
      if (slot < 0) continue;                     // a padding row: nothing to cache
      const TA* kv = proj + (size_t)t * ld + kv_col;
      TA* row = cache + (size_t)slot * (R + dr);
      float ss = 0.f;
      for (int d = lane; d < R; d += 32) {
        const float v = lt_f32(kv[d]);
        ss = fmaf(v, v, ss);
      }
      const float mul = 1.0f / sqrtf(warp_sum(ss) / (float)R + eps);
      for (int d = lane; d < R; d += 32) lt_out(row + d, lt_f32(kv[d]) * mul * __bfloat162float(kv_norm_w[d]));
      rotate_part(kv + R, row + R, dr, dims, half_layout, cs, sn, lane);
      continue;
    }
    const int h = task - 1;
    rotate_part(q + (size_t)t * ldq + (size_t)h * (dn + dr) + dn, qa + (size_t)t * ldqa + (size_t)h * (R + dr) + R, dr, dims,
                half_layout, cs, sn, lane);
  }
}

// The same for bf16 rows of 512 + 64 whose whole rotated part turns: a warp per token, nothing shared, no barrier.  Lane l holds
// the latent's columns 8 l and 256 + 8 l (16 bytes each) and entries 2 l, 2 l + 1 of every 64-wide part; the token's loads are in
// flight together.  Bound: latency, then HBM; the kernel above, a CTA per token with two-byte accesses, took 42 us for 8192 rows of
// 16 heads and 10 us for 64, this one 10 and 4.4.
constexpr int kLpHeads = 8;                            // heads in flight

__global__ void __launch_bounds__(kLtWarps * 32)
latent_prep_rows_kernel(const bf16* __restrict__ proj, int64_t ld, int kv_col, const bf16* __restrict__ q, int64_t ldq,
                        const bf16* __restrict__ kv_norm_w, const int32_t* __restrict__ positions, const int32_t* __restrict__ slots,
                        bf16* cache, bf16* qa, int64_t ldqa, int T, int H, int dn, int half_layout, const double* __restrict__ freq,
                        float mag, float eps) {
  pdl_wait_in_place();      // (the heads product started beside 8192 rows' last CTAs makes a prompt layer 2 us of 560 longer)
  constexpr int R = 512, DR = 64;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const int pos = positions[t], slot = slots[t];
  const bf16* kv = proj + (size_t)t * ld + kv_col;
  const bf16* qr = q + (size_t)t * ldq + dn + 2 * lane;
  uint4 lat[2], wn[2];
  uint32_t part[kLpHeads + 1];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    lat[i] = __ldcg(reinterpret_cast<const uint4*>(kv + i * 256 + lane * 8));
    wn[i] = ld_v4(kv_norm_w + i * 256 + lane * 8);
  }
  part[kLpHeads] = __ldcg(reinterpret_cast<const uint32_t*>(kv + R + 2 * lane));
#pragma unroll
  for (int h = 0; h < kLpHeads; ++h) part[h] = __float_as_uint(ld_cg_if(reinterpret_cast<const float*>(qr + (size_t)h * (dn + DR)), h < H));
  // lane l: the angle of pair l, formed and reduced in fp64 as above
  const double ang = (double)pos * freq[lane];
  const double turns = rint(ang * 0.15915494309189535);
  float sl, cl;
  sincosf((float)fma(-turns, 6.283185307179586, ang), &sl, &cl);
  cl *= mag;
  sl *= mag;
  // half layout: entry d turns with entry d ^ 32 by pair d % 32, so lanes 16 apart exchange; interleaved: a lane's own two entries
  float c0 = cl, s0 = sl, c1 = cl, s1 = sl;
  if (half_layout) {
    const int i = (2 * lane) & 31;
    c0 = __shfl_sync(0xffffffffu, cl, i);
    s0 = __shfl_sync(0xffffffffu, sl, i);
    c1 = __shfl_sync(0xffffffffu, cl, i + 1);
    s1 = __shfl_sync(0xffffffffu, sl, i + 1);
  }
  const bool upper = lane >= 16;
  auto turn = [&](uint32_t v) {
    const float a = bf16_lo(v), b = bf16_hi(v);
    if (!half_layout) return pack_bf16(a * c0 - b * s0, b * c0 + a * s0);
    const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 16);
    const float oa = bf16_lo(o), ob = bf16_hi(o);
    return upper ? pack_bf16(a * c0 + oa * s0, b * c1 + ob * s1) : pack_bf16(a * c0 - oa * s0, b * c1 - ob * s1);
  };
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t v[4] = {lat[i].x, lat[i].y, lat[i].z, lat[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) ss = fmaf(bf16_hi(v[e]), bf16_hi(v[e]), fmaf(bf16_lo(v[e]), bf16_lo(v[e]), ss));
  }
  const float mul = 1.0f / sqrtf(warp_sum(ss) / (float)R + eps);
  const uint32_t key = turn(part[kLpHeads]);
  if (slot >= 0) {                                     // (a padding row has nothing to cache)
    bf16* row = cache + (size_t)slot * (R + DR);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t v[4] = {lat[i].x, lat[i].y, lat[i].z, lat[i].w}, w[4] = {wn[i].x, wn[i].y, wn[i].z, wn[i].w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = pack_bf16(bf16_lo(v[e]) * mul * bf16_lo(w[e]), bf16_hi(v[e]) * mul * bf16_hi(w[e]));
      st_v4(row + i * 256 + lane * 8, make_uint4(o[0], o[1], o[2], o[3]));
    }
    *reinterpret_cast<uint32_t*>(row + R + 2 * lane) = key;
  }
  bf16* qd = qa + (size_t)t * ldqa + R + 2 * lane;
  for (int h0 = 0; h0 < H; h0 += kLpHeads) {
    uint32_t next[kLpHeads];
#pragma unroll
    for (int h = 0; h < kLpHeads; ++h) {
      const int n = h0 + kLpHeads + h;
      next[h] = __float_as_uint(ld_cg_if(reinterpret_cast<const float*>(qr + (size_t)n * (dn + DR)), n < H));
    }
#pragma unroll
    for (int h = 0; h < kLpHeads; ++h) {
      const uint32_t v = turn(part[h]);
      if (h0 + h < H) *reinterpret_cast<uint32_t*>(qd + (size_t)(h0 + h) * (R + DR)) = v;
      part[h] = next[h];
    }
  }
}

}  // namespace b200

using namespace b200;

extern "C" int b200_rms_rows(const void* x, int f32, int64_t ldx, const void* w, void* out, int64_t ldo, int T, int n,
                             float eps, void* stream) {
  B200_REQUIRE(T >= 0 && n > 0 && ldx >= n && ldo >= n, "rms_rows: bad shape T=%d n=%d", T, n);
  if (T == 0) return B200_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int grid = (T + kLtWarps - 1) / kLtWarps;
  if (f32) rms_rows_kernel<float><<<grid, kLtWarps * 32, 0, s>>>((const float*)x, ldx, (const bf16*)w, (float*)out, ldo, T, n, eps);
  else rms_rows_kernel<bf16><<<grid, kLtWarps * 32, 0, s>>>((const bf16*)x, ldx, (const bf16*)w, (bf16*)out, ldo, T, n, eps);
  return b200_check_launch("b200_rms_rows");
}

extern "C" int b200_latent_prep(const void* proj, int f32, int64_t ld, int kv_col, const void* q, int64_t ldq,
                                const void* kv_norm_w, const int32_t* positions, const int32_t* slots, void* cache,
                                void* qa, int64_t ldqa, int T, int H, int dn, int dr, int R, int dims, int half_layout,
                                const double* freq, float mag, float eps, void* stream) {
  B200_REQUIRE(T >= 0 && H > 0 && dn >= 0 && dr > 0 && R > 0 && dims > 0 && dims % 2 == 0 && dims <= dr &&
                   dims <= 2 * kLtMaxPairs,
               "latent_prep: bad shape H=%d dn=%d dr=%d R=%d dims=%d", H, dn, dr, R, dims);
  if (T == 0) return B200_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // four-byte pieces of the rotated parts, sixteen-byte ones of the latents
  auto al = [](const void* p, int n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; };
  if (!f32 && R == 512 && dr == 64 && dims == 64 && ld % 8 == 0 && kv_col % 8 == 0 && ldq % 2 == 0 && dn % 2 == 0 && ldqa % 2 == 0 &&
      al(proj, 16) && al(kv_norm_w, 16) && al(cache, 16) && al(q, 4) && al(qa, 4)) {
    const int warps = T >= 4 * sm_count() ? kLtWarps : 1;     // few rows: a CTA each, over as many SMs
    (void)launch_pdl(latent_prep_rows_kernel, dim3((T + warps - 1) / warps), dim3(warps * 32), 0, s, 1, (const bf16*)proj, ld, kv_col,
                     (const bf16*)q, ldq, (const bf16*)kv_norm_w, positions, slots, (bf16*)cache, (bf16*)qa, ldqa, T, H, dn, half_layout, freq, mag, eps);
    return b200_check_launch("b200_latent_prep");
  }
  dim3 grid(T);
  const int threads = 32 * (H + 1 < kLtWarps ? H + 1 : kLtWarps);
  if (f32)
    latent_prep_kernel<float><<<grid, threads, 0, s>>>((const float*)proj, ld, kv_col, (const float*)q, ldq,
                                                            (const bf16*)kv_norm_w, positions, slots, (float*)cache,
                                                            (float*)qa, ldqa, H, dn, dr, R, dims, half_layout, freq, mag, eps);
  else
    latent_prep_kernel<bf16><<<grid, threads, 0, s>>>((const bf16*)proj, ld, kv_col, (const bf16*)q, ldq,
                                                           (const bf16*)kv_norm_w, positions, slots, (bf16*)cache,
                                                           (bf16*)qa, ldqa, H, dn, dr, R, dims, half_layout, freq, mag, eps);
  return b200_check_launch("b200_latent_prep");
}
