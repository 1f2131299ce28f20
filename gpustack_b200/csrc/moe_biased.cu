// Routing with a choice correction and identity experts, and the combine that closes such a layer.
//
//   moe_route_biased:  s = softmax(z) over all E router outputs (fp32 logits); the K outputs with the largest
//                      s + correction are chosen (ties: the lowest index); their weights are
//                      s / (sum of the chosen s + 1e-20) * scale -- the correction steers the choice only.
//   moe_route_scored:  the same with two options: s = sigmoid(z) per output instead of the softmax, and weights that
//                      are the chosen scores as they are (times scale), not renormalised.
//                      A third form chooses by z + correction (here the router's learned bias, part of the logit) and
//                      weights with the softmax over the chosen logits alone.
//                      With groups the outputs form equal groups of neighbours: only outputs of the groups_keep groups
//                      with the largest choice scores (the best one in each) can be chosen, ties to the lowest index.
//   moe_combine_mixed: out[t] = sum_j ( id_j < n_real ? yp[pair_row[t K + j]] : w_j * x[t] ) (+ shared[t]).
//                      Routed rows arrive already multiplied by their weight (the down projection's row
//                      scale); an identity expert returns the layer input itself times the weight.  fp32 sum in a
//                      fixed order (j = 0 .. K-1, then the shared expert), fp32 output: it enters the residual.
// The pair bookkeeping between the two (moe_align: pairs grouped by expert into whole tiles) is shared with the
// other routed models; identity experts are ordinary ids there, their tiles are skipped by the expert GEMMs.
#include "common.cuh"
#include "runtime.h"
#include "../../include/b200.h"

#include <math_constants.h>

namespace b200 {

constexpr int kRbPerLane = 8;        // E <= 256
constexpr int kRbMaxTop = 16;

// (what the kernels before wrote is read past L1: a grid that became resident early has missed its invalidation)
__device__ __forceinline__ float rb_cg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float rb_cg(const bf16* p) { return __bfloat162float(__ldcg(p)); }
__device__ __forceinline__ float4 rb_cg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 rb_cg4(const bf16* p) {
  const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
  return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}

// A warp's token t: lane l holds outputs l, l + 32, ... of its logits; gc, gbest: this warp's choice scores, best of every group
__device__ __forceinline__ void rb_route(const float* __restrict__ logits, const float* __restrict__ correction,
                                         int32_t* __restrict__ topk_ids, float* __restrict__ topk_w, int t, int E, int K, float scale,
                                         int score_mode, int renormalize, int groups, int groups_keep, float* gc, float* gbest) {
  const int lane = threadIdx.x & 31;
  float s[kRbPerLane], c[kRbPerLane];
  float mx = -CUDART_INF_F;
#pragma unroll
  for (int i = 0; i < kRbPerLane; ++i) {
    const int e = lane + 32 * i;
    s[i] = e < E ? logits[e] : -CUDART_INF_F;
    mx = fmaxf(mx, s[i]);
  }
  mx = warp_max(mx);
  if (score_mode == 2) {
    // the biased logits themselves are chosen from and go into the softmax over the chosen (below)
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      if (e < E && correction != nullptr) s[i] += correction[e];
      c[i] = e < E ? s[i] : -CUDART_INF_F;
    }
  } else if (score_mode == 1) {
    // every output scored on its own; without a correction the choice is made on the logits themselves (the
    // sigmoid is monotone, and two large logits must not tie where it saturates)
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      const float z = s[i];
      s[i] = e < E ? 1.0f / (1.0f + expf(-z)) : 0.f;
      c[i] = e < E ? (correction != nullptr ? s[i] + correction[e] : z) : -CUDART_INF_F;
    }
  } else {
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      s[i] = e < E ? expf(s[i] - mx) : 0.f;
      sum += s[i];
    }
    const float inv = 1.0f / warp_sum(sum);
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      s[i] *= inv;
      c[i] = e < E ? s[i] + (correction != nullptr ? correction[e] : 0.f) : -CUDART_INF_F;
    }
  }
  if (groups > 1 && groups_keep < groups) {
    float* cs = gc;
    float* gs = gbest;
    const int n = E / groups;
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i)
      if (lane + 32 * i < E) cs[lane + 32 * i] = c[i];
    __syncwarp();
    for (int g = lane; g < groups; g += 32) {
      float b = cs[g * n];
      for (int j = 1; j < n; ++j) b = fmaxf(b, cs[g * n + j]);
      gs[g] = b;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      if (e < E) {
        const int g = e / n;
        const float mine = gs[g];
        int ahead = 0;
        for (int j = 0; j < groups; ++j) ahead += (gs[j] > mine || (gs[j] == mine && j < g)) ? 1 : 0;
        if (ahead >= groups_keep) c[i] = -CUDART_INF_F;
      }
    }
  }
  float wsum = 0.f, mine_w = 0.f, top_z = 0.f;
  int mine_id = 0;
  for (int j = 0; j < K; ++j) {
    float bv = -CUDART_INF_F, bs = 0.f;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i) {
      const int e = lane + 32 * i;
      if (e < E && c[i] > bv) { bv = c[i]; be = e; bs = s[i]; }       // ascending e: the lowest index wins a tie
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o), os = __shfl_xor_sync(0xffffffffu, bs, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ov > bv || (ov == bv && oe < be)) { bv = ov; be = oe; bs = os; }
    }
    if (be >= E) { be = j; bs = 0.f; }                                 // logits that are not numbers: still a valid id
#pragma unroll
    for (int i = 0; i < kRbPerLane; ++i)
      if (lane + 32 * i == be) c[i] = -CUDART_INF_F;                   // taken
    if (score_mode == 2) {                                             // the first choice is the largest logit
      if (j == 0) top_z = bs;
      bs = expf(bs - top_z);
    }
    wsum += bs;
    if (lane == j) { mine_id = be; mine_w = bs; }
  }
  if (lane < K) {
    topk_ids[(size_t)t * K + lane] = mine_id;
    topk_w[(size_t)t * K + lane] = (renormalize ? mine_w / (wsum + 1e-20f) : mine_w) * scale;
  }
}

__global__ void __launch_bounds__(128)
moe_route_biased_kernel(const float* __restrict__ logits, int64_t ld, const float* __restrict__ correction,
                        int32_t* __restrict__ topk_ids, float* __restrict__ topk_w, int T, int E, int K, float scale,
                        int score_mode, int renormalize, int groups, int groups_keep) {
  __shared__ float gc[4][32 * kRbPerLane], gbest[4][32 * kRbPerLane];
  const int w = threadIdx.x >> 5, t = blockIdx.x * 4 + w;
  if (t < T)
    rb_route(logits + (size_t)t * ld, correction, topk_ids, topk_w, t, E, K, scale, score_mode, renormalize, groups, groups_keep, gc[w],
             gbest[w]);
}

// The router's product and the choice in one launch, a cluster of eight CTAs per two tokens: each of its 64 warps sums the
// products of two outputs at a time with both tokens in fp32, writes the logits and leaves them in the first CTA's shared
// memory, whose first two warps choose.  A step of few tokens gives the tensor-core product one or two CTAs, a serial chain over
// the whole width (with the choice, 2048 -> 128: 11.5 us for
// 1 to 128 tokens; here 4.8 for one, 5.7 for 64, 7.3 for 128 and 12.4 for 256).  Bound: latency, then
// the router's rows through L2 once per pair of tokens.
constexpr int kRtWarps = 8, kRtCluster = 8, kRtRows = 2;

__global__ void __launch_bounds__(kRtWarps * 32)
moe_router_kernel(const bf16* __restrict__ x, int64_t ldx, const bf16* __restrict__ router, int64_t ldw, int N, int D, float* logits,
                  int64_t ldl, const float* __restrict__ correction, int32_t* __restrict__ topk_ids, float* __restrict__ topk_w, int T,
                  int E, int K, float scale, int score_mode, int renormalize, int groups, int groups_keep) {
  __shared__ float z[2][32 * kRbPerLane], gc[2][32 * kRbPerLane], gbest[2][32 * kRbPerLane];
  pdl_launch_dependents();
  cluster_sync_all();      // the first CTA has started: only then is its shared memory there to be stored into
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_ctarank();
  const int t0 = blockIdx.x / kRtCluster * 2;
  const bool two = t0 + 1 < T;
  const bf16* x0 = x + (size_t)t0 * ldx;
  const bf16* x1 = two ? x0 + ldx : x0;
  const uint32_t z0 = mapa_u32(z[0], 0);
  for (int r0 = (rank * kRtWarps + warp) * kRtRows; r0 < N; r0 += kRtCluster * kRtWarps * kRtRows) {
    float acc[kRtRows][2];
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) acc[r][0] = acc[r][1] = 0.f;
#pragma unroll 8
    for (int d = lane * 8; d < D; d += 256) {
      const uint4 u0 = ld_cg_v4(x0 + d), u1 = ld_cg_v4(x1 + d);
      const uint32_t p[4] = {u0.x, u0.y, u0.z, u0.w}, q[4] = {u1.x, u1.y, u1.z, u1.w};
#pragma unroll
      for (int r = 0; r < kRtRows; ++r) {
        const uint4 v = ld_v4(router + (size_t)min(r0 + r, N - 1) * ldw + d);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[r][0] = fmaf(bf16_lo(p[i]), bf16_lo(w[i]), acc[r][0]);
          acc[r][1] = fmaf(bf16_lo(q[i]), bf16_lo(w[i]), acc[r][1]);
          acc[r][0] = fmaf(bf16_hi(p[i]), bf16_hi(w[i]), acc[r][0]);
          acc[r][1] = fmaf(bf16_hi(q[i]), bf16_hi(w[i]), acc[r][1]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRtRows; ++r)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const float sum = warp_sum(acc[r][t]);
        if (lane != 0 || r0 + r >= N || (t == 1 && !two)) continue;
        logits[(size_t)(t0 + t) * ldl + r0 + r] = sum;
        if (r0 + r < E)
          asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(z0 + (uint32_t)(t * 32 * kRbPerLane + r0 + r) * 4u), "f"(sum) : "memory");
      }
  }
  cluster_sync_all();
  if (rank == 0 && warp < (two ? 2 : 1))
    rb_route(z[warp], correction, topk_ids, topk_w, t0 + warp, E, K, scale, score_mode, renormalize, groups, groups_keep, gc[warp], gbest[warp]);
}

// VEC: four neighbouring columns per thread (D % 4 == 0 and every row aligned for it)
template <typename TX, typename TP, bool VEC>
__global__ void __launch_bounds__(256)
moe_combine_mixed_kernel(const TP* __restrict__ yp, int64_t ldp, const int32_t* __restrict__ pair_row,
                         const int32_t* __restrict__ topk_ids, const float* __restrict__ topk_w,
                         const TX* __restrict__ x, int64_t ldx, const TP* __restrict__ shared, int64_t lds,
                         float* __restrict__ out, int64_t ldo, int T, int D, int K, int n_real) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int V = VEC ? 4 : 1;
  const size_t total = (size_t)T * D / V;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / (D / V)), d = (int)(i % (D / V)) * V;
    if constexpr (VEC) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int j = 0; j < K; ++j) {
        const int id = __ldcg(topk_ids + (size_t)t * K + j);
        if (id < n_real) {
          const float4 v = rb_cg4(yp + (size_t)__ldcg(pair_row + (size_t)t * K + j) * ldp + d);
          acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        } else {
          const float w = __ldcg(topk_w + (size_t)t * K + j);
          const float4 v = rb_cg4(x + (size_t)t * ldx + d);
          acc.x += w * v.x; acc.y += w * v.y; acc.z += w * v.z; acc.w += w * v.w;
        }
      }
      if (shared != nullptr) {
        const float4 v = rb_cg4(shared + (size_t)t * lds + d);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      *reinterpret_cast<float4*>(out + (size_t)t * ldo + d) = acc;
    } else {
      float acc = 0.f;
      for (int j = 0; j < K; ++j) {
        const int id = __ldcg(topk_ids + (size_t)t * K + j);
        if (id < n_real) acc += rb_cg(yp + (size_t)__ldcg(pair_row + (size_t)t * K + j) * ldp + d);
        else acc += __ldcg(topk_w + (size_t)t * K + j) * rb_cg(x + (size_t)t * ldx + d);
      }
      if (shared != nullptr) acc += rb_cg(shared + (size_t)t * lds + d);
      out[(size_t)t * ldo + d] = acc;
    }
  }
}

}  // namespace b200

using namespace b200;

static int rb_check(int T, int E, int K, int score_mode, int groups, int groups_keep) {
  B200_REQUIRE(T >= 0 && E >= 1 && E <= 32 * kRbPerLane && K >= 1 && K <= kRbMaxTop && K <= E,
               "moe_route_biased: unsupported E=%d K=%d (E <= %d, K <= %d)", E, K, 32 * kRbPerLane, kRbMaxTop);
  B200_REQUIRE(score_mode >= 0 && score_mode <= 2, "moe_route_biased: unknown score form %d", score_mode);
  B200_REQUIRE(groups == 0 || (groups > 0 && E % groups == 0 && groups_keep >= 1 && groups_keep <= groups && K <= groups_keep * (E / groups)),
               "moe_route_biased: %d of %d groups of %d outputs, K=%d", groups_keep, groups, E, K);
  return B200_OK;
}

extern "C" int b200_moe_route_grouped(const float* logits, int64_t ld, const float* correction, int32_t* topk_ids,
                                      float* topk_w, int T, int E, int K, float scale, int score_mode, int renormalize,
                                      int groups, int groups_keep, void* stream) {
  B200_REQUIRE(ld >= E, "moe_route_biased: row stride %lld < E=%d", (long long)ld, E);
  if (int rc = rb_check(T, E, K, score_mode, groups, groups_keep)) return rc;
  if (T == 0) return B200_OK;
  moe_route_biased_kernel<<<(T + 3) / 4, 128, 0, (cudaStream_t)stream>>>(logits, ld, correction, topk_ids, topk_w, T, E, K,
                                                                       scale, score_mode, renormalize, groups, groups_keep);
  return b200_check_launch("b200_moe_route_biased");
}

extern "C" int b200_moe_router(const void* x, int64_t ldx, const void* router, int64_t ldw, int N, int D, float* logits, int64_t ldl,
                               const float* correction, int32_t* topk_ids, float* topk_w, int T, int E, int K, float scale, int score_mode,
                               int renormalize, int groups, int groups_keep, void* stream) {
  B200_REQUIRE(D > 0 && D % 8 == 0 && ldx >= D && ldw >= D && ldx % 8 == 0 && ldw % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(router)) & 15) == 0,
               "moe_router: 16-byte aligned bf16 rows of a multiple of 8 columns required (D=%d)", D);
  B200_REQUIRE(N >= E && ldl >= N, "moe_router: %d rows for %d outputs, logits of row stride %lld", N, E, (long long)ldl);
  if (int rc = rb_check(T, E, K, score_mode, groups, groups_keep)) return rc;
  if (T == 0) return B200_OK;
  const cudaError_t e = launch_pdl_cls(kPdlMoe, moe_router_kernel, dim3((T + 1) / 2 * kRtCluster), dim3(kRtWarps * 32), 0, (cudaStream_t)stream,
                                       kRtCluster, (const bf16*)x, ldx, (const bf16*)router, ldw, N, D, logits, ldl, correction, topk_ids,
                                       topk_w, T, E, K, scale, score_mode, renormalize, groups, groups_keep);
  if (e != cudaSuccess) {
    b200_set_error("b200_moe_router: launch failed: %s", cudaGetErrorString(e));
    (void)cudaGetLastError();
    return B200_ERR_CUDA;
  }
  return b200_check_launch("b200_moe_router");
}

extern "C" int b200_moe_route_scored(const float* logits, int64_t ld, const float* correction, int32_t* topk_ids,
                                     float* topk_w, int T, int E, int K, float scale, int score_mode,
                                     int renormalize, void* stream) {
  return b200_moe_route_grouped(logits, ld, correction, topk_ids, topk_w, T, E, K, scale, score_mode, renormalize, 0, 0, stream);
}

extern "C" int b200_moe_route_biased(const float* logits, int64_t ld, const float* correction, int32_t* topk_ids,
                                     float* topk_w, int T, int E, int K, float scale, void* stream) {
  return b200_moe_route_scored(logits, ld, correction, topk_ids, topk_w, T, E, K, scale, 0, 1, stream);
}

extern "C" int b200_moe_combine_mixed(const void* yp, int p_f32, int64_t ldp, const int32_t* pair_row,
                                      const int32_t* topk_ids, const float* topk_w, const void* x, int x_f32, int64_t ldx,
                                      const void* shared, int64_t lds, float* out, int64_t ldo, int T, int D, int K,
                                      int n_real, void* stream) {
  B200_REQUIRE(T >= 0 && D > 0 && K >= 1, "moe_combine_mixed: bad shape");
  if (T == 0) return B200_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const uintptr_t xm = x_f32 ? 15 : 7, pm = p_f32 ? 15 : 7;
  const bool vec = D % 4 == 0 && ldp % 4 == 0 && ldx % 4 == 0 && lds % 4 == 0 && ldo % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(yp) | reinterpret_cast<uintptr_t>(shared)) & pm) == 0 &&
                   (reinterpret_cast<uintptr_t>(x) & xm) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  size_t blocks = ((size_t)T * D / (vec ? 4 : 1) + 255) / 256;
  if (blocks > 8192) blocks = 8192;
#define B200_CMV(TX, TP, V)                                                                                          \
  (void)launch_pdl_cls(kPdlMoe, moe_combine_mixed_kernel<TX, TP, V>, dim3((unsigned)blocks), dim3(256), 0, s, 1, (const TP*)yp, ldp, \
                       pair_row, topk_ids, topk_w, (const TX*)x, ldx, (const TP*)shared, lds, out, ldo, T, D, K, n_real)
#define B200_CM(TX, TP)                     \
  do {                                      \
    if (vec) B200_CMV(TX, TP, true);        \
    else B200_CMV(TX, TP, false);           \
  } while (0)
  if (x_f32 && p_f32) B200_CM(float, float);
  else if (x_f32) B200_CM(float, bf16);
  else if (p_f32) B200_CM(bf16, float);
  else B200_CM(bf16, bf16);
#undef B200_CM
#undef B200_CMV
  return b200_check_launch("b200_moe_combine_mixed");
}
