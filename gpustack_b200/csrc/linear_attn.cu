// Linear attention with a fixed decay per head: no softmax, no denominator, state in fp32.
//
// Per head, with the constant decay d_h:
//     S_t = d_h S_{t-1} + k_t v_t^T          (S: dk x dv, zero before a sequence's first token)
//     o_t = S_t^T q_t
// Queries, keys and values arrive as fp32 rows (the per-head preparation -- feature map, rotation, factors -- has
// been applied; rot_prep.cu); the state of slot s is S [slots][H][dv][dk] (key index fastest), so that a warp's
// loads and stores are contiguous.  A sequence whose context is empty starts from zero, whatever the slot held
// before: a slot that is handed to a new sequence needs no clearing.
//
// `linattn_scan`   runs a sequence's new rows in order (the single row of a decode step, or a short portion); grid
//                  (sequences, heads, ceil(dv / 32)): a CTA owns 32 value columns of one head's state, each of its 8
//                  warps 4 of them; lane r holds the key rows r, r + 32, ... of those columns in registers; S^T q is
//                  a warp-shuffle reduction, no block barrier per token.
// `linattn_chunk`  the same recurrence for prompt portions, 16 rows at a time without a serial dependency inside a
//                  chunk.  With the state S_0 at the chunk's start and rows t = 0 .. n-1:
//                      o_t = d^{t+1} S_0^T q_t + sum_{s<=t} d^{t-s} (k_s . q_t) v_s
//                      S_n = d^n S_0 + sum_s d^{n-1-s} k_s v_s^T
//                  Every power has a non-negative exponent (nothing is divided by a decay, so a small decay cannot
//                  overflow); all products and sums are fp32 FMAs, only the grouping of the sums differs from the
//                  serial form.  The CTA's 32 columns of S live in shared memory for the whole portion.
// The same over chunks of 128 rows side by side (chunk_tc.cuh) when the caller brings a workspace.
// `linattn_out`    closes the mixer: the heads' outputs over their root mean square -- per head without a weight, or
//                  all heads together with a weight vector -- times sigmoid(g) or silu(g) of the gate columns of the
//                  fused projection, rounded once to the activation type.
#include "chunk_tc.cuh"
#include "common.cuh"
#include "head_out.cuh"
#include "runtime.h"
#include "../../include/b200.h"

namespace b200 {

__device__ __forceinline__ float la_f32(float v) { return v; }
__device__ __forceinline__ float la_f32(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void la_store(float* p, float v) { *p = v; }
__device__ __forceinline__ void la_store(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

constexpr int kLaWarps = 8, kLaColsPerWarp = 4, kLaCols = kLaWarps * kLaColsPerWarp, kLaTok = 16;

// EPT = key rows per lane = ceil(dk / 32)
template <int EPT>
__global__ void __launch_bounds__(kLaWarps * 32)
linattn_scan_kernel(const float* __restrict__ x, int64_t ld, int q_col, int k_col, int v_col,
                    const float* __restrict__ decay, const int32_t* __restrict__ cu_seq,
                    const int32_t* __restrict__ ctx_lens, const int32_t* __restrict__ state_slots, float* S_state,
                    float* __restrict__ o_raw, int H, int dk, int dv) {
  extern __shared__ float smem[];
  float* qs = smem;                                   // [16][dk]
  float* ks = qs + kLaTok * dk;                       // [16][dk]
  float* vs = ks + kLaTok * dk;                       // [16][32]
  const int s = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
  const int slot = state_slots[s];
  if (slot < 0) return;
  const int t0 = cu_seq[s], t1 = cu_seq[s + 1];
  if (t1 <= t0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = z * kLaCols + warp * kLaColsPerWarp;
  float* Sp = S_state + ((size_t)slot * H + h) * dv * dk;
  const float d = decay[h];
  const bool fresh = ctx_lens[s] == 0;
  float S[EPT][kLaColsPerWarp];
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int row = lane + 32 * j;
#pragma unroll
    for (int c = 0; c < kLaColsPerWarp; ++c)
      S[j][c] = (!fresh && row < dk && c0 + c < dv) ? Sp[(size_t)(c0 + c) * dk + row] : 0.f;
  }
  if (t1 - t0 == 1) {
    // a decode row: no staging, no barrier; the state and the inputs are in flight together
    const float* row = x + (size_t)t0 * ld;
    float kk[EPT], qq[EPT], v[kLaColsPerWarp], num[kLaColsPerWarp];
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int r = lane + 32 * j;
      kk[j] = r < dk ? row[k_col + h * dk + r] : 0.f;
      qq[j] = r < dk ? row[q_col + h * dk + r] : 0.f;
    }
#pragma unroll
    for (int c = 0; c < kLaColsPerWarp; ++c) {
      v[c] = c0 + c < dv ? row[v_col + h * dv + c0 + c] : 0.f;
      num[c] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < EPT; ++j)
#pragma unroll
      for (int c = 0; c < kLaColsPerWarp; ++c) {
        S[j][c] = fmaf(d, S[j][c], kk[j] * v[c]);
        num[c] = fmaf(S[j][c], qq[j], num[c]);
      }
#pragma unroll
    for (int c = 0; c < kLaColsPerWarp; ++c) num[c] = warp_sum(num[c]);
    if (lane < kLaColsPerWarp && c0 + lane < dv) {
      float mine = num[0];
#pragma unroll
      for (int c = 1; c < kLaColsPerWarp; ++c) mine = lane == c ? num[c] : mine;
      o_raw[(size_t)t0 * H * dv + h * dv + c0 + lane] = mine;
    }
  } else {
    for (int ch = t0; ch < t1; ch += kLaTok) {
      const int nt = min(kLaTok, t1 - ch);
      __syncthreads();                                // every warp is done with the previous chunk
      for (int i = threadIdx.x; i < nt * dk; i += blockDim.x) {
        const int tt = i / dk, dd = i - tt * dk;
        const float* row = x + (size_t)(ch + tt) * ld;
        qs[i] = row[q_col + h * dk + dd];
        ks[i] = row[k_col + h * dk + dd];
      }
      for (int i = threadIdx.x; i < nt * kLaCols; i += blockDim.x) {
        const int tt = i / kLaCols, c = z * kLaCols + (i % kLaCols);
        vs[i] = c < dv ? x[(size_t)(ch + tt) * ld + v_col + h * dv + c] : 0.f;
      }
      __syncthreads();
      for (int tt = 0; tt < nt; ++tt) {
        float v[kLaColsPerWarp], num[kLaColsPerWarp];
#pragma unroll
        for (int c = 0; c < kLaColsPerWarp; ++c) {
          v[c] = vs[tt * kLaCols + warp * kLaColsPerWarp + c];
          num[c] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < EPT; ++j) {
          const int row = lane + 32 * j;
          if (row < dk) {
            const float kk = ks[tt * dk + row], qq = qs[tt * dk + row];
#pragma unroll
            for (int c = 0; c < kLaColsPerWarp; ++c) {
              S[j][c] = fmaf(d, S[j][c], kk * v[c]);
              num[c] = fmaf(S[j][c], qq, num[c]);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < kLaColsPerWarp; ++c) num[c] = warp_sum(num[c]);
        if (lane < kLaColsPerWarp && c0 + lane < dv) {
          float mine = num[0];
#pragma unroll
          for (int c = 1; c < kLaColsPerWarp; ++c) mine = lane == c ? num[c] : mine;
          o_raw[(size_t)(ch + tt) * H * dv + h * dv + c0 + lane] = mine;
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int row = lane + 32 * j;
    if (row < dk) {
#pragma unroll
      for (int c = 0; c < kLaColsPerWarp; ++c)
        if (c0 + c < dv) Sp[(size_t)(c0 + c) * dk + row] = S[j][c];
    }
  }
}

// ------------------------------------------------------------------------------------- chunk form
constexpr int kLcTok = 16, kLcThreads = 512;

__global__ void __launch_bounds__(kLcThreads)
linattn_chunk_kernel(const float* __restrict__ x, int64_t ld, int q_col, int k_col, int v_col,
                     const float* __restrict__ decay, const int32_t* __restrict__ cu_seq,
                     const int32_t* __restrict__ ctx_lens, const int32_t* __restrict__ state_slots, float* S_state,
                     float* __restrict__ o_raw, int H, int dk, int dv) {
  extern __shared__ float smem[];
  const int dkp = dk + 1;
  float* Ssm = smem;                                  // [dk][33]
  float* qs = Ssm + dk * 33;                          // [16][dk + 1]
  float* ks = qs + kLcTok * dkp;                      // [16][dk + 1]
  float* vs = ks + kLcTok * dkp;                      // [16][32]
  float* A = vs + kLcTok * 32;                        // [16][17]   k_s . q_t
  float* dp = A + kLcTok * 17;                        // [17]       d^0 .. d^16
  const int s = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
  const int slot = state_slots[s];
  if (slot < 0) return;
  const int t0 = cu_seq[s], t1 = cu_seq[s + 1];
  if (t1 <= t0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = z * 32;
  float* Sp = S_state + ((size_t)slot * H + h) * dv * dk;
  const bool fresh = ctx_lens[s] == 0;
  for (int i = tid; i < dk * 32; i += kLcThreads) {
    const int c = i / dk, r = i - c * dk;             // r fastest: contiguous global reads
    Ssm[r * 33 + c] = (!fresh && c0 + c < dv) ? Sp[(size_t)(c0 + c) * dk + r] : 0.f;
  }
  if (tid <= kLcTok) dp[tid] = (float)pow((double)decay[h], (double)tid);
  for (int ch = t0; ch < t1; ch += kLcTok) {
    const int nt = min(kLcTok, t1 - ch);
    __syncthreads();                                  // state update of the previous chunk done, inputs free
    for (int i = tid; i < nt * dk; i += kLcThreads) {
      const int tt = i / dk, dd = i - tt * dk;
      const float* row = x + (size_t)(ch + tt) * ld;
      qs[tt * dkp + dd] = row[q_col + h * dk + dd];
      ks[tt * dkp + dd] = row[k_col + h * dk + dd];
    }
    {
      const int tt = tid >> 5, c = c0 + (tid & 31);
      vs[tid] = (tt < nt && c < dv) ? x[(size_t)(ch + tt) * ld + v_col + h * dv + c] : 0.f;
    }
    __syncthreads();
    // (a) k_s . q_t for s <= t
    if (tid < 256) {
      const int t = tid >> 4, sx = tid & 15;
      if (t < nt && sx <= t) {
        float acc = 0.f;
        const float* kr = ks + sx * dkp;
        const float* qr = qs + t * dkp;
        for (int r = 0; r < dk; ++r) acc = fmaf(kr[r], qr[r], acc);
        A[t * 17 + sx] = acc;
      }
    }
    __syncthreads();
    // (b) outputs: thread = (row = warp, column = lane)
    if (warp < nt) {
      const int t = warp;
      float acc = 0.f;
      const float* qr = qs + t * dkp;
      for (int r = 0; r < dk; ++r) acc = fmaf(Ssm[r * 33 + lane], qr[r], acc);
      float num = dp[t + 1] * acc;
      for (int sx = 0; sx <= t; ++sx) num = fmaf(dp[t - sx] * A[t * 17 + sx], vs[sx * 32 + lane], num);
      if (c0 + lane < dv) o_raw[(size_t)(ch + t) * H * dv + h * dv + c0 + lane] = num;
    }
    __syncthreads();
    // (c) state update: S[r][c] = d^n S[r][c] + sum_s d^{n-1-s} k_s[r] v_s[c]
    for (int i = tid; i < dk * 32; i += kLcThreads) {
      const int r = i >> 5, c = i & 31;
      float acc = dp[nt] * Ssm[r * 33 + c];
      for (int sx = 0; sx < nt; ++sx) acc = fmaf(dp[nt - 1 - sx] * ks[sx * dkp + r], vs[sx * 32 + c], acc);
      Ssm[r * 33 + c] = acc;
    }
  }
  __syncthreads();
  for (int i = tid; i < dk * 32; i += kLcThreads) {
    const int c = i / dk, r = i - c * dk;
    if (c0 + c < dv) Sp[(size_t)(c0 + c) * dk + r] = Ssm[r * 33 + c];
  }
}

// The chunk form for key widths that are multiples of 4 (every real head): register tiles and 16-byte shared loads.
//   * queries are staged transposed, qT [dk][16 rows] (pitch 20), keys row-major with a pitch that keeps 16-byte alignment;
//   * S_0^T q_t: a thread owns one state column, FOUR rows of the chunk and a quarter of the key range -- one state
//     element and one 16-byte query load feed four FMAs; the four key-range quarters meet in shared memory;
//   * the state update: a thread owns FOUR key rows of one column -- one value and one 16-byte key load per chunk row
//     feed four FMAs;
//   * the next chunk's inputs travel in registers while this one is computed.
constexpr int kL4Pre = 8;            // 16 * dk / 512 elements of q and of k per thread: dk <= 256
constexpr int kL4QP = 20;            // pitch of qT

__global__ void __launch_bounds__(kLcThreads)
linattn_chunk4_kernel(const float* __restrict__ x, int64_t ld, int q_col, int k_col, int v_col,
                      const float* __restrict__ decay, const int32_t* __restrict__ cu_seq,
                      const int32_t* __restrict__ ctx_lens, const int32_t* __restrict__ state_slots, float* S_state,
                      float* __restrict__ o_raw, int H, int dk, int dv, int most_rows) {
  if (most_rows != INT32_MAX) ct_release_next();      // the other sequences' chunks, which touch nothing of these
  extern __shared__ __align__(16) float smem[];
  const int kst = dk + 4;
  float* Ssm = smem;                                  // [dk][33]
  float* qT = Ssm + ((dk * 33 + 3) & ~3);             // [dk][20]
  float* ks = qT + dk * kL4QP;                        // [16][dk + 4]
  float* vs = ks + kLcTok * kst;                      // [16][32]
  float* part = vs + kLcTok * 32;                     // [4][16][32]
  float* A = part + 4 * kLcTok * 32;                  // [16][17]
  float* dp = A + kLcTok * 17;                        // [17]
  const int s = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
  const int slot = state_slots[s];
  if (slot < 0) return;
  const int t0 = cu_seq[s], t1 = cu_seq[s + 1];
  if (t1 <= t0 || t1 - t0 > most_rows) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = z * 32;
  float* Sp = S_state + ((size_t)slot * H + h) * dv * dk;
  const bool fresh = ctx_lens[s] == 0;
  for (int i = tid; i < dk * 32; i += kLcThreads) {
    const int c = i / dk, r = i - c * dk;
    Ssm[r * 33 + c] = (!fresh && c0 + c < dv) ? Sp[(size_t)(c0 + c) * dk + r] : 0.f;
  }
  for (int i = tid; i < dk * kL4QP; i += kLcThreads) qT[i] = 0.f;     // rows of a short last chunk stay finite
  if (tid <= kLcTok) dp[tid] = (float)pow((double)decay[h], (double)tid);
  float rq[kL4Pre], rk[kL4Pre], rv = 0.f;
  auto fetch = [&](int ch, int nt) {
#pragma unroll
    for (int u = 0; u < kL4Pre; ++u) {
      const int i = tid + u * kLcThreads;
      if (i < nt * dk) {
        const int tt = i / dk, d = i - tt * dk;
        const float* row = x + (size_t)(ch + tt) * ld;
        rq[u] = row[q_col + h * dk + d];
        rk[u] = row[k_col + h * dk + d];
      }
    }
    const int tt = tid >> 5, c = c0 + (tid & 31);
    rv = (tt < nt && c < dv) ? x[(size_t)(ch + tt) * ld + v_col + h * dv + c] : 0.f;
  };
  fetch(t0, min(kLcTok, t1 - t0));
  for (int ch = t0; ch < t1; ch += kLcTok) {
    const int nt = min(kLcTok, t1 - ch);
    __syncthreads();                                  // state update of the previous chunk done, inputs free
#pragma unroll
    for (int u = 0; u < kL4Pre; ++u) {
      const int i = tid + u * kLcThreads;
      if (i < nt * dk) {
        const int tt = i / dk, d = i - tt * dk;
        qT[d * kL4QP + tt] = rq[u];
        ks[tt * kst + d] = rk[u];
      }
    }
    vs[tid] = rv;
    if (ch + kLcTok < t1) fetch(ch + kLcTok, min(kLcTok, t1 - ch - kLcTok));
    __syncthreads();
    // (a) k_s . q_t for s <= t
    if (tid < 256) {
      const int t = tid >> 4, sx = tid & 15;
      if (t < nt && sx <= t) {
        float acc = 0.f;
        const float* kr = ks + sx * kst;
        for (int r = 0; r < dk; ++r) acc = fmaf(kr[r], qT[r * kL4QP + t], acc);
        A[t * 17 + sx] = acc;
      }
    }
    // (b) S_0^T q_t: column = lane, rows 4 tg .. 4 tg + 3, key range quarter rq_
    {
      const int tg = warp & 3, rq_ = warp >> 2;
      const int r_lo = (dk * rq_) >> 2, r_hi = (dk * (rq_ + 1)) >> 2;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
      for (int r = r_lo; r < r_hi; ++r) {
        const float sv = Ssm[r * 33 + lane];
        const float4 q4 = *reinterpret_cast<const float4*>(qT + r * kL4QP + tg * 4);
        a0 = fmaf(sv, q4.x, a0);
        a1 = fmaf(sv, q4.y, a1);
        a2 = fmaf(sv, q4.z, a2);
        a3 = fmaf(sv, q4.w, a3);
      }
      float* pp = part + ((rq_ * kLcTok + tg * 4) * 32) + lane;
      pp[0] = a0; pp[32] = a1; pp[64] = a2; pp[96] = a3;
    }
    __syncthreads();
    // outputs: thread = (row = warp, column = lane); the quarters are added in a fixed order
    if (warp < nt) {
      const int t = warp;
      const float acc = (part[(0 * kLcTok + t) * 32 + lane] + part[(1 * kLcTok + t) * 32 + lane]) +
                        (part[(2 * kLcTok + t) * 32 + lane] + part[(3 * kLcTok + t) * 32 + lane]);
      float num = dp[t + 1] * acc;
      for (int sx = 0; sx <= t; ++sx) num = fmaf(dp[t - sx] * A[t * 17 + sx], vs[sx * 32 + lane], num);
      if (c0 + lane < dv) o_raw[(size_t)(ch + t) * H * dv + h * dv + c0 + lane] = num;
    }
    // (c) state update: S[r .. r+3][c] = d^n S + sum_s d^{n-1-s} k_s[r .. r+3] v_s[c]
    for (int it = tid; it < (dk >> 2) * 32; it += kLcThreads) {
      const int r = (it >> 5) << 2, c = it & 31;
      const float dn = dp[nt];
      float s0 = dn * Ssm[r * 33 + c], s1 = dn * Ssm[(r + 1) * 33 + c], s2 = dn * Ssm[(r + 2) * 33 + c],
            s3 = dn * Ssm[(r + 3) * 33 + c];
      for (int sx = 0; sx < nt; ++sx) {
        const float v = dp[nt - 1 - sx] * vs[sx * 32 + c];
        const float4 k4 = *reinterpret_cast<const float4*>(ks + sx * kst + r);
        s0 = fmaf(k4.x, v, s0);
        s1 = fmaf(k4.y, v, s1);
        s2 = fmaf(k4.z, v, s2);
        s3 = fmaf(k4.w, v, s3);
      }
      Ssm[r * 33 + c] = s0; Ssm[(r + 1) * 33 + c] = s1; Ssm[(r + 2) * 33 + c] = s2; Ssm[(r + 3) * 33 + c] = s3;
    }
  }
  __syncthreads();
  for (int i = tid; i < dk * 32; i += kLcThreads) {
    const int c = i / dk, r = i - c * dk;
    if (c0 + c < dv) Sp[(size_t)(c0 + c) * dk + r] = Ssm[r * 33 + c];
  }
}

// The fixed decay in the chunk form of chunk_tc.cuh: every weight is a power of the head's decay with a non-negative
// exponent, formed in fp64 by squaring (a decay of zero or below one's sign is as good as any) and rounded once.
__device__ __forceinline__ float la_power(float d, int n) {
  double r = 1.0, b = (double)d;
#pragma unroll
  for (int bit = 0; bit < 8; ++bit) {
    if ((n >> bit) & 1) r *= b;
    b *= b;
  }
  return (float)r;
}

struct LinearForm {
  static constexpr const char* kName = "b200_linattn_scan(chunks)";
  static constexpr bool kNorm = false;
  struct Params {
    const float* decay;
  };
  struct Scratch {
    float dp[kCtRows + 1], w[kCtRows];
  };
  static __device__ __forceinline__ void state_weights(const Params& p, const ChunkScanArgs&, Scratch& sc, int h, const ChunkPlace& at, int, float*) {
    const int t = ct_team_row();
    sc.w[t] = t < at.rows ? la_power(p.decay[h], at.rows - 1 - t) : 0.f;
  }
  struct Carry {
    float d;
    __device__ __forceinline__ Carry(const Params& p, const ChunkScanArgs&, int h, int) : d(p.decay[h]) {}
    __device__ __forceinline__ void factors(int c0, int, int rows, float2* table) const {
      const int c = c0 + (threadIdx.x & 31);
      table[threadIdx.x & 31] = make_float2(la_power(d, min(kCtRows, max(rows - c * kCtRows, 0))), 1.0f);
    }
  };
  template <int DK>
  static __device__ __forceinline__ void carry_row(const Params&, const ChunkScanArgs&, int, int, int, bool, int) {}
  static __device__ __forceinline__ void output_weights(const Params& p, const ChunkScanArgs&, Scratch& sc, int h, const ChunkPlace&, int) {
    sc.dp[ct_team_row() + 1] = la_power(p.decay[h], ct_team_row() + 1);
    if (ct_team_row() == 0) sc.dp[0] = 1.f;
  }
  static __device__ __forceinline__ float q_scale(const Params&) { return 1.0f; }
  struct Row {};
  static __device__ __forceinline__ Row row(const Params&, const Scratch&, int) { return {}; }
  static __device__ __forceinline__ float D(const Params&, const Scratch& sc, const Row&, int t, int s) { return sc.dp[t - s]; }
  // of sixteen rows from s0 on, all of them seen (`before`) or not
  static __device__ __forceinline__ void weights(const Params&, const Scratch& sc, const Row&, int t, int s0, bool, float (&d)[16]) {
#pragma unroll
    for (int e = 0; e < 16; ++e) d[e] = sc.dp[max(t - s0 - e, 0)];
  }
  static __device__ __forceinline__ float aq(const Scratch& sc, int t) { return sc.dp[t + 1]; }
  struct Finish {
    __device__ __forceinline__ Finish(const Params&, const ChunkScanArgs&, const Scratch&, int, int, const float*) {}
    __device__ __forceinline__ void apply(float (&)[32]) const {}
    __device__ __forceinline__ float one(float f) const { return f; }
  };
};

// ------------------------------------------------------------------------------------------- out
// One CTA per row.  all_heads: the H * dv outputs are normed together and multiplied by w; otherwise every head is
// divided by its own root mean square (w optional, dv entries shared by the heads).  gate_act 0 sigmoid, 1 silu.
template <typename TA>
__global__ void __launch_bounds__(256)
linattn_out_kernel(const float* __restrict__ o_raw, const TA* __restrict__ proj, int64_t ld, int gate_col,
                   const bf16* __restrict__ w, TA* out, int64_t ldo, int H, int dv, int all_heads, int gate_act,
                   float eps) {
  extern __shared__ float head_ss[];                  // [H]
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const float* o = o_raw + (size_t)t * H * dv;
  for (int h = warp; h < H; h += nw) {
    float ss = 0.f;
    for (int d = lane; d < dv; d += 32) {
      const float v = o[h * dv + d];
      ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) head_ss[h] = ss;
  }
  __syncthreads();
  float all = 0.f;
  if (all_heads) {
    for (int h = 0; h < H; ++h) all += head_ss[h];     // the same order in every thread
    all = 1.0f / sqrtf(all / (float)(H * dv) + eps);
  }
  const TA* g = proj + (size_t)t * ld + gate_col;
  for (int i = threadIdx.x; i < H * dv; i += blockDim.x) {
    const int h = i / dv;
    const float mul = all_heads ? all : 1.0f / sqrtf(head_ss[h] / (float)dv + eps);
    float v = o[i] * mul;
    if (w != nullptr) v *= __bfloat162float(w[all_heads ? i : i - h * dv]);
    const float gv = la_f32(g[i]);
    const float sg = 1.0f / (1.0f + expf(-gv));
    v *= gate_act == 1 ? gv * sg : sg;
    la_store(out + (size_t)t * ldo + i, v);
  }
}

}  // namespace b200

using namespace b200;

static int launch_chunk4(const float* x, int64_t ld, int q_col, int k_col, int v_col, const float* decay, const int32_t* cu_seq,
                         const int32_t* ctx_lens, const int32_t* state_slots, float* S, float* o_raw, int n_seqs, int H, int dk, int dv,
                         int most_rows, cudaStream_t s) {
  const size_t smem4 = sizeof(float) * ((((size_t)dk * 33 + 3) & ~(size_t)3) + (size_t)dk * kL4QP + (size_t)kLcTok * (dk + 4) +
                                        kLcTok * 32 + 4 * kLcTok * 32 + kLcTok * 17 + 32);
  if (smem4 > 48 * 1024)
    cudaFuncSetAttribute(linattn_chunk4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem4);
  linattn_chunk4_kernel<<<dim3(n_seqs, H, (dv + kLaCols - 1) / kLaCols), kLcThreads, smem4, s>>>(
      x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S, o_raw, H, dk, dv, most_rows);
  return b200_check_launch("b200_linattn_scan(chunk4)");
}

extern "C" int b200_linattn_scan(const float* x, int64_t ld, int q_col, int k_col, int v_col, const float* decay,
                                 const int32_t* cu_seq, const int32_t* ctx_lens, const int32_t* state_slots, float* S,
                                 float* o_raw, int n_seqs, int H, int dk, int dv, int max_len, void* stream) {
  B200_REQUIRE(n_seqs >= 0 && H > 0 && dk > 0 && dv > 0 && dk <= 256, "linattn_scan: bad shape H=%d dk=%d dv=%d (dk <= 256)",
               H, dk, dv);
  if (n_seqs == 0) return B200_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int Z = (dv + kLaCols - 1) / kLaCols;
  dim3 grid(n_seqs, H, Z);
  if (max_len > 2 && dk % 4 == 0) {
    // prompt portions: the chunk form (a single decode row riding in the same launch is a chunk of one)
    return launch_chunk4(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S, o_raw, n_seqs, H, dk, dv, INT32_MAX, s);
  }
  if (max_len > 2) {
    // key widths that are not multiples of 4: the element-wise chunk kernel
    const size_t smem = sizeof(float) * ((size_t)dk * 33 + 2 * (size_t)kLcTok * (dk + 1) + kLcTok * 32 + kLcTok * 17 + 32);
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(linattn_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    linattn_chunk_kernel<<<grid, kLcThreads, smem, s>>>(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S,
                                                        o_raw, H, dk, dv);
    return b200_check_launch("b200_linattn_scan(chunk)");
  }
  const size_t smem = sizeof(float) * (2 * (size_t)kLaTok * dk + kLaTok * kLaCols);
#define B200_LA(E)                                                                                              \
  linattn_scan_kernel<E><<<grid, kLaWarps * 32, smem, s>>>(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, \
                                                           state_slots, S, o_raw, H, dk, dv)
  if (dk <= 32) B200_LA(1);
  else if (dk <= 64) B200_LA(2);
  else if (dk <= 128) B200_LA(4);
  else B200_LA(8);
#undef B200_LA
  return b200_check_launch("b200_linattn_scan");
}

// The same with a workspace of b200_chunk_scan_floats(rows, n_seqs, H, dk, dv, 0) floats: sequences of more than 16 rows run with
// all their chunks side by side, the others one-pass beside them.  Shapes and alignments that the chunk kernels do not take
// run as b200_linattn_scan.
extern "C" int b200_linattn_scan_chunked(const float* x, int64_t ld, int q_col, int k_col, int v_col, const float* decay,
                                         const int32_t* cu_seq, const int32_t* ctx_lens, const int32_t* state_slots, float* S,
                                         float* o_raw, int n_seqs, int H, int dk, int dv, int max_len, int rows, float* workspace,
                                         int64_t workspace_floats, void* stream) {
  if (workspace == nullptr || rows <= 0 || n_seqs <= 0 || H <= 0 || dv <= 0 || ((uintptr_t)workspace & 15) != 0 ||
      !cs_covers(x, 4, ld, q_col, k_col, v_col, dk, dv, S, o_raw))
    return b200_linattn_scan(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S, o_raw, n_seqs, H, dk, dv, max_len,
                             stream);
  B200_REQUIRE(workspace_floats >= cs_workspace_floats(rows, n_seqs, H, dk, dv), "linattn_scan: workspace of %lld floats too small",
               (long long)workspace_floats);
  cudaStream_t s = (cudaStream_t)stream;
  const int group = (int)ct_group(rows, n_seqs, H, dk, dv, workspace_floats);
  if (group == 0)                                     // (fewer than 64 rows)
    return b200_linattn_scan(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S, o_raw, n_seqs, H, dk, dv, max_len,
                             stream);
  const int short_rows = cs_short(rows, n_seqs);
  if (short_rows > 0) {
    const int rc = launch_chunk4(x, ld, q_col, k_col, v_col, decay, cu_seq, ctx_lens, state_slots, S, o_raw, n_seqs, H, dk, dv,
                                 short_rows, s);
    if (rc != B200_OK) return rc;
  }
  const ChunkScanArgs a{x, ld, q_col, k_col, v_col, H, H, dv, cu_seq, ctx_lens, state_slots, n_seqs, short_rows, S, o_raw};
  return ct_launch<float, LinearForm>(a, {decay}, dk, rows, group, workspace, s);
}

extern "C" int b200_linattn_out(const float* o_raw, const void* proj, int f32, int64_t ld, int gate_col, const void* w,
                                void* out, int64_t ldo, int T, int H, int dv, int all_heads, int gate_act, float eps,
                                void* stream) {
  B200_REQUIRE(T >= 0 && H > 0 && dv > 0 && H <= 8192, "linattn_out: bad shape");
  B200_REQUIRE(!all_heads || w != nullptr, "linattn_out: the joint norm has a weight");
  if (T == 0) return B200_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // a norm per head keeps its heads in registers; the joint norm, and widths the other does not take, one CTA per row
  if (!all_heads && (f32 ? head_out_launch<float>(o_raw, proj, ld, gate_col, w, 0, out, ldo, T, H, dv, gate_act, eps, s)
                         : head_out_launch<bf16>(o_raw, proj, ld, gate_col, w, 0, out, ldo, T, H, dv, gate_act, eps, s)))
    return b200_check_launch("b200_linattn_out(heads)");
  const size_t smem = sizeof(float) * H;
  if (f32)
    linattn_out_kernel<float><<<T, 256, smem, s>>>(o_raw, (const float*)proj, ld, gate_col, (const bf16*)w, (float*)out, ldo,
                                                   H, dv, all_heads, gate_act, eps);
  else
    linattn_out_kernel<bf16><<<T, 256, smem, s>>>(o_raw, (const bf16*)proj, ld, gate_col, (const bf16*)w, (bf16*)out, ldo, H,
                                                  dv, all_heads, gate_act, eps);
  return b200_check_launch("b200_linattn_out");
}
