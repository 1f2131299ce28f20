// Recurrences on a matrix state per head with ONE decay per head and token, state in fp32.
//
//   state space:  S_t = g S_(t-1) + beta k_t v_t^T                      g = exp(-rate softplus(a + bias)), beta = softplus(a + bias)
//                 o_t = S_t^T q_t + skip v_t
//   delta rule:   S  <- g S_(t-1);  u = beta (v_t - S^T k_t);  S_t = S + k_t u^T;  o_t = S_t^T q_t
//                 g = exp(-rate softplus(a + bias)), beta = sigmoid(b)
// (S: dk x dv, zero before a sequence's first token; head h reads query / key head h / (H / G).)  Queries, keys and values
// arrive as fp32 rows whose heads are padded with zeros to a multiple of 4 entries (conv_rec_prep.cu); the gates' raw
// projections are fp32 rows, and everything formed from them is fp32.  The state of slot s is S [slots][H][dv][dkp] (key index
// fastest, dkp = dk rounded up to 4).  A sequence whose context is empty starts from zero, whatever its slot held.
//
// Every value column of S is a recurrence of its own, so columns are the unit of work: L lanes share C neighbouring columns,
// lane l holds the key entries 4 (i L + l) .. + 3 (i < R4) of each in registers, and a warp walks its C 32 / L columns
// through the sequence's new rows in blocks of four tokens.  Of a block, with G_j the product of its decays up to token j and D_ij
// of those behind token i up to j:
//   u_j = beta_j v_j - beta_j G_j S^T k_j - sum_(i < j) beta_j D_ij (k_i . k_j) u_i       (state space: beta_j v_j)
//   o_j = G_j S^T q_j + sum_(i <= j) D_ij (k_i . q_j) u_i,      S <- G_3 S + sum_i D_i3 k_i u_i^T
// so S^T k and S^T q of all four tokens come from the state before the block: their sums over the lanes travel together, and the
// state is scaled once for four tokens.  Token by token, as this was, each token waits for a sum over the lanes: 675 us for the delta
// rule over 4 x 2048 rows of 16 heads of 128 x 128 where blocks take 471 (fp32 pipe some 55 % busy), 450 -> 334 for the state space of
// 32 heads of 128 x 64.  Errors against 64 bits are no larger (delta rule 4 x 600 rows: outputs 1.23e-7 -> 1.16e-7, states 1.61e-7 -> 1.51e-7;
// state space 1.38e-7 -> 1.35e-7, 1.61e-7 -> 1.50e-7; rows of one sign 5.86e-8 -> 5.85e-8 and 1.43e-7 -> 1.42e-7, states 7 % less).
// What bounds it is one warp's issue: the products of a token go column by column in turn so that four chains cover an FMA's latency,
// and a token's sum over the lanes goes on a level per product that follows.  Of no use: eight warps of half the columns each (+6 %),
// key rows held over the block instead of read twice, queries a block ahead (+10 %, registers).
// Beside the four warps that walk, four warps stage rows by cp.async (16 tokens a stage), form a block's factors each, ahead of the
// walk, and write the outputs: the walk itself reads neither gates nor global memory.
// The state-space recurrence over prompts, with a workspace, runs over chunks of 64 rows side by side instead (chunk_scan.cuh).
#include "chunk_scan.cuh"
#include "common.cuh"
#include "runtime.h"
#include "../../include/b200.h"

namespace b200 {

struct GatedScanArgs {
  const float* x;
  int64_t ld;
  int q_col, k_col, v_col;
  const float* gates;              // [T][ld_g]: delta [b: H | a: H], state space [a: H]
  int64_t ld_g;
  const float* rate;               // [H]
  const float* dt_bias;            // [H]
  const float* skip;               // [H] or null
  const int32_t* cu_seq;
  const int32_t* ctx_lens;
  const int32_t* state_slots;
  float* S;
  float* o;                        // [T][H dv]
  int H, G, dkp, dv, dvp;
  int most_rows;                   // sequences with more new rows are another kernel's
};

__device__ __forceinline__ float gs_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// (decay, step) of a token from the raw gates
template <bool DELTA>
__device__ __forceinline__ float2 gs_gate(float a, float b, float rate, float bias) {
  const float sp = gs_softplus(a + bias);
  return make_float2(expf(-rate * sp), DELTA ? 1.0f / (1.0f + expf(-b)) : sp);
}

template <int L>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// the lane's shares of S^T x for C columns, a column's entries in turn with the others'
template <int R2, int C>
__device__ __forceinline__ void gs_dot(const f32x2 (&S)[C][R2], const f32x2 (&x)[R2], float (&o)[C]) {
  f32x2 p[C];
#pragma unroll
  for (int c = 0; c < C; ++c) p[c] = mul2(S[c][0], x[0]);
#pragma unroll
  for (int i = 1; i < R2; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) p[c] = fma2(S[c][i], x[i], p[c]);
#pragma unroll
  for (int c = 0; c < C; ++c) o[c] = sum2(p[c]);
}
// ... for one column, in two chains
template <int R2>
__device__ __forceinline__ float gs_dot1(const f32x2 (&S)[R2], const f32x2 (&x)[R2]) {
  f32x2 p0 = mul2(S[0], x[0]), p1 = mul2(S[1], x[1]);
#pragma unroll
  for (int i = 2; i < R2; i += 2) {
    p0 = fma2(S[i], x[i], p0);
    p1 = fma2(S[i + 1], x[i + 1], p1);
  }
  return sum2(add2(p0, p1));
}

// 4 R4 entries of a row of key entries: lane l of L takes entries 4 (i L + l) .. + 3
template <int L, int R4>
__device__ __forceinline__ void gs_row(const float* __restrict__ row, int l, f32x2 (&r)[2 * R4]) {
#pragma unroll
  for (int i = 0; i < R4; ++i) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + 4 * (i * L + l));
    r[2 * i] = t.x;
    r[2 * i + 1] = t.y;
  }
}

// 16 bytes of global memory -> shared memory, or zeros
__device__ __forceinline__ void gs_copy(float* to, const float* from, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(to)), "l"(from), "r"(there ? 16 : 0) : "memory");
}
// what rounding left of sum = a + b
__device__ __forceinline__ float gs_left(float a, float b, float sum) {
  const float t = sum - a;
  return (a - (sum - t)) + (b - t);
}

// Shares p[column][token] of the L lanes that hold the same columns -> lane l's column 0, summed over them, a level at a time: first
// l ^ 1, .. l ^ (C - 1) exchange columns, then all add.  A lane counts its columns from its own: number c is column c ^ (l % C),
// so what a lane keeps and what it gives away have the same numbers in every lane.
template <int C>
__device__ __forceinline__ void gs_level(float (&p)[C][4], int j, int level) {
  const int w = C >> (level + 1);
  if (w > 0) {
#pragma unroll
    for (int c = 0; c < w; ++c) p[c][j] += __shfl_xor_sync(0xffffffffu, p[c + w][j], w);
  } else {
    p[0][j] += __shfl_xor_sync(0xffffffffu, p[0][j], (C << level) / C);
  }
}
constexpr int gs_log2(int n) { return n <= 1 ? 0 : 1 + gs_log2(n / 2); }

constexpr int kGsWarps = 4;                            // warps that walk columns
constexpr int kGsStepWarps = 8;                        // of the single rows' kernel
constexpr int kGsTile = 4;                             // tokens of a block
constexpr int kGsHelpers = 4;                          // warps that stage rows and form the factors of a block each: blocks of a stage
constexpr int kGsStage = kGsHelpers * kGsTile;
// A block's factors in shared memory, floats: beta_j | D_j3 | G_j | what rounding left of G_j | D_ij k_i.k_j (i < j) | D_ij k_i.q_j (row j,
// i <= j) | the state's factor | c - 1 behind the block.  An error of theirs is one of every column and entry, which nothing averages
// out: decays and the last sums of the products are formed in 64 bits and rounded once, and an output's last sum takes along what its
// rounding leaves (fp32 throughout: outputs 3 to 8 % further off than token by token, 19 % over rows of one sign; all of it in 64 bits: the
// walk waits for it, 328 -> 379 us for the state space of 4 x 2048 rows).  The state is scaled by G_3 rounded to fp32.  What that
// leaves would be an error of all its entries alike, and one of decays that do not change adds up (a state left alone for 2048 tokens: 1e-5
// off, token by token 1e-6).  So the state is held as itself over a number c close to 1: the helpers, which know what was left,
// keep c, G_j is times c, D_j3 over it, and the walk multiplies by c at its end.  Multiplied by both parts of G_3 instead: the walk 471 -> 496 us.
constexpr int kGsBeta = 0, kGsD3 = 4, kGsG = 8, kGsGl = 12, kGsA = 16, kGsB = 24, kGsScale = 40, kGsRest = 41, kGsFactors = 44;

template <int L, int R4, int C>
struct GsShape {
  static constexpr int DKP = 4 * R4 * L, CPW = C * 32 / L, BUFS = DKP <= 256 ? 4 : 2;
  // stages that factors are ahead of outputs: one holds up a walk of few entries per lane (state space of 124 keys, one sequence of 2048 rows:
  // 217 us, with two 197), with two a portion of many takes longer (8 of 8 rows 11.6 and 12.3)
  static constexpr int AHEAD = C * R4 <= 4 ? 2 : 1;
  static constexpr int VW = kGsWarps * CPW;
  static constexpr int OUT = 4 * (L / C + 1);         // of a column and block: what the steps u are, and its lanes' shares of the read-outs
  static constexpr int kFloats = kGsHelpers * (BUFS * (kGsTile * (2 * DKP + VW) + kGsFactors) + (AHEAD + 1) * VW * OUT);
  static constexpr size_t kBytes = sizeof(float) * kFloats + 2 * BUFS * sizeof(uint64_t);
};

template <int L, int R4, int C, bool DELTA>
__global__ void __launch_bounds__((kGsWarps + kGsHelpers) * 32, C * R4 <= 8 ? 2 : 1)
gated_scan_kernel(GatedScanArgs a) {
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  using Sh = GsShape<L, R4, C>;
  constexpr int R2 = 2 * R4, DKP = Sh::DKP, CPW = Sh::CPW, BUFS = Sh::BUFS, VW = Sh::VW, BLOCKS = kGsHelpers, AHEAD = Sh::AHEAD;
  float* ks = smem;                                   // [BUFS][kGsStage][DKP]
  float* qs = ks + BUFS * kGsStage * DKP;             // [BUFS][kGsStage][DKP]
  float* vs = qs + BUFS * kGsStage * DKP;             // [BUFS][kGsStage][VW]
  float* fs = vs + BUFS * kGsStage * VW;              // [BUFS][BLOCKS][kGsFactors]
  float* os = fs + BUFS * BLOCKS * kGsFactors;        // [AHEAD + 1][BLOCKS][L / C + 1][VW][4]
  uint64_t* factors_full = reinterpret_cast<uint64_t*>(os + (AHEAD + 1) * BLOCKS * VW * Sh::OUT);     // [BUFS] each
  uint64_t* empty = factors_full + BUFS;
  const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int col0 = blockIdx.z * VW;
  const int slot = a.state_slots[s], t0 = a.cu_seq[s], t1 = a.cu_seq[s + 1], ctx = a.ctx_lens[s];      // (one wait)
  if (slot < 0 || t1 <= t0 || t1 - t0 > a.most_rows) return;
  const int dkp = a.dkp, rows = t1 - t0, blocks = (rows + kGsTile - 1) / kGsTile, stages = (blocks + BLOCKS - 1) / BLOCKS;
  if (tid == 0) {
    for (int i = 0; i < BUFS; ++i) {
      mbar_init(&factors_full[i], kGsHelpers);
      mbar_init(&empty[i], kGsWarps);
    }
    fence_mbar_init();
  }
  // key entries behind dkp: zeros in all buffers, written once
  if (dkp < DKP) {
    const int pad = DKP - dkp;
    for (int i = tid; i < BUFS * kGsStage * pad; i += (kGsWarps + kGsHelpers) * 32) {
      const int r = i / pad, d = dkp + i % pad;
      ks[r * DKP + d] = 0.f;
      qs[r * DKP + d] = 0.f;
    }
  }
  // the lane's columns are group .. group + C - 1, counted from its own: number c is column group + (c ^ l % C)
  const int l = lane % L, group = warp * CPW + lane / L * C, mine = group + l % C;
  float* Sp = a.S + (((size_t)slot * a.H + h) * a.dv + col0) * dkp;
  f32x2 S[C][R2];
  if (warp < kGsWarps) {                               // (on its way beside the first rows)
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int i = 0; i < R4; ++i) {
        ulonglong2 t = make_ulonglong2(0, 0);
        const int col = group + (c ^ l % C);
        if (ctx != 0 && col0 + col < a.dv && 4 * (i * L + l) < dkp) t = *reinterpret_cast<const ulonglong2*>(Sp + (size_t)col * dkp + 4 * (i * L + l));
        S[c][2 * i] = t.x;
        S[c][2 * i + 1] = t.y;
      }
  }
  __syncthreads();

  if (warp >= kGsWarps) {
    // ------------------------------------------------------------------ staging, and a block's factors per warp and stage
    const int helper = warp - kGsWarps, n = lane & 15, j = n & 3;
    // the lane's pair of rows (above the diagonal keys with keys): place n of a 4 x 4 table, of few keys place lane / 2
    constexpr bool FEW = DKP <= 32;
    const int pair_row = FEW ? lane >> 3 : n >> 2, pair_col = FEW ? lane >> 1 & 3 : j, lo = min(pair_row, pair_col), hi = max(pair_row, pair_col);
    const bool upper = pair_col > pair_row;
    const int hk = h / (a.H / a.G), v4 = min(VW, a.dvp - col0) >> 2;
    const float rate = a.rate[h], bias = a.dt_bias[h];
    const float* x = a.x + (size_t)t0 * a.ld + lane * 4;
    const int kc = a.k_col + hk * dkp, qc = a.q_col + hk * dkp, vc = a.v_col + h * a.dvp + col0;
    auto stage = [&](int st) {                        // the rows of this warp's block; those behind the portion are zeros
      const int from = (st * BLOCKS + helper) * kGsTile, to = (st % BUFS * BLOCKS + helper) * kGsTile;
#pragma unroll
      for (int r = 0; r < kGsTile; ++r) {
        const bool there = from + r < rows;
        const float* row = x + (size_t)min(from + r, rows - 1) * a.ld;
#pragma unroll
        for (int d = 0; d < DKP; d += 128)
          if (d + lane * 4 < dkp) {
            gs_copy(ks + (to + r) * DKP + d + lane * 4, row + kc + d, there);
            gs_copy(qs + (to + r) * DKP + d + lane * 4, row + qc + d, there);
          }
        if (lane < v4) gs_copy(vs + (to + r) * VW + lane * 4, row + vc, there);
      }
    };
    float ra = 0.f, rb = 0.f;
    auto raw_gates = [&](int st) {                    // lane n: token n of the stage
      const int t = st * kGsStage + n;
      if (t < rows) {
        const float* g = a.gates + (size_t)(t0 + t) * a.ld_g;
        ra = __ldcg(g + (DELTA ? a.H + h : h));
        if (DELTA) rb = __ldcg(g + h);
      }
    };
    // outputs of this warp's block: the read-out of the state before it and what its own tokens add
    const float skip = a.skip != nullptr ? a.skip[h] : 0.f;
    auto put = [&](int st) {
      mbar_wait_guarded(&empty[st % BUFS], (st / BUFS) & 1);
      const int b = st * BLOCKS + helper, at = st % BUFS * BLOCKS + helper;
      const float* f = fs + at * kGsFactors;
      const float* ob = os + (st % (AHEAD + 1) * BLOCKS + helper) * VW * Sh::OUT;
      float G[4], Gl[4], B[10];
#pragma unroll
      for (int i = 0, n = 0; i < 4; ++i) {
        G[i] = f[kGsG + i];
        Gl[i] = f[kGsGl + i];
#pragma unroll
        for (int e = 0; e <= i; ++e) B[n++] = f[kGsB + 4 * i + e];
      }
      for (int c = lane; c < VW && col0 + c < a.dv; c += 32) {
        const float4 uf = *reinterpret_cast<const float4*>(ob + c * 4);
        const float u[4] = {uf.x, uf.y, uf.z, uf.w};
        float r[2][4];                                 // two halves of the lanes' shares
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) r[e][i] = 0.f;
#pragma unroll
        for (int i = 0; i < L / C; ++i) {
          const float4 m = *reinterpret_cast<const float4*>(ob + ((i + 1) * VW + c) * 4);
          float (&h2)[4] = r[2 * i >= L / C && L > C];
          h2[0] += m.x; h2[1] += m.y; h2[2] += m.z; h2[3] += m.w;
        }
        const float* v = vs + at * kGsTile * VW + c;
        float* out = a.o + (size_t)(t0 + b * kGsTile) * a.H * a.dv + h * a.dv + col0 + c;
#pragma unroll
        for (int i = 0, n = 0; i < 4; ++i) {
          float y = B[n] * u[0], low = DELTA ? fmaf(B[n], u[0], -y) : 0.f;
          ++n;
#pragma unroll
          for (int e = 1; e <= i; ++e, ++n) {
            if (DELTA) {                               // (whose steps take values back: what their sum's rounding leaves counts too)
              const float m = B[n] * u[e], z = y + m;
              low += gs_left(y, m, z) + fmaf(B[n], u[e], -m);
              y = z;
            } else {
              y = fmaf(B[n], u[e], y);
            }
          }
          y = fmaf(skip, v[i * VW], y);
          const float R = r[0][i] + r[1][i], left = gs_left(r[0][i], r[1][i], R);
          if (DELTA) {
            const float P = G[i] * R, sum = P + y;
            low += gs_left(P, y, sum) + fmaf(Gl[i], R, fmaf(G[i], left, fmaf(G[i], R, -P)));
            y = fabsf(sum) < INFINITY ? sum + low : sum;
          } else {                                     // (a third of the instructions, and as close where the steps are not the state's)
            y = fmaf(G[i], R, fabsf(R) < INFINITY ? fmaf(Gl[i], R, fmaf(G[i], left, y)) : y);
          }
          if (b * kGsTile + i < rows) out[(size_t)i * a.H * a.dv] = y;
        }
      }
    };
    double carry = 0.0;                               // c - 1 before the stage
    auto factors = [&](int st) {
      const int at = st % BUFS * BLOCKS + helper, from = helper * kGsTile;
      const float2 gb = st * kGsStage + n < rows ? gs_gate<DELTA>(ra, rb, rate, bias) : make_float2(1.f, 0.f);   // (behind the portion the state stays)
      if (st + 1 < stages) raw_gates(st + 1);
      // lane n: the product of the four decays of its block of the stage, rounded, and what that leaves, over the product
      float g = __shfl_xor_sync(0xffffffffu, gb.x, 1), scale = gb.x * g, rest = fmaf(gb.x, g, -scale);
      g = __shfl_xor_sync(0xffffffffu, scale, 2);
      rest = fmaf(scale, __shfl_xor_sync(0xffffffffu, rest, 2), rest * g);
      rest += fmaf(scale, g, -scale * g);
      scale *= g;
      rest = scale > 1e-30f && scale < 1e30f ? rest * rcp_approx(scale) : 0.f;
      const float beside = __shfl_xor_sync(0xffffffffu, rest, 4), pair = rest + beside, others = __shfl_xor_sync(0xffffffffu, pair, 8);
      const float c = (float)carry + ((n & 4 ? beside : 0.f) + (n & 8 ? others : 0.f)), behind = c + fmaf(c, rest, rest);      // - 1
      carry = fma(carry, (double)(pair + others), carry + (double)(pair + others));
      const float g0 = __shfl_sync(0xffffffffu, gb.x, from), g1 = __shfl_sync(0xffffffffu, gb.x, from + 1),
                  g2 = __shfl_sync(0xffffffffu, gb.x, from + 2), g3 = __shfl_sync(0xffffffffu, gb.x, from + 3);
      double decay = 1.0;                             // from token lo to token hi
      if (lo < 1 && hi >= 1) decay = g1;
      if (lo < 2 && hi >= 2) decay *= g2;
      if (lo < 3 && hi >= 3) decay *= g3;
      asm volatile("cp.async.wait_group %0;" ::"n"(BUFS - AHEAD - 1) : "memory");
      __syncwarp();
      double product;
      const float* kb = ks + at * kGsTile * DKP;
      const float* qb = qs + at * kGsTile * DKP;
      if constexpr (FEW) {                             // eight lanes per row, each four keys of its products (lanes without keys: 202 -> 191 us, 16 keys)
        float dot[4] = {0.f, 0.f, 0.f, 0.f};
        const int d = (lane & 7) * 4;
        if (d < DKP) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(kb + c * DKP + d),
                             x = *reinterpret_cast<const ulonglong2*>((DELTA && c > pair_row ? kb : qb) + pair_row * DKP + d);
            dot[c] = sum2(fma2(k.y, x.y, mul2(k.x, x.x)));
          }
        }
        const bool up = lane & 4;
        double sum[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float own = up ? dot[i + 2] : dot[i], other = up ? dot[i] : dot[i + 2];
          sum[i] = own + __shfl_xor_sync(0xffffffffu, other, 4);
        }
        const double own = lane & 2 ? sum[1] : sum[0], other = lane & 2 ? sum[0] : sum[1];
        product = own + __shfl_xor_sync(0xffffffffu, other, 2);
        product += __shfl_xor_sync(0xffffffffu, product, 1);
      } else {
        float dot[16];
        {
          f32x2 d2[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) d2[i] = 0;
#pragma unroll 1
          for (int d = lane * 4; d < DKP; d += 128) {
            ulonglong2 k[4], q[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              k[i] = *reinterpret_cast<const ulonglong2*>(kb + i * DKP + d);
              q[i] = *reinterpret_cast<const ulonglong2*>(qb + i * DKP + d);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                if (c <= r) d2[r * 4 + c] = fma2(k[c].y, q[r].y, fma2(k[c].x, q[r].x, d2[r * 4 + c]));
                else if (DELTA) d2[r * 4 + c] = fma2(k[c].y, k[r].y, fma2(k[c].x, k[r].x, d2[r * 4 + c]));
              }
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) dot[i] = sum2(d2[i]);
        }
#pragma unroll
        for (int w = 8; w > 2; w >>= 1) {                // lanes n and n + 16 end with pair n
          const bool up = n & w;
#pragma unroll
          for (int i = 0; i < w; ++i) {
            const float own = up ? dot[i + w] : dot[i], other = up ? dot[i] : dot[i + w];
            dot[i] = own + __shfl_xor_sync(0xffffffffu, other, w);
          }
        }
        double sum[4] = {dot[0], dot[1], dot[2], dot[3]};
#pragma unroll
        for (int w = 2; w > 0; w >>= 1) {
          const bool up = n & w;
#pragma unroll
          for (int i = 0; i < w; ++i) {
            const double own = up ? sum[i + w] : sum[i], other = up ? sum[i] : sum[i + w];
            sum[i] = own + __shfl_xor_sync(0xffffffffu, other, w);
          }
        }
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 16);
        product = sum[0];
      }
      float* f = fs + at * kGsFactors;
      if (FEW ? !(lane & 1) : lane < 16) f[upper ? kGsA + hi * (hi - 1) / 2 + lo : kGsB + 4 * pair_row + pair_col] = (float)(decay * product);
      if (lane >= 16 && n >> 2 == helper) {
        double G = g0, D3 = 1.0;
        if (j >= 1) G *= g1;
        if (j >= 2) G *= g2;
        if (j >= 3) G *= g3;
        if (j < 1) D3 = g1;
        if (j < 2) D3 *= g2;
        if (j < 3) D3 *= g3;
        G = fma(G, (double)c, G);
        D3 = fma(D3, (double)(-behind * rcp_approx(1.f + behind)), D3);      // over 1 + behind
        const float high = (float)G;
        f[kGsBeta + j] = gb.y;
        f[kGsG + j] = high;
        f[kGsGl + j] = (float)(G - high);
        f[kGsD3 + j] = (float)D3;
        if (j == 0) {
          f[kGsScale] = scale;
          f[kGsRest] = behind;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&factors_full[st % BUFS]);
    };
    raw_gates(0);
    // a stage's factors, the outputs of the one AHEAD before it, then the rows of the next one for its buffer: none of the walk's
    // stages waits for copies, or for the outputs of less than AHEAD + 1 stages before.  A warp copies, reads and writes out its own block only.
    for (int st = AHEAD - BUFS; st < stages + AHEAD; ++st) {
      if (st >= 0 && st < stages) factors(st);
      if (st >= AHEAD) put(st - AHEAD);
      __syncwarp();                                   // a lane copies columns that others read in put(), each in as many turns as it has columns
      if (st - AHEAD + BUFS < stages) stage(st - AHEAD + BUFS);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    return;
  }

  // -------------------------------------------------------------------- the walk
  constexpr int LV = gs_log2(L), LC = gs_log2(C);
  mbar_wait_guarded(&factors_full[0], 0);             // (a stage's rows have landed when its factors are there)
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    const int at = b % (BUFS * BLOCKS);
    const float* vr = vs + at * kGsTile * VW + mine;
    const float* f = fs + at * kGsFactors;
    float* ob = os + b % ((AHEAD + 1) * BLOCKS) * VW * Sh::OUT;
    if ((b + 1) % BLOCKS == 0 && b + 1 < blocks) {    // the next stage's, a block early: at its own start 474 us, delta rule of 4 x 2048 rows
      const int st = (b + 1) / BLOCKS;
      mbar_wait_guarded(&factors_full[st % BUFS], (st / BUFS) & 1);
    }
    float v[4], p[C][4], r[C][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = vr[j * VW];
    const float4 beta = *reinterpret_cast<const float4*>(f + kGsBeta), d3 = *reinterpret_cast<const float4*>(f + kGsD3);
    // S^T k of the block's tokens, then S^T q; a token's sum over the lanes goes on a level for each product that follows
    constexpr int FIRST = DELTA ? 0 : 4;
#pragma unroll
    for (int t = FIRST; t < 8 || (DELTA && t < 4 + LV); ++t) {
      if (t < 8) {
        float d[C];
        f32x2 q[R2];
        gs_row<L, R4>((t < 4 ? ks : qs) + (at * kGsTile + (t & 3)) * DKP, l, q);
        gs_dot<R2, C>(S, q, d);
#pragma unroll
        for (int c = 0; c < C; ++c) (t < 4 ? p : r)[c][t & 3] = d[c];
      }
      if (DELTA) {
#pragma unroll
        for (int lv = 0; lv < LV; ++lv)
          if (t - 1 - lv >= 0 && t - 1 - lv < 4) gs_level<C>(p, t - 1 - lv, lv);
      }
    }
    const float scale = f[kGsScale];
    const f32x2 g4 = pack2(scale, scale);
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int i = 0; i < R2; ++i) S[c][i] = mul2(g4, S[c][i]);
    float u[4];
    if (DELTA) {
      const float4 G = *reinterpret_cast<const float4*>(f + kGsG), Gl = *reinterpret_cast<const float4*>(f + kGsGl),
                   a0 = *reinterpret_cast<const float4*>(f + kGsA);
      const float2 a1 = *reinterpret_cast<const float2*>(f + kGsA + 4);
      u[0] = beta.x * fmaf(-Gl.x, p[0][0], fmaf(-G.x, p[0][0], v[0]));
      u[1] = beta.y * fmaf(-a0.x, u[0], fmaf(-Gl.y, p[0][1], fmaf(-G.y, p[0][1], v[1])));
      u[2] = beta.z * fmaf(-a0.z, u[1], fmaf(-a0.y, u[0], fmaf(-Gl.z, p[0][2], fmaf(-G.z, p[0][2], v[2]))));
      u[3] = beta.w * fmaf(-a1.y, u[2], fmaf(-a1.x, u[1], fmaf(-a0.w, u[0], fmaf(-Gl.w, p[0][3], fmaf(-G.w, p[0][3], v[3])))));
    } else {
      u[0] = beta.x * v[0];
      u[1] = beta.y * v[1];
      u[2] = beta.z * v[2];
      u[3] = beta.w * v[3];
    }
    const float w[4] = {d3.x * u[0], d3.y * u[1], d3.z * u[2], d3.w * u[3]};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f32x2 k[R2];
      gs_row<L, R4>(ks + (at * kGsTile + j) * DKP, l, k);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float x = c ? __shfl_xor_sync(0xffffffffu, w[j], c) : w[j];
        const f32x2 x2 = pack2(x, x);
#pragma unroll
        for (int i = 0; i < R2; ++i) S[c][i] = fma2(k[i], x2, S[c][i]);
      }
      if (j < LC) {
#pragma unroll
        for (int i = 0; i < 4; ++i) gs_level<C>(r, i, j);
      }
    }
    if (l < C) *reinterpret_cast<float4*>(ob + mine * 4) = make_float4(u[0], u[1], u[2], u[3]);
    *reinterpret_cast<float4*>(ob + ((l / C + 1) * VW + mine) * 4) = make_float4(r[0][0], r[0][1], r[0][2], r[0][3]);
    if ((b + 1) % BLOCKS == 0 || b + 1 == blocks) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[b / BLOCKS % BUFS]);
    }
  }
  const float rest = fs[(blocks - 1) % (BUFS * BLOCKS) * kGsFactors + kGsRest];
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int i = 0; i < R2; ++i) {
      const float2 v = unpack2(S[c][i]);
      S[c][i] = pack2(fabsf(v.x) < INFINITY ? fmaf(v.x, rest, v.x) : v.x, fabsf(v.y) < INFINITY ? fmaf(v.y, rest, v.y) : v.y);
    }
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int i = 0; i < R4; ++i)
      if (col0 + group + (c ^ l % C) < a.dv && 4 * (i * L + l) < dkp)
        *reinterpret_cast<ulonglong2*>(Sp + (size_t)(group + (c ^ l % C)) * dkp + 4 * (i * L + l)) = make_ulonglong2(S[c][2 * i], S[c][2 * i + 1]);
}

// Single rows (a decode step): the state, the token's rows and its gates are in flight together; no staging, no barrier.
template <int L, int R4, bool DELTA>
__global__ void __launch_bounds__(kGsStepWarps * 32, 4)
gated_step_kernel(GatedScanArgs a) {
  pdl_wait();
  constexpr int R2 = 2 * R4, CPW = 32 / L, COLS = kGsStepWarps * CPW;
  const int s = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
  const int slot = a.state_slots[s];
  if (slot < 0) return;
  const int t = a.cu_seq[s];
  if (a.cu_seq[s + 1] <= t) return;
  const int lane = threadIdx.x & 31, l = lane % L, col = z * COLS + (threadIdx.x >> 5) * CPW + lane / L;
  const int hk = h / (a.H / a.G), dkp = a.dkp;
  const bool live = col < a.dv, fresh = a.ctx_lens[s] == 0;
  float* Sp = a.S + (((size_t)slot * a.H + h) * a.dv + col) * dkp;
  const float* row = a.x + (size_t)t * a.ld;
  f32x2 S[R2], k[R2], q[R2];
#pragma unroll
  for (int i = 0; i < R4; ++i) {
    const int d = 4 * (i * L + l);
    ulonglong2 ts = make_ulonglong2(0, 0), tk = ts, tq = ts;
    if (d < dkp) {
      if (live && !fresh) ts = *reinterpret_cast<const ulonglong2*>(Sp + d);
      tk = __ldcg(reinterpret_cast<const ulonglong2*>(row + a.k_col + hk * dkp + d));
      tq = __ldcg(reinterpret_cast<const ulonglong2*>(row + a.q_col + hk * dkp + d));
    }
    S[2 * i] = ts.x; S[2 * i + 1] = ts.y;
    k[2 * i] = tk.x; k[2 * i + 1] = tk.y;
    q[2 * i] = tq.x; q[2 * i + 1] = tq.y;
  }
  const float v = live ? __ldcg(row + a.v_col + h * a.dvp + col) : 0.f;
  const float* g = a.gates + (size_t)t * a.ld_g;
  const float2 gb = gs_gate<DELTA>(__ldcg(g + (DELTA ? a.H + h : h)), DELTA ? __ldcg(g + h) : 0.f, a.rate[h], a.dt_bias[h]);
  float u = gb.y * v;
  if (DELTA) u = gb.y * (v - gb.x * lanes_sum<L>(gs_dot1<R2>(S, k)));
  const f32x2 g2 = pack2(gb.x, gb.x), u2 = pack2(u, u);
#pragma unroll
  for (int i = 0; i < R2; ++i) S[i] = fma2(k[i], u2, mul2(g2, S[i]));
  const float o = lanes_sum<L>(gs_dot1<R2>(S, q));
  if (!live) return;
#pragma unroll
  for (int i = 0; i < R4; ++i) {
    const int d = 4 * (i * L + l);
    if (d < dkp) *reinterpret_cast<ulonglong2*>(Sp + d) = make_ulonglong2(S[2 * i], S[2 * i + 1]);
  }
  if (l == 0) a.o[(size_t)t * a.H * a.dv + h * a.dv + col] = a.skip != nullptr ? fmaf(a.skip[h], v, o) : o;
}

template <int L, int R4, int C, bool DELTA>
int gated_scan_launch(const GatedScanArgs& a, int n_seqs, cudaStream_t s) {
  using Sh = GsShape<L, R4, C>;
  if constexpr (Sh::kBytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(gated_scan_kernel<L, R4, C, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::kBytes);
    if (e != cudaSuccess) {
      b200_set_error("gated_scan: %zu bytes of shared memory: %s", Sh::kBytes, cudaGetErrorString(e));
      return B200_ERR_CUDA;
    }
  }
  (void)launch_pdl(gated_scan_kernel<L, R4, C, DELTA>, dim3(n_seqs, a.H, (a.dv + Sh::VW - 1) / Sh::VW), dim3((kGsWarps + kGsHelpers) * 32),
                   Sh::kBytes, s, 1, a);
  return b200_check_launch("b200_gated_scan");
}

template <int L, int R4, bool DELTA>
int gated_step_launch(const GatedScanArgs& a, int n_seqs, cudaStream_t s) {
  constexpr int COLS = kGsStepWarps * (32 / L);
  (void)launch_pdl(gated_step_kernel<L, R4, DELTA>, dim3(n_seqs, a.H, (a.dv + COLS - 1) / COLS), dim3(kGsStepWarps * 32), 0, s, 1, a);
  return b200_check_launch("b200_gated_scan(step)");
}

// Single rows have a kernel of their own.  Portions: the more columns a warp walks the fewer instructions a column costs, the fewer
// it walks the shorter a block takes, so the widest form whose CTAs still find an SM each: us for 1, 2, 3 and 4 sequences of the delta
// rule with 16 heads of 128 x 128 (2048, 1024, 1024 and 2048 rows), in CTAs of 64 columns 467, 236, 236, 468, of 32 columns 332, 169, 286, 566,
// of 16 columns 264, 219, 339, 853.  CTAs of 32 columns share an SM in pairs, which covers the start and the end of short portions: 16
// of 16 rows 28.7 in CTAs of 64 columns, 26.6 of 32, but 8 of 1024 rows 473 and 558.  A bound on the rows per portion is often that of all
// of them, so pairs are for sequences enough to fill the GPU three times (16 of 512 rows: 477 and 489) or a bound that is short.
// Few keys: a lane of two columns walks faster than one of four, whose sums over lanes and columns take longer than its products.  State
// space of 32 heads of 64 values, us token by token, in four columns a lane, in two: 16 keys, one sequence of 2048 rows 203, 221, 192, 64 of 33
// rows 59, 55, 49; 32 keys 205, 187, 152 and 59, 55, 86: of 17 to 32 keys two only where CTAs of 32 columns find an SM each.
template <int L, int R4, int C = 4>
bool gs_fits(const GatedScanArgs& a, int n_seqs) {
  constexpr int cols = GsShape<L, R4, C>::VW;
  return (int64_t)n_seqs * a.H * ((a.dv + cols - 1) / cols) <= sm_count();
}
template <bool DELTA>
int gated_scan_pick(const GatedScanArgs& a, int n_seqs, int max_len, cudaStream_t s) {
  if (max_len == 1) {
    if (a.dkp <= 32) return gated_step_launch<8, 1, DELTA>(a, n_seqs, s);
    if (a.dkp <= 64) return gated_step_launch<8, 2, DELTA>(a, n_seqs, s);
    if (a.dkp <= 96) return gated_step_launch<8, 3, DELTA>(a, n_seqs, s);
    if (a.dkp <= 128) return gated_step_launch<8, 4, DELTA>(a, n_seqs, s);
    if (a.dkp <= 256) return gated_step_launch<16, 4, DELTA>(a, n_seqs, s);
    return gated_step_launch<32, 4, DELTA>(a, n_seqs, s);
  }
  if (a.dkp <= 16) return gated_scan_launch<4, 1, 2, DELTA>(a, n_seqs, s);
  if (a.dkp <= 32) return gs_fits<8, 1, 2>(a, n_seqs) ? gated_scan_launch<8, 1, 2, DELTA>(a, n_seqs, s) : gated_scan_launch<8, 1, 4, DELTA>(a, n_seqs, s);
  if (a.dkp <= 64) return gs_fits<16, 1>(a, n_seqs) ? gated_scan_launch<16, 1, 4, DELTA>(a, n_seqs, s) : gated_scan_launch<8, 2, 4, DELTA>(a, n_seqs, s);
  if (a.dkp <= 96) return gated_scan_launch<8, 3, 4, DELTA>(a, n_seqs, s);
  if (a.dkp <= 128) {
    if (gs_fits<32, 1>(a, n_seqs)) return gated_scan_launch<32, 1, 4, DELTA>(a, n_seqs, s);
    const bool pairs = gs_fits<16, 2>(a, n_seqs) || max_len <= 64 || !gs_fits<8, 4>(a, (n_seqs + 2) / 3);
    return pairs ? gated_scan_launch<16, 2, 4, DELTA>(a, n_seqs, s) : gated_scan_launch<8, 4, 4, DELTA>(a, n_seqs, s);
  }
  if (a.dkp <= 256) return gs_fits<32, 2>(a, n_seqs) ? gated_scan_launch<32, 2, 4, DELTA>(a, n_seqs, s) : gated_scan_launch<16, 4, 4, DELTA>(a, n_seqs, s);
  return gated_scan_launch<32, 4, 4, DELTA>(a, n_seqs, s);
}

// The state-space recurrence in the chunk form: log decays of a chunk's rows summed in fp64, every exponent <= 0.  A decay of
// less than e^-10000 is zero all the same and is cut there, so that sums and their differences stay finite.
//   ws_row[dk] of a chunk: its whole decay
struct StateSpaceForm {
  static constexpr const char* kName = "b200_gated_scan(chunks)";
  static constexpr bool kVector = false;
  struct Params {
    const float* gates;
    int64_t ld_g;
    const float* rate;
    const float* dt_bias;
    const float* skip;
  };
  struct Scratch {
    double F[kCsRows];
    float beta[kCsRows], w[kCsRows], aq[kCsRows], all;
  };
  // warp 0, two rows per lane
  static __device__ __forceinline__ void sums(const Params& p, int h, const ChunkPlace& at, double (&F)[2], float (&beta)[2]) {
    const int lane = threadIdx.x & 31;
    const float rate = p.rate[h], bias = p.dt_bias[h];
    double f[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = 2 * lane + e;
      f[e] = 0.0;
      beta[e] = 0.f;
      if (t < at.rows) {
        beta[e] = gs_softplus(__ldcg(p.gates + (size_t)(at.first + t) * p.ld_g + h) + bias);
        const float lg = -rate * beta[e];
        f[e] = lg < -1.0e4f ? -1.0e4 : (double)lg;
      }
    }
    double sum = f[0] + f[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const double before = __shfl_up_sync(0xffffffffu, sum, 1);
    F[1] = sum;
    F[0] = lane ? before + f[0] : f[0];               // (not sum - f[1]: what is no number in a row stays out of the one before)
  }
  static __device__ __forceinline__ void state_weights(const Params& p, const ChunkScanArgs&, Scratch& sc, int h, const ChunkPlace& at) {
    if (threadIdx.x < 32) {
      double F[2];
      float beta[2];
      sums(p, h, at, F, beta);
      const double Fn = __shfl_sync(0xffffffffu, F[1], 31);        // rows behind the last one decay by nothing
#pragma unroll
      for (int e = 0; e < 2; ++e) sc.w[2 * threadIdx.x + e] = expf((float)(Fn - F[e])) * beta[e];
      if (threadIdx.x == 0) sc.all = expf((float)Fn);
    }
    __syncthreads();
  }
  template <int DK>
  static __device__ __forceinline__ void state_row(const ChunkScanArgs& a, const Scratch& sc, int h) {
    if (threadIdx.x == 0) a.ws_row[((size_t)blockIdx.x * a.H + h) * a.ws_row_width + DK] = sc.all;
  }
  struct Carry {
    const float* row;
    size_t step;
    float f[kCsCarryDepth];
    __device__ __forceinline__ Carry(const ChunkScanArgs& a, int h, int base, int)
        : row(a.ws_row + ((size_t)base * a.H + h) * a.ws_row_width + a.ws_row_width - 4), step((size_t)a.H * a.ws_row_width) {}
    __device__ __forceinline__ void fetch(int c0, int nc) {
#pragma unroll
      for (int u = 0; u < kCsCarryDepth; ++u)
        if (c0 + u < nc) f[u] = __ldcg(row + (c0 + u) * step);
    }
  };
  static __device__ __forceinline__ void output_weights(const Params& p, const ChunkScanArgs&, Scratch& sc, int h, const ChunkPlace& at) {
    if (threadIdx.x < 32) {
      double F[2];
      float beta[2];
      sums(p, h, at, F, beta);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * threadIdx.x + e;
        sc.F[t] = F[e];
        sc.beta[t] = beta[e];
        sc.aq[t] = expf((float)F[e]);
      }
    }
  }
  static __device__ __forceinline__ float D(const Params&, const Scratch& sc, int t, int s) { return expf((float)(sc.F[t] - sc.F[s])) * sc.beta[s]; }
  static __device__ __forceinline__ float aq(const Scratch& sc, int t) { return sc.aq[t]; }
  static __device__ __forceinline__ float4 finish(const Params& p, const Scratch&, int h, int, float4 v, float4 x) {
    const float s = p.skip != nullptr ? p.skip[h] : 0.f;
    return p.skip != nullptr ? make_float4(fmaf(s, x.x, v.x), fmaf(s, x.y, v.y), fmaf(s, x.z, v.z), fmaf(s, x.w, v.w)) : v;
  }
};

// ------------------------------------------------------------------------------------------- out
// out = RMSnorm over `parts` equal pieces of (y * silu(z)), times w[channel] -- the gate BEFORE the norm -- or, with the gate
// AFTER it, RMSnorm of the pieces of y times w[place in the piece] (one weight vector for all pieces) times silu(z).  One CTA
// per row; the row is staged in shared memory between the statistic and the product.
// four or one value(s) of the rows that kernels before this one wrote, and of weights
__device__ __forceinline__ float4 gs_cg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 gs_cg4(const bf16* p) {
  const uint2 r = __ldcg(reinterpret_cast<const uint2*>(p));
  return make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
}
__device__ __forceinline__ float gs_cg1(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float gs_cg1(const bf16* p) { return __bfloat162float(__ldcg(p)); }
__device__ __forceinline__ float4 gs_w4(const bf16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  return make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
}
__device__ __forceinline__ void gs_st1(float* p, float v) { *p = v; }
__device__ __forceinline__ void gs_st1(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
__device__ __forceinline__ void gs_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void gs_st4(bf16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }
__device__ __forceinline__ float gs_silu(float z) { return z / (1.0f + expf(-z)); }

constexpr int kGnThreads = 256;

template <typename TA, bool VEC, bool AFTER>
__global__ void __launch_bounds__(kGnThreads)
gate_norm_kernel(const float* __restrict__ y, const TA* __restrict__ proj, int64_t ld, int z_col, const bf16* __restrict__ w,
                 TA* out, int64_t ldo, int C, int parts, float eps) {
  pdl_wait();
  extern __shared__ __align__(16) float row[];        // [C], then the warps' partial sums
  __shared__ float sums[kGnThreads / 32];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NW = kGnThreads / 32, V = VEC ? 4 : 1;
  const float* yr = y + (size_t)t * C;
  const TA* zr = proj + (size_t)t * ld + z_col;
  TA* o = out + (size_t)t * ldo;
  const int W = C / parts, per = parts >= NW ? 1 : NW / parts;       // warps that share a part
  for (int p0 = 0; p0 < parts; p0 += NW / per) {
    const int p = p0 + warp / per, sub = warp % per;
    const bool live = p < parts && warp / per < NW / per;
    float ss = 0.f;
    if (live)
      for (int i = (sub * 32 + lane) * V; i < W; i += per * 32 * V) {
        const int c = p * W + i;
        if (VEC) {
          float4 v = gs_cg4(yr + c);
          if (!AFTER) {
            const float4 g = gs_cg4(zr + c);
            v.x *= gs_silu(g.x); v.y *= gs_silu(g.y); v.z *= gs_silu(g.z); v.w *= gs_silu(g.w);
          }
          *reinterpret_cast<float4*>(row + c) = v;
          ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        } else {
          const float v = AFTER ? gs_cg1(yr + c) : gs_cg1(yr + c) * gs_silu(gs_cg1(zr + c));
          row[c] = v;
          ss = fmaf(v, v, ss);
        }
      }
    ss = warp_sum(ss);
    if (per > 1) {
      if (lane == 0) sums[warp] = ss;
      __syncthreads();
      if (live) {
        ss = 0.f;
        for (int i = 0; i < per; ++i) ss += sums[warp - sub + i];    // the same order in every warp
      }
    }
    if (!live) continue;
    const float rstd = 1.0f / sqrtf(ss / (float)W + eps);
    for (int i = (sub * 32 + lane) * V; i < W; i += per * 32 * V) {  // (each thread reads back what it staged itself)
      const int c = p * W + i;
      if (VEC) {
        float4 v = *reinterpret_cast<const float4*>(row + c);
        const float4 g = gs_w4(w + (AFTER ? i : c));
        if (AFTER) {
          const float4 t = gs_cg4(zr + c);
          v.x *= gs_silu(t.x); v.y *= gs_silu(t.y); v.z *= gs_silu(t.z); v.w *= gs_silu(t.w);
        }
        gs_st4(o + c, make_float4(v.x * rstd * g.x, v.y * rstd * g.y, v.z * rstd * g.z, v.w * rstd * g.w));
      } else {
        gs_st1(o + c, row[c] * rstd * __bfloat162float(w[AFTER ? i : c]) * (AFTER ? gs_silu(gs_cg1(zr + c)) : 1.0f));
      }
    }
  }
}

// Pieces of up to 128 channels (a head): W / 4 neighbouring lanes share one, a thread holds up to N of its row's 16-byte
// groups in registers and all their loads are in flight together.  Bound by bytes in flight: N 2 where it covers the row (the
// registers of 8 leave 3 CTAs to an SM: 57 us for 8192 rows of 2048 channels, 38 of 2), and by instructions (325 a thread where the
// logistic and the root of common.cuh took 455: 31 us now; weights in registers over several rows, the next row's loads in flight: 32).
template <typename TA, bool AFTER, int N>
__global__ void __launch_bounds__(kGnThreads)
gate_norm_heads_kernel(const float* __restrict__ y, const TA* __restrict__ proj, int64_t ld, int z_col, const bf16* __restrict__ w, TA* out,
                       int64_t ldo, int C, int W, float eps) {
  pdl_wait();
  const int t = blockIdx.x, i0 = threadIdx.x * 4, step = kGnThreads * 4, lanes = W >> 2;
  const float over = 1.0f / (float)W;                  // (a power of two)
  const float* yr = y + (size_t)t * C;
  const TA* zr = proj + (size_t)t * ld + z_col;
  TA* o = out + (size_t)t * ldo;
  float4 v[N], g[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int i = i0 + n * step;
    if (n * step >= C) break;
    v[n] = g[n] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < C) {
      v[n] = gs_cg4(yr + i);
      g[n] = gs_cg4(zr + i);
    }
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int i = i0 + n * step;
    if (n * step >= C) break;
    {
      float z[4] = {g[n].x, g[n].y, g[n].z, g[n].w};
      logistic_all<true>(z, z);
      g[n] = make_float4(z[0], z[1], z[2], z[3]);
    }
    float4 x = v[n];
    if (!AFTER) { x.x *= g[n].x; x.y *= g[n].y; x.z *= g[n].z; x.w *= g[n].w; }
    float ss = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
      if (s < lanes) ss += __shfl_xor_sync(0xffffffffu, ss, s);
    if (i >= C) continue;
    const float rstd = inv_sqrt(ss * over + eps);
    const float4 c = gs_w4(w + (AFTER ? i & (W - 1) : i));
    x = make_float4(x.x * rstd * c.x, x.y * rstd * c.y, x.z * rstd * c.z, x.w * rstd * c.w);
    if (AFTER) { x.x *= g[n].x; x.y *= g[n].y; x.z *= g[n].z; x.w *= g[n].w; }
    gs_st4(o + i, x);
  }
}

// Pieces of whole warps' 128 channels in rows of up to 2048: a thread holds its two 16-byte groups in registers, their loads in flight
// together, and the warps' sums meet in shared memory once.  Bound by bytes and by the logistics' instructions (the row staged in shared
// memory, one group in flight per thread, expf and a division for each logistic: 8192 rows of 2 x 1024 channels 45 us, 33 now; of 1024
// channels 33 and 20, of 256 27 and 13).
template <typename TA, bool AFTER>
__global__ void __launch_bounds__(kGnThreads)
gate_norm_parts_kernel(const float* __restrict__ y, const TA* __restrict__ proj, int64_t ld, int z_col, const bf16* __restrict__ w, TA* out,
                       int64_t ldo, int C, int W, float eps) {
  pdl_wait();
  constexpr int NW = kGnThreads / 32, N = 2;
  __shared__ float sums[N * NW];                       // of the row's groups of 128 channels
  const int t = blockIdx.x, i0 = threadIdx.x * 4, step = kGnThreads * 4, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, per = W / 128;
  const float* yr = y + (size_t)t * C;
  const TA* zr = proj + (size_t)t * ld + z_col;
  TA* o = out + (size_t)t * ldo;
  float4 v[N], g[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int i = i0 + n * step;
    if (i >= C) break;
    v[n] = gs_cg4(yr + i);
    g[n] = gs_cg4(zr + i);
  }
#pragma unroll
  for (int n = 0; n < N; ++n) {
    if (i0 + n * step >= C) break;
    float z[4] = {g[n].x, g[n].y, g[n].z, g[n].w};
    logistic_all<true>(z, z);
    g[n] = make_float4(z[0], z[1], z[2], z[3]);
    float4& x = v[n];
    if (!AFTER) { x.x *= g[n].x; x.y *= g[n].y; x.z *= g[n].z; x.w *= g[n].w; }
    const float ss = warp_sum(fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w))));
    if (lane == 0) sums[n * NW + warp] = ss;
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const int i = i0 + n * step;
    if (i >= C) break;
    const int piece = (n * NW + warp) / per;
    float ss = 0.f;
    for (int j = 0; j < per; ++j) ss += sums[piece * per + j];
    const float rstd = inv_sqrt(ss / (float)W + eps);
    const float4 c = gs_w4(w + (AFTER ? i - piece * W : i));
    float4 x = v[n];
    x = make_float4(x.x * rstd * c.x, x.y * rstd * c.y, x.z * rstd * c.z, x.w * rstd * c.w);
    if (AFTER) { x.x *= g[n].x; x.y *= g[n].y; x.z *= g[n].z; x.w *= g[n].w; }
    gs_st4(o + i, x);
  }
}

}  // namespace b200

using namespace b200;

extern "C" int b200_gated_scan(const float* x, int64_t ld, int q_col, int k_col, int v_col, const float* gates, int64_t ld_g,
                               const float* rate, const float* dt_bias, const float* skip, const int32_t* cu_seq,
                               const int32_t* ctx_lens, const int32_t* state_slots, float* S, float* o_raw, int n_seqs, int H,
                               int G, int dk, int dv, int delta, int max_len, void* stream) {
  B200_REQUIRE(n_seqs >= 0 && H > 0 && G > 0 && H % G == 0 && dk > 0 && dv > 0 && dk <= 512,
               "gated_scan: bad shape H=%d G=%d dk=%d dv=%d (dk <= 512)", H, G, dk, dv);
  B200_REQUIRE(((ld | q_col | k_col | v_col) & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(S)) & 15) == 0,
               "gated_scan: rows, columns and state in whole 16-byte pieces");
  if (n_seqs == 0) return B200_OK;
  const GatedScanArgs a{x, ld, q_col, k_col, v_col, gates, ld_g, rate, dt_bias, skip, cu_seq, ctx_lens, state_slots, S, o_raw, H, G,
                        (dk + 3) & ~3, dv, (dv + 3) & ~3, INT32_MAX};
  cudaStream_t s = (cudaStream_t)stream;
  return delta ? gated_scan_pick<true>(a, n_seqs, max_len, s) : gated_scan_pick<false>(a, n_seqs, max_len, s);
}

// The state-space form with a workspace: portions of more than 16 rows over their chunks side by side, the others one-pass beside
// them.  The delta rule, and shapes and alignments that the chunk kernels do not take, run as b200_gated_scan.
extern "C" int b200_gated_scan_chunked(const float* x, int64_t ld, int q_col, int k_col, int v_col, const float* gates, int64_t ld_g,
                                       const float* rate, const float* dt_bias, const float* skip, const int32_t* cu_seq,
                                       const int32_t* ctx_lens, const int32_t* state_slots, float* S, float* o_raw, int n_seqs, int H,
                                       int G, int dk, int dv, int delta, int max_len, int rows, float* workspace,
                                       int64_t workspace_floats, void* stream) {
  if (delta || workspace == nullptr || rows <= 0 || n_seqs <= 0 || H <= 0 || G <= 0 || H % G != 0 || dv <= 0 ||
      ((uintptr_t)workspace & 15) != 0 || !cs_covers(x, 4, ld, q_col, k_col, v_col, dk, dv, S, o_raw))
    return b200_gated_scan(x, ld, q_col, k_col, v_col, gates, ld_g, rate, dt_bias, skip, cu_seq, ctx_lens, state_slots, S, o_raw, n_seqs, H,
                           G, dk, dv, delta, max_len, stream);
  B200_REQUIRE(workspace_floats >= cs_workspace_floats(rows, n_seqs, H, dk, dv), "gated_scan: workspace of %lld floats too small",
               (long long)workspace_floats);
  cudaStream_t s = (cudaStream_t)stream;
  const int short_rows = cs_short(rows, n_seqs);
  if (short_rows > 0) {
    const GatedScanArgs one{x, ld, q_col, k_col, v_col, gates, ld_g, rate, dt_bias, skip, cu_seq, ctx_lens, state_slots, S, o_raw, H, G,
                            dk, dv, dv, short_rows};
    const int rc = gated_scan_pick<false>(one, n_seqs, short_rows, s);
    if (rc != B200_OK) return rc;
  }
  const ChunkScanArgs a{x, ld, q_col, k_col, v_col, H, G, dv, cu_seq, ctx_lens, state_slots, n_seqs, short_rows, S, o_raw};
  return cs_launch<StateSpaceForm>(a, {gates, ld_g, rate, dt_bias, skip}, dk, rows, workspace, s);
}

extern "C" int b200_gate_norm(const float* y, const void* proj, int f32, int64_t ld, int z_col, const void* w, void* out,
                              int64_t ldo, int T, int C, int parts, int gate_after, float eps, void* stream) {
  B200_REQUIRE(T >= 0 && C > 0 && parts > 0 && C % parts == 0, "gate_norm: %d channels in %d parts", C, parts);
  if (T == 0) return B200_OK;
  const size_t smem = sizeof(float) * (size_t)C;
  cudaStream_t s = (cudaStream_t)stream;
  auto al = [](const void* p, int n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; };
  const int n = f32 ? 16 : 8;
  const bool vec = (C / parts) % 4 == 0 && ld % 4 == 0 && ldo % 4 == 0 && z_col % 4 == 0 && al(y, 16) && al(proj, n) && al(out, n) && al(w, 8);
  const int W = C / parts, lanes = W / 4;
  if (vec && lanes <= 32 && (lanes & (lanes - 1)) == 0 && C <= kGnThreads * 4 * 8) {
#define B200_GNHN(TA, A, N) \
  (void)launch_pdl(gate_norm_heads_kernel<TA, A, N>, dim3(T), dim3(kGnThreads), 0, s, 1, y, (const TA*)proj, ld, z_col, (const bf16*)w, (TA*)out, \
                   ldo, C, W, eps)
#define B200_GNH(TA, A)                                            \
  do {                                                             \
    if (C <= 2 * kGnThreads * 4) B200_GNHN(TA, A, 2);              \
    else B200_GNHN(TA, A, 8);                                      \
  } while (0)
    if (f32) { if (gate_after) B200_GNH(float, true); else B200_GNH(float, false); }
    else { if (gate_after) B200_GNH(bf16, true); else B200_GNH(bf16, false); }
#undef B200_GNH
#undef B200_GNHN
    return b200_check_launch("b200_gate_norm");
  }
  if (vec && W % 128 == 0 && C <= kGnThreads * 8) {      // (two groups per thread; with four of 4096 channels 84 us where the staged row takes 71)
#define B200_GNP(TA, A) \
  (void)launch_pdl(gate_norm_parts_kernel<TA, A>, dim3(T), dim3(kGnThreads), 0, s, 1, y, (const TA*)proj, ld, z_col, (const bf16*)w, (TA*)out, ldo, \
                   C, W, eps)
    if (f32) { if (gate_after) B200_GNP(float, true); else B200_GNP(float, false); }
    else { if (gate_after) B200_GNP(bf16, true); else B200_GNP(bf16, false); }
#undef B200_GNP
    return b200_check_launch("b200_gate_norm");
  }
  B200_REQUIRE(smem <= 48 * 1024, "gate_norm: %d channels exceed the staged row (12288)", C);
#define B200_GN(TA, V, A) \
  (void)launch_pdl(gate_norm_kernel<TA, V, A>, dim3(T), dim3(kGnThreads), smem, s, 1, y, (const TA*)proj, ld, z_col, (const bf16*)w, (TA*)out, ldo, C, \
                   parts, eps)
#define B200_GN2(TA)                                                                                     \
  do {                                                                                                   \
    if (gate_after) { if (vec) B200_GN(TA, true, true); else B200_GN(TA, false, true); }                 \
    else { if (vec) B200_GN(TA, true, false); else B200_GN(TA, false, false); }                          \
  } while (0)
  if (f32) B200_GN2(float);
  else B200_GN2(bf16);
#undef B200_GN2
#undef B200_GN
  return b200_check_launch("b200_gate_norm");
}
