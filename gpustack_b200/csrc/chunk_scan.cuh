// Matrix-state recurrences with one decay per token and head, or per token and key channel, over prompt portions: all chunks of a
// sequence side by side.
//
// With a state S (dk x dv), rows t = 0 .. n-1 of a chunk of 64 and the weights that a recurrence's `Form` supplies:
//     o_t = aq_t S_start^T q_t + sum_{s<=t} D(t, s) (k_s . q_t) v_s          S_end = a S_start + sum_s w_s k_s v_s^T
// State space and, with a decay per key channel, gated linear attention; mLSTM and linear attention run on the tensor cores
// (chunk_tc.cuh).  Three launches:
//   chunk_state   one CTA per (chunk, head, value tile): C = sum_s w_s k_s v_s^T into the workspace, [chunk][H][dk][dv]
//   chunk_carry   one CTA per (8 keys x 128 values of the state, head, sequence): walks a sequence's chunks, puts S_start in C's
//                 place and leaves the sequence's final state in its slot
//   chunk_output  one CTA per (chunk, head, value tile): k_s . q_t, then aq_t S_start^T q_t and the chunk's own rows
// Why: the one-pass form (16 rows at a time, state in shared memory) is a serial chain of short phases on (sequences x heads x
// dv / 32) CTAs -- 128 CTAs at 6 us per 16 rows for four prompts -- and idles the chip.  Chunks are independent but for the
// elementwise carry, so a portion of any length fills the chip; the price is the chunks' states through L2 (dk dv 4 bytes per
// 64 rows and head, written, carried and read once each).  Everything is fp32 FMAs as before; bound: the FMA rate
// (4 dk dv + 64 (dk + dv) per row and head) and, next to it, shared memory: a 16-byte read takes it four cycles for a warp of many
// addresses and two for a warp of one, a packed FMA (fma.rn.f32x2) a scheduler two.  So a CTA of 256 threads holds a 128 x 128 (state)
// or 64 x 128 (output) tile in which a warp shares its keys or rows and its lanes the 128 values: per key or row of 8 x 128, two reads
// of one address and one of many feed 16 packed FMAs, 64 cycles of either for the eight warps (4 x 8 tiles, two sets of keys or
// rows to a warp: 96 of reads).
// Gated linear attention, 5 ragged prompts of 6007 rows, 8 heads of 64 x 128: state 42, carry 12, output 67 us (with 4 x 8 tiles and
// the weights pair by pair 44, 12, 85; one-pass, the layer 501 us, so 155).  State space, one prompt of 2048 rows, 32 heads of
// 128 x 64: 36, 14, 79 us (one-pass 191).  The copies behind the sums and the carry's whole lines are worth a tenth (measured over
// linear attention's 4 x 2048 rows before it left: 62, 44, 104 us, without them 65, 62, 116).  Chunks of 64: with 32 the states double,
// with 128 the chunk's own rows cost more FMAs than the states save.
// Sequences of at most kCsShort rows are left to the caller's one-pass kernel (their state would cross L2 three times for
// a few rows of work).
#pragma once
#include "common.cuh"
#include "runtime.h"

namespace b200 {

constexpr int kCsRows = 64, kCsThreads = 256, kCsShort = 16, kCsAPitch = kCsRows + 4;

// What every recurrence shares: rows, sequences, state, outputs, workspace.
struct ChunkScanArgs {
  const void* x;                   // rows of TA
  int64_t ld;
  int q_col, k_col, v_col;
  int H, G, dv;                    // head h reads query / key head h / (H / G)
  const int32_t* cu_seq;
  const int32_t* ctx_lens;
  const int32_t* state_slots;
  int n_seqs;
  int short_rows;                  // sequences of at most so many rows are the one-pass kernel's (cs_short)
  float* S;                        // [slots][H][dv][dk]
  float* o;                        // [T][H dv]
  float* ws;                       // [chunks][H][dk][dv]
  float* ws_row;                   // [chunks][H][ws_row_width]: a recurrence's own carry (its Form says what)
  int ws_row_width;                // dk + 4
  float* ws_sums;                  // [chunks][H][2][64][dk]: kVector, the running sums' two parts
};

template <int ROWS>
__host__ __device__ __forceinline__ int cs_chunks(int rows, int short_rows) { return rows > short_rows ? (rows + ROWS - 1) / ROWS : 0; }

// A step of one sequence needs no one-pass launch beside the chunks: whatever the sequence's rows of a longer buffer, they are chunks.
inline int cs_short(int64_t rows, int n_seqs) { return n_seqs > 1 || rows <= kCsShort ? kCsShort : 0; }

// Chunks that the sequences of a step can have at most: the launch's grid and the workspace are sized by this.
inline int64_t cs_max_chunks(int64_t rows, int64_t n_seqs) {
  const int64_t longs = rows / (kCsShort + 1);
  return rows / kCsRows + (longs < n_seqs ? longs : n_seqs);
}
inline int64_t cs_workspace_floats(int64_t rows, int64_t n_seqs, int64_t H, int64_t dk, int64_t dv, bool vector = false) {
  return cs_max_chunks(rows, n_seqs) * H * (dk * dv + dk + 4 + (vector ? 2 * kCsRows * dk : 0));
}

// Sequence and place in it of chunk b of ROWS rows (whole warp; seq -1: no such chunk), or with b < 0 the chunks before sequence `upto`.
template <int ROWS>
__device__ __forceinline__ void cs_find(const int32_t* cu, int n_seqs, int short_rows, int b, int upto, int& seq, int& local, int& before) {
  const int lane = threadIdx.x & 31;
  seq = -1;
  local = 0;
  before = 0;
  for (int base = 0; base < n_seqs; base += 32) {
    const int s = base + lane;
    const int c = s < n_seqs ? cs_chunks<ROWS>(cu[s + 1] - cu[s], short_rows) : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (b >= 0) {
      const uint32_t hit = __ballot_sync(0xffffffffu, before + incl > b);
      if (hit) {
        const int l = __ffs(hit) - 1;
        seq = base + l;
        local = b - before - (__shfl_sync(0xffffffffu, incl, l) - __shfl_sync(0xffffffffu, c, l));
        return;
      }
    } else if (upto < base + 32) {
      before += __shfl_sync(0xffffffffu, incl - c, upto - base);
      return;
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// The chunk of a CTA of chunk_state / chunk_output.
struct ChunkPlace {
  int seq, first, rows, slot, local;
};
__device__ __forceinline__ ChunkPlace cs_place(const ChunkScanArgs& a, int* shared5) {
  if (threadIdx.x < 32) {
    int seq, local, before;
    cs_find<kCsRows>(a.cu_seq, a.n_seqs, a.short_rows, (int)blockIdx.x, 0, seq, local, before);
    if (threadIdx.x == 0) {
      shared5[0] = seq;
      if (seq >= 0) {
        const int t0 = a.cu_seq[seq] + local * kCsRows;
        shared5[1] = t0;
        shared5[2] = min(kCsRows, a.cu_seq[seq + 1] - t0);
        shared5[3] = a.state_slots[seq];
        shared5[4] = local;
      }
    }
  }
  __syncthreads();
  return {shared5[0], shared5[1], shared5[2], shared5[3], shared5[4]};
}

// ROWS x W values of column `col` on, on their way to shared memory by cp.async (row pitch PITCH, rows from `n` and columns from
// `width` on zero).
template <int ROWS, int W, int PITCH>
__device__ __forceinline__ void cs_issue(const float* x, int64_t ld, int first, int n, int col, int width, float* dst) {
  constexpr int PER = W / 4, STEP = kCsThreads / PER, ITERS = ROWS / STEP;
  const int c = ((int)threadIdx.x % PER) * 4, r0 = (int)threadIdx.x / PER;
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    const int r = r0 + i * STEP;
    const bool in = r < n && c < width;
    cp_async_16_zfill(dst + r * PITCH + c, in ? x + (size_t)(first + r) * ld + col + c : x, in);
  }
}

// Running sums of a chunk's logarithms per key channel, inclusive: F[t][k] = sum_(r <= t) lg(r, k), 256 threads: four runs of 16
// rows per channel, with 128 channels two of 32.  hi / lo: [64][DK + 4].  Ends with a barrier.
template <int DK, typename LG>
__device__ __forceinline__ void cs_channel_sums(float* hi, float* lo, double* run, LG lg) {
  constexpr int RUNS = kCsThreads / DK, ROWS = kCsRows / RUNS, P = DK + 4;
  const int k = (int)threadIdx.x % DK, r = (int)threadIdx.x / DK;
  double sum = 0.0;
#pragma unroll 4
  for (int t = r * ROWS; t < (r + 1) * ROWS; ++t) sum += (double)lg(t, k);
  run[r * DK + k] = sum;
  __syncthreads();
  double F = 0.0;
  for (int i = 0; i < r; ++i) F += run[i * DK + k];
#pragma unroll 4
  for (int t = r * ROWS; t < (r + 1) * ROWS; ++t) {
    F += (double)lg(t, k);
    const float h = (float)F;
    hi[t * P + k] = h;
    lo[t * P + k] = (float)(F - (double)h);
  }
  __syncthreads();
}
// 2^(h + l) of a sum's two parts
__device__ __forceinline__ float cs_exp2(float h, float l) { return ex2_approx(h) * fmaf(l, 0.6931471805599453f, 1.0f); }

template <int DK, int VT, bool VECTOR = false>
struct ChunkSmem {
  static constexpr int kSum = VECTOR ? kCsRows * (DK + 4) : 0;               // one part of the running sums
  static constexpr int kState = kCsRows * (DK + VT) + 2 * kSum;              // floats
  static constexpr int kTile = 32 * VT;                      // a tile of 32 state or value rows
  static constexpr int kB = kCsRows * (DK + 4) + kSum > 2 * kTile ? kCsRows * (DK + 4) + kSum : 2 * kTile;
  static constexpr int kOutput = kCsRows * (DK + 4) + kB + kTile + kCsRows * kCsAPitch + kSum;
};

// Form: `Scratch` (shared arrays of one chunk), `state_weights` and `state_row` for chunk_state, `output_weights`, aq(t), D(t, s) and
// finish() for chunk_output, `Carry` (the chunks' decays) for chunk_carry.
// A Form with kVector has one decay per KEY CHANNEL instead: with the running sums F of a chunk's base-2 logarithms per channel
// (summed in fp64, kept as two fp32 parts, so that a difference is as exact as an fp32 product of decays) the keys of the state
// are weighted by 2^(F_n - F_s), the queries of the state's part by 2^F_t, and (k_s . q_t) is a sum of k q 2^(F_t - F_s), whose
// exponents cs_vector_weights forms in parts: none of a positive number, whatever the decays are.
// The carry and the output begin while the launch before runs (programmatic launches): a carry's CTAs load their slots' states, an
// output's their queries and keys, before they wait for it (gated linear attention of 6007 rows, the layer 171 -> 162 us, with the
// states' own launch and those before it 155; of 256 to 2048 rows 2 to 4 us less).  Every CTA of chunk_state waits first and only then
// lets a carry start, so that one whose CTAs have nothing to do still comes after the one-pass kernel before the chunks.
__device__ __forceinline__ void cs_release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cs_wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <int DK, int VT, typename Form>
__global__ void __launch_bounds__(kCsThreads, 2)
chunk_state_kernel(const ChunkScanArgs a, const typename Form::Params p) {
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  __shared__ typename Form::Scratch scratch;
  __shared__ int shared5[5];
  const ChunkPlace at = cs_place(a, shared5);
  if (at.seq < 0 || at.slot < 0) return;
  const int h = blockIdx.y, v0 = blockIdx.z * VT, tid = threadIdx.x;
  float* ks = smem;                // [64][DK]
  float* vs = smem + kCsRows * DK; // [64][VT]
  const float* x = reinterpret_cast<const float*>(a.x);
  const int kcol = a.k_col + h / (a.H / a.G) * DK, vcol = a.v_col + h * a.dv + v0;
  // two halves of 32 rows: the second one is on its way while the first is summed
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    cs_issue<32, DK, DK>(x, a.ld, at.first + 32 * e, at.rows - 32 * e, kcol, DK, ks + 32 * e * DK);
    cs_issue<32, VT, VT>(x, a.ld, at.first + 32 * e, at.rows - 32 * e, vcol, a.dv - v0, vs + 32 * e * VT);
    cp_async_commit();
  }
  float* hi = vs + kCsRows * VT;   // [64][DK + 4] each, kVector only
  float* lo = hi + kCsRows * (DK + 4);
  if constexpr (Form::kVector) Form::template sums<DK>(p, a, scratch, h, at, hi, lo);
  else Form::state_weights(p, a, scratch, h, at);
  // a thread: KR keys (in pairs) x 4 values; the lanes of a group share the keys
  constexpr int LANES = VT / 4, KR = DK / (kCsThreads / LANES);
  const int vl = tid % LANES, kg = tid / LANES;
  f32x2 acc[KR / 2][4];
#pragma unroll
  for (int i = 0; i < KR / 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (e == 0) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    const int n = min(at.rows - 32 * e, 32);
    if constexpr (Form::kVector) {
      const int k = tid % DK;
      const float Fh = hi[(at.rows - 1) * (DK + 4) + k], Fl = lo[(at.rows - 1) * (DK + 4) + k];
#pragma unroll 4
      for (int s = 32 * e + tid / DK; s < 32 * e + n; s += kCsThreads / DK)
        ks[s * DK + k] *= cs_exp2(Fh - hi[s * (DK + 4) + k], Fl - lo[s * (DK + 4) + k]);
      __syncthreads();
    }
#pragma unroll 4
    for (int r = 0; r < n; ++r) {
      const int s = 32 * e + r;
      float4 v = *reinterpret_cast<const float4*>(vs + s * VT + 4 * vl);
      if constexpr (!Form::kVector) {
        const float w = scratch.w[s];
        v = make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
      }
      const f32x2 d[4] = {dup2(v.x), dup2(v.y), dup2(v.z), dup2(v.w)};
#pragma unroll
      for (int i = 0; i < KR / 4; ++i) {
        const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(ks + s * DK + KR * kg + 4 * i);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * i][j] = fma2(kk.x, d[j], acc[2 * i][j]);
          acc[2 * i + 1][j] = fma2(kk.y, d[j], acc[2 * i + 1][j]);
        }
      }
    }
  }
  float* out = a.ws + (((size_t)blockIdx.x * a.H + h) * DK + KR * kg) * a.dv + v0 + 4 * vl;
  if (v0 + 4 * vl < a.dv) {
#pragma unroll
    for (int i = 0; i < KR / 2; ++i) {
      const float2 u[4] = {unpack2(acc[i][0]), unpack2(acc[i][1]), unpack2(acc[i][2]), unpack2(acc[i][3])};
      *reinterpret_cast<float4*>(out + (size_t)(2 * i) * a.dv) = make_float4(u[0].x, u[1].x, u[2].x, u[3].x);
      *reinterpret_cast<float4*>(out + (size_t)(2 * i + 1) * a.dv) = make_float4(u[0].y, u[1].y, u[2].y, u[3].y);
    }
  }
  if constexpr (Form::kVector) {
    if (blockIdx.z == 0) {
      if (tid < DK) {
        const int i = (at.rows - 1) * (DK + 4) + tid;
        a.ws_row[((size_t)blockIdx.x * a.H + h) * a.ws_row_width + tid] = cs_exp2(hi[i], lo[i]);
      }
      float* sums = a.ws_sums + ((size_t)blockIdx.x * a.H + h) * (2 * kCsRows * DK);
      for (int i = tid; i < kCsRows * DK / 4; i += kCsThreads) {
        const int from = (4 * i / DK) * (DK + 4) + 4 * i % DK;
        *reinterpret_cast<float4*>(sums + 4 * i) = *reinterpret_cast<const float4*>(hi + from);
        *reinterpret_cast<float4*>(sums + kCsRows * DK + 4 * i) = *reinterpret_cast<const float4*>(lo + from);
      }
    }
  } else if (blockIdx.z == 0) {
    Form::template state_row<DK>(a, scratch, h);
  }
}

// 8 keys x 128 values of a head's state through a sequence's chunks: a warp's row of a chunk is 512 contiguous bytes, eight
// chunks are in flight.
constexpr int kCsCarryKeys = 8, kCsCarryDepth = 8;

template <int DK, typename Form>
__global__ void __launch_bounds__(kCsThreads)
chunk_carry_kernel(const ChunkScanArgs a, const typename Form::Params p) {
  __shared__ float tile[128][kCsCarryKeys + 1];
  __shared__ int base;
  const int s = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int t0 = a.cu_seq[s], t1 = a.cu_seq[s + 1], nc = cs_chunks<kCsRows>(t1 - t0, a.short_rows), slot = a.state_slots[s];
  if (nc == 0 || slot < 0) return;
  if (tid < 32) {
    int q, l, before;
    cs_find<kCsRows>(a.cu_seq, a.n_seqs, a.short_rows, -1, s, q, l, before);
    if (tid == 0) base = before;
  }
  const int k0 = (blockIdx.x % (DK / kCsCarryKeys)) * kCsCarryKeys, v0 = (blockIdx.x / (DK / kCsCarryKeys)) * 128;
  float* Sp = a.S + ((size_t)slot * a.H + h) * a.dv * DK;
  const bool fresh = a.ctx_lens[s] == 0;
  for (int i = tid; i < 128 * kCsCarryKeys; i += kCsThreads) {
    const int v = i / kCsCarryKeys, k = i % kCsCarryKeys;     // k fastest: the slot's layout, whole 32-byte sectors
    tile[v][k] = (!fresh && v0 + v < a.dv) ? __ldcg(Sp + (size_t)(v0 + v) * DK + k0 + k) : 0.f;
  }
  cs_wait_before();
  cs_release_next();                                  // (behind the wait: an output's CTA finds the chunks' states complete)
  __syncthreads();
  const int v = (tid & 31) * 4, k = tid >> 5;
  float4 S = make_float4(tile[v][k], tile[v + 1][k], tile[v + 2][k], tile[v + 3][k]);
  const bool live = v0 + v < a.dv;
  const size_t step = (size_t)a.H * DK * a.dv;
  float* C = a.ws + ((size_t)base * a.H + h) * DK * a.dv + (size_t)(k0 + k) * a.dv + v0 + v;
  typename Form::Carry carry(a, h, base, k0 + k);
  constexpr int U = kCsCarryDepth;
  for (int c0 = 0; c0 < nc; c0 += U) {
    float4 in[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (live && c0 + u < nc) in[u] = __ldcg(reinterpret_cast<const float4*>(C + (size_t)(c0 + u) * step));
    carry.fetch(c0, nc);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c0 + u >= nc) break;
      const float f = carry.f[u];
      if (live) {
        *reinterpret_cast<float4*>(C + (size_t)(c0 + u) * step) = S;
        S = make_float4(fmaf(f, S.x, in[u].x), fmaf(f, S.y, in[u].y), fmaf(f, S.z, in[u].z), fmaf(f, S.w, in[u].w));
      }
    }
  }
  __syncthreads();
  tile[v][k] = S.x; tile[v + 1][k] = S.y; tile[v + 2][k] = S.z; tile[v + 3][k] = S.w;
  __syncthreads();
  for (int i = tid; i < 128 * kCsCarryKeys; i += kCsThreads) {
    const int vv = i / kCsCarryKeys, kk = i % kCsCarryKeys;
    if (v0 + vv < a.dv) Sp[(size_t)(v0 + vv) * DK + k0 + kk] = tile[vv][kk];
  }
}

// How chunk_output's threads share the 64 rows x VT values: VT / 4 lanes side by side are a group, a thread has 4 values of the
// group's rows, which lie in pairs (2 g, 2 g + 1) + i * BLOCK.  Queries and weights lie transposed, [key or row][64], a
// group's rows side by side, so that one read serves a whole group (half the price of one with addresses of its own) and its pairs
// are the operands of packed FMAs.
template <int VT>
struct CsRows {
  static constexpr int kLanes = VT / 4, kGroups = kCsThreads / kLanes, kRows = kCsRows / kGroups, kPairs = kRows / 2, kBlock = 2 * kGroups;
  static __device__ __forceinline__ int place(int t) { return t % kBlock / 2 * kRows + t / kBlock * 2 + (t & 1); }
};

// a group's rows of one key or row: its pairs
template <int VT>
__device__ __forceinline__ void cs_pairs(const float* p, f32x2 (&out)[CsRows<VT>::kPairs]) {
#pragma unroll
  for (int i = 0; i < CsRows<VT>::kPairs; i += 2) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + 2 * i);
    out[i] = v.x;
    out[i + 1] = v.y;
  }
}

// acc += weights^T V over the chunk's own rows of block I0.  A row sees those up to itself -- the rest is left out, not multiplied by
// zero, so that a value that is no number reaches no earlier row.
template <int VT, int I0>
__device__ __forceinline__ void cs_own_rows(f32x2 (&acc)[CsRows<VT>::kPairs][4], const float* A, const float* V, int g, int vl) {
  using R = CsRows<VT>;
#pragma unroll 4
  for (int r = 0; r < R::kBlock; ++r) {
    const int s = R::kBlock * I0 + r;
    const float4 v = *reinterpret_cast<const float4*>(V + s * VT + 4 * vl);
    const f32x2 d[4] = {dup2(v.x), dup2(v.y), dup2(v.z), dup2(v.w)};
    f32x2 w[R::kPairs];
    cs_pairs<VT>(A + s * kCsAPitch + R::kRows * g, w);
    if (r <= 2 * g) {
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[I0][j] = fma2(w[I0], d[j], acc[I0][j]);
    } else if (r == 2 * g + 1) {
      const float u = unpack2(w[I0]).y, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 o = unpack2(acc[I0][j]);
        acc[I0][j] = pack2(o.x, fmaf(u, vv[j], o.y));
      }
    }
#pragma unroll
    for (int i = I0 + 1; i < R::kPairs; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(w[i], d[j], acc[i][j]);
  }
}

// The weights k_s . q_t of a recurrence with a decay per key channel, transposed into A, and the queries' part of the state into qs
// ([key][64] in the order of `place`, times 2^F_t).  Rows are taken in 16 blocks of four.  Within a block the sums are formed term by
// term, with the decay between the two rows.  Between two blocks the decay comes in three factors, from s to the end of its
// block, from there to the end of the one before t's, and on to t: no exponent is positive, only the middle one
// belongs to a pair of blocks, and 4 x 4 sums share it.  (With an exponential for each of the 2080 pairs of rows and each channel,
// and both rows and their sums read for it, these weights alone kept shared memory busy for 12.3k of the kernel's 31k cycles.)
// On entry the queries in qs, the keys in B, the sums in hi / lo, all [64][DK + 4]; hi and lo are used up.
template <int DK, int VT>
__device__ __forceinline__ void cs_vector_weights(float* qs, float* B, float* hi, float* lo, float* A, bool zero_start) {
  using R = CsRows<VT>;
  constexpr int P = DK + 4, QUADS = DK / 4;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  {
    // the blocks' own weights: 16 lanes share the channels of a block
    const int b = tid >> 4, c = tid & 15;
    float sum[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) sum[i] = 0.f;
#pragma unroll
    for (int e = 0; e < QUADS / 16; ++e) {
      float q[4][4], k[4][4], h[4][4], l[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int from = (4 * b + i) * P + 4 * (c + 16 * e);
        *reinterpret_cast<float4*>(q[i]) = *reinterpret_cast<const float4*>(qs + from);
        *reinterpret_cast<float4*>(k[i]) = *reinterpret_cast<const float4*>(B + from);
        *reinterpret_cast<float4*>(h[i]) = *reinterpret_cast<const float4*>(hi + from);
        *reinterpret_cast<float4*>(l[i]) = *reinterpret_cast<const float4*>(lo + from);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j)
#pragma unroll
          for (int u = 0; u < 4; ++u)
            sum[i * (i + 1) / 2 + j] = fmaf(q[i][u] * k[j][u], ex2_approx((h[i][u] - h[j][u]) + (l[i][u] - l[j][u])), sum[i * (i + 1) / 2 + j]);
    }
    float mine = 0.f;
    int to = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        float v = sum[i * (i + 1) / 2 + j];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (c == i * (i + 1) / 2 + j) {
          mine = v;
          to = (4 * b + j) * kCsAPitch + R::place(4 * b + i);
        }
      }
    if (c < 10) A[to] = mine;
  }
  __syncthreads();
  // a lane has two rows (one of each half), a warp every eighth quad of channels: rows of pitch DK + 4 are read without conflicts
  constexpr int ITEMS = QUADS / 8 * 2;
  float qe[ITEMS][4], qt[ITEMS][4];
#pragma unroll
  for (int e = 0; e < ITEMS; ++e) {
    const int t = lane + 32 * (e & 1), k0 = 4 * (warp + 8 * (e >> 1)), from = t * P + k0, end = (t | 3) * P + k0, start = ((t & ~3) - 1) * P + k0;
    float q[4], k[4], h[4], l[4], eh[4], el[4], sh[4] = {0.f, 0.f, 0.f, 0.f}, sl[4] = {0.f, 0.f, 0.f, 0.f};
    *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(qs + from);
    *reinterpret_cast<float4*>(k) = *reinterpret_cast<const float4*>(B + from);
    *reinterpret_cast<float4*>(h) = *reinterpret_cast<const float4*>(hi + from);
    *reinterpret_cast<float4*>(l) = *reinterpret_cast<const float4*>(lo + from);
    *reinterpret_cast<float4*>(eh) = *reinterpret_cast<const float4*>(hi + end);
    *reinterpret_cast<float4*>(el) = *reinterpret_cast<const float4*>(lo + end);
    if (t >= 4) {
      *reinterpret_cast<float4*>(sh) = *reinterpret_cast<const float4*>(hi + start);
      *reinterpret_cast<float4*>(sl) = *reinterpret_cast<const float4*>(lo + start);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      k[u] *= cs_exp2(eh[u] - h[u], el[u] - l[u]);
      qe[e][u] = q[u] * cs_exp2(h[u] - sh[u], l[u] - sl[u]);
      qt[e][u] = zero_start ? 0.f : q[u] * cs_exp2(h[u], l[u]);
    }
    *reinterpret_cast<float4*>(B + from) = *reinterpret_cast<const float4*>(k);
  }
  // the sums at the blocks' ends: a warp has two of them
  constexpr int EK = DK / 32;                        // a lane's channels of a row
  float e_h[2][EK], e_l[2][EK];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int u = 0; u < EK; ++u) {
      e_h[i][u] = hi[(4 * (2 * warp + i) + 3) * P + lane + 32 * u];
      e_l[i][u] = lo[(4 * (2 * warp + i) + 3) * P + lane + 32 * u];
    }
  __syncthreads();
  float* Eh = lo;                                    // [16][DK + 4] each
  float* El = lo + 16 * P;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int u = 0; u < EK; ++u) {
      Eh[(2 * warp + i) * P + lane + 32 * u] = e_h[i][u];
      El[(2 * warp + i) * P + lane + 32 * u] = e_l[i][u];
    }
#pragma unroll
  for (int e = 0; e < ITEMS; ++e) {
    const int t = lane + 32 * (e & 1), k0 = 4 * (warp + 8 * (e >> 1));
    *reinterpret_cast<float4*>(hi + t * P + k0) = *reinterpret_cast<const float4*>(qe[e]);
#pragma unroll
    for (int u = 0; u < 4; ++u) qs[(k0 + u) * kCsRows + R::place(t)] = qt[e][u];
  }
  __syncthreads();
  {
    // 120 pairs of blocks; two lanes share a pair's channels, and start at different ones where their rows lie in the same banks
    const int half = tid & 1, u = min(tid >> 1, 119);
    int bt = 1;
    while (bt * (bt + 1) / 2 <= u) ++bt;
    const int bs = u - bt * (bt - 1) / 2;
    f32x2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 1
    for (int d = 0; d < QUADS / 2; ++d) {
      const int c = 4 * (2 * ((d + (bs >> 1)) & (QUADS / 2 - 1)) + half);
      const float4 sh = *reinterpret_cast<const float4*>(Eh + (bt - 1) * P + c), sl = *reinterpret_cast<const float4*>(El + (bt - 1) * P + c),
                   eh = *reinterpret_cast<const float4*>(Eh + bs * P + c), el = *reinterpret_cast<const float4*>(El + bs * P + c);
      const f32x2 m0 = pack2(ex2_approx((sh.x - eh.x) + (sl.x - el.x)), ex2_approx((sh.y - eh.y) + (sl.y - el.y))),
                  m1 = pack2(ex2_approx((sh.z - eh.z) + (sl.z - el.z)), ex2_approx((sh.w - eh.w) + (sl.w - el.w)));
      ulonglong2 k[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(B + (4 * bs + j) * P + c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ulonglong2 q = *reinterpret_cast<const ulonglong2*>(hi + (4 * bt + i) * P + c);
        q.x = mul2(q.x, m0);
        q.y = mul2(q.y, m1);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma2(q.y, k[j].y, fma2(q.x, k[j].x, acc[i][j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 z = unpack2(acc[i][j]);
        v[i] = z.x + z.y;
      }
      const float a0 = __shfl_xor_sync(0xffffffffu, half ? v[0] : v[2], 1), a1 = __shfl_xor_sync(0xffffffffu, half ? v[1] : v[3], 1);
      if (tid < 240)
        *reinterpret_cast<float2*>(A + (4 * bs + j) * kCsAPitch + R::place(4 * bt + 2 * half)) =
            half ? make_float2(v[2] + a0, v[3] + a1) : make_float2(v[0] + a0, v[1] + a1);
    }
  }
}

template <int DK, int VT, typename Form>
__global__ void __launch_bounds__(kCsThreads, 2)
chunk_output_kernel(const ChunkScanArgs a, const typename Form::Params p) {
  extern __shared__ __align__(16) float smem[];
  __shared__ typename Form::Scratch scratch;
  __shared__ int shared5[5];
  const ChunkPlace at = cs_place(a, shared5);
  if (at.seq < 0 || at.slot < 0) return;
  const int h = blockIdx.y, v0 = blockIdx.z * VT, tid = threadIdx.x, n = at.rows;
  using R = CsRows<VT>;
  constexpr int QP = DK + 4, TILE = ChunkSmem<DK, VT>::kTile;
  float* qs = smem;                                  // [64][DK + 4]
  float* X = qs + kCsRows * QP;                      // ring of three tiles of 32 rows; the keys [64][DK + 4] first lie on tiles 1 and 2
  float* B = X + TILE;
  float* A = B + ChunkSmem<DK, VT, Form::kVector>::kB;              // [64][68], a row for each s
  float* hi = A + kCsRows * kCsAPitch;               // [64][DK + 4] each, kVector only; lo behind the keys, until the ring takes the place
  float* lo = B + kCsRows * QP;
  const float* x = reinterpret_cast<const float*>(a.x);
  const int hg = h / (a.H / a.G), vcol = a.v_col + h * a.dv + v0;
  const bool zero_start = at.local == 0 && a.ctx_lens[at.seq] == 0;
  const float* C = a.ws + ((size_t)blockIdx.x * a.H + h) * DK * a.dv;
  // tiles in the order of their use: the state's rows (none for a zero start), then the chunk's own values
  const int n_state = zero_start ? 0 : DK / 32;
  auto tile_at = [&](int i) { return X + (i % 3) * TILE; };
  auto issue = [&](int i) {
    if (i < n_state) {
      cs_issue<32, VT, VT>(C, a.dv, 32 * i, 32, v0, a.dv - v0, tile_at(i));
    } else if (i == n_state) {
      cs_issue<32, VT, VT>(x, a.ld, at.first, n, vcol, a.dv - v0, tile_at(i));
    } else if (i == n_state + 1) {
      cs_issue<32, VT, VT>(x, a.ld, at.first + 32, n - 32, vcol, a.dv - v0, tile_at(i));
    }
    cp_async_commit();
  };
  {
    cs_issue<kCsRows, DK, QP>(x, a.ld, at.first, n, a.q_col + hg * DK, DK, qs);
    cs_issue<kCsRows, DK, QP>(x, a.ld, at.first, n, a.k_col + hg * DK, DK, B);
    cs_wait_before();
    if constexpr (Form::kVector) {                   // as chunk_state left them
      const float* sums = a.ws_sums + ((size_t)blockIdx.x * a.H + h) * (2 * kCsRows * DK);
      cs_issue<kCsRows, DK, QP>(sums, DK, 0, kCsRows, 0, DK, hi);
      cs_issue<kCsRows, DK, QP>(sums, DK, kCsRows, kCsRows, 0, DK, lo);
    }
    cp_async_commit();
    issue(0);
    if constexpr (!Form::kVector) Form::output_weights(p, a, scratch, h, at);
  }
  cp_async_wait<1>();
  __syncthreads();
  if constexpr (Form::kVector) {
    cs_vector_weights<DK, VT>(qs, B, hi, lo, A, zero_start);
  } else {
    const int tg = tid >> 4, vg = tid & 15;
    // k_s . q_t: rows t = tg + 16 i, columns s = vg + 16 j, j <= i; even and odd entries summed apart
    f32x2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 2
    for (int d = 0; d < DK; d += 4) {
      ulonglong2 q[4], k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        q[i] = *reinterpret_cast<const ulonglong2*>(qs + (tg + 16 * i) * QP + d);
        k[i] = *reinterpret_cast<const ulonglong2*>(B + (vg + 16 * i) * QP + d);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) acc[i][j] = fma2(q[i].y, k[j].y, fma2(q[i].x, k[j].x, acc[i][j]));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const int t = tg + 16 * i, s = vg + 16 * j;
        const float2 z = unpack2(acc[i][j]);
        A[s * kCsAPitch + R::place(t)] = (s <= t && t < n) ? Form::D(p, scratch, t, s) * (z.x + z.y) : 0.f;
      }
    if (!zero_start) {                               // the queries, [key][64]
      constexpr int ITEMS = DK / 32 * 2;
      const int warp = tid >> 5, lane = tid & 31;
      float4 v[ITEMS];
#pragma unroll
      for (int e = 0; e < ITEMS; ++e) v[e] = *reinterpret_cast<const float4*>(qs + (lane + 32 * (e & 1)) * QP + 4 * (warp + 8 * (e >> 1)));
      __syncthreads();
#pragma unroll
      for (int e = 0; e < ITEMS; ++e) {
        float* to = qs + 4 * (warp + 8 * (e >> 1)) * kCsRows + R::place(lane + 32 * (e & 1));
        to[0] = v[e].x;
        to[kCsRows] = v[e].y;
        to[2 * kCsRows] = v[e].z;
        to[3 * kCsRows] = v[e].w;
      }
    }
  }
  const int g = tid / R::kLanes, vl = tid % R::kLanes;
  f32x2 acc[R::kPairs][4];
#pragma unroll
  for (int i = 0; i < R::kPairs; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  // tile i: landed, and tile i - 1 used by every thread, so tile i + 2 may take its place (behind the first barrier the keys
  // are used as well)
  auto next_tile = [&](int i) {
    if (i == 0 || i == n_state + 1) cp_async_wait<0>();
    else cp_async_wait<1>();
    __syncthreads();
    if (i == 0) issue(1);
    if (i + 2 <= n_state + 1) issue(i + 2);
    return tile_at(i);
  };
#pragma unroll 1
  for (int i = 0; i < n_state; ++i) {
    const float* T = next_tile(i);
#pragma unroll 4
    for (int d = 0; d < 32; ++d) {
      f32x2 q[R::kPairs];
      cs_pairs<VT>(qs + (32 * i + d) * kCsRows + R::kRows * g, q);
      const float4 v = *reinterpret_cast<const float4*>(T + d * VT + 4 * vl);
      const f32x2 b[4] = {dup2(v.x), dup2(v.y), dup2(v.z), dup2(v.w)};
#pragma unroll
      for (int u = 0; u < R::kPairs; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[u][j] = fma2(q[u], b[j], acc[u][j]);
    }
  }
  if (!zero_start) {
#pragma unroll
    for (int i = 0; i < R::kPairs; ++i) {
      const int t = R::kBlock * i + 2 * g;
      const f32x2 f = pack2(Form::aq(scratch, t), Form::aq(scratch, t + 1));
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = mul2(acc[i][j], f);
    }
  }
  constexpr int HALF = R::kPairs / 2;                // blocks in each half of the rows
  const float* V0 = next_tile(n_state);
  cs_own_rows<VT, 0>(acc, A, V0, g, vl);
  if constexpr (HALF == 2) cs_own_rows<VT, 1>(acc, A, V0, g, vl);
  const float* V1 = next_tile(n_state + 1) - 32 * VT;
  cs_own_rows<VT, HALF>(acc, A, V1, g, vl);
  if constexpr (HALF == 2) cs_own_rows<VT, 3>(acc, A, V1, g, vl);
  const int v = v0 + 4 * vl;
  if (v >= a.dv) return;
#pragma unroll
  for (int i = 0; i < R::kPairs; ++i) {
    const float2 u[4] = {unpack2(acc[i][0]), unpack2(acc[i][1]), unpack2(acc[i][2]), unpack2(acc[i][3])};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = R::kBlock * i + 2 * g + e;
      if (t >= n) continue;
      const float4 mine = *reinterpret_cast<const float4*>((i < HALF ? V0 : V1) + t * VT + 4 * vl);
      const float4 sum = e ? make_float4(u[0].y, u[1].y, u[2].y, u[3].y) : make_float4(u[0].x, u[1].x, u[2].x, u[3].x);
      *reinterpret_cast<float4*>(a.o + (size_t)(at.first + t) * a.H * a.dv + h * a.dv + v) = Form::finish(p, scratch, h, t, sum, mine);
    }
  }
}

// Row layout and shapes that the three kernels take; everything else stays on the one-pass kernels.
inline bool cs_covers(const void* x, int elem, int64_t ld, int q_col, int k_col, int v_col, int dk, int dv, const void* S, const void* o) {
  const uintptr_t al = 4 * (uintptr_t)elem - 1;
  return (dk == 64 || dk == 128) && dv % 4 == 0 && ld % 4 == 0 && q_col % 4 == 0 && k_col % 4 == 0 && v_col % 4 == 0 &&
         ((uintptr_t)x & al) == 0 && ((uintptr_t)S & 15) == 0 && ((uintptr_t)o & 15) == 0;
}

template <int DK, int VT, typename Form>
int cs_launch_shape(const ChunkScanArgs& a, const typename Form::Params& p, int64_t rows, cudaStream_t s) {
  const int64_t chunks = cs_max_chunks(rows, a.n_seqs);
  const dim3 grid((unsigned)chunks, a.H, (a.dv + VT - 1) / VT);
  const int sb = ChunkSmem<DK, VT, Form::kVector>::kState * 4, ob = ChunkSmem<DK, VT, Form::kVector>::kOutput * 4;
  cudaError_t e = cudaFuncSetAttribute(chunk_state_kernel<DK, VT, Form>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_output_kernel<DK, VT, Form>, cudaFuncAttributeMaxDynamicSharedMemorySize, ob);
  if (e != cudaSuccess) {
    b200_set_error("chunk scan: %d bytes of shared memory: %s", ob, cudaGetErrorString(e));
    return B200_ERR_CUDA;
  }
  (void)launch_pdl(chunk_state_kernel<DK, VT, Form>, grid, dim3(kCsThreads), (size_t)sb, s, 1, a, p);
  (void)launch_pdl(chunk_carry_kernel<DK, Form>, dim3(DK / kCsCarryKeys * ((a.dv + 127) / 128), a.H, a.n_seqs), dim3(kCsThreads), 0, s, 1, a, p);
  (void)launch_pdl(chunk_output_kernel<DK, VT, Form>, grid, dim3(kCsThreads), (size_t)ob, s, 1, a, p);
  return b200_check_launch(Form::kName);
}

template <typename Form>
int cs_launch(ChunkScanArgs a, const typename Form::Params& p, int dk, int64_t rows, float* ws, cudaStream_t s) {
  const int64_t chunks = cs_max_chunks(rows, a.n_seqs);
  if (chunks == 0) return B200_OK;
  a.ws = ws;
  a.ws_row = ws + chunks * a.H * dk * a.dv;
  a.ws_row_width = dk + 4;
  a.ws_sums = a.ws_row + chunks * a.H * (dk + 4);
  if (dk == 64) return a.dv <= 64 ? cs_launch_shape<64, 64, Form>(a, p, rows, s) : cs_launch_shape<64, 128, Form>(a, p, rows, s);
  return a.dv <= 64 ? cs_launch_shape<128, 64, Form>(a, p, rows, s) : cs_launch_shape<128, 128, Form>(a, p, rows, s);
}

}  // namespace b200
