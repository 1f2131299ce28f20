// Matrix-state recurrences with one decay per token and head over prompt portions, all chunks of a sequence side by side, on the
// tensor cores with the precision of fp32.
//
// With a state S (dk x dv), rows t = 0 .. n-1 of a chunk of 128 and the weights that a recurrence's `Form` supplies:
//     o_t = aq_t S_start^T q_t + sum_{s<=t} D(t, s) (k_s . q_t) v_s          S_end = a S_start + b sum_s w_s k_s v_s^T
// Three launches:
//   ct_state   (chunk, head, value tile): C = sum_s k_s (w_s v_s)^T into the workspace
//   ct_carry   one thread per eight keys of a value column, head and sequence: walks a sequence's chunks, puts S_start's terms in C's
//              place and leaves the sequence's final state in its slot
//   ct_output  (chunk, head, value tile): scores Q K^T, Q S_start^T, and the weighted scores times V
// Precision: an fp32 number is the sum of three bf16 numbers (8 + 8 + 8 bits), so a product of two is formed from the six pairs of terms
// whose exponents matter, every pair exact and summed in fp32 by tcgen05.mma; what is a bf16 number is one term.  The instruction
// cuts its accumulator to 24 bits (it does not round), so the small pairs come first and few instructions meet an accumulator at
// its full size, and ct_uncut adds back what is lost on average.  Relative errors against 64 bits, by fp32 FMAs and here: states of
// 4 x 2048 rows of linear attention 2.3e-7 and 1.1e-7; mLSTM over 4000 ragged fp32 rows, outputs 2.2e-7 and 1.4e-7, states 1.3e-7 and
// 1.2e-7.
// Why: the same sums by fp32 FMAs were bound by the FMA pipe and by shared-memory reads (mLSTM, 7 ragged prompts of 7919 rows, 8 heads of
// 128 x 128: state 70, carry 68, output 135 us; here, one launch after the other, 26, 17 and 52 us.  Linear attention over fp32 rows,
// 4 x 2048: 62, 44, 104 us; here 32, 11, 63; with each launch begun while the one before runs, the chain takes 2 to 5 us less).
// Chunks of 128 rows are the matrix instructions' own height and halve the chunks' states.  What bounds it: the chain of an item --
// keys converted, scores, the state's part, values converted, their part -- beside a few hundred cycles for every conversion, copy and
// wait in it: tensor pipe 13 (state) to 28 % (output) active, issue slots 41 to 47 %, DRAM 15 to 33 %, waits on memory and at barriers
// first among the stalls (8 converting warps instead of 16, 16 columns of the output per store: 39, 12, 69 us).
#pragma once
#include <type_traits>

#include "chunk_scan.cuh"
#include "common.cuh"
#include "runtime.h"

namespace b200 {

constexpr int kCtRows = 128, kCtHalf = 64;
// one CTA per SM walks the items: 16 warps convert operands, 8 read tensor memory (and form the items' weights), one issues the
// products, one copies the chunks' first states, one finds the items
constexpr int kCtConvWarps = 16, kCtReadWarps = 8, kCtConv = kCtConvWarps * 32, kCtMma = kCtConvWarps + kCtReadWarps, kCtCopy = kCtMma + 1,
              kCtFind = kCtCopy + 1, kCtThreads = (kCtFind + 2) * 32;
constexpr int kCtCarryThreads = 256, kCtDepth = 8, kCtTable = 32;      // chunks in flight in the carry; chunks per table of factors

// ------------------------------------------------------------------------------------------- operands
// Two fp32 numbers -> the next bf16 term of each (packed) and what is left of them.
__device__ __forceinline__ uint32_t ct_term(float& a, float& b) {
  const uint32_t h = pack_bf16(a, b);
  const float2 r = unpack2(sub2(pack2(a, b), pack2(bf16_lo(h), bf16_hi(h))));
  a = r.x;
  b = r.y;
  return h;
}
// two bf16 numbers held as fp32, packed
__device__ __forceinline__ uint32_t ct_high(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
__device__ __forceinline__ void ct_st8(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ bool ct_finite(float x) { return fabsf(x) < 3.38e38f; }   // rounds to a finite bf16

// Operand tiles in shared memory: blocks of 64 rows x 64 columns, [64][128 bytes] with the 128-byte swizzle, a term's blocks behind one
// another.  Blocks one below the other are a panel of more rows, blocks side by side more panels; the same bytes serve as a K-major
// operand (rows x columns) and as an MN-major one (columns x rows).
//
// Two blocks on their way from global memory through a converting thread's registers: columns c .. c + 3 of rows r and r + 32
template <typename TA>
struct CtBlocks {
  static constexpr bool kExact = sizeof(TA) == 2;
  typedef typename std::conditional<kExact, uint2, float4>::type Raw;
  Raw raw[2][2];
  __device__ __forceinline__ static int column() { return ((int)threadIdx.x & 15) * 4; }
  __device__ __forceinline__ static int row() { return ((int)threadIdx.x >> 4) & 31; }
  // block 1 begins `next` numbers behind block 0; rows and columns that are not there are zeros
  __device__ __forceinline__ void load(const TA* src, int64_t ld, int64_t next, int rows0, int rows1, int cols0, int cols1) {
    const TA* at = src + (int64_t)row() * ld + column();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int left = column() < (u ? cols1 : cols0) ? (u ? rows1 : rows0) - row() : 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        raw[u][i] = Raw{};
        if (32 * i < left) raw[u][i] = *reinterpret_cast<const Raw*>(at + u * next + (int64_t)(32 * i) * ld);
      }
    }
  }
  __device__ __forceinline__ float4 value(int u, int i) const {
    if constexpr (kExact) return make_float4(bf16_lo(raw[u][i].x), bf16_hi(raw[u][i].x), bf16_lo(raw[u][i].y), bf16_hi(raw[u][i].y));
    else return raw[u][i];
  }
  // whether this thread's numbers are bf16 numbers: one term each
  __device__ __forceinline__ bool one_term() const {
    if constexpr (kExact) {
      return true;
    } else {
      uint32_t low = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 v = raw[i >> 1][i & 1];
        low |= __float_as_uint(v.x) | __float_as_uint(v.y) | __float_as_uint(v.z) | __float_as_uint(v.w);
      }
      return (low & 0xffffu) == 0;
    }
  }
  // where this thread's part of a block lies (row + 32 is 4 KB on, the next block 8 KB)
  __device__ __forceinline__ static uint32_t place() {
    const int r = row(), c = column();
    return (uint32_t)(r * 128 + (((c >> 3) ^ (r & 7)) << 4) + ((c >> 2) & 1) * 8);
  }
};
constexpr uint32_t kCtBlock = 8192;
__device__ __forceinline__ void ct_put(uint32_t at, uint32_t term_bytes, float4 v) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const uint32_t a = ct_term(v.x, v.y), b = ct_term(v.z, v.w);
    ct_st8(at + t * term_bytes, a, b);
  }
}
template <typename TA>
__device__ __forceinline__ void ct_store(const CtBlocks<TA>& b, int blocks, uint32_t base, uint32_t term_bytes, bool one_term = false) {
  const uint32_t at = base + CtBlocks<TA>::place();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (u >= blocks) break;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t to = at + u * kCtBlock + i * 4096;
      if constexpr (CtBlocks<TA>::kExact) ct_st8(to, b.raw[u][i].x, b.raw[u][i].y);
      else if (one_term) ct_st8(to, ct_high(b.raw[u][i].x, b.raw[u][i].y), ct_high(b.raw[u][i].z, b.raw[u][i].w));
      else ct_put(to, term_bytes, b.raw[u][i]);
    }
  }
}

// An infinite number (or one that rounds to one) has no three terms: every product with it is no number, where an fp32 FMA may give an
// infinite one.  What comes out of the products not finite is formed again by FMAs, in its place; that there is such is told by adding up
// zero times the results, which is zero for finite ones alone.  (With every value of 4 x 2048 rows
// infinite, 8 heads of 128 x 128: 51 ms; with every key no number, which ends a sum, 4 ms.)
struct CtFinite {
  f32x2 sum = 0ull;
  __device__ __forceinline__ void add(float a, float b) { sum = fma2(pack2(a, b), 0ull, sum); }
  __device__ __forceinline__ bool all() const {
    const float2 v = unpack2(sum);
    return v.x + v.y == 0.f;
  }
};
__device__ __forceinline__ bool ct_number(float x) { return fabsf(x) < INFINITY; }
// k . q; sum of w_s k_s v_s over rows, until it is no number
template <typename TA>
__device__ __noinline__ float ct_dot(const TA* q, const TA* k, int dk) {
  float acc = 0.f;
  for (int i = 0; i < dk; ++i) acc = fmaf((float)q[i], (float)k[i], acc);
  return acc;
}
template <typename TA>
__device__ __noinline__ float ct_rows_sum(const TA* k, int64_t ld, const TA* v, int64_t ld_v, const float* w, int rows) {
  float acc = 0.f;
  for (int s = 0; s < rows && acc == acc; ++s) acc = fmaf((float)k[s * ld] * w[s], (float)v[s * ld_v], acc);
  return acc;
}

// A sum that left the products is cut towards zero once per instruction; what that loses on average, sums of one sign and of both taken
// together, is added back (measured, with and without: mean deviation of outputs -1.0e-7 to -2.3e-7 -> +-8e-8, of states -4e-8 to -8e-8
// -> +-3e-8; their relative error to two thirds of that of fp32 FMAs, where rows of one sign stood at up to 1.9 times without).
__device__ __forceinline__ float ct_uncut(float x) { return fmaf(x, 5.0e-8f, x); }

// One pair of terms over KS steps of 16, or all pairs (i, j) of 1 <= i + j <= 2, smallest first: the low words of the descriptors
// and their steps in 16-byte units; A's terms in shared memory (A_TMEM: in tensor memory, a_step columns per step).  One thread.
template <bool A_TMEM, int KS>
__device__ __forceinline__ void ct_pair(uint32_t d, uint64_t a, uint32_t a_step, uint64_t b, uint32_t b_step, uint32_t idesc, uint32_t& acc) {
#pragma unroll
  for (int k = 0; k < KS; ++k) {
    if constexpr (A_TMEM) umma_bf16_ts(d, (uint32_t)a + k * a_step, b + k * b_step, idesc, acc);
    else umma_bf16(d, a + k * a_step, b + k * b_step, idesc, acc);
    acc = 1u;
  }
}
template <bool A_TMEM, int NA, int NB, int KS>
__device__ __forceinline__ void ct_small(uint32_t d, uint64_t a, uint32_t a_term, uint32_t a_step, uint64_t b, uint32_t b_term, uint32_t b_step,
                                         uint32_t idesc, uint32_t& acc) {
#pragma unroll 1
  for (int order = 2; order >= 1; --order)
#pragma unroll 1
    for (int i = order < NB ? 0 : order - NB + 1; i < NA && i <= order; ++i)
      ct_pair<A_TMEM, KS>(d, a + i * a_term, a_step, b + (order - i) * b_term, b_step, idesc, acc);
}
// bytes (a multiple of 16) of global memory -> shared memory
__device__ __forceinline__ void ct_copy(uint32_t to, const void* from, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(from), "r"(bytes),
               "r"(smem_u32(bar))
               : "memory");
}
constexpr uint32_t kCtAmn = 1u << 15, kCtBmn = 1u << 16;      // instruction descriptor: operand is MN-major

// ------------------------------------------------------------------------------------------- places
inline int64_t ct_max_chunks(int64_t rows, int64_t n_seqs) {
  const int64_t longs = rows / (kCsShort + 1);
  return rows / kCtRows + (longs < n_seqs ? longs : n_seqs);
}

// The items of a CTA that walks (chunk, head, value tile) triples `step` apart: the next one from `item` on that there is (items:
// none).  Whole warp.
struct CtItem {
  int item, chunk, h, v0;
  ChunkPlace at;
  int fresh;
};
template <int VT>
__device__ __forceinline__ CtItem ct_next(const ChunkScanArgs& a, int items, int item, int step) {
  const int tiles = (a.dv + VT - 1) / VT, per = a.H * tiles;
  CtItem r{items};
  for (; item < items; item += step) {
    int seq, local, before;
    cs_find<kCtRows>(a.cu_seq, a.n_seqs, a.short_rows, item / per, 0, seq, local, before);
    if (seq < 0) break;                               // the chunks that there are come first
    const int slot = a.state_slots[seq], first = a.cu_seq[seq], end = a.cu_seq[seq + 1], ctx = a.ctx_lens[seq];      // (one wait)
    if (slot < 0) continue;
    const int t0 = first + local * kCtRows;
    r.item = item;
    r.chunk = item / per;
    r.h = item % per / tiles;
    r.v0 = item % tiles * VT;
    r.at = {seq, t0, min(kCtRows, end - t0), slot, local};
    r.fresh = ctx == 0;
    break;
  }
  return r;
}
// `rows` rows of `bytes` on their way to L2, so that the loads that wait for one another further on wait for L2 alone.  Whole warp.
__device__ __forceinline__ void ct_prefetch(const void* at, int64_t pitch, int rows, int bytes) {
  const int lines = (bytes + 127) / 128;
  for (int i = threadIdx.x & 31; i < rows * lines; i += 32)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(at) + (i / lines) * pitch + (i % lines) * 128));
}

__device__ __forceinline__ void ct_named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
// whether it holds in all of them
__device__ __forceinline__ bool ct_named_all(int id, int threads, bool v) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %3, 0;\n\tbar.red.and.pred q, %1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
               : "=r"(r)
               : "r"(id), "r"(threads), "r"((uint32_t)v)
               : "memory");
  return r != 0;
}
// A warpgroup's share of the registers that the block was launched with (28 warps of 72): 16 converting warps of 64, 8 reading ones of 88,
// 4 others of 72.
template <int N>
__device__ __forceinline__ void ct_more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void ct_fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int kCtConvRegs = 64, kCtReadRegs = 88;
constexpr int kCtBarConv = 1, kCtBarRead = 2, kCtBarTeam = 3, kCtBarTerms = 4;      // named barriers

// The first four reading warps form an item's weights, a row each: inclusive sums and running maxima over the rows (`parts`: four
// numbers in shared memory).  What is no number in a row stays out of the rows before.
constexpr int kCtTeam = 128;
__device__ __forceinline__ int ct_team_row() { return (int)threadIdx.x & (kCtTeam - 1); }
template <bool MAX>
__device__ __forceinline__ double ct_team_scan(double v, double* parts) {
  const int lane = threadIdx.x & 31, w = ct_team_row() >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = MAX ? fmax(v, u) : v + u;
  }
  if (lane == 31) parts[w] = v;
  ct_named_barrier(kCtBarTeam, kCtTeam);
  double before = parts[0];
#pragma unroll
  for (int i = 1; i < 3; ++i)
    if (i < w) before = MAX ? fmax(before, parts[i]) : before + parts[i];
  return w == 0 ? v : MAX ? fmax(before, v) : before + v;
}

// An exponent's two parts: what is left of a double after rounding to fp32 is kept beside it, so that a sum or difference of two
// is as exact as the fp32 it ends in.
struct CtExp {
  float h, l;
};
__device__ __forceinline__ CtExp ct_exp(double v) {
  const float h = (float)v;
  return {h, (float)(v - (double)h)};
}

// The launches of a chain begin while the one before runs, on the SMs that it leaves free: set-up, places and, without a normaliser, the
// first item's scores are behind them when it ends.  A grid that began early has missed the launch-time L1 invalidation: what the
// chain's kernels write is read past L1.  Every CTA of the second and third launch waits, so that each launch's end is the end of
// all before it.  Small steps are what it is for, whose code comes from DRAM three times over (L2 cold; launched one after the other
// -> so; by FMAs over 64 rows): linear attention of 128 rows, 4 heads, 45 -> 30 (38) us, of 1024 rows, 8 heads, 46 -> 38 (44); mLSTM of 200
// fp32 rows 51 -> 44 (51).  With a normaliser nothing can be formed before the carry's rows are there, and a step of more than an
// item per SM releases the output at the carry's end (its CTAs, apart from the start, take longer for 4 x 2048 fp32 rows of 32 heads:
// 476 -> 487; released at the end 479).
__device__ __forceinline__ void ct_release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void ct_wait_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The items of a CTA, found ahead of their use (three loads deep).
constexpr int kCtAhead = 4;
constexpr int kCtUsers = kCtConvWarps + kCtReadWarps + 1;      // warps that release an item (the copying one is done before the products are)
struct CtQueue {
  CtItem item[kCtAhead];
  uint64_t full[kCtAhead], free[kCtAhead];
};
__device__ __forceinline__ void ct_queue_init(CtQueue& q) {
  for (int i = 0; i < kCtAhead; ++i) {
    mbar_init(&q.full[i], 1);
    mbar_init(&q.free[i], kCtUsers);
  }
}
__device__ __forceinline__ CtItem ct_item(CtQueue& q, int it) {
  mbar_wait_guarded(&q.full[it % kCtAhead], (it / kCtAhead) & 1);
  return q.item[it % kCtAhead];
}
// a warp is done (lane 0 tells)
__device__ __forceinline__ void ct_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// what this warp stored in shared memory is there for the products
__device__ __forceinline__ void ct_stored(uint64_t* bar) {
  fence_proxy_async();
  ct_arrive(bar);
}
__device__ __forceinline__ void ct_wait(uint64_t* bar, int it) {
  mbar_wait_guarded(bar, it & 1);
  tc_fence_after();
}
// barriers are initialised by the first thread before this; ends with the whole block knowing the address
__device__ __forceinline__ uint32_t ct_tmem(uint32_t* at, uint32_t columns) {
  if (threadIdx.x >> 5 == kCtMma) {
    tmem_alloc(at, columns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *at;
}
__device__ __forceinline__ void ct_end(uint32_t tmem, uint32_t columns) {
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x >> 5 == kCtMma) {
    tc_fence_after();
    tmem_dealloc(tmem, columns);
  }
}

// ------------------------------------------------------------------------------------------- shared memory
template <int DK, int VT, typename TA>
struct CtSmem {
  static constexpr int kIn = sizeof(TA) == 2 ? 1 : 3;                        // terms of what the rows hold
  // state: two halves of 64 rows of keys and of weighted values.  With 64 keys the instruction's other 64 rows read on into what
  // follows and go nowhere.
  static constexpr int kStateK = kIn * DK * 128, kStateV = 3 * VT * 128, kStateHalf = kStateK + kStateV;
  static constexpr int kSums = 32 * DK * 4;
  static constexpr int kState = 2 * kStateHalf + kSums + 1024;
  // output: panels of 64 columns of Q and K, of S, halves of 64 rows of V.  Three terms: two regions of two stages that change roles
  // with every item, Q's and then V's, K's and then S's
  static constexpr int kPanels = DK / 64, kPanel = kCtRows * 128, kVHalf = VT * 128;
  static constexpr bool kApart = kIn == 1;            // one term: room for Q, K, V and S apart
  static constexpr int kStage = kApart ? kPanel : kIn * kPanel > 3 * VT * 128 ? kIn * kPanel : 3 * VT * 128;
  static constexpr int kStatePanel = kApart ? 3 * VT * 128 : kStage;
  static constexpr int kOperands = kApart ? 6 * kStage + 2 * kStatePanel : 4 * kStage;
  static constexpr int kTurn = kCtReadWarps * 2048, kOutput = kOperands + kTurn + 1024;
  // where an item's panels of Q, K and S and halves of V lie
  __device__ __forceinline__ static uint32_t q(int it, int i) { return (kApart ? 0 : (it & 1) * 2 * kStage) + i * kStage; }
  __device__ __forceinline__ static uint32_t k(int it, int i) { return (kApart ? 2 * kStage : ((it & 1) ^ 1) * 2 * kStage) + i * kStage; }
  __device__ __forceinline__ static uint32_t s(int it, int i) { return kApart ? 6 * kStage + i * kStatePanel : k(it, i); }
  __device__ __forceinline__ static uint32_t v(int it, int i) { return kApart ? 4 * kStage + i * kStage : q(it, i); }
};
__device__ __forceinline__ uint8_t* ct_align(uint8_t* p) {
  return p + (-smem_u32(p) & 1023u);                  // (by an offset: the compiler still sees shared memory)
}

// ------------------------------------------------------------------------------------------- workspace
// The state of a chunk and head in the workspace, dk dv 6 bytes: three planes [dk / 64][dv][128 bytes] of bf16 terms, each row of 128
// bytes swizzled by its number as an operand panel is, so that a panel is one copy.  Before the carry the first two planes hold
// the chunk's own C in fp32: what will be term 0 and term 1 of eight neighbouring keys, 16 bytes each, are four keys of C each.
__device__ __forceinline__ size_t ct_plane(int dk, int dv) { return (size_t)dk * dv * 2; }
// byte in a plane where eight keys from 8 k8 on of value v lie
__device__ __forceinline__ size_t ct_in_plane(int v, int k8, int dv) {
  return (size_t)((k8 >> 3) * dv + v) * 128 + (size_t)(((k8 & 7) ^ (v & 7)) << 4);
}

// ------------------------------------------------------------------------------------------- state
// Two accumulators per item -- the small pairs of terms and the second half's large ones; the first half's large ones -- and two
// sets of them: an item's products run while the item before leaves tensor memory.
template <int DK, int VT, typename TA, typename Form>
__global__ void __launch_bounds__(kCtThreads, 1)
ct_state_kernel(const ChunkScanArgs a, const typename Form::Params p, int items) {
  extern __shared__ uint8_t ct_raw[];
  __shared__ CtQueue queue;
  __shared__ typename Form::Scratch scratch[2];
  __shared__ uint64_t weight_full[2], half_full[2], half_done[2], sum_full[2], sum_free[2];
  __shared__ uint32_t tmem_at, one_term[2];
  typedef CtSmem<DK, VT, TA> L;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t smem = smem_u32(ct_align(ct_raw));
  const TA* x = reinterpret_cast<const TA*>(a.x);
  ct_release_next();
  if (tid == 0) {
    ct_queue_init(queue);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&weight_full[i], kCtTeam / 32);
      mbar_init(&half_full[i], kCtConvWarps);
      mbar_init(&half_done[i], 1);
      mbar_init(&sum_full[i], 1);
      mbar_init(&sum_free[i], kCtReadWarps);
    }
    fence_mbar_init();
  }
  const uint32_t tmem = ct_tmem(&tmem_at, 4 * VT);
  if (warp < kCtConvWarps) {
    ct_fewer_registers<kCtConvRegs>();
    float* sums = reinterpret_cast<float*>(ct_align(ct_raw) + 2 * L::kStateHalf);
    typedef CtBlocks<TA> Blocks;
    Blocks kt, vt;
    auto load_k = [&](const CtItem& w, int e) {
      const int n = w.at.rows - kCtHalf * e;
      kt.load(x + (int64_t)(w.at.first + kCtHalf * e) * a.ld + a.k_col + w.h * DK, a.ld, 64, n, DK == 128 ? n : 0, 64, 64);
    };
    CtItem now = ct_item(queue, 0);
    if (now.item < items) load_k(now, 0);
    for (int it = 0; now.item < items; ++it) {
      const typename Form::Scratch& sc = scratch[it & 1];
      float4 ksum[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
      CtItem then{items};
#pragma unroll 1
      for (int e = 0; e < 2; ++e) {
        const uint32_t ks = smem + e * L::kStateHalf, vs = ks + L::kStateK;
        const int n = now.at.rows - kCtHalf * e, width = a.dv - now.v0;
        vt.load(x + (int64_t)(now.at.first + kCtHalf * e) * a.ld + a.v_col + now.h * a.dv + now.v0, a.ld, 64, n, VT == 128 ? n : 0, width,
                width - 64);
        if (it) ct_wait(&half_done[e], it - 1);       // the item before has used this half
        if (e == 0) mbar_wait_guarded(&weight_full[it & 1], (it >> 1) & 1);
        // values of one term leave the weights to the keys: half the products
        const bool one = L::kIn == 3 && ct_named_all(kCtBarTerms, kCtConv, vt.one_term());
        if (L::kIn == 1) {
          ct_store(kt, DK / 64, ks, DK * 128);
        } else {
          if (tid == 0) one_term[e] = one;
          const uint32_t at = ks + Blocks::place();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float w = one ? sc.w[kCtHalf * e + kt.row() + 32 * i] : 1.f;
#pragma unroll
            for (int u = 0; u < DK / 64; ++u) {
              float4 k = kt.value(u, i);
              k = make_float4(k.x * w, k.y * w, k.z * w, k.w * w);
              ct_put(at + u * kCtBlock + i * 4096, DK * 128, k);
            }
          }
        }
        if constexpr (Form::kNorm) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float w = sc.w[kCtHalf * e + kt.row() + 32 * i];
#pragma unroll
            for (int u = 0; u < DK / 64; ++u) {
              const float4 k = kt.value(u, i);
              ksum[u] = make_float4(fmaf(w, k.x, ksum[u].x), fmaf(w, k.y, ksum[u].y), fmaf(w, k.z, ksum[u].z), fmaf(w, k.w, ksum[u].w));
            }
          }
        }
        if (e) then = ct_item(queue, it + 1);
        if (!e || then.item < items) load_k(e ? then : now, e ^ 1);
        if (one) {
          ct_store(vt, VT / 64, vs, VT * 128, true);
        } else {
          const uint32_t at = vs + Blocks::place();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float w = sc.w[kCtHalf * e + vt.row() + 32 * i];
#pragma unroll
            for (int u = 0; u < VT / 64; ++u) {
              float4 v = vt.value(u, i);
              v = make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
              ct_put(at + u * kCtBlock + i * 4096, VT * 128, v);
            }
          }
        }
        ct_stored(&half_full[e]);
      }
      if (now.v0 == 0) {
        if constexpr (Form::kNorm) {                  // the keys' own sum: a thread's rows, then the row groups
          float* row = a.ws_row + ((size_t)now.chunk * a.H + now.h) * a.ws_row_width;
#pragma unroll
          for (int u = 0; u < DK / 64; ++u) *reinterpret_cast<float4*>(sums + kt.row() * DK + 64 * u + kt.column()) = ksum[u];
          ct_named_barrier(kCtBarConv, kCtConv);
          if (tid < DK) {
            double n = 0.0;                           // (fp32 sums of 32 groups are further off than the one-pass form's)
#pragma unroll 8
            for (int g = 0; g < 32; ++g) n += (double)sums[g * DK + tid];
            row[tid] = (float)n;
          }
          ct_named_barrier(kCtBarConv, kCtConv);
        }
      }
      ct_arrive(&queue.free[it % kCtAhead]);
      now = then;
    }
  } else if (warp < kCtConvWarps + kCtReadWarps) {
    ct_more_registers<kCtReadRegs>();
    // lane = key, columns = values: a warp stores two 64-byte pieces of a row
    const int w = warp - kCtConvWarps, k = (w & 3) * 32 + lane;
    const size_t plane = ct_plane(DK, a.dv);
    // an item ahead: the last item of its buffer has used its weights once its sums are complete (they are all that the converting
    // warps read of it; the chunk's row of factors goes to the workspace from here)
    auto weigh = [&](const CtItem& next, int it) {
      if (w >= kCtTeam / 32 || next.item >= items) return;
      float* row = a.ws_row + ((size_t)next.chunk * a.H + next.h) * a.ws_row_width + DK;
      Form::state_weights(p, a, scratch[it & 1], next.h, next.at, next.fresh, next.v0 == 0 ? row : nullptr);
      ct_arrive(&weight_full[it & 1]);
    };
    CtItem now = ct_item(queue, 0);
    weigh(now, 0);
    for (int it = 0; now.item < items; ++it) {
      const int buf = it & 1;
      const CtItem then = ct_item(queue, it + 1);
      ct_named_barrier(kCtBarRead, kCtReadWarps * 32);                // the item before, whose weights these replace, is behind every warp
      weigh(then, it + 1);
      mbar_wait_guarded(&sum_full[buf], (it >> 1) & 1);
      tc_fence_after();
      constexpr int PER = VT / 2;
      const int v0 = now.v0 + (w >> 2) * PER;
      uint8_t* C = reinterpret_cast<uint8_t*>(a.ws) + ((size_t)now.chunk * a.H + now.h) * 3 * plane;
      const uint32_t t0 = tmem + ((uint32_t)((w & 3) * 32) << 16) + buf * 2 * VT + (w >> 2) * PER;
      if ((w & 3) * 32 < DK) {
#pragma unroll 1
        for (int c0 = 0; c0 < PER; c0 += 16) {
          uint32_t r[16], s[16];
          tmem_ld_32x16(t0 + c0, r);
          tmem_ld_32x16(t0 + VT + c0, s);
          tmem_ld_wait();
          uint8_t* out = C + ((k >> 2) & 1) * plane + (size_t)((k >> 6) * a.dv + v0 + c0) * 128 + (k & 3) * 4;
          const int k8 = (k >> 3) & 7;                // (v0 + c0 is a multiple of 8)
          CtFinite finite;
#pragma unroll
          for (int c = 0; c < 16; ++c) r[c] = __float_as_uint(ct_uncut(__uint_as_float(r[c]) + __uint_as_float(s[c])));
#pragma unroll
          for (int c = 0; c < 16; c += 2) finite.add(__uint_as_float(r[c]), __uint_as_float(r[c + 1]));
#pragma unroll
          for (int c = 0; c < 16; ++c)
            if (v0 + c0 + c < a.dv) *reinterpret_cast<uint32_t*>(out + c * 128 + ((k8 ^ (c & 7)) << 4)) = r[c];
          if (!finite.all()) {
#pragma unroll 1
            for (int c = 0; c < 16 && v0 + c0 + c < a.dv; ++c) {
              float* C_kv = reinterpret_cast<float*>(out + c * 128 + ((k8 ^ (c & 7)) << 4));
              if (!ct_number(*C_kv))
                *C_kv = ct_rows_sum(x + (int64_t)now.at.first * a.ld + a.k_col + now.h * DK + k, a.ld,
                                    x + (int64_t)now.at.first * a.ld + a.v_col + now.h * a.dv + v0 + c0 + c, a.ld, scratch[buf].w, now.at.rows);
            }
          }
        }
      }
      tc_fence_before();
      ct_arrive(&sum_free[buf]);
      ct_arrive(&queue.free[it % kCtAhead]);
      now = then;
    }
  } else if (warp == kCtMma) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, VT) | kCtAmn | kCtBmn;
      for (int it = 0;; ++it) {
        const CtItem now = ct_item(queue, it);
        if (now.item >= items) break;
        const int buf = it & 1;
        if (it >= 2) mbar_wait_guarded(&sum_free[buf], ((it >> 1) - 1) & 1);
        const uint32_t d0 = tmem + buf * 2 * VT, d1 = d0 + VT;
        uint32_t acc0 = 0;
        for (int e = 0; e < 2; ++e) {
          ct_wait(&half_full[e], it);
          if (e == 0 || now.at.rows > kCtHalf) {
            const uint64_t da = umma_desc_mn_sw128(smem + e * L::kStateHalf, kCtHalf * 128, 1024),
                           db = umma_desc_mn_sw128(smem + e * L::kStateHalf + L::kStateK, kCtHalf * 128, 1024);
            if (L::kIn == 3 && one_term[e]) ct_small<false, L::kIn, 1, 4>(d0, da, DK * 8, 128, db, VT * 8, 128, idesc, acc0);
            else ct_small<false, L::kIn, 3, 4>(d0, da, DK * 8, 128, db, VT * 8, 128, idesc, acc0);
            uint32_t acc1 = e;
            ct_pair<false, 4>(e ? d0 : d1, da, 128, db, 128, idesc, acc1);
          }
          umma_commit(&half_done[e]);
        }
        umma_commit(&sum_full[buf]);
        mbar_arrive(&queue.free[it % kCtAhead]);
      }
    }
    __syncwarp();
  } else if (warp == kCtFind) {
    for (int it = 0, item = (int)blockIdx.x;; ++it) {
      const CtItem next = ct_next<VT>(a, items, item, (int)gridDim.x);
      const int buf = it % kCtAhead;
      if (it >= kCtAhead) mbar_wait_guarded(&queue.free[buf], (it / kCtAhead - 1) & 1);
      if (lane == 0) queue.item[buf] = next;
      ct_arrive(&queue.full[buf]);
      if (next.item >= items) break;
      const int w = min(VT, a.dv - next.v0) * (int)sizeof(TA);
      ct_prefetch(x + (int64_t)next.at.first * a.ld + a.k_col + next.h * DK, a.ld * sizeof(TA), next.at.rows, DK * (int)sizeof(TA));
      ct_prefetch(x + (int64_t)next.at.first * a.ld + a.v_col + next.h * a.dv + next.v0, a.ld * sizeof(TA), next.at.rows, w);
      item = next.item + (int)gridDim.x;
    }
    ct_wait_before();                                 // (the short sequences' one-pass kernel, beside which this one runs)
  }
  ct_end(tmem, 4 * VT);
}

// ------------------------------------------------------------------------------------------- carry
template <int DK, typename Form>
__global__ void __launch_bounds__(kCtCarryThreads)
ct_carry_kernel(const ChunkScanArgs a, const typename Form::Params p, bool early) {
  __shared__ int base;
  __shared__ float2 table[kCtTable];                  // a chunk's factors: of the state so far, of the chunk's own part
  const int s = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int t0 = a.cu_seq[s], t1 = a.cu_seq[s + 1], nc = cs_chunks<kCtRows>(t1 - t0, a.short_rows), slot = a.state_slots[s];
  if (early) ct_release_next();
  if (nc == 0 || slot < 0) {
    ct_wait_before();
    return;
  }
  if (tid < 32) {
    int q, l, before;
    cs_find<kCtRows>(a.cu_seq, a.n_seqs, a.short_rows, -1, s, q, l, before);
    if (tid == 0) base = before;
  }
  __syncthreads();
  const int i = (blockIdx.x * kCtCarryThreads + tid) * 8;           // eight keys of a value column
  const bool live = i < a.dv * DK, fresh = a.ctx_lens[s] == 0;
  float4* Sp = reinterpret_cast<float4*>(a.S + ((size_t)slot * a.H + h) * a.dv * DK + i);
  float4 S[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  if (live && !fresh) { S[0] = Sp[0]; S[1] = Sp[1]; }
  const size_t plane = ct_plane(DK, a.dv), step = (size_t)a.H * 3 * plane;
  uint8_t* C = reinterpret_cast<uint8_t*>(a.ws) + ((size_t)base * a.H + h) * 3 * plane + ct_in_plane(i / DK, i % DK / 8, a.dv);
  ct_wait_before();
  typename Form::Carry carry(p, a, h, base);
  for (int c0 = 0; c0 < nc; c0 += kCtDepth) {
    float4 in[kCtDepth][2];
#pragma unroll
    for (int u = 0; u < kCtDepth; ++u)
      if (live && c0 + u < nc) {
        const uint8_t* from = C + (size_t)(c0 + u) * step;
        in[u][0] = __ldcg(reinterpret_cast<const float4*>(from));
        in[u][1] = __ldcg(reinterpret_cast<const float4*>(from + plane));
      }
    if (c0 % kCtTable == 0) {
      __syncthreads();
      if (tid < 32) carry.factors(c0, nc, t1 - t0, table);
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < kCtDepth; ++u) {
      if (c0 + u >= nc) break;
      const float2 f = table[(c0 + u) % kCtTable];
      if (live) {
        float4 x = S[0], y = S[1];
        uint8_t* to = C + (size_t)(c0 + u) * step;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          uint4 r;
          r.x = ct_term(x.x, x.y); r.y = ct_term(x.z, x.w); r.z = ct_term(y.x, y.y); r.w = ct_term(y.z, y.w);
          *reinterpret_cast<uint4*>(to + e * plane) = r;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
          S[e] = make_float4(fmaf(f.x, S[e].x, f.y * in[u][e].x), fmaf(f.x, S[e].y, f.y * in[u][e].y), fmaf(f.x, S[e].z, f.y * in[u][e].z),
                             fmaf(f.x, S[e].w, f.y * in[u][e].w));
      }
    }
  }
  if (!early) ct_release_next();
  if (live) { Sp[0] = S[0]; Sp[1] = S[1]; }
  if (blockIdx.x == 0) Form::template carry_row<DK>(p, a, h, base, nc, fresh, slot);
}

// ------------------------------------------------------------------------------------------- output
// Values that are no finite bf16 number are left out of the products (zero times one would reach the rows before) and join the rows
// from their own on one by one.
//
// q . a value's row of the state's terms in the workspace, until it is no number
template <typename TA>
__device__ __noinline__ float ct_state_dot(const TA* q, const uint8_t* S, size_t plane, int v, int dk, int dv) {
  float acc = 0.f;
  for (int k = 0; k < dk && acc == acc; ++k) {
    const unsigned short* at = reinterpret_cast<const unsigned short*>(S + ct_in_plane(v, k >> 3, dv)) + (k & 7);
    float x = __uint_as_float((uint32_t)__ldcg(at) << 16);
    if (ct_number(x))                                 // (behind an infinite first term stand none)
      x += __uint_as_float((uint32_t)__ldcg(at + plane / 2) << 16) + __uint_as_float((uint32_t)__ldcg(at + plane) << 16);
    acc = fmaf((float)q[k], x, acc);
  }
  return acc;
}

// Products of an item in their order: scores (the small pairs of terms and the first panel's large ones into one accumulator, the
// second panel's into the other), Q S_start^T, and the weighted scores times V.  While the state's part is formed, the weights are;
// while the values' part is, the next item's queries are converted.
template <int DK, int VT, typename TA, typename Form>
__global__ void __launch_bounds__(kCtThreads, 1)
ct_output_kernel(const ChunkScanArgs a, const typename Form::Params p, int items) {
  extern __shared__ uint8_t ct_raw[];
  __shared__ CtQueue queue;
  __shared__ typename Form::Scratch scratch[2];
  __shared__ uint64_t key_full[2], state_full[2], value_full[2], score_done, state_done, value_done, weight_full, out_free;
  __shared__ uint32_t tmem_at, special[kCtAhead][4], one_term[2];
  __shared__ float den_of[2][Form::kNorm ? 3 * kCtRows : 1];
  typedef CtSmem<DK, VT, TA> L;
  constexpr int NP = L::kPanels, OC = VT / 2;         // panels of keys; a reading thread's value columns
  constexpr bool kTwo = NP == 2 || L::kIn == 3;       // the scores have a second accumulator
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TA* x = reinterpret_cast<const TA*>(a.x);
  const uint32_t smem = smem_u32(ct_align(ct_raw));
  if (tid == 0) {
    ct_queue_init(queue);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&key_full[i], kCtConvWarps);
      mbar_init(&state_full[i], 1);
      mbar_init(&value_full[i], kCtConvWarps);
    }
    mbar_init(&score_done, 1);
    mbar_init(&state_done, 1);
    mbar_init(&value_done, 1);
    mbar_init(&weight_full, kCtReadWarps);
    mbar_init(&out_free, kCtReadWarps);
    fence_mbar_init();
  }
  const uint32_t t_s = ct_tmem(&tmem_at, 512), t_o = t_s + 256;      // two accumulators of scores, later the weights' terms; the state's part, the values'
  auto from_state = [](const CtItem& w) { return w.at.local > 0 || !w.fresh; };
  if (warp < kCtConvWarps) {
    ct_fewer_registers<kCtConvRegs>();
    // an item's tiles in their order: NP panels of queries, NP of keys, two halves of values; one is on its way while another is stored
    typedef CtBlocks<TA> Blocks;
    constexpr int TILES = 2 * NP + 2;
    Blocks tiles[2];
    auto load = [&](Blocks& b, const CtItem& w, int i) {
      if (i < 2 * NP) {
        const int col = (i < NP ? a.q_col : a.k_col) + w.h * DK + 64 * (i % NP);
        b.load(x + (int64_t)w.at.first * a.ld + col, a.ld, 64 * a.ld, w.at.rows, w.at.rows - 64, 64, 64);
      } else {
        const int n = w.at.rows - kCtHalf * (i - 2 * NP), width = a.dv - w.v0;
        b.load(x + (int64_t)(w.at.first + kCtHalf * (i - 2 * NP)) * a.ld + a.v_col + w.h * a.dv + w.v0, a.ld, 64, n, VT == 128 ? n : 0,
               width, width - 64);
      }
    };
    CtItem now = ct_item(queue, 0);
    if (now.item < items) load(tiles[0], now, 0);
    if constexpr (Form::kNorm) ct_wait_before();
    for (int it = 0; now.item < items; ++it) {
      CtItem then{items};
      float old[4];                                   // kNorm: n_start . q of a thread's rows
#pragma unroll 1
      for (int i0 = 0; i0 < TILES; i0 += 2) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int i = i0 + b;
          Blocks& tile = tiles[b];
          if (i + 1 == TILES) then = ct_item(queue, it + 1);
          if (i + 1 < TILES || then.item < items) load(tiles[b ^ 1], i + 1 < TILES ? now : then, i + 1 < TILES ? i + 1 : 0);
          if (i < 2 * NP) {
            // (three terms: the queries take the place of the state in the item before, whose part is complete; the keys that of its
            // values)
            if (L::kApart && i == 0 && it) ct_wait(&state_done, it - 1);
            if (i == NP && it) ct_wait(L::kApart ? &score_done : &value_done, it - 1);
            ct_store(tile, 2, smem + (i < NP ? L::q(it, i) : L::k(it, i - NP)), L::kPanel);
            if (Form::kNorm && i < NP) {
              const bool start = from_state(now);
              float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
              if (start)
                n = __ldcg(reinterpret_cast<const float4*>(a.ws_row + ((size_t)now.chunk * a.H + now.h) * a.ws_row_width + 64 * i + tile.column()));
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                const float4 q = tile.value(r >> 1, r & 1);
                old[r] = start ? fmaf(q.x, n.x, fmaf(q.y, n.y, fmaf(q.z, n.z, fmaf(q.w, n.w, i ? old[r] : 0.f)))) : 0.f;
              }
              if (i == NP - 1) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
#pragma unroll
                  for (int o = 8; o > 0; o >>= 1) old[r] += __shfl_xor_sync(0xffffffffu, old[r], o);
                  if ((tid & 15) == 0) den_of[it & 1][2 * kCtRows + 64 * (r >> 1) + 32 * (r & 1) + tile.row()] = old[r];
                }
              }
            }
            if (i >= NP) ct_stored(&key_full[i - NP]);
          } else {
            const int e = i - 2 * NP;
            // values that are no finite bf16 number are left out (zero times one would reach the rows before) and noted
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const float4 v = tile.value(r >> 1, r & 1);
              if (!(ct_finite(v.x) && ct_finite(v.y) && ct_finite(v.z) && ct_finite(v.w))) {
                const int at = kCtHalf * e + tile.row() + 32 * (r & 1);
                atomicOr(&special[it % kCtAhead][at >> 5], 1u << (at & 31));
                const float4 f = make_float4(ct_finite(v.x) ? v.x : 0.f, ct_finite(v.y) ? v.y : 0.f, ct_finite(v.z) ? v.z : 0.f,
                                             ct_finite(v.w) ? v.w : 0.f);
                if constexpr (Blocks::kExact) tile.raw[r >> 1][r & 1] = make_uint2(pack_bf16(f.x, f.y), pack_bf16(f.z, f.w));
                else tile.raw[r >> 1][r & 1] = f;
              }
            }
            if (!L::kApart && e == 0) ct_wait(&state_done, it);        // the queries are used
            if (L::kApart && e == 0 && it) ct_wait(&value_done, it - 1);
            const bool one = L::kIn == 1 || ct_named_all(kCtBarTerms, kCtConv, tile.one_term());
            if (tid == 0) one_term[e] = one;
            if (e == 0 || now.at.rows > kCtHalf) ct_store(tile, VT / 64, smem + L::v(it, e), L::kVHalf, one);
            ct_stored(&value_full[e]);
          }
        }
      }
      ct_arrive(&queue.free[it % kCtAhead]);
      now = then;
    }
  } else if (warp < kCtConvWarps + kCtReadWarps) {
    ct_more_registers<kCtReadRegs>();
    const int w0 = warp - kCtConvWarps, t = (w0 & 3) * 32 + lane, part = w0 >> 2;      // a thread's row and half of the columns
    const uint32_t lane_off = (uint32_t)((w0 & 3) * 32) << 16;
    const float q_scale = Form::q_scale(p);
    float* turn = reinterpret_cast<float*>(ct_align(ct_raw) + L::kOperands + w0 * 2048);   // 32 columns of 16 rows on their way to whole lines
    // an item ahead, while the values' part of the one before is formed
    auto weigh = [&](const CtItem& next, int it) {
      if (w0 < kCtTeam / 32 && next.item < items) Form::output_weights(p, a, scratch[it & 1], next.h, next.at, next.chunk);
    };
    CtItem now = ct_item(queue, 0);
    if constexpr (Form::kNorm) ct_wait_before();
    weigh(now, 0);
    for (int it = 0; now.item < items; ++it) {
      const typename Form::Scratch& sc = scratch[it & 1];
      const int n = now.at.rows, h = now.h;
      float* den = den_of[it & 1];
      ct_named_barrier(kCtBarRead, kCtReadWarps * 32);                // the weights are there, the item before is behind every warp
      const typename Form::Row row = Form::row(p, sc, t);
      ct_wait(&score_done, it);
      // sixteen scores at a time become three terms of eight columns, in columns of their own that have been read
      float own = 0.f;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const int s0 = 64 * part + 16 * c;
        const uint32_t at = t_s + lane_off + s0;
        uint32_t r[16];
        if (s0 <= (w0 & 3) * 32 + 31) {               // (whole warp) some of them are seen
          uint32_t r1[16];
          tmem_ld_32x16(at, r);
          if constexpr (kTwo) tmem_ld_32x16(at + 128, r1);
          float d[16];
          Form::weights(p, sc, row, t, s0, s0 + 15 < (w0 & 3) * 32, d);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float z = kTwo ? __uint_as_float(r[e]) + __uint_as_float(r1[e]) : __uint_as_float(r[e]);
            if constexpr (!Form::kNorm) z = ct_uncut(z);        // (with a normaliser it divides out)
            const float w = (s0 + e <= t && t < n) ? d[e] * (z * q_scale) : 0.f;
            if (Form::kNorm) own += w;
            r[e] = __float_as_uint(w);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) r[e] = 0;
        }
        uint32_t term[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float x0 = __uint_as_float(r[2 * e]), x1 = __uint_as_float(r[2 * e + 1]);
#pragma unroll
          for (int i = 0; i < 3; ++i) term[i][e] = ct_term(x0, x1);
        }
        tmem_st_32x8(at, term[0]);
        tmem_st_32x8(at + 8, term[1]);
        tmem_st_32x8(at + 128, term[2]);
      }
      if constexpr (Form::kNorm) {
        if (!ct_number(own) && t < n) {               // an infinite key or query: scores by FMAs
          const TA* qk = x + (size_t)now.at.first * a.ld + h * DK;
          own = 0.f;
#pragma unroll 1
          for (int s = 64 * part; s < min(64 * part + 64, t + 1) && own == own; ++s)
            own += Form::D(p, sc, row, t, s) * (ct_dot(qk + (size_t)t * a.ld + a.q_col, qk + (size_t)s * a.ld + a.k_col, DK) * q_scale);
        }
        den[part * kCtRows + t] = own;
      }
      tmem_st_wait();
      tc_fence_before();
      // (before the products of this item can end, behind which the next item's values arrive: what was noted about these is seen)
      mbar_wait_guarded(&value_full[0], it & 1);
      mbar_wait_guarded(&value_full[1], it & 1);
      ct_arrive(&weight_full);
      const CtItem then = ct_item(queue, it + 1);
      weigh(then, it + 1);
      if constexpr (Form::kNorm) ct_named_barrier(kCtBarRead, kCtReadWarps * 32);      // both halves' sums
      const uint32_t* sp = special[it % kCtAhead];
      const bool odd = (sp[0] | sp[1] | sp[2] | sp[3]) != 0, live = t < n, start = from_state(now);
      const float f = start ? Form::aq(sc, t) * q_scale : 0.f;
      const typename Form::Finish finish(p, a, sc, h, t, den);
      const TA* mine = x + (size_t)(now.at.first + (live ? t : 0)) * a.ld;
      ct_wait(&value_done, it);
#pragma unroll 1
      for (int c0 = 0; c0 < OC; c0 += 32) {
        const int v = now.v0 + part * OC + c0;
        float o[32];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          uint32_t r[16], r1[16];
          tmem_ld_32x16(t_o + VT + lane_off + part * OC + c0 + 16 * b, r);
          tmem_ld_32x16(t_o + lane_off + part * OC + c0 + 16 * b, r1);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) o[16 * b + e] = ct_uncut(start ? fmaf(__uint_as_float(r1[e]), f, __uint_as_float(r[e])) : __uint_as_float(r[e]));
        }
        CtFinite finite;
#pragma unroll
        for (int e = 0; e < 32; e += 2) finite.add(o[e], o[e + 1]);
        const bool bad = live && !finite.all();
        if (odd && live) {
          const int g = h * DK;
#pragma unroll 1
          for (int s = 0; s <= t; ++s) {
            if (!((sp[s >> 5] >> (s & 31)) & 1)) continue;
            const TA* vr = x + (size_t)(now.at.first + s) * a.ld + a.v_col + h * a.dv + v;
            const float ps = Form::D(p, sc, row, t, s) *
                             (ct_dot(mine + a.q_col + g, x + (size_t)(now.at.first + s) * a.ld + a.k_col + g, DK) * q_scale);
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (v + e < a.dv && !ct_finite((float)vr[e])) o[e] = fmaf(ps, (float)vr[e], o[e]);
          }
        }
        if (live) finish.apply(o);
        // sixteen rows at a time: eight lanes store a line of a row
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          __syncwarp();
          if (lane >> 4 == b)
#pragma unroll
            for (int e = 0; e < 8; ++e)
              *reinterpret_cast<float4*>(turn + (lane & 15) * 32 + ((e ^ lane) & 7) * 4) = make_float4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
          __syncwarp();
          const int col = v + 4 * (lane & 7);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r_ = 4 * e + (lane >> 3), row_ = (w0 & 3) * 32 + 16 * b + r_;
            if (row_ < n && col < a.dv)
              *reinterpret_cast<float4*>(a.o + (size_t)(now.at.first + row_) * a.H * a.dv + h * a.dv + col) =
                  *reinterpret_cast<const float4*>(turn + r_ * 32 + ((lane ^ r_) & 7) * 4);
          }
        }
        if (__any_sync(0xffffffffu, bad)) {
          __syncwarp();                               // (a row is written by eight lanes)
          if (bad) {
            ct_wait_before();                         // (long since true)
            const int g = h * DK;
            const size_t plane = ct_plane(DK, a.dv);
            const uint8_t* S = reinterpret_cast<const uint8_t*>(a.ws) + ((size_t)now.chunk * a.H + h) * 3 * plane;
            float* to = a.o + (size_t)(now.at.first + t) * a.H * a.dv + h * a.dv + v;
            uint32_t again = 0;                       // columns that may yet be numbers
#pragma unroll 1
            for (int e = 0; e < 32 && v + e < a.dv; ++e) {
              if (ct_number(to[e])) continue;
              const float z = start ? ct_state_dot(mine + a.q_col + g, S, plane, v + e, DK, a.dv) * f : 0.f;
              to[e] = z;
              again |= z == z ? 1u << e : 0u;
            }
#pragma unroll 1
            for (int s = 0; s <= t && again; ++s) {
              const TA* vr = x + (size_t)(now.at.first + s) * a.ld + a.v_col + h * a.dv + v;
              const float ps = Form::D(p, sc, row, t, s) *
                               (ct_dot(mine + a.q_col + g, x + (size_t)(now.at.first + s) * a.ld + a.k_col + g, DK) * q_scale);
              for (uint32_t m = again; m; m &= m - 1) {
                const int e = __ffs(m) - 1;
                const float z = fmaf(ps, (float)vr[e], to[e]);
                to[e] = z;
                if (z != z) again &= ~(1u << e);
              }
            }
            for (; again; again &= again - 1) {
              float* z = to + __ffs(again) - 1;
              *z = finish.one(*z);
            }
          }
        }
      }
      tc_fence_before();
      ct_arrive(&out_free);
      ct_arrive(&queue.free[it % kCtAhead]);
      now = then;
    }
  } else if (warp == kCtMma) {
    if (lane == 0) {
      for (int it = 0;; ++it) {
        const CtItem now = ct_item(queue, it);
        if (now.item >= items) break;
        constexpr uint32_t q_term = L::kPanel / 16, s_term = VT * 8, v_term = L::kVHalf / 16;
        auto q = [&](int e) { return umma_desc_k_sw128(smem + L::q(it, e)); };
        auto k = [&](int e) { return umma_desc_k_sw128(smem + L::k(it, e)); };
        auto st = [&](int e) { return umma_desc_k_sw128(smem + L::s(it, e)); };
        auto v = [&](int e) { return umma_desc_mn_sw128(smem + L::v(it, e), kCtHalf * 128, 1024); };
        {
          constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
          uint32_t acc = 0, acc1 = 0;
          for (int e = 0; e < NP; ++e) {
            ct_wait(&key_full[e], it);
            ct_small<false, L::kIn, L::kIn, 4>(t_s, q(e), q_term, 2, k(e), q_term, 2, idesc, acc);
          }
          if constexpr (NP == 2) ct_pair<false, 4>(t_s, q(0), 2, k(0), 2, idesc, acc);
          ct_pair<false, 4>(kTwo ? t_s + 128 : t_s, q(NP - 1), 2, k(NP - 1), 2, idesc, acc1);
          umma_commit(&score_done);
        }
        if (it) ct_wait(&out_free, it - 1);
        {
          constexpr uint32_t idesc = umma_idesc_bf16(128, VT);
          uint32_t acc = 0;
          for (int e = 0; e < NP; ++e) {
            ct_wait(&state_full[e], it);
            if (from_state(now)) ct_small<false, L::kIn, 3, 4>(t_o, q(e), q_term, 2, st(e), s_term, 2, idesc, acc);
          }
          if (from_state(now))
            for (int e = 0; e < NP; ++e) ct_pair<false, 4>(t_o, q(e), 2, st(e), 2, idesc, acc);
          umma_commit(&state_done);
        }
        ct_wait(&weight_full, it);
        {
          constexpr uint32_t idesc = umma_idesc_bf16(128, VT) | kCtBmn;
          const int halves = now.at.rows > kCtHalf ? 2 : 1;
          uint32_t acc = 0;
          for (int e = 0; e < 2; ++e) {
            ct_wait(&value_full[e], it);
            if (e < halves) {
              const uint32_t w = t_s + 64 * e;        // a term's eight columns of sixteen rows: 0, 8, 128 columns behind theirs
              const bool three = !one_term[e];
              ct_pair<true, 4>(t_o + VT, w + 128, 16, v(e), 128, idesc, acc);
              if (three) {
                ct_pair<true, 4>(t_o + VT, w + 8, 16, v(e) + v_term, 128, idesc, acc);
                ct_pair<true, 4>(t_o + VT, w, 16, v(e) + 2 * v_term, 128, idesc, acc);
              }
              ct_pair<true, 4>(t_o + VT, w + 8, 16, v(e), 128, idesc, acc);
              if (three) ct_pair<true, 4>(t_o + VT, w, 16, v(e) + v_term, 128, idesc, acc);
            }
          }
          for (int e = 0; e < halves; ++e) ct_pair<true, 4>(t_o + VT, t_s + 64 * e, 16, v(e), 128, idesc, acc);
          umma_commit(&value_done);
        }
        mbar_arrive(&queue.free[it % kCtAhead]);
      }
    }
    __syncwarp();
  } else if (warp == kCtCopy) {
    if (lane == 0) {                                  // the state's panels, where the keys were
      const size_t plane = ct_plane(DK, a.dv);
      ct_wait_before();
      for (int it = 0;; ++it) {
        const CtItem now = ct_item(queue, it);
        if (now.item >= items) break;
        const uint8_t* S = reinterpret_cast<const uint8_t*>(a.ws) + ((size_t)now.chunk * a.H + now.h) * 3 * plane;
        const uint32_t bytes = min(VT, a.dv - now.v0) * 128;
        const bool start = from_state(now);
        if (!L::kApart) mbar_wait_guarded(&score_done, it & 1);        // the keys are used
        else if (it) mbar_wait_guarded(&state_done, (it - 1) & 1);
        for (int e = 0; e < NP; ++e) {
          if (start) {
            mbar_expect_tx(&state_full[e], 3 * bytes);
            for (int i = 0; i < 3; ++i)
              ct_copy(smem + L::s(it, e) + i * VT * 128, S + i * plane + (size_t)(e * a.dv + now.v0) * 128, bytes, &state_full[e]);
          } else {
            mbar_arrive(&state_full[e]);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kCtFind) {
    for (int it = 0, item = (int)blockIdx.x;; ++it) {
      const CtItem next = ct_next<VT>(a, items, item, (int)gridDim.x);
      const int buf = it % kCtAhead;
      if (it >= kCtAhead) mbar_wait_guarded(&queue.free[buf], (it / kCtAhead - 1) & 1);
      if (lane < 4) special[buf][lane] = 0;
      if (lane == 0) queue.item[buf] = next;
      ct_arrive(&queue.full[buf]);
      if (next.item >= items) break;
      const TA* row = x + (int64_t)next.at.first * a.ld;
      const int g = next.h * DK, w = min(VT, a.dv - next.v0) * (int)sizeof(TA);
      ct_prefetch(row + a.q_col + g, a.ld * sizeof(TA), next.at.rows, DK * (int)sizeof(TA));
      ct_prefetch(row + a.k_col + g, a.ld * sizeof(TA), next.at.rows, DK * (int)sizeof(TA));
      ct_prefetch(x + (int64_t)next.at.first * a.ld + a.v_col + next.h * a.dv + next.v0, a.ld * sizeof(TA), next.at.rows, w);
      item = next.item + (int)gridDim.x;
    }
  }
  ct_end(t_s, 512);
}

// Its size for `chunks` chunks: the states, then every chunk's row of factors.  A workspace of cs_workspace_floats holds the chunks of
// 64 rows in fp32, which is less than those of 128 rows need where portions are short (64 x 128 rows in 256 sequences: by a fifth);
// then the sequences run in groups, one after the other, as many in each as it has room for.
inline int64_t ct_state_floats(int64_t chunks, int64_t H, int64_t dk, int64_t dv) { return (chunks * H * dk * dv / 2 * 3 + 3) / 4 * 4; }
inline int64_t ct_group(int64_t rows, int64_t n_seqs, int64_t H, int64_t dk, int64_t dv, int64_t floats) {
  auto fits = [&](int64_t n) {
    const int64_t chunks = ct_max_chunks(rows, n);
    return ct_state_floats(chunks, H, dk, dv) + chunks * H * (dk + 4) <= floats;
  };
  if (fits(n_seqs)) return n_seqs;
  int64_t n = 0;                                      // (sizes grow with n)
  for (int64_t step = (int64_t)1 << 32; step > 0; step >>= 1)
    if (n + step < n_seqs && fits(n + step)) n += step;
  return n;
}

// ------------------------------------------------------------------------------------------- launch
template <typename K>
inline int ct_allow(K kernel, int bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) return B200_OK;
  b200_set_error("chunk scan: %d bytes of shared memory: %s", bytes, cudaGetErrorString(e));
  return B200_ERR_CUDA;
}

template <int DK, int VT, typename TA, typename Form>
int ct_launch_shape(const ChunkScanArgs& a, const typename Form::Params& p, int64_t rows, bool beside, cudaStream_t s) {
  const int64_t items = ct_max_chunks(rows, a.n_seqs) * a.H * ((a.dv + VT - 1) / VT);
  constexpr int sb = CtSmem<DK, VT, TA>::kState, ob = CtSmem<DK, VT, TA>::kOutput;
  B200_REQUIRE(items < INT32_MAX - 65536, "chunk scan: too many chunks");
  int rc = ct_allow(ct_state_kernel<DK, VT, TA, Form>, sb);
  if (rc == B200_OK) rc = ct_allow(ct_output_kernel<DK, VT, TA, Form>, ob);
  if (rc != B200_OK) return rc;
  const int grid = (int)(items < sm_count() ? items : sm_count());
  if (beside) (void)launch_pdl(ct_state_kernel<DK, VT, TA, Form>, dim3(grid), dim3(kCtThreads), (size_t)sb, s, 1, a, p, (int)items);
  else ct_state_kernel<DK, VT, TA, Form><<<grid, kCtThreads, sb, s>>>(a, p, (int)items);
  const dim3 carry((DK * a.dv / 8 + kCtCarryThreads - 1) / kCtCarryThreads, a.H, a.n_seqs);
  const bool early = !Form::kNorm || items <= sm_count();
  (void)launch_pdl(ct_carry_kernel<DK, Form>, carry, dim3(kCtCarryThreads), 0, s, 1, a, p, early);
  (void)launch_pdl(ct_output_kernel<DK, VT, TA, Form>, dim3(grid), dim3(kCtThreads), (size_t)ob, s, 1, a, p, (int)items);
  return b200_check_launch(Form::kName);
}

// group: sequences per walk (ct_group).  The sequences of at most a.short_rows rows are in a one-pass kernel launched just before: it writes
// other slots and rows than the chunks.  Where sequences of 48 rows or fewer on average say that there are such, the chunks begin
// beside it (one portion of 2048 rows beside 64 single ones, mLSTM, 2 heads of 64 x 64: 62.5 -> 52.7 us, by FMAs 59.4; four of 512
// without any, 8 heads of 128 x 128, would take 58.3 instead of 56.3).
template <typename TA, typename Form>
int ct_launch(ChunkScanArgs a, const typename Form::Params& p, int dk, int64_t rows, int group, float* ws, cudaStream_t s) {
  a.ws = ws;
  a.ws_row_width = dk + 4;
  int rc = B200_OK;
  bool beside = a.short_rows > 0 && rows <= 48 * (int64_t)a.n_seqs;
  for (int left = a.n_seqs; left > 0 && rc == B200_OK; left -= group) {
    a.n_seqs = left < group ? left : group;
    const int64_t chunks = ct_max_chunks(rows, a.n_seqs);
    if (chunks == 0) break;
    a.ws_row = ws + ct_state_floats(chunks, a.H, dk, a.dv);
    if (dk == 64) rc = a.dv <= 64 ? ct_launch_shape<64, 64, TA, Form>(a, p, rows, beside, s) : ct_launch_shape<64, 128, TA, Form>(a, p, rows, beside, s);
    else rc = a.dv <= 64 ? ct_launch_shape<128, 64, TA, Form>(a, p, rows, beside, s) : ct_launch_shape<128, 128, TA, Form>(a, p, rows, beside, s);
    beside = false;
    a.cu_seq += group;
    a.ctx_lens += group;
    a.state_slots += group;
  }
  return rc;
}

}  // namespace b200
