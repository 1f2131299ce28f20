// Latent attention of prompt portions in the absorbed form on the 5th-generation tensor cores: every head of a query row
// scores against the SAME cached row per token, [latent: 512 | rotated key part: 64], and takes the latent as its value.
//
// The (query row, head) pairs are the M rows of the products.  A PAIR of CTAs (tcgen05 cta_group::2) owns 256 of them -- 256 / H
// query rows with all their heads, 128 pairs per CTA -- and ONE HALF (256 columns) of the values: the fp32 accumulator
// [128][256] and two score buffers [128][96] live in a CTA's tensor memory, which the whole 512 columns would fill alone.  The
// scores are therefore computed once per value half (576 + 256 products per key instead of 576 / 2 + 256); what that buys is
// that nothing but the query tile (144 KB) has to stay in shared memory, and that each CTA stages only half of every key
// block: with single CTAs the blocks' way through L2, not the tensor cores, would be the bound.
//
//   warp 4    query tile (once per work item) and keys: per block of 96 keys a CTA stages ITS 48 keys as three units of 192
//             columns (18 KB) through a ring of three.  One copy brings a page's 16 rows of a unit: the tensor map has the
//             eight-row group outermost, so every group of a unit is 3 KB behind the one before, as a K-major operand wants it;
//   warp 6    values: its 128 of the half's 256 columns of all 96 keys, three units of 32 keys (8 KB), read MN-major straight from
//             the row layout, one copy per page.  A unit that reaches past the sequence's last key is copied with plain loads
//             and zeros behind it: probability zero times a stale page's content must not be no number;
//   warp 5    MMA issuer (leading CTA): S = Q K^T (M 256, N 96), O += P V (M 256, N 256, P from tensor memory);
//             S of block j + 1 is issued before P of block j is waited for;
//   warps 0-3 softmax: thread = pair.  Base-2 online softmax whose reference is the running maximum, so that a row's largest
//             probability is exactly 1 in bf16, P in bf16 over the score columns, l the sum of P as it was rounded, O / (l + sink)
//             at the end.  (A reference that moves by more than 2^8 only, as in the other tensor-core attention kernels, rounds the
//             largest probability like any other: the error of P V over 512 to 2048 keys is 1.4 to 1.6 times as large.  The rescaling it
//             saves, 25 us of the whole layer's 573 for 4 x 2048 rows of 16 heads, is not worth that.)
// Persistent: one pair of CTAs per two SMs walks the heaviest-first (tile, sub-tile, half) list back and forth; barriers, tensor
// memory and rings live for the whole kernel, so an item's epilogue overlaps the next one's loads and first scores.
// Bound: the products' reads of shared memory.  With both operands there, S of a block (36 instructions of 256 x 96 x 16) takes 3700
// cycles of the block's 5000, where the tensor pipe needs 1730 for it: the 256 query rows of every instruction leave shared memory
// at about 64 bytes a cycle.  (The same queries held in tensor memory: 2270 cycles; but they fill what a second score buffer and the
// accumulators need, and two of nine slabs there, in turns with the scores, cost more in waits than they save, 498 -> 528 us.)  Rings of
// three to six units take the same time; few copies matter: blocks of 128 keys in nine slabs of 8 KB, 52 copies of 2 KB each per
// block, took 458 us for 4 x 2048 rows of 16 heads where these took 430.  Now, with the reference that moves at every new maximum, 421
// us with L2 cold, the tensor pipe 53 % active (mma.sync kernel: 1940 us).
#include "common.cuh"
#include "runtime.h"
#include "../../include/b200.h"

#include <math.h>

namespace b200 {

constexpr int kLtThreads = 224;
constexpr int kLtR = 512, kLtW = 576, kLtSlabs = kLtW / 64, kLtKeys = 96, kLtHalfCols = 256;
constexpr int kLtPage = 16, kLtKPages = kLtKeys / kLtPage / 2, kLtVPages = 2;      // pages per key unit and per value unit
constexpr int kLtQSlab = 128 * 128;                    // [128 pairs][128 B]
constexpr int kLtUnitSlabs = 3, kLtKUnits = kLtSlabs / kLtUnitSlabs, kLtKGroup = kLtUnitSlabs * 1024;
constexpr int kLtKPageBytes = 2 * kLtKGroup;           // [2 groups][3 slabs][8 rows][128 B]
constexpr int kLtKUnit = kLtKPages * kLtKPageBytes;    // 18,432
constexpr int kLtKSlots = 3;
constexpr int kLtVPageBytes = 2 * kLtPage * 128;       // [2 column groups][16 rows][128 B]
constexpr int kLtVUnit = kLtVPages * kLtVPageBytes;    // 8,192
constexpr int kLtVUnits = kLtKeys / kLtPage / kLtVPages;
constexpr int kLtOffK = kLtSlabs * kLtQSlab;           // 147,456
constexpr int kLtOffV = kLtOffK + kLtKSlots * kLtKUnit;
constexpr int kLtOffBar = kLtOffV + kLtVUnits * kLtVUnit;     // 227,328
constexpr int kLtSmemBytes = kLtOffBar + 256 + 1024;
constexpr int kLtColS = 256, kLtColStep = 128;         // O: columns [0, 256), S0 from 256, S1 from 384

__device__ __forceinline__ void umma_bf16_ts_2sm(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Tiled loads of either CTA of a pair that complete on the leading CTA's barrier (tma_load_2d_2sm with more coordinates)
__device__ __forceinline__ void tma_load_3d_2sm(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar) & 0xFEFFFFFFu), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_2sm(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar) & 0xFEFFFFFFu), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// K-major, 128-byte swizzle, eight-row groups `sbo` bytes apart
__device__ __forceinline__ uint64_t lt_desc_k(uint32_t addr, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// registers -> 32 lanes x 16 columns of tensor memory
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

struct LtArgs {
  const bf16* cache;
  const int32_t* block_table;
  int max_blocks;
  const int32_t* cu_q;
  const int32_t* ctx_lens;
  const int32_t* tile_seq;
  const int32_t* tile_q0;
  int num_tiles, subs, tpi;        // sub-tiles per tile, query rows per item (256 / H)
  const float* sink;
  bf16* out;
  int64_t ldo;
  int H;
  float scale_log2;
};

__global__ void __launch_bounds__(kLtThreads, 1)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const LtArgs a) {
  extern __shared__ uint8_t lt_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lt_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kLtOffBar);
  // on the leader: what both CTAs' copies and softmax warps complete; in each CTA: what the leader's commits release
  uint64_t* q_full = bars;             // leader
  uint64_t* q_empty = bars + 1;        // each
  uint64_t* k_full = bars + 2;         // [3] leader
  uint64_t* k_empty = bars + 5;        // [3] each
  uint64_t* v_full = bars + 8;         // [3] leader
  uint64_t* v_empty = bars + 11;       // [3] each
  uint64_t* s_full = bars + 14;        // [2] each
  uint64_t* p_full = bars + 16;        // [2] leader
  uint64_t* p_empty = bars + 18;       // each
  uint64_t* o_full = bars + 19;        // each
  uint64_t* o_empty = bars + 20;       // leader
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int crank = (int)cluster_ctarank();
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    mbar_init(q_full, 2);
    mbar_init(q_empty, 1);
    for (int i = 0; i < kLtKSlots; ++i) {
      mbar_init(&k_full[i], 2);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < kLtVUnits; ++i) {
      mbar_init(&v_full[i], 2);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);        // one per softmax warp of the pair; one barrier per score buffer
    }
    mbar_init(p_empty, 1);
    mbar_init(o_full, 1);
    mbar_init(o_empty, 8);
    fence_mbar_init();
  }
  if (warp == 5) {
    tmem_alloc_2sm(tmem_slot, 512);
    tmem_relinquish_2sm();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  struct Work {
    int seq, half, q0, q_begin, q_len, ctx, total_len, n_blocks;     // n_blocks 0: a sub-tile without query rows
  };
  const int total_work = a.num_tiles * a.subs * 2;
  auto load_work = [&](int w) {
    Work m;
    if (w >= total_work) w = total_work - 1;
    m.half = w & 1;
    const int t = (w >> 1) / a.subs, sub = (w >> 1) - t * a.subs;
    m.seq = __ldg(a.tile_seq + t);
    m.q0 = __ldg(a.tile_q0 + t) + sub * a.tpi;
    m.q_begin = __ldg(a.cu_q + m.seq);
    m.q_len = __ldg(a.cu_q + m.seq + 1) - m.q_begin;
    m.ctx = __ldg(a.ctx_lens + m.seq);
    m.total_len = m.ctx + m.q_len;
    const int kv_end = min(m.total_len, m.ctx + m.q0 + a.tpi);
    m.n_blocks = m.q0 < m.q_len ? (kv_end + kLtKeys - 1) / kLtKeys : 0;
    return m;
  };
  const int n_cl = gridDim.x >> 1, cl = blockIdx.x >> 1;
  const int n_rounds = (total_work + n_cl - 1) / n_cl;
  auto work_of = [&](int rd) { return rd * n_cl + ((rd & 1) ? n_cl - 1 - cl : cl); };

  if (warp == 4) {
    // ------------------------------------------------------------------ queries and keys
    int slot = 0;
    uint32_t phase = 0, it = 0;
    Work nxt = load_work(work_of(0));
    for (int rd = 0; rd < n_rounds; ++rd) {
      const Work m = nxt;
      nxt = load_work(work_of(rd + 1));
      if (work_of(rd) >= total_work) break;
      if (m.n_blocks == 0) continue;
      if (lane == 0) {
        if (it > 0) mbar_wait_guarded(q_empty, (it - 1) & 1);
        mbar_expect_tx_cluster(mapa_u32(q_full, 0), kLtSlabs * kLtQSlab);
        const int row = (m.q_begin + m.q0) * a.H + crank * 128;
        for (int s = 0; s < kLtSlabs; ++s) tma_load_2d_2sm(smem + s * kLtQSlab, &tmap_q, q_full, s * 64, row, kEvictFirst);
      }
      const int n_pages = (m.total_len + kLtPage - 1) / kLtPage;
      const int32_t* bt = a.block_table + (size_t)m.seq * a.max_blocks;
      constexpr int AHEAD = 32 / kLtKPages;            // blocks whose pages the lanes hold
      int mine = 0;
      for (int j = 0, f = 0; j < m.n_blocks; ++j, f = f + 1 == AHEAD ? 0 : f + 1) {
        if (f == 0) {                                  // the pages of this CTA's half of the next blocks
          const int page = (j + lane / kLtKPages) * (2 * kLtKPages) + crank * kLtKPages + lane % kLtKPages;
          mine = page < n_pages ? __ldg(bt + page) : 0;
        }
        int group[kLtKPages];
#pragma unroll
        for (int p = 0; p < kLtKPages; ++p) group[p] = __shfl_sync(0xffffffffu, mine, f * kLtKPages + p) * (kLtPage / 8);
        if (lane == 0) {
#pragma unroll
          for (int u = 0; u < kLtKUnits; ++u) {
            mbar_wait_guarded(&k_empty[slot], phase ^ 1);
            mbar_expect_tx_cluster(mapa_u32(&k_full[slot], 0), kLtKUnit);
            uint8_t* dst = smem + kLtOffK + slot * kLtKUnit;
#pragma unroll
            for (int p = 0; p < kLtKPages; ++p)
              tma_load_4d_2sm(dst + p * kLtKPageBytes, &tmap_k, &k_full[slot], 0, 0, u * kLtUnitSlabs, group[p]);
            if (++slot == kLtKSlots) { slot = 0; phase ^= 1; }
          }
        }
        __syncwarp();
      }
      ++it;
    }
  } else if (warp == 6) {
    // ------------------------------------------------------------------ values
    uint32_t gb = 0;
    Work nxt = load_work(work_of(0));
    for (int rd = 0; rd < n_rounds; ++rd) {
      const Work m = nxt;
      nxt = load_work(work_of(rd + 1));
      if (work_of(rd) >= total_work) break;
      const int n_pages = (m.total_len + kLtPage - 1) / kLtPage;
      const int32_t* bt = a.block_table + (size_t)m.seq * a.max_blocks;
      const int col = m.half * kLtHalfCols + crank * 128;
      constexpr int PAGES = kLtKeys / kLtPage, AHEAD = 32 / PAGES;
      int mine = 0;
      for (int j = 0, f = 0; j < m.n_blocks; ++j, ++gb, f = f + 1 == AHEAD ? 0 : f + 1) {
        if (f == 0) {
          const int page = j * PAGES + lane;
          mine = page < n_pages ? __ldg(bt + page) : 0;
        }
#pragma unroll
        for (int u = 0; u < kLtVUnits; ++u) {
          int rows[kLtVPages];
#pragma unroll
          for (int p = 0; p < kLtVPages; ++p) rows[p] = __shfl_sync(0xffffffffu, mine, f * PAGES + u * kLtVPages + p) * kLtPage;
          uint8_t* dst = smem + kLtOffV + u * kLtVUnit;
          const int key0 = j * kLtKeys + u * (kLtVPages * kLtPage);
          if (key0 + kLtVPages * kLtPage <= m.total_len) {
            if (lane == 0) {
              mbar_wait_guarded(&v_empty[u], (gb & 1) ^ 1);
              mbar_expect_tx_cluster(mapa_u32(&v_full[u], 0), kLtVUnit);
#pragma unroll
              for (int p = 0; p < kLtVPages; ++p) tma_load_3d_2sm(dst + p * kLtVPageBytes, &tmap_v, &v_full[u], 0, rows[p], col / 64);
            }
          } else {
            mbar_wait_guarded(&v_empty[u], (gb & 1) ^ 1);
            const uint32_t base = smem_u32(dst);
#pragma unroll 4
            for (int i = lane; i < kLtVPages * kLtPage * 16; i += 32) {      // 16 chunks of 16 bytes per key: 8 of each column group
              const int r = i >> 4, c = i & 15, p = r >> 4, pr = r & 15;
              uint4 v = make_uint4(0, 0, 0, 0);
              if (key0 + r < m.total_len) v = ld_cg_v4(a.cache + (size_t)((p ? rows[1] : rows[0]) + pr) * kLtW + col + c * 8);
              st_shared_v4(base + p * kLtVPageBytes + (c >> 3) * (kLtPage * 128) + pr * 128 + (((c & 7) ^ (pr & 7)) << 4), v);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_u32(&v_full[u], 0));
          }
          __syncwarp();
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer (leading CTA)
    if (crank == 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(256, kLtKeys);
      constexpr uint32_t idesc_o = umma_idesc_bf16_bmn(256, kLtHalfCols);
      const uint32_t q_addr = smem_u32(smem), k_addr0 = smem_u32(smem + kLtOffK), v_addr0 = smem_u32(smem + kLtOffV);
      int slot = 0;
      uint32_t phase = 0;
      auto issue_s = [&](uint32_t gb) {
        const uint32_t d = tmem_base + kLtColS + (gb & 1) * kLtColStep;
        for (int u = 0; u < kLtKUnits; ++u) {
          mbar_wait_guarded(&k_full[slot], phase);
          tc_fence_after();
          const uint32_t qa = q_addr + u * kLtUnitSlabs * kLtQSlab, ka = k_addr0 + slot * kLtKUnit;
#pragma unroll
          for (int k = 0; k < 4 * kLtUnitSlabs; ++k)
            umma_bf16_2sm(d, umma_desc_k_sw128(qa + (k >> 2) * kLtQSlab + (k & 3) * 32),
                          lt_desc_k(ka + (k >> 2) * 1024 + (k & 3) * 32, kLtKGroup), idesc_s, (u | k) != 0);
          umma_commit_2sm_mc(&k_empty[slot], 3);
          if (++slot == kLtKSlots) { slot = 0; phase ^= 1; }
        }
        umma_commit_2sm_mc(&s_full[gb & 1], 3);
      };
      uint32_t gb = 0, it = 0;
      Work nxt = load_work(work_of(0));
      for (int rd = 0; rd < n_rounds; ++rd) {
        const int n_blocks = nxt.n_blocks;
        nxt = load_work(work_of(rd + 1));
        if (work_of(rd) >= total_work) break;
        if (n_blocks == 0) continue;
        mbar_wait_guarded(q_full, it & 1);
        tc_fence_after();
        issue_s(gb);
        if (n_blocks == 1) umma_commit_2sm_mc(q_empty, 3);
        for (int j = 0; j < n_blocks; ++j, ++gb) {
          // the other buffer holds P of the block before, whose PV product was issued before these scores
          if (j + 1 < n_blocks) {
            issue_s(gb + 1);
            if (j + 2 == n_blocks) umma_commit_2sm_mc(q_empty, 3);
          }
          mbar_wait_guarded(&p_full[gb & 1], (gb >> 1) & 1);
          tc_fence_after();
          if (j == 0 && it > 0) {
            mbar_wait_guarded(o_empty, (it - 1) & 1);
            tc_fence_after();
          }
          const uint32_t p_col = tmem_base + kLtColS + (gb & 1) * kLtColStep;
#pragma unroll
          for (int u = 0; u < kLtVUnits; ++u) {
            mbar_wait_guarded(&v_full[u], gb & 1);
            tc_fence_after();
            const uint32_t va = v_addr0 + u * kLtVUnit;
#pragma unroll
            for (int k = 0; k < kLtVPages; ++k)
              umma_bf16_ts_2sm(tmem_base, p_col + (u * kLtVPages + k) * 8, umma_desc_mn_sw128(va + k * kLtVPageBytes, kLtPage * 128, 1024),
                               idesc_o, (j | u | k) != 0);
            umma_commit_2sm_mc(&v_empty[u], 3);
          }
          umma_commit_2sm_mc(p_empty, 3);
        }
        umma_commit_2sm_mc(o_full, 3);
        ++it;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax / epilogue (warps 0..3 of both CTAs)
    const int pair = crank * 128 + warp * 32 + lane, tok = pair / a.H, head = pair - tok * a.H;
    const uint32_t t_lane = tmem_base + ((uint32_t)(warp * 32) << 16);
    const bool wide = (reinterpret_cast<uintptr_t>(a.out) & 31u) == 0 && a.ldo % 16 == 0;
    const uint32_t p_full_at[2] = {mapa_u32(&p_full[0], 0), mapa_u32(&p_full[1], 0)};
    const uint32_t o_empty_at = mapa_u32(o_empty, 0);
    uint32_t gb = 0, it = 0;
    Work nxt = load_work(work_of(0));
    for (int rd = 0; rd < n_rounds; ++rd) {
      const Work m = nxt;
      nxt = load_work(work_of(rd + 1));
      if (work_of(rd) >= total_work) break;
      if (m.n_blocks == 0) continue;
      const int qi = m.q0 + tok, qpos = m.ctx + qi;
      const bool valid = qi < m.q_len;
      float m_used = -INFINITY, l = 0.f;
      for (int j = 0; j < m.n_blocks; ++j, ++gb) {
        const uint32_t s_col = t_lane + kLtColS + (gb & 1) * kLtColStep;
        mbar_wait_guarded(&s_full[gb & 1], (gb >> 1) & 1);
        tc_fence_after();
        uint32_t s[3][32];
#pragma unroll
        for (int c = 0; c < 3; ++c) tmem_ld_32x32(s_col + c * 32, s[c]);
        tmem_ld_wait();
        const int kv0 = j * kLtKeys;
        if (kv0 + kLtKeys - 1 > m.ctx + m.q0 || kv0 + kLtKeys > m.total_len) {
          const int last = min(qpos, m.total_len - 1) - kv0;
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > last) s[c][i] = 0xff800000u;
        }
        float mx = -INFINITY;
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) mx = fmaxf(mx, __uint_as_float(s[c][i]));
        mx *= a.scale_log2;
        float alpha = 1.f;
        bool rescale = false;
        if (mx > m_used) {
          alpha = ex2_approx(m_used - mx);
          m_used = mx;
          l *= alpha;
          rescale = j > 0;
        }
        const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
        float sum = 0.f;
        uint32_t pk[2][32];                            // 48 columns of bf16 pairs
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = ex2_approx(fmaf(__uint_as_float(s[c][i]), a.scale_log2, neg_m));
            const float p1 = ex2_approx(fmaf(__uint_as_float(s[c][i + 1]), a.scale_log2, neg_m));
            const uint32_t both = pack_bf16(p0, p1);
            sum += bf16_lo(both) + bf16_hi(both);
            pk[c >> 1][(c & 1) * 16 + (i >> 1)] = both;
          }
        l += sum;
        if (__any_sync(0xffffffffu, rescale)) {        // (implies j > 0) the block before's product has retired
          mbar_wait_guarded(p_empty, (gb - 1) & 1);
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < kLtHalfCols / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(t_lane + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(t_lane + c * 32, o);
          }
          tmem_st_wait();
        }
        tmem_st_32x32(s_col, pk[0]);
        tmem_st_32x16(s_col + 32, pk[1]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(p_full_at[gb & 1]);
      }
      mbar_wait_guarded(o_full, it & 1);
      tc_fence_after();
      if (a.sink != nullptr && m_used > -INFINITY) l += exp2f(a.sink[head] * 1.4426950408889634f - m_used);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* orow = a.out + (size_t)(m.q_begin + qi) * a.ldo + (size_t)head * kLtR + m.half * kLtHalfCols;
#pragma unroll 1
      for (int c = 0; c < kLtHalfCols / 32; c += 2) {
        uint32_t o[2][32];
        tmem_ld_32x32(t_lane + c * 32, o[0]);
        tmem_ld_32x32(t_lane + c * 32 + 32, o[1]);
        tmem_ld_wait();
        if (c + 2 >= kLtHalfCols / 32) {               // O is in registers: the next item may overwrite the accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(o_empty_at);
        }
        if (valid) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint4 w[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(o[e][8 * v + i]) * inv;
              w[v] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
            }
            bf16* dst = orow + (c + e) * 32;
            if (wide) {
              st_v8(dst, w[0], w[1]);
              st_v8(dst + 16, w[2], w[3]);
            } else {
#pragma unroll
              for (int v = 0; v < 4; ++v) st_v4(dst + v * 8, w[v]);
            }
          }
        }
      }
      ++it;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, 512);
  }
}

}  // namespace b200

using namespace b200;

// The tensor-core kernel takes 512 + 64 wide rows, heads that divide 128 and tiles of whole 256-pair items; the queries' rows
// contiguous over the heads, pages of 16 rows.  Everything else goes to b200_latent_attn_prefill.
extern "C" int b200_latent_attn_prefill_rows(const void* qa, int64_t ldq, int rows, const void* cache, int num_blocks, int page,
                                             const int32_t* block_table, int max_blocks, const int32_t* cu_q, const int32_t* ctx_lens,
                                             const int32_t* tile_seq, const int32_t* tile_q0, int n_tiles, int tile_rows,
                                             const float* sink, void* out, int64_t ldo, int H, int R, int dr, float scale,
                                             void* stream) {
  const DeviceInfo& d = device_info();
  if (R != kLtR || dr != kLtW - kLtR || H <= 0 || 128 % H != 0 || tile_rows <= 0 || (tile_rows * H) % 256 != 0 || page != kLtPage ||
      ldq != (int64_t)H * kLtW || rows <= 0 || num_blocks <= 0 || n_tiles <= 0 || ldo % 8 != 0 ||
      (reinterpret_cast<uintptr_t>(out) & 15) != 0 || (reinterpret_cast<uintptr_t>(qa) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(cache) & 15) != 0 || !d.valid || d.cc_major != 10)
    return b200_latent_attn_prefill(qa, ldq, cache, page, block_table, max_blocks, cu_q, ctx_lens, tile_seq, tile_q0, n_tiles, tile_rows,
                                    sink, out, ldo, H, R, dr, scale, stream);
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(latent_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLtSmemBytes);
    if (e != cudaSuccess) {
      b200_set_error("latent_attn(tc): cudaFuncSetAttribute(smem=%d): %s", kLtSmemBytes, cudaGetErrorString(e));
      return B200_ERR_CUDA;
    }
    attr_set = true;
  }
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_bf16_2d(&tq, qa, (uint64_t)rows * H, kLtW, kLtW, 128, 64);
  if (rc) return rc;
  const uint64_t cache_rows = (uint64_t)num_blocks * kLtPage, row_bytes = kLtW * 2;
  {
    const uint64_t dims[4] = {64, 8, kLtSlabs, cache_rows / 8}, strides[3] = {row_bytes, 128, 8 * row_bytes};
    const uint32_t box[4] = {64, 8, kLtUnitSlabs, 2};
    if ((rc = make_tmap_bf16_nd(&tk, cache, 4, dims, strides, box))) return rc;
  }
  {
    const uint64_t dims[3] = {64, cache_rows, kLtSlabs}, strides[2] = {row_bytes, 128};
    const uint32_t box[3] = {64, kLtPage, 2};
    if ((rc = make_tmap_bf16_nd(&tv, cache, 3, dims, strides, box))) return rc;
  }
  const LtArgs a{(const bf16*)cache, block_table, max_blocks, cu_q, ctx_lens, tile_seq, tile_q0, n_tiles, tile_rows * H / 256, 256 / H,
                 sink, (bf16*)out, ldo, H, scale * 1.4426950408889634f};
  const long long items = (long long)n_tiles * a.subs * 2;
  const int sms = d.sm_count > 0 ? d.sm_count : 148;
  const int pairs = (int)(items < sms / 2 ? items : sms / 2);
  cudaError_t e = launch_pdl(latent_attn_tc_kernel, dim3(pairs * 2), dim3(kLtThreads), (size_t)kLtSmemBytes, (cudaStream_t)stream, 2, tq, tk,
                             tv, a);
  if (e != cudaSuccess) {
    b200_set_error("b200_latent_attn_prefill(tc): launch failed: %s", cudaGetErrorString(e));
    (void)cudaGetLastError();
    return B200_ERR_CUDA;
  }
  return b200_check_launch("b200_latent_attn_prefill(tc)");
}
