// flash-attention forward for sm_100a, the default tile: O = softmax(Q K^T * scale [+ causal mask]) V, LSE optional. Two
// query tiles of 128 rows of one (batch, head) slice per work item, KV blocks of 128 keys, softmax as in fa_fwd_sm100.cuh (a
// warpgroup per tile, thread t owns row t), the same arithmetic in the same order.
//
// What paces a tile is its chain S = Q K^T -> softmax -> O += P V -> next S. With P written over its S (fa_fwd_sm100.cuh)
// the next S of a tile cannot start before its P V has read P, so a tile waits for both products (1024 tensor cycles and
// the hand-offs between one issuing thread and two warpgroups, about 1480 cycles in an event trace) after every softmax
// (2010 cycles), and the tensor pipe idles for 40 % of the time. Here P has columns of its own (tensor memory: S buffers,
// P0, P1, O0, O1; at 128 columns of V that leaves ONE S buffer, which the tiles fill in turn): the threads of a tile load
// their scores into registers and hand the buffer back at once (s_free), so that the next S runs under the softmax and
// is there when the threads come for it. S and P V are issued by a warp each: a wait that is already over costs a thread
// 80 cycles, a commit 65, a blocked issue hundreds, and in one thread that time adds up to more than the pipe's queue
// covers (measured: this layout with one issuing warp 4500 cycles per block, 3490 before, 3000 with two).
// Sustained / in a short burst, before and now, us (d = 128 fp16, bf16 where causal and not 4096): B=8 H=16 L=4096 1080 -> 944 /
// 928 -> 815; causal 597 -> 544 / 516 -> 472; B=1 H=16 L=16384 causal 1123 -> 965 / 1000 -> 844; B=4 H=16 L=2999 causal
// 188 -> 175 / 178 -> 160; B=2 H=16 Lq=1024 Lkv=9000 causal 155 -> 123; B=1 H=32 L=8192 d=64 805 -> 731. Work items of one
// short block gain little (2000 slices of L=64: 55 -> 54 at d=128, 47.4 / 47.4 at d=64). What bounds it now: the power limit
// (the SM clock falls to 1.4 GHz under it) and the exponentials of both tiles beside the rest of the softmax (2500 cycles per
// block for the pair, of which this form takes 3000).
//
// The work list has two forms. SINGLE: a grid of one CTA per work item, latest query block first. Otherwise one CTA per SM
// walks a static list: what a CTA costs once -- launch, tensor-memory allocation, barrier set-up, the Q load, the first S
// before any softmax can start, and at the end a last P V and an epilogue under which nothing else runs -- is paid once
// per SM, the Q tiles of the next work item are loaded as soon as the last S MMA of the current one has read them, the
// next item's first S goes ahead of the current one's last P V, and one query tile's epilogue runs under the other tile's
// GEMMs and its own next S.
//
// Work list of the persistent form: items are (slice, V-column chunk, block of 256 query rows). Pairs of items of equal
// total cost (k-th heaviest and k-th lightest query block of a slice under a causal mask) are handed out round-robin, so
// every CTA gets the same work up to one pair, and neighbouring CTAs work on the same slice (K and V shared in L2).
// Replaces the reference kernels flashattn_fwd_regfuse (csrc/kernels/attention/regfuse/regfuse.h:48-455) and
// flashattn_fwd_smemfuse (csrc/kernels/attention/smemfuse/smemfuse.h:61-614), like fa_fwd_sm100.cuh.
//
// No wait can be circular: S(g) of the CTA's g-th block (a block of one tile) waits for the scores of the buffer's last
// product to be read, which waits for that tile's previous block only, i.e. for P V before it; K of block r + 1 precedes V of
// block r in the ring, and either is released by the product that reads it. K and V tiles report to barriers of their own
// although they share the slots: a warp that waits for one kind only must not find the barrier a phase behind or ahead.
//
// Ring order: within a work item K of block j + 1 precedes V of block j (entries K0, K1 V0, K2 V1, ..., V of the last block), and
// an item's entries follow those of the item before. With K of the next item ahead of the last V as well, a ring of three
// entries gave the V of a one-block item its slot only when the second tile's S of that item was complete, which at 128 columns
// of V (one score buffer) is when the first tile starts on its scores: the load (3000 cycles from DRAM) then ended after the
// softmax (1000 slices of Lq=256 Lkv=128 at d = 128 39.9 -> 37.3 us).
// Items of one block are also bound by instruction fetch: every role runs its per-item code once per block, the SM
// sub-partitions hold 32 KB of it, and neighbouring SMs stall together. Hence one copy of each loader, two decodes of an item
// in the softmax threads instead of five, and multiplications for the divisions of the decode (2000 slices of L=64 at d = 64
// 49.5 -> 47.4 us, 4000 of them 94 -> 88; 512 of L=512 causal 61.3 -> 58.6).
#pragma once

#include "fa_fwd_sm100.cuh"
#include "fast_div.cuh"

namespace ab200 {

enum FaPersistTag : int { kTagQFree = 8, kTagOFree = 9, kTagSFree = 10 };

struct FaFwdPersistParams {
  FaFwdParams f;
  int nqb;      // blocks of 256 query rows per slice
  int ndv;      // V-column chunks
  int n_super;  // pairs of work items: BH * ndv * ceil(nqb / 2)
  FastDiv by_npair, by_ndv;  // ceil(nqb / 2), ndv
};

struct FaFwdItem {
  int bh, dv_off, m_base;
  int nblk[2];
  int nmax;
};

// Output staging: where shared memory has room beside the operands (for both finished tiles with a K / V ring of up to three
// entries at d = 128, for a box of each with four), a tile's rows are written there (16-bit, 128-byte swizzle) and leave through TMA stores, one per warp and
// 64-column box (32 rows each, so no warp waits for another). A thread storing its own row writes 32-byte pieces of 32
// different rows per instruction, which keeps the softmax warps from the next item's first block for as long as a
// couple of KV blocks take.
template <class Cfg>
struct FaFwdPersistLayout {
  static constexpr int O_BOX_BYTES = Cfg::BM * 128;  // 128 rows x 64 columns
#ifdef AB200_FA_FWD_NO_STAGE_O  // build option for comparisons: every thread stores its own row
  static constexpr int STAGE_BOXES = 0;
#else
  static constexpr int room(int boxes) { return Cfg::SMEM_BYTES + 2 * boxes * O_BOX_BYTES <= 232448; }
  static constexpr int STAGE_BOXES = Cfg::DV % 64 != 0 ? 0 : room(Cfg::DV / 64) ? Cfg::DV / 64 : room(1) ? 1 : 0;
#endif
  static constexpr bool STAGE_O = STAGE_BOXES > 0;
  static constexpr int O_STAGE_BYTES = STAGE_BOXES * O_BOX_BYTES;  // per tile
  static constexpr int SMEM_BYTES = Cfg::SMEM_BYTES + 2 * O_STAGE_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory overflow");
  // Tensor memory (columns): score buffers, P of both tiles, O of both tiles.
  static constexpr int S_BUFS = 2 * (128 + 64 + Cfg::DV) <= 512 ? 2 : 1;
  static constexpr int P_COL = S_BUFS * 128;
  static constexpr int O_COL = P_COL + 2 * 64;
  static constexpr int COLS_USED = O_COL + 2 * Cfg::DV;
  static constexpr int TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
  static_assert(COLS_USED <= 512, "tensor memory");
};

template <class Cfg, bool SINGLE>
__global__ void __launch_bounds__(Cfg::NTHREADS, 1)
fa_fwd_persist_sm100_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                            const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                            const FaFwdPersistParams pp) {
  static_assert(Cfg::NQ == 2 && Cfg::SPLIT == 1 && Cfg::NMMA == 1 && Cfg::EXP_EMU == 0 && Cfg::EXP_H2 == 0,
                "the persistent kernel is built for the default tile only");
  static_assert(Cfg::DV <= 128, "the epilogue holds a whole output row in registers");
  static_assert(Cfg::NSTAGE >= 2, "K of the next block is loaded before V of the current one");
  constexpr int DQK = Cfg::DQK, DV = Cfg::DV, NQ = 2, NSTAGE = Cfg::NSTAGE;
  constexpr bool BF16 = Cfg::BF16;
  constexpr int BM = Cfg::BM, BN = Cfg::BN;
  const FaFwdParams& p = pp.f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + NQ * Cfg::Q_TILE_BYTES;
  using Lay = FaFwdPersistLayout<Cfg>;
  constexpr bool STAGE_O = Lay::STAGE_O;
  constexpr int S_BUFS = Lay::S_BUFS;
  uint8_t* sO = smem + Cfg::SMEM_TILES;  // [2] finished tiles, or boxes of them, on their way out (STAGE_O only)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::SMEM_TILES + 2 * Lay::O_STAGE_BYTES);
  uint64_t* q_full = bars;                   // [2] Q tile landed
  uint64_t* q_free = q_full + NQ;            // [2] the item's last S MMA of the tile is complete
  uint64_t* k_full = q_free + NQ;            // [NSTAGE] a K tile landed in the slot
  uint64_t* v_full = k_full + NSTAGE;        // [NSTAGE] a V tile did
  uint64_t* kv_empty = v_full + NSTAGE;      // [NSTAGE]
  uint64_t* s_full = kv_empty + NSTAGE;      // [2] per tile
  uint64_t* s_free = s_full + NQ;            // [2] per score buffer: its scores are in registers
  uint64_t* p_full = s_free + NQ;            // [2]
  uint64_t* o_done = p_full + NQ;            // [2]
  uint64_t* o_free = o_done + NQ;            // [2] the finished tile's O is in the softmax threads' registers
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(o_free + NQ);
  CtaAbort* ab = reinterpret_cast<CtaAbort*>(tmem_base_slot + 1);
  constexpr int kBars = 7 * NQ + 3 * NSTAGE;
  static_assert(kBars * 8 + 16 <= Cfg::BARRIER_BYTES, "barrier area");
  static_assert(NSTAGE <= 16, "the producer keeps two bits per ring entry in a word");

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  constexpr int kSWarp = 4 * NQ;
  constexpr int kPvWarp = 4 * NQ + 1;
  constexpr int kTmaWarp = 4 * NQ + 2;

  const int nblk_all = (p.Lkv + BN - 1) / BN;
  const int npair = (pp.nqb + 1) / 2;
  const int n_steps = SINGLE ? 1 : 2 * ((pp.n_super + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x));
  // u-th work item of this CTA; false if there is none at this position
  auto get_item = [&](int u, FaFwdItem& it) -> bool {
    // heavy block first: under a causal mask the late query blocks see the most keys
    int qb;
    if constexpr (SINGLE) {
      qb = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);
      it.bh = static_cast<int>(blockIdx.z);
      it.dv_off = static_cast<int>(blockIdx.y) * DV;
    } else {
      const int sidx = (u >> 1) * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
      if (sidx >= pp.n_super) return false;
      const int sl = fast_div(sidx, pp.by_npair);
      const int j = sidx - sl * npair;
      qb = (u & 1) ? j : pp.nqb - 1 - j;
      if ((u & 1) && qb == pp.nqb - 1 - j) return false;  // odd number of blocks: the middle one is alone
      it.bh = fast_div(sl, pp.by_ndv);
      it.dv_off = (sl - it.bh * pp.ndv) * DV;
    }
    it.m_base = qb * (BM * NQ);
    it.nmax = 0;
#pragma unroll
    for (int s = 0; s < NQ; ++s) {
      int n = nblk_all;
      if (p.causal) {
        const int last_col = it.m_base + s * BM + (BM - 1) + (p.Lkv - p.Lq);
        const int nc = last_col < 0 ? 0 : last_col / BN + 1;
        n = nc < n ? nc : n;
      }
      if (it.m_base + s * BM >= p.Lq) n = 0;  // tile entirely past the end of Q
      it.nblk[s] = n;
      it.nmax = n > it.nmax ? n : it.nmax;
    }
    return true;
  };

  // (a barrier per thread: one after another they cost a short call 0.2 us)
  static_assert(kBars <= 64, "set up by the first two warps");
  if (threadIdx.x < kBars) {
    uint64_t* bar = bars + threadIdx.x;
    const bool by_warps = (bar >= s_free && bar < s_free + NQ) || (bar >= p_full && bar < p_full + NQ) || bar >= o_free;
    mbar_init(bar, by_warps ? 4 : 1);
    if (threadIdx.x == 0) ab->flag = 0;
    fence_mbar_init();
  }
  if (warp == kSWarp) {
    tmem_alloc(tmem_base_slot, Lay::TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;

  if (warp >= kSWarp) {
    // 384 threads start with 168 registers each; the softmax threads take 208 (a 128-column score row), which
    // leaves this warpgroup 88: 256 x 208 + 128 x 88 = 384 x 168. (setmaxnreg.inc waits, with no limit, until the
    // registers it asks for have been released: the two numbers must add up to no more than the CTA was given.)
    static_assert(256 * 208 + 128 * 88 <= 384 * 168, "register split of the warpgroups");
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == kTmaWarp) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0) {
        bool ok = true;
        int t = 0;                 // ring items issued so far (all work items)
        int n_k = 0, n_v = 0;      // K and V tiles of them (event trace)
        int nq_loaded[NQ] = {0, 0};
        uint32_t k_loads = 0, v_loads = 0;   // bit per slot: odd number of K / V tiles so far; 16 bits higher: any
        auto load_q = [&](const FaFwdItem& it, int s) {
          if (it.nblk[s] == 0 || !ok) return;
          AB200_TR(3, n_k - 1, 4 + 2 * s);
          // the tile's buffer is free once the previous item's last S MMA of this tile has read it
          if (nq_loaded[s] > 0) ok = mbar_wait(&q_free[s], (nq_loaded[s] - 1) & 1, ab, kTagQFree);
          if (!ok) return;
          AB200_TR(3, n_k - 1, 5 + 2 * s);
          mbar_expect_tx(&q_full[s], Cfg::Q_TILE_BYTES);
#pragma unroll
          for (int c = 0; c < DQK / 64; ++c)
            tma_load_3d(sQ + s * Cfg::Q_TILE_BYTES + c * (BM * 128), &tmQ, &q_full[s], c * 64, it.m_base + s * BM, it.bh);
          ++nq_loaded[s];
        };
        auto slot_free = [&]() -> uint8_t* {
          const int slot = t % NSTAGE;
          const int use = t / NSTAGE;
          if (ok && use > 0) ok = mbar_wait(&kv_empty[slot], (use - 1) & 1, ab, kTagKvEmpty);
          return sKV + slot * Cfg::KV_SLOT_BYTES;
        };
        auto load_k = [&](const FaFwdItem& it, int j) {
          uint8_t* dst = slot_free();
          if (!ok) return;
          AB200_TR(3, n_k, 1);
          uint64_t* bar = &k_full[t % NSTAGE];
          k_loads = (k_loads ^ (1u << (t % NSTAGE))) | (0x10000u << (t % NSTAGE));
          mbar_expect_tx(bar, Cfg::K_TILE_BYTES);
#pragma unroll
          for (int c = 0; c < DQK / 64; ++c) tma_load_3d(dst + c * (BN * 128), &tmK, bar, c * 64, j * BN, it.bh);
          ++t;
          ++n_k;
        };
        auto load_v = [&](const FaFwdItem& it, int j) {
          uint8_t* dst = slot_free();
          if (!ok) return;
          AB200_TR(3, n_v, 3);
          uint64_t* bar = &v_full[t % NSTAGE];
          v_loads = (v_loads ^ (1u << (t % NSTAGE))) | (0x10000u << (t % NSTAGE));
          mbar_expect_tx(bar, Cfg::V_TILE_BYTES);
#pragma unroll
          for (int c = 0; c < DV / 64; ++c) tma_load_3d(dst + c * (BN * 128), &tmV, bar, it.dv_off + c * 64, j * BN, it.bh);
          ++t;
          ++n_v;
        };
        for (int u = 0; u < n_steps && ok; ++u) {
          FaFwdItem it;
          if (!get_item(u, it) || it.nmax == 0) continue;
          for (int j = 0; j <= it.nmax && ok; ++j) {
            if (j < it.nmax) load_k(it, j);
            if (j > 0) {
              if (ok) load_v(it, j - 1);
            } else {
              for (int s = 0; s < NQ; ++s) load_q(it, s);
            }
          }
        }
        if (!ok) {
          // abort path: let the copies already issued land before this CTA's shared memory is released
          for (int s = 0; s < NQ; ++s)
            if (nq_loaded[s] > 0) mbar_wait_drain(&q_full[s], (nq_loaded[s] - 1) & 1, 2000000ull);
          for (int slot = 0; slot < NSTAGE; ++slot) {
            if ((k_loads >> (16 + slot)) & 1u) mbar_wait_drain(&k_full[slot], ~(k_loads >> slot) & 1u, 2000000ull);
            if ((v_loads >> (16 + slot)) & 1u) mbar_wait_drain(&v_full[slot], ~(v_loads >> slot) & 1u, 2000000ull);
          }
        }
      }
    } else if (warp == kSWarp) {
      // ------------------------------------------------------------------ S = Q K^T (converged warp, one elected lane)
      constexpr uint32_t idesc_qk = umma_idesc(BM, BN, BF16, false, false);
      const uint32_t q_desc = umma_desc_lo(smem_u32(sQ), 16), kv_desc = umma_desc_lo(smem_u32(sKV), 16);
      bool ok = true;
      int base = 0, r = 0;                  // ring slot of the work item's first entry; blocks so far
      uint32_t phases = 0;                  // bit per slot: phase of its next K tile
      int n_s = 0;                          // products so far
      int n_tile[NQ] = {0, 0};              // of either tile
      int n_items[NQ] = {0, 0};             // work items with at least one block, per tile, before the current one
      for (int u = 0; u < n_steps && ok; ++u) {
        FaFwdItem it;
        if (!get_item(u, it)) continue;
        int slot = base;  // of the block's K tile: entry 0 of the work item, then 2 j - 1
        for (int j = 0; j < it.nmax && ok; ++j) {
          ok = mbar_wait_warp(&k_full[slot], (phases >> slot) & 1u, ab, kTagKvFull);
          phases ^= 1u << slot;
          if (lane == 0) AB200_TR(2, r, 0);
          const uint32_t kd = kv_desc + ((slot * Cfg::KV_SLOT_BYTES) >> 4);
          const int last_user = it.nblk[1] > j ? 1 : 0;
#pragma unroll
          for (int s = 0; s < NQ; ++s) {
            if (it.nblk[s] <= j || !ok) continue;
            if (j == 0) ok = mbar_wait_warp(&q_full[s], n_items[s] & 1, ab, kTagQ);
            if (lane == 0) AB200_TR(2, r, 1 + 3 * s);
            // the buffer's scores are in the registers of the threads that read them last
            const int before = S_BUFS == 1 ? n_s : n_tile[s];
            if (ok && before > 0) ok = mbar_wait_warp(&s_free[S_BUFS == 1 ? 0 : s], (before - 1) & 1, ab, kTagSFree);
            // With a score buffer per tile nothing else holds the tiles apart, and once both softmaxes are in step each slows the
            // other's exponentials (event trace: 2070 -> 2290 cycles). Tile 1 starts a long item when tile 0 has written its first
            // P: 8 slices of L=4500 at d = 64 60 -> 58 us, persistent 20 of L=4000 206 -> 195. Short items lose that wait (100 of
            // L=700 causal 30.5 -> 31.2); without a mask they gain 2 % in the grid form from following tile 0's reads instead (200
            // of L=768 67.5 -> 64.5 us), but lose up to 5 % with one, and in the persistent form.
            if (S_BUFS == 2 && s == 1 && it.nblk[0] > j && ok) {
              if (it.nblk[0] >= 8) {
                if (j == 0) ok = mbar_wait_warp(&p_full[0], (n_tile[0] - 1) & 1, ab, kTagPFull);
              } else if (SINGLE && !p.causal) {
                ok = mbar_wait_warp(&s_free[0], (n_tile[0] - 1) & 1, ab, kTagSFree);
              }
            }
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) AB200_TR(2, r, 2 + 3 * s);
            const uint32_t qd = q_desc + ((s * Cfg::Q_TILE_BYTES) >> 4);
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < DQK / 16; ++ks) {
                const uint32_t off = ((ks >> 2) * (BM * 128) + (ks & 3) * 32) >> 4;
                umma_ss(tmem_base + (S_BUFS == 1 ? 0 : s * 128), umma_desc(qd + off), umma_desc(kd + off), idesc_qk, ks > 0 ? 1u : 0u);
              }
              tc_commit(&s_full[s]);
              if (s == last_user) tc_commit(&kv_empty[slot]);
              if (j + 1 == it.nblk[s]) tc_commit(&q_free[s]);
            }
            __syncwarp();
            if (lane == 0) AB200_TR(2, r, 3 + 3 * s);
            ++n_s;
            ++n_tile[s];
          }
          slot += j == 0 ? 1 : 2;
          ++r;
          if (slot >= NSTAGE) slot -= NSTAGE;
        }
        base = (base + 2 * it.nmax) % NSTAGE;
#pragma unroll
        for (int s = 0; s < NQ; ++s)
          if (it.nblk[s] > 0) ++n_items[s];
      }
    } else if (warp == kPvWarp) {
      // ------------------------------------------------------------------ O += P V (converged warp, one elected lane)
      constexpr uint32_t idesc_pv = umma_idesc(BM, DV, BF16, false, true);
      const uint32_t kv_desc = umma_desc_lo(smem_u32(sKV), BN * 128);
      bool ok = true;
      int base = 0;           // ring slot of the work item's first entry
      uint32_t phases = 0;    // bit per slot: phase of its next V tile
      int n_tile[NQ] = {0, 0}, n_items[NQ] = {0, 0}, r = 0;
      for (int u = 0; u < n_steps && ok; ++u) {
        FaFwdItem it;
        if (!get_item(u, it)) continue;
        int slot = (base + (it.nmax > 1 ? 2 : 1)) % NSTAGE;  // of the block's V tile: entry 2 j + 2, the last one 2 nmax - 1
        for (int j = 0; j < it.nmax && ok; ++j) {
          ok = mbar_wait_warp(&v_full[slot], (phases >> slot) & 1u, ab, kTagKvFull);
          phases ^= 1u << slot;
          if (lane == 0) AB200_TR(4, r, 0);
          const uint32_t vd = kv_desc + ((slot * Cfg::KV_SLOT_BYTES) >> 4);
          const int last_user = it.nblk[1] > j ? 1 : 0;
#pragma unroll
          for (int s = 0; s < NQ; ++s) {
            if (it.nblk[s] <= j || !ok) continue;
            // the first P V of an item overwrites O: the previous item's epilogue must have read it
            if (j == 0 && n_items[s] > 0) ok = mbar_wait_warp(&o_free[s], (n_items[s] - 1) & 1, ab, kTagOFree);
            if (ok) ok = mbar_wait_warp(&p_full[s], n_tile[s] & 1, ab, kTagPFull);
            if (!ok) break;
            tc_fence_after();
            if (lane == 0) AB200_TR(4, r, 1 + 2 * s);
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < BN / 16; ++ks)
                umma_ts(tmem_base + Lay::O_COL + s * DV, tmem_base + Lay::P_COL + s * 64 + ks * 8, umma_desc(vd + ((ks * 2048) >> 4)),
                        idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
              tc_commit(&o_done[s]);
              if (s == last_user) tc_commit(&kv_empty[slot]);
            }
            __syncwarp();
            if (lane == 0) AB200_TR(4, r, 2 + 2 * s);
            ++n_tile[s];
          }
          ++r;
          slot += j + 2 < it.nmax ? 2 : 1;
          if (slot >= NSTAGE) slot -= NSTAGE;
        }
        base = (base + 2 * it.nmax) % NSTAGE;
#pragma unroll
        for (int s = 0; s < NQ; ++s)
          if (it.nblk[s] > 0) ++n_items[s];
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int s = warp >> 2;                    // query tile of this warpgroup
    const int row_in_tile = threadIdx.x & 127;  // TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32);
    const uint32_t tS = tmem_addr(tmem_base, lane_base, S_BUFS == 1 ? 0 : s * 128);
    const uint32_t tP = tmem_addr(tmem_base, lane_base, Lay::P_COL + s * 64);
    const uint32_t tO = tmem_addr(tmem_base, lane_base, Lay::O_COL + s * DV);
    uint64_t* my_s_free = &s_free[S_BUFS == 1 ? 0 : s];
    const int causal_shift = p.Lkv - p.Lq;
    bool ok = true;
    int cs = 0;  // blocks of this tile in the work items before the current one (phase base of s_full / o_done)
    for (int u = 0; u < n_steps && ok; ++u) {
      FaFwdItem it;
      if (!get_item(u, it)) continue;
      const int n_my = s == 0 ? it.nblk[0] : it.nblk[1];  // (a select: indexing by s would put the item in local memory)
      const int row = it.m_base + s * BM + row_in_tile;
      const int m_tile = it.m_base + s * BM;
      auto out_row = [&](const FaFwdItem& of) -> uint16_t* {
        return reinterpret_cast<uint16_t*>(p.o) + (static_cast<size_t>(of.bh) * p.Lq + row) * p.dv_total + of.dv_off;
      };
      auto lse_row = [&](const FaFwdItem& of) -> float* {
        return (p.lse != nullptr && of.dv_off == 0) ? p.lse + static_cast<size_t>(of.bh) * p.Lq + row : nullptr;
      };
      if (n_my == 0) {
        // no visible key at all for this tile (causal with Lkv < Lq), or the tile lies past the end of Q
        if (row < p.Lq) {
          uint16_t* orow = out_row(it);
          const uint32_t zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
          for (int c = 0; c < DV; c += 16) st_global_v8(orow + c, zero);
          if (float* l = lse_row(it)) *l = -INFINITY;
        }
        continue;
      }
      float m_ref = -INFINITY;  // reference maximum (raw score units) the exponentials are taken against
      float l_sum = 0.f;        // running sum of exp
      for (int j = 0; j < n_my; ++j) {
        if (row_in_tile == 0) AB200_TR(s, cs + j, 0);
        ok = mbar_wait_warp(&s_full[s], (cs + j) & 1, ab, kTagSFull);
        if (!ok) break;
        if (row_in_tile == 0) AB200_TR(s, cs + j, 1);
        tc_fence_after();
        float sv[BN];
        {
          uint32_t* r = reinterpret_cast<uint32_t*>(sv);
          tmem_ld32(tS + 0, r + 0);
          tmem_ld32(tS + 32, r + 32);
          tmem_ld32(tS + 64, r + 64);
          tmem_ld32(tS + 96, r + 96);
          tc_wait_ld();
        }
        // the scores are in registers: the next product may overwrite their buffer
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(my_s_free);
        if (row_in_tile == 0) AB200_TR(s, cs + j, 2);
        const int n0 = j * BN;
        // masking: keys past Lkv (ragged tail) and, under causal, keys j > i + shift
        const bool tail_blk = (n0 + BN > p.Lkv);
        const bool diag_blk = p.causal && (n0 + BN - 1 > m_tile + causal_shift);
        if (tail_blk || diag_blk) {
          int limit = p.Lkv - n0;  // columns [limit, BN) are masked
          if (p.causal) {
            const int cl = row + causal_shift - n0 + 1;
            limit = cl < limit ? cl : limit;
          }
#pragma unroll
          for (int c = 0; c < BN; ++c)
            if (c >= limit) sv[c] = -INFINITY;
        }
        // row maximum: four independent chains of three-input maxima
        float mA = sv[0], mB = sv[1], mC = sv[2], mD = sv[3];
#pragma unroll
        for (int c = 4; c < BN - 4; c += 8) {
          mA = fmax3(mA, sv[c], sv[c + 1]);
          mB = fmax3(mB, sv[c + 2], sv[c + 3]);
          mC = fmax3(mC, sv[c + 4], sv[c + 5]);
          mD = fmax3(mD, sv[c + 6], sv[c + 7]);
        }
        mA = fmax3(mA, sv[BN - 4], sv[BN - 3]);
        mB = fmax3(mB, sv[BN - 2], sv[BN - 1]);
        const float m_blk = fmaxf(fmaxf(mA, mB), fmaxf(mC, mD));

        // P V of this tile's previous block: O may be rescaled, and P overwritten, once it is complete
        if (j > 0) {
          ok = mbar_wait_warp(&o_done[s], (cs + j - 1) & 1, ab, kTagODone);
          if (!ok) break;
          tc_fence_after();
        }
        if (row_in_tile == 0) AB200_TR(s, cs + j, 3);
        // Lazy rescale: keep the old reference unless the maximum grew by more than 2^8 in the exp2 domain.
        bool need = (j == 0) || ((m_blk - m_ref) * p.scale_log2 > Cfg::RESCALE_LOG2);
        if (m_blk == -INFINITY) need = false;
        if (__any_sync(0xffffffffu, need)) {
          float alpha = 1.0f;
          if (need) {
            alpha = (m_ref == -INFINITY) ? 0.0f : ex2_approx((m_ref - m_blk) * p.scale_log2);
            m_ref = m_blk;
            l_sum *= alpha;
          }
          if (j > 0) {
#pragma unroll
            for (int c0 = 0; c0 < DV; c0 += 32) {
              uint32_t r[32];
              tmem_ld32(tO + c0, r);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st32(tO + c0, r);
            }
          }
        }
        const float neg_m = (m_ref == -INFINITY) ? 0.0f : -m_ref * p.scale_log2;
        // P = exp2(S * scale_log2 - m * scale_log2): packed FMA, MUFU ex2, four packed partial sums
        const uint64_t sl2 = f2_pack(p.scale_log2, p.scale_log2);
        const uint64_t nm2 = f2_pack(neg_m, neg_m);
        uint64_t acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t pk[BN / 4];
#pragma unroll
          for (int c = 0; c < BN / 2; c += 2) {
            const int cc = h * (BN / 2) + c;
            float x0, x1;
            f2_unpack(ffma2(f2_pack(sv[cc], sv[cc + 1]), sl2, nm2), x0, x1);
            const float e0 = ex2_approx(x0), e1 = ex2_approx(x1);
            acc[(c >> 1) & 3] = fadd2(acc[(c >> 1) & 3], f2_pack(e0, e1));
            pk[c >> 1] = pack2<BF16>(e0, e1);
          }
          tmem_st32(tP + h * (BN / 4), pk);
        }
        {
          float a0, a1;
          f2_unpack(fadd2(fadd2(acc[0], acc[1]), fadd2(acc[2], acc[3])), a0, a1);
          l_sum += a0 + a1;
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[s]);
        if (row_in_tile == 0) AB200_TR(s, cs + j, 4);
      }
      if (!ok) break;
      // epilogue: O / l -> global, lse. O goes to registers first so that the next item's first P V may overwrite it.
      ok = mbar_wait_warp(&o_done[s], (cs + n_my - 1) & 1, ab, kTagODone);
      if (!ok) break;
      tc_fence_after();
      if (row_in_tile == 0) AB200_TR(s, cs + n_my - 1, 5);
      const float inv_l = l_sum > 0.f ? 1.0f / l_sum : 0.f;
      FaFwdItem io;  // decoded again (persistent form): only the tile's row and block count stay live across the block loop
      get_item(u, io);
      {
        uint32_t r[DV];
#pragma unroll
        for (int c0 = 0; c0 < DV; c0 += 32) tmem_ld32(tO + c0, r + c0);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_free[s]);
        if (row_in_tile == 0) AB200_TR(s, cs + n_my - 1, 6);
        if constexpr (STAGE_O) {
#pragma unroll
          for (int b0 = 0; b0 < DV / 64; b0 += Lay::STAGE_BOXES) {
            // this warp's earlier stores must have read the staging rows before they are written again
            if (lane == 0) tma_store_wait_read0();
            __syncwarp();
            uint8_t* stage = sO + s * Lay::O_STAGE_BYTES + row_in_tile * 128;
#pragma unroll
            for (int i = b0 * 64; i < (b0 + Lay::STAGE_BOXES) * 64; i += 8) {
              uint4 v;
              v.x = pack2<BF16>(__uint_as_float(r[i + 0]) * inv_l, __uint_as_float(r[i + 1]) * inv_l);
              v.y = pack2<BF16>(__uint_as_float(r[i + 2]) * inv_l, __uint_as_float(r[i + 3]) * inv_l);
              v.z = pack2<BF16>(__uint_as_float(r[i + 4]) * inv_l, __uint_as_float(r[i + 5]) * inv_l);
              v.w = pack2<BF16>(__uint_as_float(r[i + 6]) * inv_l, __uint_as_float(r[i + 7]) * inv_l);
              const int chunk16 = (i & 63) >> 3;
              *reinterpret_cast<uint4*>(stage + ((i >> 6) - b0) * Lay::O_BOX_BYTES + ((chunk16 ^ (row_in_tile & 7)) << 4)) = v;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const int row0 = m_tile + (warp & 3) * 32;
              if (row0 < p.Lq) {  // rows past the end of Q are clipped by the store
#pragma unroll
                for (int b = 0; b < Lay::STAGE_BOXES; ++b)
                  tma_store_3d(&tmO, sO + s * Lay::O_STAGE_BYTES + b * Lay::O_BOX_BYTES + (warp & 3) * (32 * 128),
                               io.dv_off + (b0 + b) * 64, row0, io.bh);
                tma_store_commit();
              }
            }
          }
        } else if (row < p.Lq) {
          uint16_t* orow = out_row(io);
#pragma unroll
          for (int i = 0; i < DV; i += 16) {
            uint32_t v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
              v[e] = pack2<BF16>(__uint_as_float(r[i + 2 * e]) * inv_l, __uint_as_float(r[i + 2 * e + 1]) * inv_l);
            st_global_v8(orow + i, v);
          }
        }
      }
      if (row < p.Lq)
        if (float* l = lse_row(io)) *l = (l_sum > 0.f) ? (m_ref * p.scale + __logf(l_sum)) : -INFINITY;
      if (row_in_tile == 0) AB200_TR(s, cs + n_my - 1, 7);
      cs += n_my;
    }
    if (STAGE_O && lane == 0) tma_store_wait0();  // all output written before the CTA's shared memory is released
  }

  // common tail: every role gets here, also after an aborted wait
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == kSWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Lay::TMEM_COLS);
  }
}

}  // namespace ab200
