// flash-attention forward for a handful of query rows (decoding: up to 16 new positions against a long K / V cache).
//
// What bounds it: reading K and V once. A key costs 64 d FLOP with 16 rows and 4 d bytes, 16 FLOP per byte of K and V, a
// sixteenth of what the tensor cores need to be the limit (1640 TFLOP/s over 6.53 TB/s), so the tile of 128 query rows of fa_fwd_sm100.cuh does nothing but fetch: one CTA per (batch, head) slice,
// one block of 128 keys (64 KB) per 1.8 us of serial S -> softmax -> P V chain. Here
//   * the keys of a slice are split over the CTAs of a thread-block cluster (1, 4 or 8, by the number of keys); each keeps its own maximum, sum and accumulator, and the cluster combines them through
//     distributed shared memory at the end: one launch, no scratch memory;
//   * a CTA streams blocks of 64 keys (128 at d = 64; K and V together, 32 KB) by TMA through a ring of three, two CTAs
//     per SM: 192 KB on the way per SM;
//   * each of four warps takes a quarter of a block's keys on its own (mma.sync m16n8k16: the query rows are the 16 rows of the
//     tile, where a tcgen05 tile would pad them to 128 and need two trips through tensor memory); the warps meet again
//     only after the last block.
// Same arithmetic as the large tiles: fp32 scores, maxima, sums and accumulators, P rounded to the storage type.
//
// Measured (B200, bf16, causal, cold caches, against the 256-row tile of one CTA per slice): BH = 32, Lq = 1, Lkv = 16384,
// d = 128: 45 us = 5.95 TB/s against 230 us; d = 64: 26.5 us. BH = 1, Lkv = 32768, d = 128: 33 us against 450.
// BH = 256, Lkv = 4096, d = 128: 83 us = 6.5 TB/s. Distance to 64-bit results 2.5e-4 / 2.1e-3 (fp16 / bf16, 2-norm), the
// large tile 2.9e-4 / 2.4e-3: its running maximum may lag by 2^8, this one's does not.
#pragma once

#include "fa_fwd_sm100.cuh"
#include "ptx_pair.cuh"

namespace ab200 {

enum FaDecodeTag : int { kTagDecFull = 81, kTagDecEmpty = 82 };

template <int D_, bool BF16_>
struct FaDecodeConfig {
  static constexpr int D = D_;
  static constexpr bool BF16 = BF16_;
  static constexpr int MAX_ROWS = 16;
  static constexpr int NWARPS = 4;            // consumers
  static constexpr int KT = D == 128 ? 1 : 2;  // groups of 16 keys per warp and block: 32 KB of K and V per block
  static constexpr int BN = 16 * KT * NWARPS;  // keys per block
  static constexpr int NSTAGE = 3;
  static constexpr int NTHREADS = 32 * NWARPS + 32;
  static constexpr int TILE_BYTES = BN * D * 2;  // one K or V tile
  static constexpr int RING_BYTES = NSTAGE * 2 * TILE_BYTES;
  // after the last block the ring holds the warps' partial rows, then the CTA's: [NWARPS][16][D] and [16][D] floats
  static constexpr int PART_BYTES = (NWARPS + 1) * MAX_ROWS * D * 4;
  static_assert(PART_BYTES <= RING_BYTES, "the partial results live in the ring");
  static constexpr int SMEM_BYTES = RING_BYTES + 1024 + 256 + 2 * (NWARPS + 1) * MAX_ROWS * 4;
  static_assert(D == 64 || D == 128, "head dimension");
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// C[16x8] += A[16x16] * B[16x8], fp32 accumulator.
template <bool BF16>
__device__ __forceinline__ void mma_m16n8k16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if constexpr (BF16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

// grid (cluster size, 1, BH), cluster (cluster size, 1, 1): CTA x of a slice takes every cluster-size-th share of the blocks.
template <class Cfg>
__global__ void __launch_bounds__(Cfg::NTHREADS, 2)
fa_decode_sm100_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const void* q_ptr,
                       const FaFwdParams p) {
  constexpr int D = Cfg::D, BN = Cfg::BN, KT = Cfg::KT, NSTAGE = Cfg::NSTAGE, NW = Cfg::NWARPS, ROWS = Cfg::MAX_ROWS;
  constexpr bool BF16 = Cfg::BF16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES);  // [NSTAGE]
  uint64_t* empty = full + NSTAGE;                                       // [NSTAGE]
  CtaAbort* ab = reinterpret_cast<CtaAbort*>(empty + NSTAGE);
  float* part_o = reinterpret_cast<float*>(smem);                                      // [NW + 1][ROWS][D]
  float* part_m = reinterpret_cast<float*>(smem + Cfg::RING_BYTES + 256);              // [NW + 1][ROWS], exp2 units
  float* part_l = part_m + (NW + 1) * ROWS;                                            // [NW + 1][ROWS]

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int bh = blockIdx.z;
  const int nsplit = gridDim.x;
  const int nblk = (p.Lkv + BN - 1) / BN;
  const int b0 = static_cast<int>(static_cast<long long>(nblk) * blockIdx.x / nsplit);
  const int b1 = static_cast<int>(static_cast<long long>(nblk) * (blockIdx.x + 1) / nsplit);

  if (threadIdx.x == 0) {
    for (int i = 0; i < NSTAGE; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], NW);
    }
    ab->flag = 0;
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == NW) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      bool ok = true;
      int t = 0;
      for (int b = b0; b < b1; ++b, ++t) {
        const int slot = t % NSTAGE, use = t / NSTAGE;
        if (use > 0) ok = mbar_wait(&empty[slot], (use - 1) & 1, ab, kTagDecEmpty);
        if (!ok) break;
        uint8_t* dk = smem + slot * 2 * Cfg::TILE_BYTES;
        mbar_expect_tx(&full[slot], 2 * Cfg::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) tma_load_3d(dk + c * (BN * 128), &tmK, &full[slot], c * 64, b * BN, bh);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_3d(dk + Cfg::TILE_BYTES + c * (BN * 128), &tmV, &full[slot], c * 64, b * BN, bh);
      }
      if (!ok) {  // abort path: let the copies already issued land before this CTA's shared memory is released
        for (int slot = 0; slot < NSTAGE; ++slot)
          if (t > slot) mbar_wait_drain(&full[slot], ((t - 1 - slot) / NSTAGE) & 1, 2000000ull);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ consumers: warp w owns keys [16 KT w, 16 KT (w + 1))
    const int g = lane >> 2, t4 = lane & 3;
    uint32_t qa[D / 16][4];  // A fragments of Q: rows g and g + 8
    {
      const uint32_t* qrow = reinterpret_cast<const uint32_t*>(q_ptr) + static_cast<size_t>(bh) * p.Lq * (D / 2);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const int c = ks * 8 + t4;
        qa[ks][0] = g < p.Lq ? qrow[g * (D / 2) + c] : 0u;
        qa[ks][1] = g + 8 < p.Lq ? qrow[(g + 8) * (D / 2) + c] : 0u;
        qa[ks][2] = g < p.Lq ? qrow[g * (D / 2) + c + 4] : 0u;
        qa[ks][3] = g + 8 < p.Lq ? qrow[(g + 8) * (D / 2) + c + 4] : 0u;
      }
    }
    float oacc[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) oacc[n][i] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY;  // running maxima of rows g, g + 8, raw score units
    float l0 = 0.f, l1 = 0.f;              // this lane's share of the row sums
    // keys row i may see: [0, limit_i)
    const int lim0 = p.causal ? min(p.Lkv, g + p.Lkv - p.Lq + 1) : p.Lkv;
    const int lim1 = p.causal ? min(p.Lkv, g + 8 + p.Lkv - p.Lq + 1) : p.Lkv;
    const int lim_all = p.causal ? p.Lkv - p.Lq + 1 : p.Lkv;  // keys every row sees
    const uint32_t ring = smem_u32(smem);
    // ldmatrix row and 16-byte chunk of this lane: K as is (keys x d), V transposed (d x keys)
    const int k_row = warp * 16 * KT + (lane & 7) + ((lane >> 4) & 1) * 8, k_chunk = (lane >> 3) & 1;
    const int v_row = warp * 16 * KT + (lane & 7) + ((lane >> 3) & 1) * 8, v_chunk = lane >> 4;
    bool ok = true;
    for (int b = b0, t = 0; b < b1; ++b, ++t) {
      const int slot = t % NSTAGE;
      ok = mbar_wait_warp(&full[slot], (t / NSTAGE) & 1, ab, kTagDecFull);
      if (!ok) break;
      const uint32_t sk = ring + slot * 2 * Cfg::TILE_BYTES, sv = sk + Cfg::TILE_BYTES;
      // S = Q K^T, two accumulator chains per tile of eight keys where there are only two such tiles
      constexpr int NC = KT == 1 ? 2 : 1;
      float sc[NC][2 * KT][4] = {};
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const int chunk = (ks & 3) * 2 + k_chunk;
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
          uint32_t kb[4];
          ldmatrix_x4(sk + (ks >> 2) * (BN * 128) + (kt * 16 + k_row) * 128 + ((chunk ^ (k_row & 7)) << 4), kb);
          mma_m16n8k16<BF16>(sc[ks % NC][2 * kt], qa[ks], kb[0], kb[1]);
          mma_m16n8k16<BF16>(sc[ks % NC][2 * kt + 1], qa[ks], kb[2], kb[3]);
        }
      }
      float(&s)[2 * KT][4] = sc[0];
      if constexpr (NC == 2) {
#pragma unroll
        for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[n][i] += sc[NC - 1][n][i];
      }
      const int key0 = b * BN + warp * 16 * KT;
      if (key0 + 16 * KT > lim_all) {
#pragma unroll
        for (int n = 0; n < 2 * KT; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (key0 + n * 8 + 2 * t4 + (i & 1) >= (i < 2 ? lim0 : lim1)) s[n][i] = -INFINITY;
      }
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int n = 0; n < 2 * KT; ++n) {
        mx0 = fmax3(mx0, s[n][0], s[n][1]);
        mx1 = fmax3(mx1, s[n][2], s[n][3]);
      }
#pragma unroll
      for (int d = 1; d < 4; d <<= 1) {
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, d));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, d));
      }
      if (__any_sync(0xffffffffu, mx0 > m0 || mx1 > m1)) {
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
        const float a0 = m0 == -INFINITY ? 0.f : ex2_approx((m0 - n0) * p.scale_log2);
        const float a1 = m1 == -INFINITY ? 0.f : ex2_approx((m1 - n1) * p.scale_log2);
        m0 = n0;
        m1 = n1;
        l0 *= a0;
        l1 *= a1;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {
          oacc[n][0] *= a0;
          oacc[n][1] *= a0;
          oacc[n][2] *= a1;
          oacc[n][3] *= a1;
        }
      }
      const float c0 = m0 == -INFINITY ? 0.f : -m0 * p.scale_log2, c1 = m1 == -INFINITY ? 0.f : -m1 * p.scale_log2;
#pragma unroll
      for (int kt = 0; kt < KT; ++kt) {
        float e[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) e[n][i] = ex2_approx(fmaf(s[2 * kt + n][i], p.scale_log2, i < 2 ? c0 : c1));
        l0 += (e[0][0] + e[0][1]) + (e[1][0] + e[1][1]);
        l1 += (e[0][2] + e[0][3]) + (e[1][2] + e[1][3]);
        const uint32_t pa[4] = {pack2<BF16>(e[0][0], e[0][1]), pack2<BF16>(e[0][2], e[0][3]), pack2<BF16>(e[1][0], e[1][1]),
                                pack2<BF16>(e[1][2], e[1][3])};
        // O += P V
#pragma unroll
        for (int n2 = 0; n2 < D / 16; ++n2) {
          const int chunk = (n2 & 3) * 2 + v_chunk;
          uint32_t vb[4];
          ldmatrix_x4_trans(sv + (n2 >> 2) * (BN * 128) + (kt * 16 + v_row) * 128 + ((chunk ^ (v_row & 7)) << 4), vb);
          mma_m16n8k16<BF16>(oacc[2 * n2], pa, vb[0], vb[1]);
          mma_m16n8k16<BF16>(oacc[2 * n2 + 1], pa, vb[2], vb[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[slot]);
    }
    // the four lanes of a row add their sums; maxima in exp2 units from here on
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, d);
      l1 += __shfl_xor_sync(0xffffffffu, l1, d);
    }
    // every consumer has read its last block before the ring is written
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
    if (t4 == 0) {
      part_m[warp * ROWS + g] = m0 * p.scale_log2;
      part_m[warp * ROWS + g + 8] = m1 * p.scale_log2;
      part_l[warp * ROWS + g] = l0;
      part_l[warp * ROWS + g + 8] = l1;
    }
    float* po = part_o + warp * ROWS * D;
#pragma unroll
    for (int n = 0; n < D / 8; ++n) {
      if (g < p.Lq) *reinterpret_cast<float2*>(po + g * D + n * 8 + 2 * t4) = make_float2(oacc[n][0], oacc[n][1]);
      if (g + 8 < p.Lq) *reinterpret_cast<float2*>(po + (g + 8) * D + n * 8 + 2 * t4) = make_float2(oacc[n][2], oacc[n][3]);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
    // the CTA's rows: the four warps' partial results on the common maximum
    for (int i = threadIdx.x; i < p.Lq * D; i += 32 * NW) {
      const int r = i / D;
      float m = part_m[r];
#pragma unroll
      for (int w = 1; w < NW; ++w) m = fmaxf(m, part_m[w * ROWS + r]);
      float acc = 0.f, l = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float f = m == -INFINITY ? 0.f : ex2_approx(part_m[w * ROWS + r] - m);
        acc = fmaf(f, part_o[w * ROWS * D + i], acc);
        l = fmaf(f, part_l[w * ROWS + r], l);
      }
      part_o[NW * ROWS * D + i] = acc;
      if (i % D == 0) {
        part_m[NW * ROWS + r] = m;
        part_l[NW * ROWS + r] = l;
      }
    }
  }

  // the slice's rows: the cluster's partial results, every CTA a share of the columns. All threads of all CTAs get here,
  // also after an aborted wait, so the two cluster barriers always complete.
  __syncwarp();
  cluster_sync();
  {
    const uint32_t a_o = smem_u32(part_o + NW * ROWS * D), a_m = smem_u32(part_m + NW * ROWS), a_l = smem_u32(part_l + NW * ROWS);
    const int npairs = p.Lq * (D / 2);
    for (int i = blockIdx.x * Cfg::NTHREADS + threadIdx.x; i < npairs; i += nsplit * Cfg::NTHREADS) {
      const int r = i / (D / 2);
      float m = -INFINITY;
      for (int c = 0; c < nsplit; ++c) m = fmaxf(m, ld_shared_cluster_f32(mapa_shared(a_m + 4 * r, c)));
      float x = 0.f, y = 0.f, l = 0.f;
      for (int c = 0; c < nsplit; ++c) {
        const float mc = ld_shared_cluster_f32(mapa_shared(a_m + 4 * r, c));
        const float f = m == -INFINITY ? 0.f : ex2_approx(mc - m);
        const uint32_t src = mapa_shared(a_o + 8 * i, c);
        x = fmaf(f, ld_shared_cluster_f32(src), x);
        y = fmaf(f, ld_shared_cluster_f32(src + 4), y);
        l = fmaf(f, ld_shared_cluster_f32(mapa_shared(a_l + 4 * r, c)), l);
      }
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      const size_t row = static_cast<size_t>(bh) * p.Lq + r;
      reinterpret_cast<uint32_t*>(p.o)[row * (D / 2) + (i % (D / 2))] = pack2<BF16>(x * inv, y * inv);
      if (p.lse != nullptr && i % (D / 2) == 0) p.lse[row] = l > 0.f ? m * 0.6931471805599453f + __logf(l) : -INFINITY;
    }
  }
  cluster_sync();  // no CTA leaves while another may still read its shared memory
}

}  // namespace ab200
