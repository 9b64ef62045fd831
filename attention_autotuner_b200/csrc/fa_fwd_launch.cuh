// Host launcher for fa_fwd_sm100_kernel: argument checks, tensor maps, grid, timing loop.
// Plays the role of the reference's generated launch shims
// (csrc/kernels/attention/regfuse/profile_code.py:28-76: profile() and kernel_entry()).
#pragma once

#include <math.h>

#include <stdlib.h>

#include "fa_decode_sm100.cuh"
#include "fa_fwd_form.cuh"
#include "fa_fwd_pair_sm100.cuh"
#include "fa_fwd_persist_sm100.cuh"
#include "fa_fwd_sm100.cuh"
#include "host_common.cuh"

namespace ab200 {

struct FaFwdArgs {
  const void* q;  // [BH, Lq, dqk]
  const void* k;  // [BH, Lkv, dqk]
  const void* v;  // [BH, Lkv, dv]
  void* o;        // [BH, Lq, dv]
  float* lse;     // [BH, Lq] or nullptr
  int BH, Lq, Lkv, dv;
  float scale;
  int causal;
};

// The default tile (two query tiles, up to 128 V columns, no softmax variant) is fa_fwd_persist_sm100.cuh's, in two forms of the
// grid with the same bits.
template <class Cfg>
constexpr bool fa_fwd_default_tile() {
  return Cfg::NQ == 2 && Cfg::SPLIT == 1 && Cfg::NMMA == 1 && Cfg::EXP_EMU == 0 && Cfg::EXP_H2 == 0 && Cfg::DV <= 128 && Cfg::NSTAGE >= 2;
}
template <class Cfg, bool SINGLE = false>
int fa_fwd_persist_launch(const FaFwdArgs& a, cudaStream_t stream);

// Every other tile, and work items of very few blocks: a grid of one CTA per 128 * NQ query rows.
template <class Cfg>
int fa_fwd_variant_launch(const FaFwdArgs& a, cudaStream_t stream) {
  if (!a.q || !a.k || !a.v || !a.o) return fail(kErrInvalidArgument, "fa_fwd: null tensor pointer");
  if (a.BH <= 0 || a.Lq <= 0 || a.Lkv <= 0) return fail(kErrInvalidArgument, "fa_fwd: sizes must be positive");
  if (a.BH > 65535) return fail(kErrInvalidArgument, "fa_fwd: batch*heads %d exceeds 65535", a.BH);
  if (a.dv % Cfg::DV != 0) return fail(kErrUnsupported, "fa_fwd: dv %d is not a multiple of the tile's %d", a.dv, Cfg::DV);
  if (!(a.scale > 0.f) || !isfinite(a.scale)) return fail(kErrInvalidArgument, "fa_fwd: scale must be positive and finite");
  if (!aligned16(a.q) || !aligned16(a.k) || !aligned16(a.v) || !aligned32(a.o))
    return fail(kErrInvalidArgument, "fa_fwd: inputs must be 16-byte aligned and the output 32-byte aligned");

  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = check_prior_status("fa_fwd"))) return rc;
  if ((rc = bind_device_of(a.q, "fa_fwd"))) return rc;
  if ((rc = make_tmap_3d(&tq, a.q, Cfg::BF16, Cfg::DQK, a.Lq, a.BH, 64, Cfg::BM))) return rc;
  if ((rc = make_tmap_3d(&tk, a.k, Cfg::BF16, Cfg::DQK, a.Lkv, a.BH, 64, Cfg::BN))) return rc;
  if ((rc = make_tmap_3d(&tv, a.v, Cfg::BF16, a.dv, a.Lkv, a.BH, 64, Cfg::BN))) return rc;

  FaFwdParams p;
  p.o = a.o;
  p.lse = a.lse;
  p.dv_total = a.dv;
  p.Lq = a.Lq;
  p.Lkv = a.Lkv;
  p.causal = a.causal ? 1 : 0;
  p.scale = a.scale;
  p.scale_log2 = a.scale * 1.4426950408889634f;

  auto kernel = &fa_fwd_sm100_kernel<Cfg>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
  if (e != cudaSuccess) return fail(kErrCuda, "fa_fwd: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  dim3 grid((a.Lq + Cfg::BM * Cfg::NQ - 1) / (Cfg::BM * Cfg::NQ), a.dv / Cfg::DV, a.BH);
  kernel<<<grid, Cfg::NTHREADS, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, p);
  return check_launch("fa_fwd launch");
}

// The grid form of any tile. Items of one KV block (two where there is one query tile) have nothing to overlap and stay with
// the kernel whose P lies over S: it has fewer hand-offs. That kernel / the other in us, d = 64 where not stated: 2 slices of
// L=128 4.9 / 5.4, d=128 6.1 / 6.4, 100 of L=100 5.2 / 5.9, 4 of Lq=1000 Lkv=100 6.5 / 6.6, 1 of Lq=44 Lkv=255 6.4 / 6.7; with
// more blocks 16 of Lq=1024 Lkv=256 7.8 / 7.8, Lkv=384 9.5 / 9.2, 4 of L=256 d=128 9.3 / 8.7, 8 of L=512 11.1 / 10.6. Same bits.
template <class Cfg>
int fa_fwd_launch(const FaFwdArgs& a, cudaStream_t stream) {
  if constexpr (fa_fwd_default_tile<Cfg>()) {
    const bool few_blocks = a.Lkv <= Cfg::BN || (a.Lq <= Cfg::BM && a.Lkv <= 2 * Cfg::BN);
    if (!few_blocks) return fa_fwd_persist_launch<Cfg, true>(a, stream);
  }
  return fa_fwd_variant_launch<Cfg>(a, stream);
}

// ATTN_B200_FA_FWD_FORM in the environment overrides the choice between the two forms of the kernel for every shape
// they both cover: "grid" (one CTA per 256 query rows) or "persistent" (one CTA per SM walking a work list).
inline int fa_fwd_form_requested() {  // 0: automatic, 1: grid, 2: persistent
  const char* s = getenv("ATTN_B200_FA_FWD_FORM");
  if (s == nullptr) return 0;
  if (s[0] == 'g') return 1;
  if (s[0] == 'p') return 2;
  return 0;
}

inline int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return 148;
  return sms;
}

// Launcher of the default tile: one CTA per SM (fewer when there is less work) walking the work list, or one per work item.
template <class Cfg, bool SINGLE>
int fa_fwd_persist_launch(const FaFwdArgs& a, cudaStream_t stream) {
  if (!a.q || !a.k || !a.v || !a.o) return fail(kErrInvalidArgument, "fa_fwd: null tensor pointer");
  if (a.BH <= 0 || a.Lq <= 0 || a.Lkv <= 0) return fail(kErrInvalidArgument, "fa_fwd: sizes must be positive");
  if (a.BH > 65535) return fail(kErrInvalidArgument, "fa_fwd: batch*heads %d exceeds 65535", a.BH);
  if (a.dv % Cfg::DV != 0) return fail(kErrUnsupported, "fa_fwd: dv %d is not a multiple of the tile's %d", a.dv, Cfg::DV);
  if (!(a.scale > 0.f) || !isfinite(a.scale)) return fail(kErrInvalidArgument, "fa_fwd: scale must be positive and finite");
  if (!aligned16(a.q) || !aligned16(a.k) || !aligned16(a.v) || !aligned32(a.o))
    return fail(kErrInvalidArgument, "fa_fwd: inputs must be 16-byte aligned and the output 32-byte aligned");

  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = check_prior_status("fa_fwd"))) return rc;
  if ((rc = bind_device_of(a.q, "fa_fwd"))) return rc;
  if ((rc = make_tmap_3d(&tq, a.q, Cfg::BF16, Cfg::DQK, a.Lq, a.BH, 64, Cfg::BM))) return rc;
  if ((rc = make_tmap_3d(&tk, a.k, Cfg::BF16, Cfg::DQK, a.Lkv, a.BH, 64, Cfg::BN))) return rc;
  if ((rc = make_tmap_3d(&tv, a.v, Cfg::BF16, a.dv, a.Lkv, a.BH, 64, Cfg::BN))) return rc;
  CUtensorMap to = tv;  // stands in where the output is not staged
  using Lay = FaFwdPersistLayout<Cfg>;
  if (Lay::STAGE_O && (rc = make_tmap_3d(&to, a.o, Cfg::BF16, a.dv, a.Lq, a.BH, 64, 32))) return rc;  // a warp stores its 32 rows

  FaFwdPersistParams pp;
  pp.f.o = a.o;
  pp.f.lse = a.lse;
  pp.f.dv_total = a.dv;
  pp.f.Lq = a.Lq;
  pp.f.Lkv = a.Lkv;
  pp.f.causal = a.causal ? 1 : 0;
  pp.f.scale = a.scale;
  pp.f.scale_log2 = a.scale * 1.4426950408889634f;
  pp.nqb = (a.Lq + Cfg::BM * Cfg::NQ - 1) / (Cfg::BM * Cfg::NQ);
  pp.ndv = a.dv / Cfg::DV;
  const long long n_super = static_cast<long long>(a.BH) * pp.ndv * ((pp.nqb + 1) / 2);
  if (n_super > 0x3fffffffLL) return fail(kErrInvalidArgument, "fa_fwd: too many tiles");
  pp.n_super = static_cast<int>(n_super);
  pp.by_npair = make_fast_div((pp.nqb + 1) / 2);
  pp.by_ndv = make_fast_div(pp.ndv);

  auto kernel = &fa_fwd_persist_sm100_kernel<Cfg, SINGLE>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::SMEM_BYTES);
  if (e != cudaSuccess) return fail(kErrCuda, "fa_fwd: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const int sms = sm_count();
  const dim3 grid = SINGLE ? dim3(pp.nqb, pp.ndv, a.BH) : dim3(pp.n_super < sms ? pp.n_super : sms);
  kernel<<<grid, Cfg::NTHREADS, Lay::SMEM_BYTES, stream>>>(tq, tk, tv, to, pp);
  return check_launch("fa_fwd launch");
}

// Launcher of the decoding kernel (up to 16 query rows, head dimensions 64 and 128, the same for q, k and v).
// CTAs (a cluster) per slice are chosen by the number of blocks alone: the order in which a slice's partial results are
// added, and so its output to the last bit, must not depend on how many other slices are in the launch (sharding by slices
// gives the same bits on any number of ranks). Measured at d = 128, 1 / 4 / 8 CTAs: BH = 32, Lkv = 16384:
// 117 / 45.1 / 45.2 us; BH = 16, Lkv = 32768: 223 / 65 / 46.9; BH = 64, Lkv = 8192: 64.6 / 44.6 / 47.2; BH = 256, Lkv = 4096:
// 80.0 / 82.8 / 91; BH = 512, Lkv = 2048: 79.6 / 87 / 114, Lkv = 256: 18.5 / 36 / 70. Four lose little with many slices and
// win most of what there is with few; eight where a cache is long enough to hide the larger cluster.
inline int fa_decode_split(int nblk) { return nblk >= 256 ? 8 : nblk >= 32 ? 4 : 1; }

template <int D, bool BF16>
int fa_decode_launch(const FaFwdArgs& a, cudaStream_t stream) {
  using Cfg = FaDecodeConfig<D, BF16>;
  if (!a.q || !a.k || !a.v || !a.o) return fail(kErrInvalidArgument, "fa_fwd: null tensor pointer");
  if (a.BH <= 0 || a.Lq <= 0 || a.Lkv <= 0) return fail(kErrInvalidArgument, "fa_fwd: sizes must be positive");
  if (a.BH > 65535) return fail(kErrInvalidArgument, "fa_fwd: batch*heads %d exceeds 65535", a.BH);
  if (a.dv != D || a.Lq > Cfg::MAX_ROWS) return fail(kErrUnsupported, "fa_fwd: not a decoding shape");
  if (!(a.scale > 0.f) || !isfinite(a.scale)) return fail(kErrInvalidArgument, "fa_fwd: scale must be positive and finite");
  if (!aligned16(a.q) || !aligned16(a.k) || !aligned16(a.v) || !aligned32(a.o))
    return fail(kErrInvalidArgument, "fa_fwd: inputs must be 16-byte aligned and the output 32-byte aligned");
  CUtensorMap tk, tv;
  int rc;
  if ((rc = check_prior_status("fa_fwd"))) return rc;
  if ((rc = bind_device_of(a.q, "fa_fwd"))) return rc;
  if ((rc = make_tmap_3d(&tk, a.k, BF16, D, a.Lkv, a.BH, 64, Cfg::BN))) return rc;
  if ((rc = make_tmap_3d(&tv, a.v, BF16, D, a.Lkv, a.BH, 64, Cfg::BN))) return rc;
  FaFwdParams p;
  p.o = a.o;
  p.lse = a.lse;
  p.dv_total = D;
  p.Lq = a.Lq;
  p.Lkv = a.Lkv;
  p.causal = a.causal ? 1 : 0;
  p.scale = a.scale;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  auto kernel = &fa_decode_sm100_kernel<Cfg>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
  if (e != cudaSuccess) return fail(kErrCuda, "fa_fwd: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const int c = fa_decode_split((a.Lkv + Cfg::BN - 1) / Cfg::BN);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(c, 1, a.BH);
  cfg.blockDim = dim3(Cfg::NTHREADS, 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = c;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kernel, tk, tv, a.q, p);
  if (e != cudaSuccess) return fail(kErrCuda, "fa_fwd: %s", cudaGetErrorString(e));
  return check_launch("fa_fwd launch");
}

// What the persistent form saves lies at the boundaries of the work items. fa_fwd_form.cuh has the rule.
template <class Cfg>
bool fa_fwd_picks_persistent(const FaFwdArgs& a) {
  if constexpr (fa_fwd_default_tile<Cfg>()) {
    static_assert(Cfg::NQ * Cfg::BM == 256 && Cfg::BN == 128, "the rule's items and blocks");
    const int form = fa_fwd_form_requested();
    const long long slices = static_cast<long long>(a.BH) * (a.dv / Cfg::DV);
    return form == 2 || (form == 0 && fa_form_persistent(slices, a.Lq, a.Lkv, a.causal != 0, sm_count()));
  }
  return false;
}

template <class Cfg>
bool fa_fwd_is_decode(const FaFwdArgs& a) {
  return fa_decode_shape(Cfg::DQK, a.dv, a.Lq, a.Lkv) && fa_fwd_form_requested() == 0;
}

template <class Cfg>
int fa_fwd_launch_auto(const FaFwdArgs& a, cudaStream_t stream) {
  if constexpr (Cfg::DQK == 64 || Cfg::DQK == 128) {
    if (fa_fwd_is_decode<Cfg>(a)) return fa_decode_launch<Cfg::DQK, Cfg::BF16>(a, stream);
  }
  if constexpr (fa_fwd_default_tile<Cfg>()) {
    if (fa_fwd_picks_persistent<Cfg>(a)) return fa_fwd_persist_launch<Cfg>(a, stream);
  }
  return fa_fwd_launch<Cfg>(a, stream);
}

// Launcher of the CTA-pair kernel: clusters of two CTAs along x, each cluster a 512-row block of queries.
template <class Cfg>
int fa_fwd_pair_launch(const FaFwdArgs& a, cudaStream_t stream) {
  if (!a.q || !a.k || !a.v || !a.o) return fail(kErrInvalidArgument, "fa_fwd: null tensor pointer");
  if (a.BH <= 0 || a.Lq <= 0 || a.Lkv <= 0) return fail(kErrInvalidArgument, "fa_fwd: sizes must be positive");
  if (a.BH > 65535) return fail(kErrInvalidArgument, "fa_fwd: batch*heads %d exceeds 65535", a.BH);
  if (a.dv % Cfg::DV != 0) return fail(kErrUnsupported, "fa_fwd: dv %d is not a multiple of the tile's %d", a.dv, Cfg::DV);
  if (!(a.scale > 0.f) || !isfinite(a.scale)) return fail(kErrInvalidArgument, "fa_fwd: scale must be positive and finite");
  if (!aligned16(a.q) || !aligned16(a.k) || !aligned16(a.v) || !aligned32(a.o))
    return fail(kErrInvalidArgument, "fa_fwd: inputs must be 16-byte aligned and the output 32-byte aligned");

  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = check_prior_status("fa_fwd"))) return rc;
  if ((rc = bind_device_of(a.q, "fa_fwd"))) return rc;
  if ((rc = make_tmap_3d(&tq, a.q, Cfg::BF16, Cfg::DQK, a.Lq, a.BH, 64, Cfg::BM))) return rc;
  if ((rc = make_tmap_3d(&tk, a.k, Cfg::BF16, Cfg::DQK, a.Lkv, a.BH, 64, Cfg::BN / 2))) return rc;  // half of the keys
  if ((rc = make_tmap_3d(&tv, a.v, Cfg::BF16, a.dv, a.Lkv, a.BH, 64, Cfg::BN))) return rc;          // half of the columns

  FaFwdParams p;
  p.o = a.o;
  p.lse = a.lse;
  p.dv_total = a.dv;
  p.Lq = a.Lq;
  p.Lkv = a.Lkv;
  p.causal = a.causal ? 1 : 0;
  p.scale = a.scale;
  p.scale_log2 = a.scale * 1.4426950408889634f;

  auto kernel = &fa_fwd_pair_sm100_kernel<Cfg>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
  if (e != cudaSuccess) return fail(kErrCuda, "fa_fwd: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const int rows_per_pair = 2 * Cfg::BM * Cfg::NQ;
  dim3 grid(2 * ((a.Lq + rows_per_pair - 1) / rows_per_pair), a.dv / Cfg::DV, a.BH);
  kernel<<<grid, Cfg::NTHREADS, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, p);
  return check_launch("fa_fwd launch");
}

// One warm-up launch, then enough launches to fill about 100 ms; returns ms per launch, -1 on error.
template <class F>
float profile_loop(F&& launch_once, cudaStream_t stream) {
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return -1.f;
  float ms = -1.f;
  do {
    cudaEventRecord(e0, stream);
    if (launch_once() != kOk) break;
    if (cudaEventRecord(e1, stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) break;
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    int repeats = t > 0.f ? static_cast<int>(ceilf(100.0f / t)) : 100;
    if (repeats < 1) repeats = 1;
    if (repeats > 2000) repeats = 2000;
    cudaEventRecord(e0, stream);
    bool bad = false;
    for (int i = 0; i < repeats; ++i)
      if (launch_once() != kOk) { bad = true; break; }
    if (bad) break;
    if (cudaEventRecord(e1, stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) break;
    if (cudaGetLastError() != cudaSuccess) break;
    cudaEventElapsedTime(&t, e0, e1);
    int det = 0;
    if (read_device_status(1, &det) != 0) break;
    ms = t / repeats;
  } while (0);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return ms;
}

}  // namespace ab200
