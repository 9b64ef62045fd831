"""Attention forward with the KV blocks of a work item split over a cluster (FaFwdSplitConfig in csrc/fa_fwd_sm100.cuh):
cluster sizes 2, 4 and 8, uneven shares, tiles and rows that see nothing of a share, against the CPU fp32 oracle and the
unsplit form.

Tolerances as in test_gpu_attention.py: the arithmetic of a block is the same, the shares are combined in fp32."""
import pytest
import torch

from oracle import oracle
from test_gpu_attention import rand_qkv, run_capi

pytestmark = pytest.mark.gpu

DT = {"fp16": torch.float16, "bf16": torch.bfloat16}

# B, H, Lq, Lkv: 8 CTAs (2 items) over 8, 9 and 24 blocks; 4 over 5 blocks; 2 over 2 blocks; one tile of the two empty
# (Lq <= 128); a piece of a prompt against a longer cache; fewer keys than queries (rows that see nothing, causal)
SHAPES = [(1, 2, 256, 1024), (1, 1, 300, 1100), (1, 2, 219, 2964), (2, 8, 257, 600), (1, 40, 200, 256), (1, 4, 17, 1000),
          (1, 2, 600, 400), (1, 3, 1000, 1000)]


@pytest.mark.parametrize("dtype_name", ["fp16", "bf16"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dqk,dv", [(64, 64), (128, 128), (64, 128), (128, 64)])
def test_split_keys(lib, monkeypatch, dtype_name, causal, dqk, dv):
    for i, (B, H, Lq, Lkv) in enumerate(SHAPES):
        q, k, v = rand_qkv(200 + i, B, H, Lq, Lkv, dqk, dv, DT[dtype_name])
        o, lse = run_capi(lib, q, k, v, dqk ** -0.5, causal)
        oref, lref = oracle.attention_fwd(q, k, v, dqk ** -0.5, causal)
        fin = torch.isfinite(lref)
        oref = torch.where(fin[..., None], oref, torch.zeros(()))  # a row that sees no key: zeros
        st = oracle.error_stats(o, oref)
        assert oracle.within(st, dtype_name, scale_by_peak=True), ((B, H, Lq, Lkv), st)
        assert torch.equal(torch.isfinite(lse), fin) and (lse[fin] - lref[fin]).abs().max().item() < 1e-3
        monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", "grid")
        o2, _ = run_capi(lib, q, k, v, dqk ** -0.5, causal)
        monkeypatch.delenv("ATTN_B200_FA_FWD_FORM")
        # two roundings of P and one of O apart, relative to the peak
        assert (o.float() - o2.float()).abs().max().item() <= (4 if dtype_name == "fp16" else 32) * 2.0 ** -10 * max(1.0, o2.abs().max().item())


def test_growing_peaks_and_a_share_far_below_the_others(lib):
    """The maximum of one share decides every weight: shares whose scores lie 100 units below contribute nothing, and a
    share of all-equal scores its mean."""
    q, k, v = rand_qkv(9, 1, 2, 200, 2048, 128, 128, torch.float16)
    k = k * torch.cat([torch.full((1024,), 0.01), torch.linspace(0.1, 4.0, 1024)]).half()[None, None, :, None]
    for kk in (k, k.flip(2)):
        o, lse = run_capi(lib, q, kk, v, 128 ** -0.5, False)
        oref, lref = oracle.attention_fwd(q, kk, v, 128 ** -0.5, False)
        assert oracle.within(oracle.error_stats(o, oref), "fp16", scale_by_peak=True)
        assert (lse - lref).abs().max().item() < 1e-3
