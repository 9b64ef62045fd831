"""Attention forward, work items of one KV block (two with a single query tile): the grid form runs them on the kernel whose P lies
over S (csrc/fa_fwd_sm100.cuh), the persistent form on the default tile's kernel (csrc/fa_fwd_persist_sm100.cuh). Which of them
a call takes depends on its number of slices, so both give the same bits; the items around them are where the persistent form's
ring and its work list go from one item to the next."""
import ctypes

import pytest
import torch

from attention_autotuner_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu


def forward(q, k, v, causal):
    lib = _lib.load()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    o = torch.full((*q.shape[:3], v.shape[3]), 7.0, device="cuda", dtype=q.dtype)
    lse = torch.full(q.shape[:3], 7.0, device="cuda")
    B, H, Lq, d = q.shape
    _lib.check(lib.attn_b200_fa_fwd(P(q), P(k), P(v), P(o), P(lse), B, H, Lq, k.shape[2], d, v.shape[3],
                                    _lib.F16 if q.dtype == torch.float16 else _lib.BF16, d ** -0.5, int(causal), None))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return o, lse


# one tile or two, one block (two with one tile), causal rows without a key in the first tile or in several work items
SHAPES = [(Lq, Lkv, causal) for Lq, Lkv in ((17, 1), (64, 64), (128, 128), (100, 255), (128, 256), (200, 100), (256, 128), (300, 128), (513, 7))
          for causal in (False, True)]


@pytest.mark.parametrize("dqk,dv,dtype", [(64, 64, torch.bfloat16), (128, 128, torch.float16), (128, 192, torch.bfloat16)])
@pytest.mark.parametrize("Lq,Lkv,causal", SHAPES)
def test_both_kernels_give_the_same_bits(monkeypatch, Lq, Lkv, causal, dqk, dv, dtype):
    BH = 450  # three work items per SM and a remainder
    g = torch.Generator("cuda").manual_seed(Lq + Lkv)
    q, k, v = (torch.randn(1, BH, n, d, generator=g, device="cuda").to(dtype) for n, d in ((Lq, dqk), (Lkv, dqk), (Lkv, dv)))
    got = {}
    for form in ("grid", "persistent"):
        monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", form)
        got[form] = forward(q, k, v, causal)
    (og, lg), (op, lp) = got["grid"], got["persistent"]
    assert torch.equal(og, op) and torch.equal(lg, lp)
    seen = torch.arange(Lq) + (Lkv - Lq) >= 0 if causal else torch.ones(Lq, dtype=torch.bool)
    assert (op[:, :, ~seen] == 0).all() and torch.isneginf(lp[:, :, ~seen]).all()
    pick = [0, BH // 2, BH - 1]
    oref, lref = oracle.attention_fwd(*(t[:, pick].cpu() for t in (q, k, v)), dqk ** -0.5, causal)
    assert oracle.within(oracle.error_stats(op[:, pick].cpu()[:, :, seen], oref[:, :, seen]), "fp16" if dtype == torch.float16 else "bf16")
    assert (lp[:, pick].cpu()[:, :, seen] - lref[:, :, seen]).abs().max().item() < 1e-3
