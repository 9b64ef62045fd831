"""The forward's default tile (csrc/fa_fwd_persist_sm100.cuh): S = Q K^T and O += P V are issued by warps of their own, scores are
read out of one or two buffers that the query tiles fill in turn, and K of the next block precedes V of the current one in the
ring. What can go wrong depends on how blocks and work items follow each other, on the depth of the ring and on the score
buffers (one at 128 columns of V, two at 64)."""
import ctypes

import pytest
import torch

from attention_autotuner_b200 import _lib
from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.autotuner.configs import AttnConfig
from attention_autotuner_b200.autotuner.runtime import Runtime, compile_parallel
from oracle import oracle

pytestmark = pytest.mark.gpu


def make(seed, BH, Lq, Lkv, d, dtype):
    g = torch.Generator("cuda").manual_seed(seed)
    return [torch.randn(1, BH, n, d, generator=g, device="cuda").to(dtype) for n in (Lq, Lkv, Lkv)]


def forward(q, k, v, causal):
    lib = _lib.load()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    o = torch.full_like(q, 7.0)
    lse = torch.full(q.shape[:3], 7.0, device="cuda")
    B, H, Lq, d = q.shape
    _lib.check(lib.attn_b200_fa_fwd(P(q), P(k), P(v), P(o), P(lse), B, H, Lq, k.shape[2], d, d,
                                    _lib.F16 if q.dtype == torch.float16 else _lib.BF16, d ** -0.5, int(causal), None))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return o, lse


# one tile only, a second tile with a block more or none, items of one to three blocks, several items per SM, keys that
# end inside a block, causal rows without a key
SHAPES = [(300, 64, 64, False), (300, 128, 129, False), (300, 129, 128, True), (200, 256, 256, True), (160, 300, 290, True),
          (150, 513, 513, True), (320, 17, 400, False), (150, 384, 100, True), (5, 2300, 2300, True), (3, 200, 2050, False),
          (3, 128, 256, True), (3, 129, 256, False), (3, 128, 257, False)]


@pytest.mark.parametrize("form", ["grid", "persistent"])
@pytest.mark.parametrize("d,dtype", [(64, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("BH,Lq,Lkv,causal", SHAPES)
def test_sequences_of_blocks(monkeypatch, form, d, dtype, BH, Lq, Lkv, causal):
    monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", form)
    q, k, v = make(5, BH, Lq, Lkv, d, dtype)
    o, lse = forward(q, k, v, causal)
    pick = sorted({0, 1, BH // 2, BH - 1})  # the oracle on some slices; the others by their bits, in launches of their own
    oref, lref = oracle.attention_fwd(*(t[:, pick].cpu() for t in (q, k, v)), d ** -0.5, causal)
    seen = torch.arange(Lq) + (Lkv - Lq) >= 0 if causal else torch.ones(Lq, dtype=torch.bool)
    assert oracle.within(oracle.error_stats(o[:, pick].cpu()[:, :, seen], oref[:, :, seen]), "fp16" if dtype == torch.float16 else "bf16")
    assert (lse[:, pick].cpu()[:, :, seen] - lref[:, :, seen]).abs().max().item() < 1e-3
    assert (o[:, :, ~seen] == 0).all() and torch.isinf(lse[:, :, ~seen]).all()
    for b in range(0, BH, max(1, BH // 7)):
        ob, lb = forward(*(t[:, b:b + 1].contiguous() for t in (q, k, v)), causal)
        assert torch.equal(ob[:, 0], o[:, b]) and torch.equal(lb[:, 0], lse[:, b])


def test_ring_depths_give_the_same_bits():
    """Two to five ring entries, in both forms of the grid (an entry less staging, or none, with more entries)."""
    arch = B200()
    configs = [AttnConfig(256, 128, 128, 128, q_tiles=2, kv_stages=n, dv_chunk=128, dtype="fp16", persistent=form)
               for n in (2, 3, 4, 5) for form in (0, 1)]
    assert all(name is not None for name in compile_parallel(configs, arch))
    for BH, Lq, Lkv, causal in ((160, 300, 290, True), (150, 100, 300, False), (4, 1000, 1000, True)):
        q, k, v = make(6, BH, Lq, Lkv, 128, torch.float16)
        want, _ = forward(q, k, v, causal)
        for cfg in configs:
            o = torch.full_like(q, 7.0)
            Runtime(arch, cfg).apply([q, k, v, o], q.device, causal=causal, scale=128 ** -0.5)
            torch.cuda.synchronize()
            assert torch.equal(o, want), (cfg, BH, Lq, Lkv, causal)
