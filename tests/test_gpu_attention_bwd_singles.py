"""Attention backward without a causal mask, where row blocks are dealt one by one (fa_bwd_singles in csrc/fa_bwd_launch.cuh):
several blocks per SM with a ragged last one (in the dQ kernel and in the dK/dV kernel, at both head dimensions), and fewer
blocks than SMs. Oracle and tolerances as in test_gpu_attention_bwd.py."""
import pytest
import torch

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.ops.attention_interface import flash_attn_func
from oracle import oracle

pytestmark = pytest.mark.gpu


DT = {"fp16": torch.float16, "bf16": torch.bfloat16}


def singles(BH, n, sms=148):
    """fa_bwd_singles of the launcher without a causal mask."""
    items, pairs = BH * n, BH * ((n + 1) // 2)
    return -(-items // sms) < 2 * -(-pairs // sms)


# the kernels whose row blocks are dealt one by one: (dQ, by query blocks of 128; dK/dV, by key blocks)
@pytest.mark.parametrize("dtype_name", ["fp16", "bf16"])
@pytest.mark.parametrize("B,H,Lq,Lkv,d,form", [(4, 13, 600, 600, 64, (True, True)), (1, 52, 600, 500, 128, (True, False)),
                                               (1, 52, 500, 600, 128, (False, True)), (1, 3, 257, 130, 64, (True, True))])
def test_single_blocks(lib, B, H, Lq, Lkv, d, form, dtype_name):
    assert tuple(singles(B * H, -(-n // 128)) for n in (Lq, Lkv)) == form
    g = torch.Generator().manual_seed(Lq + d)
    q, do = (torch.randn(B, H, Lq, d, generator=g).to(DT[dtype_name]) for _ in range(2))
    k, v = (torch.randn(B, H, Lkv, d, generator=g).to(DT[dtype_name]) for _ in range(2))
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    flash_attn_func(qd, kd, vd, B200(), False, d ** -0.5).backward(do.cuda())
    for got, want in zip((qd.grad, kd.grad, vd.grad), oracle.attention_bwd(q, k, v, do, d ** -0.5, False)):
        st = oracle.error_stats(got.cpu(), want)
        assert oracle.within(st, dtype_name, scale_by_peak=True), st
