"""Attention backward without a causal mask, where row blocks are dealt one by one (fa_bwd_singles in csrc/fa_bwd_launch.cuh):
several blocks per SM with a ragged last one, and fewer blocks than SMs. Oracle and tolerances as in test_gpu_attention_bwd.py."""
import pytest
import torch

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.ops.attention_interface import flash_attn_func
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Lq,Lkv,d", [(4, 13, 600, 600, 64), (1, 52, 600, 500, 128), (1, 3, 257, 130, 64)])
def test_single_blocks(lib, B, H, Lq, Lkv, d):
    g = torch.Generator().manual_seed(Lq + d)
    q, do = (torch.randn(B, H, Lq, d, generator=g).half() for _ in range(2))
    k, v = (torch.randn(B, H, Lkv, d, generator=g).half() for _ in range(2))
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    flash_attn_func(qd, kd, vd, B200(), False, d ** -0.5).backward(do.cuda())
    for got, want in zip((qd.grad, kd.grad, vd.grad), oracle.attention_bwd(q, k, v, do, d ** -0.5, False)):
        st = oracle.error_stats(got.cpu(), want)
        assert oracle.within(st, "fp16", scale_by_peak=True), st
