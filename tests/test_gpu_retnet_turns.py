"""The CTA-pair chain kernels (csrc/chain_pair_sm100.cuh): Z is handed back as soon as it has been read (one buffer at 256 output
columns, two at 128), W goes into two buffers in turn, and a work item's output is staged in slots of the operand ring. What
can go wrong depends on how blocks and work items follow each other: items of one block and more, several items per cluster,
rows past the end in one CTA of a pair or in both."""
import ctypes

import pytest
import torch

from attention_autotuner_b200 import _lib
from oracle import oracle

pytestmark = pytest.mark.gpu


def P(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def run(q, k, v, do, mask, decay):
    lib = _lib.load()
    B, H, L, dqk = q.shape
    dv = v.shape[3]
    o, dq, dk, dvo = (torch.full_like(t, float("nan")) for t in (v, q, k, v))
    r = torch.full((B, H, L), float("nan"), device="cuda")
    _lib.check(lib.attn_b200_ret_fwd(P(q), P(k), P(v), P(mask), P(o), P(r), B, H, L, L, dqk, dv, _lib.F16, dqk ** -0.5, P(decay), 1, None))
    _lib.check(lib.attn_b200_ret_bwd(P(q), P(k), P(v), P(mask), P(do), P(r), P(dq), P(dk), P(dvo), None, B, H, L, L, dqk, dv, _lib.F16,
                                     dqk ** -0.5, P(decay), 1, None))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return o, r, dq, dk, dvo


@pytest.mark.parametrize("form", ["decay", "mask"])
@pytest.mark.parametrize("dqk,dv", [(128, 128), (256, 512)])
@pytest.mark.parametrize("B,H,L", [(50, 2, 120), (40, 4, 264), (30, 2, 520), (3, 2, 1304)])
def test_sequences_of_blocks(form, dqk, dv, B, H, L):
    g = torch.Generator("cuda").manual_seed(L)
    q, k, v, do = (torch.randn(B, H, L, d, generator=g, device="cuda").half() for d in (dqk, dqk, dv, dv))
    gam = torch.tensor([1 - 2.0 ** -(5 + h) for h in range(H)], device="cuda")
    i = torch.arange(L, device="cuda")
    maskf = torch.where(i[:, None] >= i[None, :], gam[:, None, None] ** (i[:, None] - i[None, :]).clamp(min=0), torch.zeros((), device="cuda"))
    mask = maskf.half() if form == "mask" else None
    decay = gam if form == "decay" else None
    got = run(q, k, v, do, mask, decay)
    ref = (mask.float() if form == "mask" else maskf).cpu()
    for b in (0, B // 2, B - 1):  # the oracle on some batch entries; others by their bits, in launches of their own
        args = [t[b:b + 1].cpu() for t in (q, k, v)]
        oref, rref = oracle.retnet_fwd(*args, ref, dqk ** -0.5)
        assert oracle.within(oracle.error_stats(got[0][b:b + 1].cpu(), oref), "fp16", scale_by_peak=True)
        assert ((got[1][b:b + 1].cpu() - rref).abs() / rref).max().item() < 1e-4
        grads = oracle.retnet_bwd(*args, ref, do[b:b + 1].cpu(), dqk ** -0.5)
        for mine, want in zip(got[2:], grads):
            assert oracle.within(oracle.error_stats(mine[b:b + 1].cpu(), want), "fp16", scale_by_peak=True)
    for b in range(0, B, max(1, B // 5)):
        one = run(*(t[b:b + 1].contiguous() for t in (q, k, v, do)), mask, decay)
        assert all(torch.equal(x[0], y[b]) for x, y in zip(one, got))


@pytest.mark.parametrize("L,offset", [(128, 0), (136, 0), (144, 8), (272, 0)])
def test_mask_rows_of_any_alignment(L, offset):
    """Rows of the mask that start at multiples of 32 bytes are read by 32, others by 16: same values either way."""
    B, H, dqk, dv = 2, 2, 128, 256
    g = torch.Generator("cuda").manual_seed(3)
    q, k, v, do = (torch.randn(B, H, L, d, generator=g, device="cuda").half() for d in (dqk, dqk, dv, dv))
    store = torch.zeros(H * L * L + 16, device="cuda", dtype=torch.float16)
    mask = store[offset:offset + H * L * L].view(H, L, L)  # offset 8: 16 bytes past a multiple of 32
    mask.copy_(0.3 * torch.randn(H, L, L, generator=g, device="cuda"))
    mask.tril_()
    got = run(q, k, v, do, mask, None)
    ref = mask.float().cpu()
    args = [t.cpu() for t in (q, k, v)]
    oref, rref = oracle.retnet_fwd(*args, ref, dqk ** -0.5)
    assert oracle.within(oracle.error_stats(got[0].cpu(), oref), "fp16", scale_by_peak=True)
    for mine, want in zip(got[2:], oracle.retnet_bwd(*args, ref, do.cpu(), dqk ** -0.5)):
        assert oracle.within(oracle.error_stats(mine.cpu(), want), "fp16", scale_by_peak=True)
    wide = mask.clone()  # the same values at the start of an allocation
    assert all(torch.equal(x, y) for x, y in zip(got, run(q, k, v, do, wide, None)))
