"""``RetNetAttnFunc``: same entry point as the reference's python/ops/retnet_interface.py:57.

    o = RetNetAttnFunc(q, k, v, mask, device_type, causal=False, scale=None, decay=None)
    o.backward(do)            # dq, dk, dv; no gradient for mask, r is a constant (ref_op.py:11)

q, k [B,H,L,dqk], v [B,H,Lkv,dv], mask [H,Lq,Lkv], all fp16 (bf16 also accepted). ``scale=None`` keeps the
reference's unscaled scores. ``decay`` (tensor of H per-head gammas) replaces the mask tensor by
M[h,i,j] = gamma_h^(i-j) (i >= j) built inside the kernel; ``mask`` may then be None. With a mask
tensor, ``causal=True`` declares it lower triangular so the kernels skip the blocks above the diagonal
(the reference accepts the argument and ignores it)."""
import torch

from ._checks import check_like, check_mask_decay, check_qkv
from ._native import TRIES, arch_token, ops, resolve_ret, ret_plan


def _plan_or_none(op, arch, q, v, causal, decay):
    try:
        return ret_plan(op, arch, q, v, causal, decay)
    except (AttributeError, IndexError):
        return None  # not tensors: the checks say so


def _call(native_call, device_type, q, k, v, mask, causal, scale, decay):
    """native_call(plan), with the checks and the plan's resolution where the first try declines."""
    plan = _plan_or_none("ret", device_type, q, v, causal, decay)
    out = native_call(plan) if plan is not None else None
    for _ in range(TRIES):
        if out is not None:
            return out
        check_qkv("RetNetAttnFunc", q, k, v)
        check_mask_decay("RetNetAttnFunc", q, k, mask, decay)
        out = native_call(resolve_ret(device_type, q, k, v, mask, causal, scale, decay))
    if out is None:
        raise RuntimeError("RetNetAttnFunc: the tuning cache keeps changing while the call is being prepared")
    return out


def retnet_forward(q, k, v, mask, device_type, causal=False, scale=None, decay=None):
    """The forward launch without autograd: returns (o, r, mask, decay) with mask / decay as the kernels took them
    (contiguous, decay as fp32 on the device). r = max(sum_j |S~|, 1) per row is what the backward needs."""
    s = 1.0 if scale is None else scale
    native = ops()
    return _call(lambda plan: native.retnet_fwd_raw(q, k, v, mask, decay, plan, s, causal), device_type, q, k, v, mask, causal,
                 scale, decay)


def retnet_backward(q, k, v, mask, do, r, device_type, causal=False, scale=None, decay=None):
    """The backward launches without autograd: (dq, dk, dv) from the tensors of retnet_forward. r is a constant
    (python/utils/ref_op.py:11 detaches it)."""
    check_qkv("RetNetAttnFunc backward", q, k, v)
    check_mask_decay("RetNetAttnFunc backward", q, k, mask, decay)
    check_like("RetNetAttnFunc backward", "dO", do, (*q.shape[:3], v.shape[3]), q.dtype, q.device)
    check_like("RetNetAttnFunc backward", "r", r, q.shape[:3], torch.float32, q.device)
    return ops().retnet_bwd_raw(q, k, v, mask, do, r, decay, ret_plan("ret_bwd", device_type, q, v, causal, decay),
                                arch_token(device_type), 1.0 if scale is None else scale, causal)


def retnet_chunkwise(q, k, v, decay, device_type=None, scale=None):
    """Chunkwise (recurrent-state) RetNet forward: o[i] = scale * sum_{j <= i} decay_h^(i-j) (q_i . k_j) v_j, the
    unnormalised retention of the reference's recurrent kernel (csrc/kernels/retnet/recurrent/recurrent.h:427-463),
    evaluated chunk by chunk with the state in tensor memory: the cost grows with L, not L^2. Forward only.
    q, k [B,H,L,dqk] (dqk 128 or 256), v [B,H,L,dv], fp16 or bf16 on one CUDA device; ``decay``: H per-head gammas.
    With few (batch, head) slices and a long sequence the library cuts the sequence into segments that run at once
    (attn_b200_ret_chunk_fwd_ws); the scratch for the segment states is allocated here."""
    s = 1.0 if scale is None else scale
    out = ops().chunkwise(q, k, v, decay, s)
    if out is None:
        check_qkv("retnet_chunkwise", q, k, v)
        check_mask_decay("retnet_chunkwise", q, k, None, decay)
        if k.shape[2] != q.shape[2]:
            raise ValueError(f"retnet_chunkwise: q and k must have the same length, got {q.shape[2]} and {k.shape[2]}")
        raise ValueError(f"retnet_chunkwise: head dimension of q/k must be 128 or 256, got {q.shape[3]}")
    return out


def RetNetAttnFunc(q, k, v, mask, device_type, causal=False, scale=None, decay=None):
    s = 1.0 if scale is None else scale
    native = ops()
    token = arch_token(device_type)

    def go(plan):
        return native.retnet(q, k, v, mask, decay, plan, _plan_or_none("ret_bwd", device_type, q, v, causal, decay), token, s, causal)

    return _call(go, device_type, q, k, v, mask, causal, scale, decay)


class RetNetAttn(torch.autograd.Function):
    """The reference's autograd class (python/ops/retnet_interface.py:8-55). Its ``apply`` goes through the native node
    (csrc/host/torch_ops.cpp: RetNode); ``forward`` and ``backward`` are that node's for classes derived from this one."""

    @staticmethod
    def forward(ctx, q, k, v, mask, device_type, *opts):
        causal = bool(opts[0]) if len(opts) > 0 else False
        scale = opts[1] if len(opts) > 1 else None
        decay = opts[2] if len(opts) > 2 else None
        q, k, v = [x.contiguous() for x in [q, k, v]]
        o, r, maskr, decayr = retnet_forward(q, k, v, mask, device_type, causal, scale, decay)
        ctx.save_for_backward(q, k, v, maskr, r, decayr)
        ctx.device_type = device_type
        ctx.opts = (causal, scale)
        ctx.n_extra = len(opts)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, mask, r, decay = ctx.saved_tensors
        causal, scale = ctx.opts
        dq, dk, dv = retnet_backward(q, k, v, mask, do, r, ctx.device_type, causal, scale, decay)
        return (dq, dk, dv, None, None) + (None,) * ctx.n_extra

    @classmethod
    def apply(cls, *args, **kwargs):
        if cls is RetNetAttn:
            return RetNetAttnFunc(*args, **kwargs)
        return super().apply(*args, **kwargs)
