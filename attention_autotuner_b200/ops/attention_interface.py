"""``flash_attn_func``: same entry point as the reference's python/ops/attention_interface.py:60.

    o = flash_attn_func(q, k, v, device_type, causal=False, softmax_scale=None, return_lse=False)

q [B,H,Lq,dqk], k [B,H,Lkv,dqk], v [B,H,Lkv,dv], fp16 or bf16 CUDA tensors. ``softmax_scale=None`` keeps
the reference's fixed 0.125 (attention_interface.py / ref_op.py:3). The reference accepts ``causal`` and
ignores it (csrc/kernels/attention/regfuse/regfuse.h:59-60); here it masks key j > i + (Lkv - Lq).
Backward is empty in the reference (attention_interface.py:38-39: autograd gets None). Here it runs the
flash-attention backward kernels (csrc/fa_bwd_kv_sm100.cuh, csrc/fa_bwd_sm100.cuh) when q, k and v share a head dimension of 64 or 128, and
raises for every other shape instead of returning None.
"""
import ctypes

import torch

from .. import _lib
from ._checks import check_like, check_qkv
from ._native import TRIES, attn_plan, ops, resolve_attn


def flash_attn_func(q, k, v, device_type, causal=False, softmax_scale=None, return_lse=False):
    scale = 0.125 if softmax_scale is None else softmax_scale
    native = ops()
    try:
        plan = attn_plan(device_type, q, v, causal)
    except (AttributeError, IndexError):
        plan = None  # not tensors: the checks below say so
    out = native.attn(q, k, v, plan, scale, causal, return_lse) if plan is not None else None
    for _ in range(TRIES):
        if out is not None:
            return out
        # first call for these head dimensions, a changed tuning cache, or arguments the kernels do not take (raises)
        check_qkv("flash_attn_func", q, k, v)
        plan = resolve_attn(device_type, q, k, v, causal, softmax_scale)
        out = native.attn(q, k, v, plan, scale, causal, return_lse)
    if out is None:
        raise RuntimeError("flash_attn_func: the tuning cache keeps changing while the call is being prepared")
    return out


class MultiHeadAttnFunc(torch.autograd.Function):
    """The reference's autograd class (python/ops/attention_interface.py:8-39). Its ``apply`` goes through the native node
    (csrc/host/torch_ops.cpp: AttnNode); ``forward`` and ``backward`` are that node's for classes derived from this one."""

    @staticmethod
    def forward(ctx, q, k, v, device_type, causal=False, softmax_scale=None, return_lse=False):
        needs_grad = any(ctx.needs_input_grad[:3])
        with torch.no_grad():
            out = flash_attn_func(q, k, v, device_type, causal, softmax_scale, return_lse or needs_grad)
        o, lse = out if return_lse or needs_grad else (out, None)
        if needs_grad:
            ctx.save_for_backward(q.contiguous(), k.contiguous(), v.contiguous(), o, lse)
        ctx.device_type = device_type
        ctx.scale = 0.125 if softmax_scale is None else float(softmax_scale)
        ctx.causal = bool(causal)
        if return_lse:
            ctx.mark_non_differentiable(lse)
            return o, lse
        return o

    @staticmethod
    def backward(ctx, do, *unused):
        q, k, v, o, lse = ctx.saved_tensors
        B, H, Lq, d = q.shape
        Lkv = k.shape[2]
        if not (k.shape[3] == d and v.shape[3] == d and d in (64, 128)):
            raise NotImplementedError(f"attention backward needs one head dimension of 64 or 128 for q, k and v "
                                      f"(got {d}, {k.shape[3]}, {v.shape[3]})")
        if ctx.causal and Lq != Lkv:
            raise NotImplementedError("causal attention backward needs Lq == Lkv")
        check_like("flash_attn_func backward", "dO", do, o.shape, o.dtype, o.device)
        do = do.contiguous()
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        P = lambda t: ctypes.c_void_p(t.data_ptr())
        with torch.cuda.device(q.device):
            stream = ctypes.c_void_p(torch.cuda.current_stream(q.device).cuda_stream)
            _lib.check(_lib.load().attn_b200_fa_bwd(P(q), P(k), P(v), P(o), P(do), P(lse), P(dq), P(dk), P(dv), B, H, Lq, Lkv,
                                                    d, 0 if q.dtype == torch.float16 else 1, ctx.scale, int(ctx.causal),
                                                    stream))
        return dq, dk, dv, None, None, None, None

    @classmethod
    def apply(cls, *args, **kwargs):
        if cls is MultiHeadAttnFunc:
            return flash_attn_func(*args, **kwargs)
        return super().apply(*args, **kwargs)
