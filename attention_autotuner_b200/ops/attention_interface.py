"""``flash_attn_func``: same entry point as the reference's python/ops/attention_interface.py:60.

    o = flash_attn_func(q, k, v, device_type, causal=False, softmax_scale=None, return_lse=False)

q [B,H,Lq,dqk], k [B,H,Lkv,dqk], v [B,H,Lkv,dv], fp16 or bf16 CUDA tensors. ``softmax_scale=None`` keeps
the reference's fixed 0.125 (attention_interface.py / ref_op.py:3). The reference accepts ``causal`` and
ignores it (csrc/kernels/attention/regfuse/regfuse.h:59-60); here it masks key j > i + (Lkv - Lq).
Backward is empty in the reference (attention_interface.py:38-39: autograd gets None). Here it runs the
flash-attention backward kernels (csrc/fa_bwd_kv_sm100.cuh, csrc/fa_bwd_sm100.cuh) when q, k and v share a head dimension of 64 or 128, and
raises for every other shape instead of returning None.
"""
from ._checks import check_qkv
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


class MultiHeadAttnFunc:
    """The reference's autograd class (python/ops/attention_interface.py:8-39); its node is native here
    (csrc/host/torch_ops.cpp: AttnNode)."""
    apply = staticmethod(flash_attn_func)
