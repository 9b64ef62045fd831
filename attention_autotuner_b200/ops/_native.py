"""The native operator layer (csrc/host/torch_ops.cpp, built into _torch_ops.so) and the plans it is called with.

A plan names the per-configuration library entry point that serves a call. It is resolved by the tuner exactly as before
(tuning-cache file, search, or the built-in tile) and remembered per (operation, device limits, head dimensions, dtype,
mask form) together with everything the choice was read from: the cache files' modification times and the environment variables.
The native layer compares those on every call (two ``stat`` calls) and refuses a stale plan, so a cache entry written
by this or another process takes effect at the next call, as it did when the tuner ran on every call."""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import threading

import torch

from .. import _lib, build
from ..autotuner.base_tunner import cache_dir
from ..autotuner.runtime import KernelError, Runtime
from ..autotuner.tunner import AttnTunner, RetBwdTunner, RetTunner, is_decoding

_ENV = ["ATTN_B200_CACHE_DIR", "ATTN_B200_AUTOTUNE"]
TRIES = 16  # attempts at a call that no change of the tuning cache overtakes; each change costs one

_lock = threading.Lock()
_module = None
_plans: dict = {}
_archs: list = []  # device descriptions seen by RetNet calls: the backward resolves its plan with the forward's


def _address(fn) -> int:
    return ctypes.cast(fn, ctypes.c_void_p).value


def ops():
    """The native module; raises if it has not been built from the present sources (python -m attention_autotuner_b200.build)."""
    global _module
    if _module is not None:
        return _module
    with _lock:
        if _module is None:
            path = build.OPS_PATH
            if not os.path.exists(path):
                raise RuntimeError(f"{path} is missing: build it with `python -m attention_autotuner_b200.build`. "
                                   "There is no fallback.")
            loader = importlib.machinery.ExtensionFileLoader("_torch_ops", path)
            mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_torch_ops", loader))
            loader.exec_module(mod)
            if getattr(mod, "source_hash", None) != build._ops_hash():
                # it calls the C entry points by signatures of its own: a stale one would call them with wrong arguments
                raise RuntimeError(f"{path} was built from other sources or for another PyTorch: build it again with "
                                   "`python -m attention_autotuner_b200.build`")
            lib = _lib.load()
            mod.init(KernelError, _lib.AttnB200Error, _resolve_bwd, _address(lib.attn_b200_last_error),
                     _address(lib.attn_b200_fa_bwd), _address(lib.attn_b200_ret_chunk_workspace_bytes),
                     _address(lib.attn_b200_ret_chunk_fwd_ws))
            _module = mod
    return _module


def _set_entry(plan, tuner, cfg):
    rt = Runtime(tuner.arch, cfg)
    lib = rt._lib()
    ops().set_entry(plan, _address(lib.kernel_entry_ex), _address(lib.last_error), rt.libname)
    return plan


def _resolve(tuner, key):
    """Plan of the configuration the tuner picks. Remembered unless the pick was neither read from the tuning cache nor
    the built-in tile by request (then the tuner is asked again next time, as a failed search should be).

    The plan is stamped before the cache is read, and the choice is made again if an entry was written in the meantime
    (by the search itself, or by another process while this one was compiling the library)."""
    native = ops()
    for _ in range(TRIES):
        plan = native.make_plan(0, 0, "", tuner.cache_candidates(), _ENV)
        if tuner.cache_path != cache_dir():  # another folder since the tuner was made
            tuner.cache_path = cache_dir()
            continue
        cached = tuner.check_cache()
        _set_entry(plan, tuner, tuner.tune() if cached is None else cached)
        if native.plan_fresh(plan):
            if cached is not None or os.environ.get("ATTN_B200_AUTOTUNE", "1") == "0":
                _plans[key] = plan
            return plan
    raise RuntimeError("the tuning cache keeps changing while a call is being prepared")


def _key(op, arch, dqk, dv, dtype, flag):
    # of the device description: what names the cache file and the library, and the limits that bound the tiles
    return (op, type(arch), getattr(arch, "compute_capability", ""), getattr(arch, "smem_cap", None),
            getattr(arch, "tmem_columns", None), dqk, dv, dtype, flag)


def _attn_key(arch, q, v, causal):
    op = "attn_decode" if is_decoding(q.shape, v.shape) else "attn"
    return _key(op, arch, q.shape[-1], v.shape[-1], q.dtype, bool(causal))


def attn_plan(arch, q, v, causal):
    return _plans.get(_attn_key(arch, q, v, causal))


def resolve_attn(arch, q, k, v, causal, scale):
    o = torch.empty(*q.shape[:3], v.shape[3], device=q.device, dtype=q.dtype)  # a search times the kernels on these tensors
    tuner = AttnTunner(arch=arch, torch_array=[q.detach().contiguous(), k.detach().contiguous(), v.detach().contiguous(), o],
                       scale=scale, causal=causal)
    if is_decoding(q.shape, v.shape):
        plan = _set_entry(ops().make_plan(0, 0, "", [], ["ATTN_B200_FA_FWD_FORM"]), tuner, tuner.tune())  # no cache entry in it
        _plans[_attn_key(arch, q, v, causal)] = plan
        return plan
    return _resolve(tuner, _attn_key(arch, q, v, causal))


def _ret_flag(causal, has_decay):
    return "decay" if has_decay else bool(causal)  # what the tuner's cache key depends on


def ret_plan(op, arch, q, v, causal, decay):
    return _plans.get(_key(op, arch, q.shape[-1], v.shape[-1], q.dtype, _ret_flag(causal, decay is not None)))


def resolve_ret(arch, q, k, v, mask, causal, scale, decay):
    q, k, v = (t.detach().contiguous() for t in (q, k, v))
    mask = mask.detach().contiguous() if mask is not None else None
    if decay is not None:
        decay = decay.detach().to(device=q.device, dtype=torch.float32).contiguous().reshape(-1)
    o = torch.empty(*q.shape[:3], v.shape[3], device=q.device, dtype=q.dtype)
    r = torch.empty(q.shape[:3], device=q.device, dtype=torch.float32)
    tuner = RetTunner(arch=arch, torch_array=[q, k, v, mask, o, r], scale=scale, causal=causal, decay=decay)
    return _resolve(tuner, _key("ret", arch, q.shape[-1], v.shape[-1], q.dtype, _ret_flag(causal, decay is not None)))


def arch_token(arch) -> int:
    """Small integer under which the backward finds the device description of its forward."""
    for i, a in enumerate(_archs):
        if a is arch or (type(a) is type(arch) and a.__dict__ == arch.__dict__):
            return i
    with _lock:
        _archs.append(arch)
        return len(_archs) - 1


def _resolve_bwd(token, arr, scale, causal, decay):
    """Called by the native backward when it has no valid plan: arr = [q, k, v, mask, do, r, dq, dk, dv, scratch]."""
    arch = _archs[token]
    key = _key("ret_bwd", arch, arr[0].shape[-1], arr[2].shape[-1], arr[0].dtype, _ret_flag(causal, decay is not None))
    plan = _plans.get(key)
    if plan is not None and ops().plan_fresh(plan):
        return plan
    return _resolve(RetBwdTunner(arch=arch, torch_array=list(arr), scale=scale, causal=causal, decay=decay), key)
