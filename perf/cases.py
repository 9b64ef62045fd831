"""Performance cases: the operators of this package as a training or serving program calls them.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs on the GPU, as a program has them before the call
    run(state)           one pass through the public operator; returns every output
    work(case)           bytes and operations one pass cannot do without
    tolerance(case)      how far another correct implementation at the same precision may be away

A case is a dict: ``op`` (attn, attn_train, retnet, retnet_train, chunkwise), the sizes B, H, Lq, Lkv, dqk, dv, the
data type, ``causal`` for attention and ``form`` ("decay": per-head gammas, "mask": the mask tensor) for RetNet.
"""
import math
import os

import torch

# the built-in tile configurations wherever the tuning cache has no entry: no search inside a timed program
os.environ.setdefault("ATTN_B200_AUTOTUNE", "0")

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.ops.attention_interface import flash_attn_func
from attention_autotuner_b200.ops.retnet_interface import RetNetAttnFunc, retnet_chunkwise

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _attn(name, B, H, Lq, Lkv, d, dtype, causal, train=False):
    return dict(name=name, op="attn_train" if train else "attn", B=B, H=H, Lq=Lq, Lkv=Lkv, dqk=d, dv=d, dtype=dtype,
                causal=causal)


def _ret(name, op, B, H, L, dqk, dv, dtype="fp16", form="decay"):
    return dict(name=name, op=op, B=B, H=H, Lq=L, Lkv=L, dqk=dqk, dv=dv, dtype=dtype, form=form)


def listed():
    return [
        # the smallest benchmark configuration: a short batch at head dimension 64, latency and launch cost
        _attn("attn_small", 2, 4, 512, 512, 64, "fp16", False),
        # the headline configuration: a full encoder batch
        _attn("attn_square", 8, 16, 4096, 4096, 128, "fp16", False),
        # prefill of a few prompts of an odd length
        _attn("attn_prefill_ragged", 4, 16, 2999, 2999, 128, "bf16", True),
        # prefill of one long prompt
        _attn("attn_prefill_long", 1, 16, 16384, 16384, 128, "bf16", True),
        # one decoding step of a few sequences against long caches
        _attn("attn_decode", 2, 16, 1, 16384, 128, "bf16", True),
        # a training step of the headline configuration (output and all gradients)
        _attn("attn_train_square", 8, 16, 4096, 4096, 128, "fp16", False, train=True),
        # a training step of a small causal model, ragged length, head dimension 64
        _attn("attn_train_ragged", 4, 12, 1500, 1500, 64, "bf16", True, train=True),
        # RetNet forward over one short prompt, parallel form
        _ret("retnet_short", "retnet", 1, 8, 500, 256, 512),
        # the RetNet training configuration with the per-head decay
        _ret("retnet_train_decay", "retnet_train", 8, 8, 2048, 256, 512),
        # the same model with the mask handed over as a tensor, a smaller batch
        _ret("retnet_train_mask", "retnet_train", 4, 8, 2048, 256, 512, form="mask"),
        # RetNet forward, recurrent form: a batch of documents, and one long document
        _ret("chunkwise_batch", "chunkwise", 8, 8, 2048, 256, 512),
        _ret("chunkwise_long", "chunkwise", 1, 8, 16384, 256, 512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_DRAW_FLOPS = 1.0e12  # about a quarter of the largest listed case
_DRAW_ELEMS = 1 << 27  # elements of the largest tensor: that of the largest listed case is 2^26, of a mask 2^25


def _draw_once(rng):
    kind = rng.choice(("square", "square", "extend", "decode", "train", "train", "retnet", "retnet_train", "chunkwise"))
    dtype = rng.choice(("fp16", "bf16"))
    if kind in ("square", "extend", "decode", "train"):
        d = rng.choice((64, 128))
        B, H = _log_int(rng, 1, 16), rng.choice((1, 4, 8, 12, 16, 32))
        if kind == "square":  # prefill or encoder, any length
            Lq = Lkv = _log_int(rng, 64, 16384)
        elif kind == "extend":  # a piece of a prompt against a longer cache
            Lq = _log_int(rng, 16, 2048)
            Lkv = Lq + _log_int(rng, 64, 16384)
        elif kind == "decode":  # one or a few new positions against a cache
            Lq = rng.choice((1, 1, 1, 2, 4, 8))
            Lkv = _log_int(rng, 256, 32768)
        else:
            Lq = Lkv = _log_int(rng, 128, 8192)
        causal = True if kind in ("extend", "decode") else rng.choice((False, True))
        return _attn("", B, H, Lq, Lkv, d, dtype, causal, train=kind == "train")
    if kind == "chunkwise":
        return _ret("", "chunkwise", _log_int(rng, 1, 8), rng.choice((4, 8, 16)), _log_int(rng, 128, 16384),
                    *rng.choice(((256, 512), (128, 256), (128, 128))), dtype=dtype)
    # parallel form: fp16 and the head dimensions whose libraries the build makes
    form = rng.choice(("decay", "decay", "mask"))
    L = _log_int(rng, 128, 4096)
    if form == "mask":
        L = 8 * (L // 8)  # the operator reads the mask tensor's rows by 16 bytes
    return _ret("", kind, _log_int(rng, 1, 8), rng.choice((4, 8, 16)), L, *rng.choice(((256, 512), (256, 512), (64, 64))),
                form=form)


def draw(rng):
    while True:
        case = _draw_once(rng)
        elems = case["B"] * case["H"] * max(case["Lq"], case["Lkv"]) * max(case["dqk"], case["dv"])
        # the parallel RetNet form is bounded by all its pairs, which a plain implementation walks
        full = 2 * case["B"] * case["H"] * case["Lq"] * case["Lkv"] * (case["dqk"] + case["dv"])
        if elems <= _DRAW_ELEMS and max(full, work(case)["flops"]) <= _DRAW_FLOPS:
            del case["name"]
            return case


def _gammas(H):
    return 1.0 - torch.pow(2.0, -5.0 - torch.arange(H, dtype=torch.float64) % 8)


def prepare(case, seed):
    dt = _DTYPES[case["dtype"]]
    g = torch.Generator("cuda").manual_seed(seed)
    B, H, Lq, Lkv, dqk, dv = (case[n] for n in ("B", "H", "Lq", "Lkv", "dqk", "dv"))

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).to(dt)

    train = case["op"].endswith("_train")
    st = dict(op=case["op"], arch=B200(), scale=dqk ** -0.5)
    st["q"], st["k"], st["v"] = normal(B, H, Lq, dqk), normal(B, H, Lkv, dqk), normal(B, H, Lkv, dv)
    if train:
        st["do"] = normal(B, H, Lq, dv)
        for n in ("q", "k", "v"):
            st[n].requires_grad_(True)
    if case["op"].startswith("attn"):
        st["causal"] = case["causal"]
    else:
        gam = _gammas(H)
        st["decay"], st["mask"] = gam.to(device="cuda", dtype=torch.float32), None
        if case.get("form") == "mask":
            i = torch.arange(Lq, device="cuda", dtype=torch.float32)
            diff = i[:, None] - i[None, :]
            log_g = torch.log(gam).to(device="cuda", dtype=torch.float32)[:, None, None]
            st["mask"] = torch.where(diff >= 0, torch.exp(log_g * diff.clamp(min=0)), torch.zeros(())).to(dt)
            st["decay"] = None
    return st


def run(st):
    q, k, v, arch, scale = st["q"], st["k"], st["v"], st["arch"], st["scale"]
    if st["op"] == "chunkwise":
        return retnet_chunkwise(q, k, v, st["decay"], arch, scale=scale)
    if st["op"].startswith("attn"):
        o = flash_attn_func(q, k, v, arch, st["causal"], scale)
    else:
        o = RetNetAttnFunc(q, k, v, st["mask"], arch, True, scale, st["decay"])
    if not st["op"].endswith("_train"):
        return o
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), st["do"])


def work(case):
    """Bytes: every input once, every output once. Operations: attention and the mask form of RetNet by the unmasked
    pairs of positions (backward: five products for attention, five for RetNet). With a constant decay per head only
    the row sums of the absolute scores need all the pairs; every other product is counted in whichever of the two
    forms is cheaper, over the pairs or through the [dqk, dv] state with chunks of 128 positions."""
    B, H, Lq, Lkv, dqk, dv = (case[n] for n in ("B", "H", "Lq", "Lkv", "dqk", "dv"))
    n = B * H
    qb, kb, vb, ob = (2 * n * x for x in (Lq * dqk, Lkv * dqk, Lkv * dv, Lq * dv))
    train = case["op"].endswith("_train")
    byts = qb + kb + vb + ob
    if train:  # dO comes in, three gradients go out
        byts += ob + qb + kb + vb
    if case["op"].startswith("attn"):
        pairs = Lq * Lkv
        if case["causal"]:  # query i sees the keys up to i + Lkv - Lq; Lkv >= Lq in every case
            pairs = Lq * (Lkv - Lq) + Lq * (Lq + 1) // 2
        flops = 2 * n * pairs * (dqk + dv)
        if train:
            flops += 10 * n * pairs * dqk
        return dict(bytes=byts, flops=flops)
    pairs = Lq * (Lq + 1) // 2
    if case.get("form") == "mask":
        byts += 2 * H * Lq * Lkv
        flops = 2 * n * pairs * (dqk + dv)
        if train:
            flops += 2 * n * pairs * (3 * dqk + 2 * dv)
        return dict(bytes=byts, flops=flops)
    byts += 4 * H
    inner = Lq * (min(Lq, 128) + 1) // 2  # pairs inside chunks of 128 positions
    state = 2 * Lq * dqk * dv  # one product with the state, or one update of it
    fwd = min(2 * pairs * (dqk + dv), 2 * inner * (dqk + dv) + 2 * state)
    if case["op"] == "chunkwise":
        return dict(bytes=byts, flops=n * fwd)
    flops = 2 * pairs * dqk + min(2 * pairs * dv, fwd)  # the row sums, then the retention product
    if train:
        # dV, dK and dQ: dV and dK share one state, dQ has its own, so three products with a state and two updates
        flops += min(2 * pairs * (3 * dqk + 2 * dv), 2 * inner * (3 * dqk + 2 * dv) + 5 * state)
    return dict(bytes=byts, flops=n * flops)


def tolerance(case):
    """Four times the distance from the same formulas in 64 bits, measured over the listed and drawn cases. fp16: at most
    4.3e-4 in the 2-norm (gradients of attention; outputs 3e-4, chunkwise 3.9e-4) and 1.2e-2 in one element; bf16: at
    most 3.6e-3 and 6.0e-2. One element is compared with the larger of its value and the result's root mean square."""
    return {"rel": 1.7e-3, "max": 4.8e-2} if case["dtype"] == "fp16" else {"rel": 1.44e-2, "max": 0.24}
