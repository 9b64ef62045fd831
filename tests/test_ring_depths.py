"""The attention forward's K / V ring: every depth that the tuner's feasibility check accepts builds, in every form of the grid, and
gives the same bits. The number of entries sets how many barriers a CTA has, and with them the barrier area's size."""
import pytest
import torch

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.autotuner.configs import AttnConfig
from attention_autotuner_b200.autotuner.runtime import Runtime, compile_parallel
from attention_autotuner_b200.autotuner.tunner import AttnTunner


def deep(q_tiles, kv_stages, **kw):
    return AttnConfig(128 * q_tiles, 128, 64, 64, q_tiles=q_tiles, kv_stages=kv_stages, dv_chunk=64, dtype="fp16", **kw)


def test_every_accepted_depth_builds(tmp_path):
    arch = B200()
    z = [torch.zeros(1, 1, 1, 64, dtype=torch.float16)] * 4
    accepted = [n for n in range(2, 20) if AttnTunner(arch, z).validate_kernel(deep(2, n))]
    assert accepted[-1] == 12
    # 5 entries are the last that the smallest barrier area holds; the automatic form instantiates both forms of the grid
    configs = [deep(2, 6), deep(2, 9), deep(2, 12), deep(1, 13)]
    assert AttnTunner(arch, z).validate_kernel(configs[-1]) and not AttnTunner(arch, z).validate_kernel(deep(1, 14))
    names = compile_parallel(configs, arch, tmp_dir=str(tmp_path))
    assert all(names), [c for c, n in zip(configs, names) if n is None]


@pytest.mark.gpu
@pytest.mark.parametrize("BH,Lq,Lkv,causal", [(160, 300, 290, True), (150, 100, 2000, False), (4, 1900, 1900, True), (300, 64, 64, False)])
def test_deep_rings_give_the_same_bits(BH, Lq, Lkv, causal):
    """4 entries against depths that the forward's barrier area is enlarged for, work items shorter and longer than the ring."""
    arch = B200()
    g = torch.Generator("cuda").manual_seed(6)
    q, k, v = (torch.randn(1, BH, n, 64, generator=g, device="cuda").half() for n in (Lq, Lkv, Lkv))
    configs = [deep(2, n, persistent=form) for form in (0, 1) for n in (4, 6, 9, 12)]
    assert all(compile_parallel(configs, arch))
    want = None
    for cfg in configs:
        o = torch.full_like(q, 7.0)
        rt = Runtime(arch, cfg)
        rt.apply([q, k, v, o], q.device, causal=causal, scale=0.125)
        torch.cuda.synchronize()
        assert rt.device_status() == 0
        want = o if want is None else want
        assert torch.equal(o, want), cfg
