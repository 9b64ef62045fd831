"""Which configuration, and which plan of the native operator layer, serves a call; without a GPU. A decoding call (up to 16
query rows, csrc/fa_decode_sm100.cuh) takes the default one, neither searched for nor read from or written to the tuning
cache, and kept apart from that of longer calls."""
import json
import os
import re
import subprocess

import pytest
import torch

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.autotuner import tunner
from attention_autotuner_b200.autotuner.configs import AttnConfig
from attention_autotuner_b200.autotuner.tunner import AttnTunner
from attention_autotuner_b200.build import CSRC


def tensors(Lq, d, dv=None, dt=torch.bfloat16, Lkv=512):
    q, k = torch.zeros(1, 2, Lq, d, dtype=dt), torch.zeros(1, 2, Lkv, d, dtype=dt)
    return [q, k, torch.zeros(1, 2, Lkv, dv or d, dtype=dt), torch.zeros(1, 2, Lq, dv or d, dtype=dt)]


class Searched(Exception):
    pass


@pytest.fixture
def searching(monkeypatch, tmp_path):
    """Searches enabled, as with a GPU; one that starts raises Searched. Returns the cache's folder."""
    def start(*_a, **_k):
        raise Searched
    monkeypatch.setenv("ATTN_B200_CACHE_DIR", str(tmp_path))
    monkeypatch.setenv("ATTN_B200_AUTOTUNE", "1")
    monkeypatch.delenv("ATTN_B200_FA_FWD_FORM", raising=False)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(AttnTunner, "compile_parallel", start)
    return tmp_path


@pytest.fixture
def asked(monkeypatch):
    """Plans without libraries: the configurations whose library was asked for, in order."""
    from attention_autotuner_b200.ops import _native
    configs = []

    class Library:
        def __init__(self, arch, config):
            self.libname = str(config)
            configs.append(config)

        def _lib(self):
            class L:
                kernel_entry_ex = last_error = None
            return L

    _native.ops()
    monkeypatch.setattr(_native, "Runtime", Library)
    monkeypatch.setattr(_native, "_address", lambda fn: 0)
    monkeypatch.setattr(_native, "_plans", {})
    return configs


@pytest.mark.parametrize("Lq,d", [(1, 64), (1, 128), (16, 64), (16, 128)])
def test_a_decoding_call_neither_searches_nor_stores(searching, monkeypatch, Lq, d):
    t = AttnTunner(B200(), tensors(Lq, d), causal=True)
    assert t.tune() == t.default_config() and t.tune(force=True) == t.default_config()
    assert os.listdir(searching) == []
    # a cached configuration that forces a form of the grid does not keep it from the decoding kernel
    cached = AttnConfig(256, 128, d, d, q_tiles=2, kv_stages=4, dv_chunk=d, persistent=1, dtype="bf16")
    with open(t._cache_file(), "w") as f:
        json.dump(cached.to_dict(), f)
    assert t.tune() == t.default_config() and t.default_config().substitution_map()["launcher"] == "fa_fwd_launch_auto"
    # calls the large tiles serve: one row more, other head dimensions, a form asked for
    assert AttnTunner(B200(), tensors(17, d), causal=True).tune() == cached
    with pytest.raises(Searched):
        AttnTunner(B200(), tensors(Lq, d, 192), causal=True).tune()
    monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", "grid")
    assert AttnTunner(B200(), tensors(Lq, d), causal=True).tune() == cached


def test_the_plan_of_a_decoding_call_is_its_own(searching, asked, monkeypatch):
    from attention_autotuner_b200.ops import _native
    arch = B200()
    one, many = tensors(1, 128), tensors(17, 128)
    cached = AttnConfig(256, 128, 128, 128, q_tiles=2, kv_stages=3, dv_chunk=128, cta_pair=1, dtype="bf16")
    plan = _native.resolve_attn(arch, *one[:3], True, 1.0)
    assert asked[-1] == AttnTunner(arch, one).default_config() and _native.attn_plan(arch, one[0], one[2], True) is plan
    assert _native.attn_plan(arch, many[0], many[2], True) is None
    with open(AttnTunner(arch, many, causal=True)._cache_file(), "w") as f:
        json.dump(cached.to_dict(), f)
    assert _native.resolve_attn(arch, *many[:3], True, 1.0) is _native.attn_plan(arch, many[0], many[2], True)
    assert asked[-1] == cached and _native.ops().plan_fresh(plan)
    # a form asked for in the environment ends the decoding plan
    monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", "persistent")
    assert not _native.ops().plan_fresh(plan) and _native.attn_plan(arch, one[0], one[2], True) is not plan


def test_device_descriptions_with_other_limits_have_plans_of_their_own(asked, monkeypatch, tmp_path):
    from attention_autotuner_b200.ops import _native
    monkeypatch.setenv("ATTN_B200_CACHE_DIR", str(tmp_path))
    monkeypatch.setenv("ATTN_B200_AUTOTUNE", "0")
    q, k, v, _o = tensors(256, 128)
    wide, small, few = B200(), B200(), B200()
    small.smem_cap = 160 * 1024  # a K / V ring of two entries beside two query tiles, or one query tile
    few.tmem_columns = 256       # no room for two query tiles
    plans = []
    for arch in (wide, small, few):
        assert _native.attn_plan(arch, q, v, True) is None
        plans.append(_native.resolve_attn(arch, q, k, v, True, 1.0))
        assert AttnTunner(arch, [q, k, v, v]).validate_kernel(asked[-1])
    assert len({str(c) for c in asked}) == 3
    assert [_native.attn_plan(a, q, v, True) for a in (wide, small, few)] == plans
    assert _native.attn_plan(B200(), q, v, True) is plans[0]


def test_an_entry_written_while_a_plan_is_made_is_not_taken_as_seen(asked, monkeypatch, tmp_path):
    """Another process stores an entry while this one compiles the library of the choice it has read before."""
    from attention_autotuner_b200.ops import _native
    monkeypatch.setenv("ATTN_B200_CACHE_DIR", str(tmp_path))
    monkeypatch.setenv("ATTN_B200_AUTOTUNE", "0")
    arch, (q, k, v, o) = B200(), tensors(256, 128)
    path = AttnTunner(arch, [q, k, v, o], causal=True)._cache_file()
    entries = [AttnConfig(256, 128, 128, 128, q_tiles=2, kv_stages=s, dv_chunk=128, persistent=p, dtype="bf16") for s, p in ((3, 0), (3, 1))]
    left = list(entries)
    library = _native.Runtime

    def slow(arch, config):
        if left:
            with open(path, "w") as f:
                json.dump(left[0].to_dict(), f)
            os.utime(path, ns=(len(left), len(left)))
            left.pop(0)
        return library(arch, config)

    monkeypatch.setattr(_native, "Runtime", slow)
    plan = _native.resolve_attn(arch, q, k, v, True, 1.0)
    assert asked == [AttnTunner(arch, [q, k, v, o]).default_config(), *entries]
    assert _native.attn_plan(arch, q, v, True) is plan and _native.ops().plan_fresh(plan)


def test_an_operator_prepares_again_what_a_change_has_overtaken(monkeypatch):
    from torch._subclasses.fake_tensor import FakeTensorMode

    from attention_autotuner_b200.ops import attention_interface, retnet_interface
    with FakeTensorMode():
        q = torch.empty(1, 2, 64, 128, dtype=torch.float16, device="cuda")
    for declined in (2, 1000):
        class Native:
            attn = retnet = staticmethod(lambda *a: next(answers))

        for mod, resolve in ((attention_interface, "resolve_attn"), (retnet_interface, "resolve_ret")):
            monkeypatch.setattr(mod, "ops", lambda: Native)
            monkeypatch.setattr(mod, resolve, lambda *a: "plan")
        calls = (lambda: attention_interface.flash_attn_func(q, q, q, B200()),
                 lambda: retnet_interface.RetNetAttnFunc(q, q, q, None, B200(), decay=torch.ones(2)))
        for call in calls:
            answers = iter([None] * declined + ["out"])
            if declined == 2:
                assert call() == "out"
            else:
                with pytest.raises(RuntimeError, match="keeps changing"):
                    call()


PROGRAM = r"""
#include "fa_fwd_form.cuh"
#include <cstdio>
int main() {
  int dqk, dv, lq, lkv;
  while (scanf("%d %d %d %d", &dqk, &dv, &lq, &lkv) == 4) printf("%d\n", ab200::fa_decode_shape(dqk, dv, lq, lkv) ? 1 : 0);
}
"""


def test_the_rule_is_the_launchers(tmp_path):
    (tmp_path / "rule.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(tmp_path / "rule.cpp"), "-o", str(tmp_path / "rule")], check=True)
    shapes = [(dqk, dv, lq, lkv) for dqk in (64, 128, 192, 256) for dv in (64, 128, 256) for lq in range(1, 19) for lkv in (1, 16, 255, 256, 257, 9000)]
    out = subprocess.run([str(tmp_path / "rule")], input="\n".join(" ".join(map(str, x)) for x in shapes), capture_output=True, text=True, check=True)
    got = [x == "1" for x in out.stdout.split()]
    assert got == [tunner.is_decoding((1, 1, lq, dqk), (1, 1, lkv, dv)) for dqk, dv, lq, lkv in shapes]
    taken = {x for x, g in zip(shapes, got) if g}
    # the kernel's tile holds 16 rows; more than 12 with few keys were slower on it at d = 128 (16 rows, 128 keys, 2048 slices:
    # 69.6 us against 55.3)
    with open(os.path.join(CSRC, "fa_decode_sm100.cuh")) as f:
        assert max(x[2] for x in taken) <= int(re.search(r"int MAX_ROWS = (\d+);", f.read()).group(1))
    assert (128, 128, 16, 257) in taken and (128, 128, 12, 16) in taken and (64, 64, 16, 16) in taken
    assert not {(128, 128, 16, 16), (128, 128, 13, 256)} & taken
