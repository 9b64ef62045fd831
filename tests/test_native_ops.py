"""The native operator layer (csrc/host/torch_ops.cpp): staleness of plans without a GPU; autograd errors and strided
gradients through the operators on one."""
import os

import pytest
import torch


def test_plan_goes_stale_with_its_files_and_environment(tmp_path, monkeypatch):
    from attention_autotuner_b200.ops import _native
    native = _native.ops()
    f = tmp_path / "best.json"
    monkeypatch.delenv("ATTN_B200_X", raising=False)
    plan = native.make_plan(0, 0, "lib", [str(f), str(tmp_path / "other.json")], ["ATTN_B200_X"])
    assert native.plan_fresh(plan)
    monkeypatch.setenv("ATTN_B200_X", "1")
    assert not native.plan_fresh(plan)
    monkeypatch.delenv("ATTN_B200_X")
    assert native.plan_fresh(plan)
    f.write_text("{}")
    assert not native.plan_fresh(plan)
    plan = native.make_plan(0, 0, "lib", [str(f)], [])
    assert native.plan_fresh(plan)
    os.utime(f, ns=(1, 1))
    assert not native.plan_fresh(plan)
    assert not native.plan_fresh(None)


def test_an_extension_made_from_something_else_is_refused(monkeypatch):
    from attention_autotuner_b200 import build
    from attention_autotuner_b200.ops import _native
    module = _native.ops()
    monkeypatch.setattr(_native, "_module", None)
    assert type(_native.ops()) is type(module)
    monkeypatch.setattr(_native, "_module", None)
    monkeypatch.setattr(build, "_ops_hash", lambda: "0")
    with pytest.raises(RuntimeError, match="other sources"):
        _native.ops()


def test_a_build_replaces_the_extension_whole_or_not_at_all(monkeypatch, tmp_path):
    import subprocess

    from attention_autotuner_b200 import build
    path = tmp_path / "_torch_ops.so"
    path.write_text("old")
    monkeypatch.setattr(build, "OPS_PATH", str(path))
    for status, left in ((1, "old"), (0, "new")):
        def compiler(cmd, **_k):
            out = cmd[cmd.index("-o") + 1]
            with open(out, "w") as f:
                f.write("half")
            assert path.read_text() == "old"  # what another process would load now
            with open(out, "w") as f:
                f.write("new")
            return subprocess.CompletedProcess(cmd, status, "", "")

        monkeypatch.setattr(build.subprocess, "run", compiler)
        if status:
            with pytest.raises(RuntimeError):
                build.build_torch_ops()
        else:
            build.build_torch_ops()
        assert path.read_text() == left
        assert sorted(os.listdir(tmp_path)) == ["_torch_ops.so"] + ([] if status else ["_torch_ops.so.srchash"])


def test_a_plan_reads_the_environment_under_the_gil(monkeypatch):
    """os.environ assignments of other threads run setenv under the GIL, so getenv has to as well. A plan with many variables,
    the last one changed: no other thread gets to run while the call looks at them and declines."""
    import sys
    import threading
    import time

    from torch._subclasses.fake_tensor import FakeTensorMode

    from attention_autotuner_b200.ops import _native
    native = _native.ops()
    with FakeTensorMode():  # passes the checks of a CUDA tensor; a declined call launches nothing
        q = torch.empty(1, 2, 64, 64, dtype=torch.float16, device="cuda")
    decay = torch.ones(2)
    names = [f"ATTN_B200_X{i}" for i in range(100000)]
    plan = native.make_plan(1, 1, "lib", [], names)
    monkeypatch.setenv(names[-1], "1")
    turns, stop = [0], threading.Event()

    def other():
        while not stop.is_set():
            turns[0] += 1
            time.sleep(0)

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1000.0)  # a thread gives the GIL away on its own or not at all
    thread = threading.Thread(target=other)
    thread.start()
    try:
        time.sleep(0.05)
        for call in (lambda: native.attn(q, q, q, plan, 1.0, False, False),
                     lambda: native.retnet(q, q, q, None, decay, plan, None, 0, 1.0, True),
                     lambda: native.retnet_fwd_raw(q, q, q, None, decay, plan, 1.0, True), lambda: native.plan_fresh(plan) or None):
            time.sleep(0.01)
            before = turns[0]
            out = call()
            after = turns[0]
            assert out is None and before > 0 and after == before
    finally:
        stop.set()
        sys.setswitchinterval(interval)
        thread.join()


def test_declines_what_the_python_checks_word():
    from attention_autotuner_b200.arch import B200
    from attention_autotuner_b200.ops import _native
    from attention_autotuner_b200.ops.attention_interface import flash_attn_func
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttnFunc, retnet_chunkwise
    native = _native.ops()
    q = torch.zeros(1, 2, 8, 128, dtype=torch.float16)  # not on a CUDA device
    plan = native.make_plan(0, 0, "lib", [], [])
    assert native.attn(q, q, q, plan, 1.0, False, False) is None
    assert native.retnet(q, q, q, None, torch.ones(2), plan, None, 0, 1.0, True) is None
    assert native.chunkwise(q, q, q, torch.ones(2), 1.0) is None
    for call in (lambda: flash_attn_func(q, q, q, B200()), lambda: flash_attn_func(None, q, q, B200()),
                 lambda: RetNetAttnFunc(q, q, q, None, B200(), decay=torch.ones(2)),
                 lambda: retnet_chunkwise(q, q, q, torch.ones(2))):
        with pytest.raises(ValueError):
            call()


def test_the_operators_classes_are_autograd_functions_to_derive_from():
    from attention_autotuner_b200.ops.attention_interface import MultiHeadAttnFunc
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttn
    for base in (MultiHeadAttnFunc, RetNetAttn):
        assert issubclass(base, torch.autograd.Function)

        class Derived(base):
            @staticmethod
            def forward(ctx, x):
                return 2 * x

            @staticmethod
            def backward(ctx, g):
                return 3 * g

        x = torch.ones(2, requires_grad=True)
        y = Derived.apply(x)
        y.sum().backward()
        assert torch.equal(y, torch.full((2,), 2.0)) and torch.equal(x.grad, torch.full((2,), 3.0))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["attention", "mask", "decay"])
def test_a_derived_class_computes_what_the_operator_does(form):
    from attention_autotuner_b200.arch import B200
    from attention_autotuner_b200.ops.attention_interface import MultiHeadAttnFunc, flash_attn_func
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttn, RetNetAttnFunc
    q, k, v, do = (torch.randn(1, 64, 2, 64, device="cuda").half().transpose(1, 2) for _ in range(4))
    if form == "attention":
        base, func, args = MultiHeadAttnFunc, flash_attn_func, (B200(), True, 0.125)
    elif form == "mask":
        base, func, args = RetNetAttn, RetNetAttnFunc, (torch.rand(2, 64, 64, device="cuda").half().tril(), B200(), True)
    else:
        base, func, args = RetNetAttn, RetNetAttnFunc, (None, B200(), True, 0.125, torch.tensor([0.97, 0.99]))

    class Derived(base):
        pass

    results = []
    for call in (func, base.apply, Derived.apply):
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v)]
        o = call(*leaves, *args)
        results.append((o.detach(), *torch.autograd.grad(o, leaves, do)))
        with torch.no_grad():
            assert torch.equal(call(*leaves, *args), o)
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    if form == "attention":
        o, lse = Derived.apply(q.detach().requires_grad_(True), k, v, *args, True)
        assert o.requires_grad and not lse.requires_grad
        assert torch.equal(lse, flash_attn_func(q, k, v, *args, True)[1])


@pytest.mark.gpu
def test_backward_errors_keep_their_class_and_strided_gradients_are_taken():
    from attention_autotuner_b200.arch import B200
    from attention_autotuner_b200.ops.attention_interface import flash_attn_func
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttnFunc
    g = torch.Generator("cuda").manual_seed(3)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda").half()

    q, k, v = (normal(1, 2, 100, 64).requires_grad_(True) for _ in range(3))
    k2, v2 = (normal(1, 2, 40, 64).requires_grad_(True) for _ in range(2))
    o = flash_attn_func(q, k2, v2, B200(), True, 0.125)
    with pytest.raises(NotImplementedError):
        o.backward(torch.ones_like(o))
    # dO as an expanded and as a transposed tensor gives the gradients of its contiguous copy
    for call in (lambda: flash_attn_func(q, k, v, B200(), True, 0.125),
                 lambda: RetNetAttnFunc(q, k, v, None, B200(), True, 0.125, torch.tensor([0.97, 0.99]))):
        o = call()
        for do in (normal(1, 2, 64, 100).transpose(2, 3), normal(1, 2, 1, 64).expand(1, 2, 100, 64)):
            got = torch.autograd.grad(o, (q, k, v), do, retain_graph=True)
            want = torch.autograd.grad(o, (q, k, v), do.contiguous(), retain_graph=True)
            assert all(torch.equal(a, b) for a, b in zip(got, want))
    # inference mode and no_grad give the same output without a node
    with torch.no_grad():
        assert torch.equal(flash_attn_func(q, k, v, B200(), True, 0.125), flash_attn_func(q, k, v, B200(), True, 0.125))
        assert flash_attn_func(q, k, v, B200(), True, 0.125).grad_fn is None
    o1, lse = flash_attn_func(q, k, v, B200(), True, 0.125, True)
    assert o1.requires_grad and not lse.requires_grad


@pytest.mark.gpu
def test_forward_mode_duals_are_refused_not_dropped():
    import torch.autograd.forward_ad as fwAD
    from attention_autotuner_b200.arch import B200
    from attention_autotuner_b200.ops.attention_interface import flash_attn_func
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttnFunc
    q, k, v, t = (torch.randn(1, 2, 64, 64, device="cuda").half() for _ in range(4))
    with fwAD.dual_level(), torch.no_grad():
        d = fwAD.make_dual(q, t)
        with pytest.raises(RuntimeError):
            flash_attn_func(d, k, v, B200(), True, 0.125)
        with pytest.raises(RuntimeError):
            RetNetAttnFunc(k, d, v, None, B200(), True, 0.125, torch.tensor([0.97, 0.99]))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["mask", "decay"])
def test_a_mask_or_decay_alone_takes_the_call_through_the_node(form):
    import torch.autograd.forward_ad as fwAD
    from attention_autotuner_b200.arch import B200
    from attention_autotuner_b200.ops.retnet_interface import RetNetAttnFunc
    q, k, v = (torch.randn(1, 2, 64, 64, device="cuda").half() for _ in range(3))
    factor = torch.rand(2, 64, 64, device="cuda").half() if form == "mask" else torch.tensor([0.97, 0.99], device="cuda")

    def call(f, q=q):
        return RetNetAttnFunc(q, k, v, f, B200(), False, 0.125) if form == "mask" else RetNetAttnFunc(q, k, v, None, B200(), True, 0.125, f)

    want = call(factor)
    assert not want.requires_grad
    with fwAD.dual_level(), pytest.raises(RuntimeError):
        call(fwAD.make_dual(factor, torch.ones_like(factor)))
    learned = factor.clone().requires_grad_(True)
    got = call(learned)
    assert got.requires_grad and torch.equal(got, want)
    # the gradient of q is that of a constant mask or decay; the factor itself gets none
    do = torch.randn_like(want)
    qg, qh = (q.clone().requires_grad_(True) for _ in range(2))
    call(learned, qg).backward(do)
    call(factor, qh).backward(do)
    assert torch.equal(qg.grad, qh.grad) and learned.grad is None
    with torch.no_grad():
        assert not call(learned).requires_grad
