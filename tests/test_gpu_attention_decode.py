"""Attention forward with up to 16 query rows (csrc/fa_decode_sm100.cuh): every cluster size of the split over the keys,
ragged last blocks, rows without a visible key, against the CPU fp32 oracle and against the large-tile kernel.

Tolerances as in test_gpu_attention.py (the arithmetic is the same: P rounded to the storage type, fp32 elsewhere)."""
import pytest
import torch

from attention_autotuner_b200.arch import B200
from attention_autotuner_b200.ops.attention_interface import flash_attn_func
from oracle import oracle
from test_gpu_attention import check, rand_qkv, run_capi

pytestmark = pytest.mark.gpu

DT = {"fp16": torch.float16, "bf16": torch.bfloat16}

# B, H, Lq, Lkv: one key; one short of, exactly and one past a block (64 keys at d = 128, 128 at d = 64); more rows than
# keys (rows that see nothing under the causal mask); the last row count; clusters of 1, of 4 (from 32 blocks) and of 8 (from
# 256) at both head dimensions, with uneven shares
SHAPES = [(1, 2, 1, 1), (1, 2, 16, 5), (1, 3, 3, 63), (2, 1, 16, 64), (1, 2, 8, 129), (2, 80, 1, 300), (3, 10, 1, 2049),
          (1, 2, 9, 4160), (1, 1, 16, 2176), (1, 1, 2, 16385), (1, 1, 1, 32800),
          # at d = 128 more than 12 rows with up to 256 keys stay on the large tile
          (1, 2, 12, 5), (2, 1, 12, 64), (1, 2, 13, 256), (1, 2, 16, 257)]


@pytest.mark.parametrize("dtype_name", ["fp16", "bf16"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d", [64, 128])
def test_small_query_counts(lib, monkeypatch, dtype_name, causal, d):
    for i, (B, H, Lq, Lkv) in enumerate(SHAPES):
        q, k, v = rand_qkv(100 + i, B, H, Lq, Lkv, d, d, DT[dtype_name])
        o, lse = run_capi(lib, q, k, v, d ** -0.5, causal)
        oref, lref = oracle.attention_fwd(q, k, v, d ** -0.5, causal)
        oref = torch.where(torch.isfinite(lref)[..., None], oref, torch.zeros(()))  # a row that sees no key: zeros
        st = oracle.error_stats(o, oref)
        assert oracle.within(st, dtype_name, scale_by_peak=True), ((B, H, Lq, Lkv), st)
        fin = torch.isfinite(lref)
        assert torch.equal(torch.isfinite(lse), fin) and (lse[fin] - lref[fin]).abs().max().item() < 1e-3
        # the large tile on the same inputs (17 rows and more always take it)
        monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", "grid")
        o2, _ = run_capi(lib, q, k, v, d ** -0.5, causal)
        monkeypatch.delenv("ATTN_B200_FA_FWD_FORM")
        # two roundings of P and one of O apart, relative to the peak
        assert (o.float() - o2.float()).abs().max().item() <= (4 if dtype_name == "fp16" else 32) * 2.0 ** -10 * max(1.0, o2.abs().max().item())


def test_first_row_count_of_the_large_tile(lib):
    q, k, v = rand_qkv(5, 2, 2, 17, 700, 128, 128, torch.float16)
    o, lse = run_capi(lib, q, k, v, 128 ** -0.5, True)
    check(o, lse, q, k, v, 128 ** -0.5, True, "fp16")


def test_operator_takes_strided_views_and_growing_peaks(lib):
    """A decoding step reads a slice of a preallocated cache; scores that grow along the keys rescale at every block."""
    g = torch.Generator().manual_seed(3)
    cache_k = torch.randn(2, 4, 1024, 128, generator=g).half()
    cache_v = torch.randn(2, 4, 1024, 128, generator=g).half()
    q = torch.randn(2, 4, 1, 128, generator=g).half()
    k = cache_k * torch.linspace(0.1, 3.0, 1024).half()[None, None, :, None]
    n = 901
    o, lse = flash_attn_func(q.cuda(), k.cuda()[:, :, :n], cache_v.cuda()[:, :, :n], B200(), True, 128 ** -0.5, return_lse=True)
    oref, lref = oracle.attention_fwd(q, k[:, :, :n], cache_v[:, :, :n], 128 ** -0.5, True)
    assert oracle.within(oracle.error_stats(o.cpu(), oref), "fp16", scale_by_peak=True)
    assert (lse.cpu() - lref).abs().max().item() < 1e-3


@pytest.mark.parametrize("d", [64, 128])
def test_a_slice_has_the_same_bits_in_any_launch(lib, d):
    q, k, v = rand_qkv(11, 12, 1, 3, 5000, d, d, torch.bfloat16)
    o, lse = run_capi(lib, q, k, v, d ** -0.5, True)
    for n in (1, 5):
        o1, lse1 = run_capi(lib, q[:n], k[:n], v[:n], d ** -0.5, True)
        assert torch.equal(o1, o[:n]) and torch.equal(lse1, lse[:n])


def in_64_bits(q, k, v, scale):
    """Causal attention in 64 bits, on the GPU."""
    s = q.double() @ k.double().transpose(-1, -2) * scale
    i, j = torch.arange(q.shape[2], device=q.device)[:, None], torch.arange(k.shape[2], device=q.device)[None]
    return torch.softmax(s.masked_fill(j > i + k.shape[2] - q.shape[2], float("-inf")), -1) @ v.double()


@pytest.mark.parametrize("dtype_name,spacing", [("fp16", 2.0 ** -10), ("bf16", 2.0 ** -7)])
@pytest.mark.parametrize("d", [64, 128])
def test_no_further_from_64_bits_than_the_large_tile(lib, monkeypatch, dtype_name, spacing, d):
    """2-norm of the error over that of the result. P and the output are each rounded once to the storage type: at most
    spacing / sqrt(12) relative as a root mean square (a value at the bottom of its binade), so sqrt(2) times that together.
    The large tile's P may be relative to a maximum that lags by 2^8, the decoding kernel's is not: it is the closer one, by 5
    to 30 % where measured; 2 % are left for the randomness of a small output."""
    for i, (B, H, Lq, Lkv) in enumerate([(1, 8, 8, 300), (2, 8, 4, 3000), (1, 8, 16, 9000), (2, 4, 4, 20000)]):
        q, k, v = (t.cuda() for t in rand_qkv(40 + i, B, H, Lq, Lkv, d, d, DT[dtype_name]))
        want = in_64_bits(q, k, v, d ** -0.5)
        errors = []
        for form in ("", "grid"):
            monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", form)
            o = flash_attn_func(q, k, v, B200(), True, d ** -0.5)
            errors.append(((o.double() - want).norm() / want.norm()).item())
        assert errors[0] <= (spacing * spacing / 6) ** 0.5 and errors[0] <= 1.02 * errors[1], ((B, H, Lq, Lkv), errors)


@pytest.mark.parametrize("dtype_name", ["fp16", "bf16"])
@pytest.mark.parametrize("causal", [False, True])
def test_infinities_and_nan_as_the_large_tile_has_them(lib, monkeypatch, dtype_name, causal):
    nan, inf = float("nan"), float("inf")
    for name, pos, value in (("q", (0, 0, 1, 3), nan), ("q", (0, 0, 1, 3), inf), ("k", (0, 1, 5, 3), nan), ("k", (0, 0, 70, 3), inf),
                             ("k", (0, 0, 70, 3), -inf), ("k", (0, 0, slice(None), 3), -inf), ("v", (0, 1, 290, 3), nan),
                             ("v", (0, 0, 5, 3), -inf)):
        t = dict(zip("qkv", rand_qkv(9, 1, 2, 4, 300, 128, 128, DT[dtype_name])))
        t[name][pos] = value
        monkeypatch.delenv("ATTN_B200_FA_FWD_FORM", raising=False)
        o, lse = run_capi(lib, t["q"], t["k"], t["v"], 128 ** -0.5, causal)
        monkeypatch.setenv("ATTN_B200_FA_FWD_FORM", "grid")
        o2, lse2 = run_capi(lib, t["q"], t["k"], t["v"], 128 ** -0.5, causal)
        for a, b in ((o, o2), (lse, lse2)):
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isposinf(), b.isposinf()) and torch.equal(a.isneginf(), b.isneginf())
            both = torch.isfinite(a)
            # as in test_small_query_counts: two roundings of P and one of O apart (outputs here are below 1)
            assert (a[both].float() - b[both].float()).abs().max().item() <= (4 if dtype_name == "fp16" else 32) * 2.0 ** -10
