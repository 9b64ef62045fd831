"""The rule between the two forms of the attention forward's grid (csrc/fa_fwd_form.cuh), compiled for the host: it takes the
faster form of measured shapes, and the persistent one wherever slices of one work item each share an SM."""
import random
import subprocess

from attention_autotuner_b200.autotuner.cost_model import forward_is_persistent
from attention_autotuner_b200.build import CSRC

# slices, Lq, Lkv, causal, grid us, persistent us; measured on a B200 (148 SMs) at d = 128, the forms at least 4 % apart
MEASURED = [
    (2000, 64, 64, 0, 74.29, 53.28), (2000, 64, 64, 1, 75.43, 53.27), (400, 256, 256, 0, 32.69, 25.13), (1000, 256, 256, 0, 73.31, 58.34),
    (2000, 130, 130, 0, 118.75, 95.91), (512, 512, 512, 0, 108.9, 101.3), (512, 512, 512, 1, 93.9, 80.6), (96, 1300, 1300, 1, 85.1, 75.5),
    (12, 5000, 5000, 1, 122.0, 90.0), (80, 512, 512, 1, 23.76, 21.58), (24, 2000, 4000, 1, 113.14, 106.44), (300, 600, 600, 0, 103.3, 124.8),
    (40, 2048, 2048, 0, 106.8, 135.5), (40, 2048, 2048, 1, 71.5, 84.0), (20, 4000, 4000, 0, 197.6, 260.0), (20, 4000, 4000, 1, 122.7, 144.0),
    (52, 1280, 1280, 0, 51.0, 90.0), (52, 1280, 1280, 1, 46.0, 61.0), (60, 2700, 2700, 0, 253.6, 302.0), (60, 2700, 2700, 1, 153.9, 160.9),
    (100, 700, 700, 0, 51.0, 61.4), (100, 700, 700, 1, 35.2, 49.2), (200, 768, 768, 1, 65.7, 73.8), (100, 1792, 1792, 0, 168.5, 185.2),
]

PROGRAM = r"""
#include "fa_fwd_form.cuh"
#include <cstdio>
int main() {
  long long slices; int lq, lkv, causal, sms;
  while (scanf("%lld %d %d %d %d", &slices, &lq, &lkv, &causal, &sms) == 5)
    printf("%d\n", ab200::fa_form_persistent(slices, lq, lkv, causal != 0, sms) ? 1 : 0);
}
"""


def test_the_faster_form_is_picked(tmp_path):
    (tmp_path / "form.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, str(tmp_path / "form.cpp"), "-o", str(tmp_path / "form")], check=True)

    def persistent(calls):
        text = "\n".join(" ".join(map(str, c)) for c in calls)
        return [x == "1" for x in subprocess.run([str(tmp_path / "form")], input=text, capture_output=True, text=True, check=True).stdout.split()]

    for row, got in zip(MEASURED, persistent([(*row[:4], 148) for row in MEASURED])):
        assert got == (row[5] < row[4]), row
    # one item per slice: nothing to balance, the persistent form's overlap counts as soon as an SM has a second item
    one = [(n, lq, lkv, c, sms) for sms in (132, 148) for n in (1, 7, 148, 149, 300, 65535) for lq in (17, 200, 256)
           for lkv in (lq, 700, 5000) for c in (0, 1)]
    for call, got in zip(one, persistent(one)):
        assert got == (call[0] > call[4]), call
    # the cost model's copy of the rule
    rng = random.Random(1)
    calls = [(rng.choice((1, 8, 37, 148, 512, 4000)), rng.randint(17, 6000), rng.randint(1, 12000), rng.randint(0, 1), rng.choice((132, 148)))
             for _ in range(3000)]
    assert persistent(calls) == [forward_is_persistent(n, lq, lkv, bool(c), sms) for n, lq, lkv, c, sms in calls]
    # long items, rows that see no key, the largest sizes
    edge = [(512, 16384, 16384, 0, 148), (512, 16384, 16384, 1, 148), (4, 2000, 3, 1, 148), (65535, 2 ** 31 - 1, 2 ** 31 - 1, 1, 148)]
    assert persistent(edge)[:2] == [False, False] and len(persistent(edge)) == len(edge)
