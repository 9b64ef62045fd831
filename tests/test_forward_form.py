"""The rule between the two forms of the attention forward's grid (csrc/fa_fwd_form.cuh), compiled for the host: it takes the
faster form of measured shapes, and the persistent one wherever slices of one work item each share an SM."""
import random
import subprocess

from attention_autotuner_b200.autotuner.cost_model import forward_is_persistent
from attention_autotuner_b200.build import CSRC

# slices, Lq, Lkv, causal, grid us, persistent us; measured on a B200 (148 SMs) at d = 128, the forms at least 4 % apart
MEASURED = [
    (2000, 64, 64, 0, 73.4, 52.5), (2000, 64, 64, 1, 73.9, 52.5), (400, 256, 256, 0, 30.0, 22.0),
    (400, 256, 256, 1, 29.5, 23.1), (1000, 256, 256, 0, 65.6, 48.2), (1000, 256, 256, 1, 65.7, 48.6),
    (2000, 130, 130, 0, 115.4, 82.3), (2000, 130, 130, 1, 112.0, 82.3), (512, 512, 512, 0, 89.4, 78.9),
    (512, 512, 512, 1, 78.5, 65.5), (96, 1300, 1300, 1, 70.3, 65.6), (12, 5000, 5000, 1, 95.8, 70.2),
    (80, 512, 512, 0, 22.2, 19.6), (80, 512, 512, 1, 19.8, 16.9), (24, 2000, 4000, 1, 89.7, 82.0),
    (24, 2000, 4000, 0, 104.4, 99.9), (300, 600, 600, 0, 83.0, 99.4), (300, 600, 600, 1, 69.4, 79.8),
    (40, 2048, 2048, 0, 86.4, 103.5), (40, 2048, 2048, 1, 57.9, 67.7), (20, 4000, 4000, 0, 157.6, 198.0),
    (20, 4000, 4000, 1, 97.5, 111.0), (52, 1280, 1280, 0, 42.4, 68.4), (52, 1280, 1280, 1, 38.0, 50.6),
    (60, 2700, 2700, 0, 202.1, 224.7), (60, 2700, 2700, 1, 127.1, 133.4), (100, 700, 700, 0, 41.8, 49.6),
    (100, 700, 700, 1, 31.4, 41.8), (200, 768, 768, 1, 57.1, 65.0), (100, 1792, 1792, 0, 143.8, 151.4),
    (96, 512, 4096, 1, 115.3, 123.1), (148, 2048, 2048, 0, 263.7, 249.5), (148, 2048, 2048, 1, 174.9, 160.9),
    (128, 4096, 4096, 0, 894.0, 826.6), (128, 4096, 4096, 1, 496.6, 460.4), (64, 2999, 2999, 1, 157.1, 150.4),
    (64, 1024, 1024, 0, 35.9, 32.6), (64, 1024, 1024, 1, 33.2, 28.2), (32, 2048, 2048, 0, 59.2, 56.8),
    (32, 2048, 2048, 1, 51.1, 38.5), (16, 3000, 3000, 0, 80.6, 77.0), (16, 3000, 3000, 1, 54.5, 46.1),
    (48, 1500, 1500, 0, 49.5, 47.2), (48, 1500, 1500, 1, 45.1, 36.2), (150, 900, 900, 0, 85.9, 91.0),
    (150, 900, 900, 1, 63.1, 73.7), (300, 384, 384, 0, 44.9, 39.5), (300, 384, 384, 1, 42.3, 36.9),
    (700, 300, 300, 0, 90.8, 67.9), (700, 300, 300, 1, 83.6, 61.4), (37, 1700, 1700, 1, 46.2, 36.1),
    (74, 1024, 2048, 1, 62.8, 58.0), (8, 4500, 4500, 0, 64.7, 110.0), (8, 4500, 4500, 1, 58.1, 61.8),
    (148, 1000, 1000, 0, 78.0, 72.7), (148, 1000, 1000, 1, 63.9, 58.4), (90, 2300, 2300, 0, 209.3, 237.3),
    (90, 2300, 2300, 1, 133.7, 148.6), (30, 1024, 4096, 1, 54.0, 90.5), (30, 1024, 4096, 0, 54.6, 96.7),
]
# where the rule takes the slower one, at most 13 % behind
MISSED = [(96, 512, 4096, 0, 107.5, 121.4), (256, 1024, 1024, 1, 100.6, 105.3)]

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
    for row, got in zip(MISSED, persistent([(*row[:4], 148) for row in MISSED])):
        assert (row[5] if got else row[4]) <= 1.13 * min(row[4:]), row
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
