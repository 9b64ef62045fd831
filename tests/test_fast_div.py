"""Division by a launch constant (csrc/fast_div.cuh), compiled for the host: the attention forward's work list is decoded with it."""
import subprocess

from attention_autotuner_b200.build import CSRC

PROGRAM = r"""
#include "fast_div.cuh"
#include <cstdio>
#include <random>
int main() {
  const long long top = 0x7fffffffLL;
  std::mt19937_64 rng(1);
  auto check = [&](long long n, int d) {
    if (n < 0 || n > top) return true;
    if (ab200::fast_div(static_cast<int>(n), ab200::make_fast_div(d)) == n / d) return true;
    printf("%lld / %d\n", n, d);
    return false;
  };
  bool ok = true;
  for (int k = 0; k < 4000; ++k) {
    const int bits = 1 + static_cast<int>(rng() % 31);
    const int d = k < 1200 ? k + 1 : k < 1231 ? (k == 1200 ? 0x7fffffff : 1 << (k - 1201)) : 1 + static_cast<int>(rng() % ((1ull << bits) - 1));
    for (long long q : {0LL, 1LL, 2LL, top / d - 1, top / d, static_cast<long long>(rng() % (top / d + 1))})
      for (long long off : {-1LL, 0LL, 1LL, static_cast<long long>(d) - 1}) ok = check(q * d + off, d) && ok;
    ok = check(top, d) && check(static_cast<long long>(rng() % (top + 1)), d) && ok;
  }
  printf(ok ? "ok\n" : "bad\n");
}
"""


def test_quotients_are_exact(tmp_path):
    (tmp_path / "d.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, str(tmp_path / "d.cpp"), "-o", str(tmp_path / "d")], check=True)
    assert subprocess.run([str(tmp_path / "d")], capture_output=True, text=True, check=True).stdout == "ok\n"
