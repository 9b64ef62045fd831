"""The order of work of the persistent kernels (csrc/work_order.cuh), compiled for the host: in each order every (row
block, slice) is taken exactly once, whatever the number of workers, and the chosen order loads no worker more than pairs
of row blocks would, under a causal mask and without one; and the limit on the operands in flight."""
import subprocess

from attention_autotuner_b200.build import CSRC

PROGRAM = r"""
#define __host__
#define __device__
#include "work_order.cuh"
#include <cstdio>
#include <vector>
using namespace ab200;
// most loaded worker, or -1 if an item is missed, taken twice or out of range; items of rank k cost nrb - k under a causal
// mask (triangular), all the same without one
static long run(const WorkList& w, int slices, int workers, bool triangular = true) {
  std::vector<char> seen(static_cast<size_t>(w.nrb) * slices, 0);
  long worst = 0;
  size_t n = 0;
  for (int c = 0; c < workers; ++c) {
    long load = 0;
    for (int u = 0; u < w.steps(workers); ++u) {
      int k = -1, s = -1;
      if (!w.step(u, c, workers, k, s)) continue;
      if (k < 0 || k >= w.nrb || s < 0 || s >= slices || seen[static_cast<size_t>(s) * w.nrb + k]++) return -1;
      load += triangular ? w.nrb - k : 1;
      ++n;
    }
    if (load > worst) worst = load;
  }
  return n == seen.size() ? worst : -1;
}
int main() {
  const int nrbs[] = {1, 2, 3, 6, 7, 12, 16, 33}, slices[] = {1, 2, 7, 16, 64, 129}, workers[] = {1, 2, 5, 74, 148};
  for (int nrb : nrbs) for (int sl : slices) for (int full : workers) {
    long load[3];
    for (int order = 0; order < 3; ++order) {
      const WorkList w = work_list(order, sl, nrb);
      const int grid = w.units < full ? w.units : full;
      load[order] = run(w, sl, grid);
      if (load[order] < 0) { printf("order %d nrb %d slices %d workers %d\n", order, nrb, sl, full); return 1; }
    }
    const int pick = pick_work_order(sl, nrb, full, true, 1e3);
    if (load[pick] > load[kOrderPairs]) { printf("pick nrb %d slices %d workers %d\n", nrb, sl, full); return 1; }
    // operands of the slices in flight beyond half of L2: pairs, whatever the balance
    const int in_flight = sl < full ? sl : full;
    if (pick_work_order(sl, nrb, full, true, 51e6 / in_flight) != kOrderPairs ||
        pick_work_order(sl, nrb, full, true, 49e6 / in_flight) != pick) {
      printf("limit nrb %d slices %d workers %d\n", nrb, sl, full);
      return 1;
    }
    // equal costs: slice after slice or in pairs, whichever loads the busiest worker least
    const int flat = pick_work_order(sl, nrb, full, false, 1e9);
    long even[2];
    for (int order : {kOrderSlices, kOrderPairs}) {
      const WorkList w = work_list(order, sl, nrb);
      even[order] = run(w, sl, w.units < full ? w.units : full, false);
    }
    if (flat > kOrderPairs || even[flat] != (even[0] < even[1] ? even[0] : even[1])) {
      printf("flat nrb %d slices %d workers %d\n", nrb, sl, full);
      return 1;
    }
  }
  return 0;
}
"""


def test_every_item_once_and_no_worker_above_the_pairs(tmp_path):
    src = tmp_path / "order.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "order"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
