// Order in which the persistent chain kernels take their work: the row blocks (128 or 256 rows) of every slice, dealt to the
// workers (CTAs, or CTA pairs) of the grid by position. Three orders, chosen per launch by pick_work_order:
//
//   kOrderSlices  one item at a time, slice after slice. For items of equal cost (no causal mask) the most loaded worker
//                 holds ceil(items / workers).
//   kOrderPairs   pairs (k-th heaviest, k-th lightest row block of a slice) of equal cost, slice after slice: balanced up
//                 to one pair under a causal mask, and neighbouring workers share a slice's streamed operands in L2. With
//                 few pairs per worker that unit is coarse: 16 pairs use 16 workers where 32 items could use 32.
//   kOrderSnake   all items, heaviest row blocks of every slice first, dealt forwards and backwards in turn. The remainder
//                 is then made of the lightest items. A worker's neighbours are on other slices, so operands are re-read
//                 from DRAM if those of the slices in flight do not fit in L2.
// Measured: RetNet forward B=1 H=8 L=500 (dqk 256, dv 512; 32 items, 16 pairs, 74 CTA pairs) 20.5 us a pass with pairs, 14.4 to
// 15.7 with the items one by one. The attention kernels do not use this structure. The persistent forward keeps its pairs (a
// snake order cost it 4 %: spills in the softmax loop, K and V of all slices in flight out of L2) and leaves the shapes that
// pairs balance badly to its grid form. In the backward the order evaluated at run time cost the dQ kernel 5 % (B=8 H=32 L=1795
// d=64: 442 -> 466 us), so its single blocks are a specialisation of the kernels (fa_bwd_singles).
#pragma once

namespace ab200 {

enum WorkOrder : int { kOrderSlices = 0, kOrderPairs = 1, kOrderSnake = 2 };

// The order as the kernels evaluate it, in every role at every item: one division, selects instead of branches (a branch
// per order made the 128-register kernels spill).
struct WorkList {
  int nrb;    // row blocks per slice; rank 0 is the heaviest under a causal mask
  int units;  // what is dealt: items, or pairs of them; below 2^30
  int per;    // units per slice (pairs, slices) or per rank (snake)
  int pair;   // 1: units are pairs
  int snake;  // 1: rank by rank, every other round backwards

  // positions a worker has to ask step() for
  __host__ __device__ int steps(int workers) const { return ((units + workers - 1) / workers) << pair; }
  // Item at position u of a worker: rank k of its row block and slice; false if there is none at this position.
  __host__ __device__ bool step(int u, int worker, int workers, int& k, int& slice) const {
    const int i = (u >> pair) * workers + ((u & snake) ? workers - 1 - worker : worker);
    if (i >= units) return false;
    const int q = i / per, r = i - q * per;
    const int j = snake ? q : r;
    slice = snake ? r : q;
    k = (u & pair) ? nrb - 1 - j : j;
    return !((u & pair) && k == j);  // the middle row block of an odd count is its own partner
  }
};

inline WorkList work_list(int order, int slices, int nrb) {
  const int npair = (nrb + 1) / 2;
  if (order == kOrderPairs) return WorkList{nrb, slices * npair, npair, 1, 0};
  if (order == kOrderSnake) return WorkList{nrb, slices * nrb, slices, 0, 1};
  return WorkList{nrb, slices * nrb, nrb, 0, 0};
}

// triangular: row blocks of a slice cost from one column block up to all of them (else all the same).
// slice_bytes: operands streamed for one slice.
// Pairs unless the other order loads the busiest worker less; under a causal mask also only where the operands of the
// slices in flight stay in one half of L2 (with 200 MB of them the RetNet backward at B=8 H=8 L=2048 took 1184 us instead
// of 1111).
inline int pick_work_order(int slices, int nrb, int workers, bool triangular, double slice_bytes) {
  const long long pairs = static_cast<long long>(slices) * ((nrb + 1) / 2), items = static_cast<long long>(slices) * nrb;
  const long long pair_rounds = (pairs + workers - 1) / workers, item_rounds = (items + workers - 1) / workers;
  if (!triangular) return item_rounds < 2 * pair_rounds ? kOrderSlices : kOrderPairs;
  const double waste = static_cast<double>(pair_rounds) * workers / (0.5 * items);
  const bool in_l2 = slice_bytes * (slices < workers ? slices : workers) <= 50e6;
  return waste > 1.02 && in_l2 ? kOrderSnake : kOrderPairs;
}

inline WorkList make_work_list(int slices, int nrb, int workers, bool triangular, double slice_bytes) {
  return work_list(pick_work_order(slices, nrb, workers, triangular, slice_bytes), slices, nrb);
}

}  // namespace ab200
