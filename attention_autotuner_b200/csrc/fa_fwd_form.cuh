// Which kernel, and which form of the grid, serves an attention forward: rules on sizes alone, also compiled for the host by
// their tests.
#pragma once

namespace ab200 {

// The decoding kernel (fa_decode_sm100.cuh): one head dimension of 64 or 128 for q, k and v and up to 16 query rows, the rows of
// its tile. At d = 128 its warps' partial rows are added at the end at a cost that grows with the rows, which a few keys do
// not hide: more than 12 rows with up to 256 keys stay on the large tile. Decoding kernel / large tile in us, bf16, 1, 148 and
// 2048 slices: Lq = 16, Lkv = 128 9.8 / 7.2, 10.2 / 8.2, 69.6 / 55.3; Lq = 16, Lkv = 256 10.2 / 8.2, 10.2 / 10.2, 85.3 / 77.8 (but
// 512 slices 22.5 / 26.1); Lq = 16, Lkv = 512 12.3 / 12.3, 12.3 / 13.4, 115 / 130; Lq = 12, Lkv = 128 8.2 / 7.2, 8.2 / 8.2, 59.4 / 55.3, Lkv = 256
// 9.2 / 8.2, 10.2 / 10.2, 75.5 / 77.8. With 8 rows, and at d = 64 with any, it is the faster one or at most 1 us behind at every
// size measured (1 to 2048 slices, 16 to 4096 keys). The number of slices has no part in the rule: a slice has the same
// bits in any launch.
inline bool fa_decode_shape(int dqk, int dv, int Lq, int Lkv) {
  if (dv != dqk || Lq > 16) return false;
  return dqk == 64 || (dqk == 128 && (Lq <= 12 || Lkv > 256));
}

// Time of both forms in units of one KV block of one item (128 keys against 256 rows, about 1.8 us at d = 128), as the busiest
// SM spends it:
//   * grid form: a CTA per item, given out as SMs become free. An item costs its blocks and 2.6 more for set-up and epilogue.
//     Items of equal cost: rounds of them. Under a causal mask they run from `first` to `last` blocks (heaviest ones first):
//     the mean load of an SM and 0.6 of the heaviest item, but no more than rounds of the heaviest.
//   * persistent form: one CTA per SM, pairs (heaviest with lightest item of a slice; the middle one of an odd count alone)
//     dealt in turn. What overlaps between items leaves 1.0 per item, and 2.0 once per launch. The busiest SM has only pairs,
//     unless the deal moves by one position of the slice's list per round (sms and the list's length without a common
//     factor), as it does with one item per slice: then its share of middle items.
// Constants fitted to 292 measurements of both forms of an earlier kernel, whose products of a tile waited for one another (10 to
// 2000 slices, Lq 64 to 4500, Lkv to 4096, d = 64 and 128, with and without a mask); over 138 measurements of the present one
// (8 to 2000 slices, Lq 64 to 5000, Lkv to 5000) the form picked is 0.2 % slower than the faster one on average, 13 % at worst.
// Comparing the rounds of pairs with those of items instead, whatever the blocks of an item, cost the earlier kernel 4.6 %
// on average and up to 42 %: with one item per slice both forms hold the same items, and short items gain most at their
// boundaries.
// Measured grid / persistent in us, without a mask (causal); d = 128 where not stated:
//   persistent:  2000 slices of L=64 73.4 / 52.5 (73.9 / 52.5), 1000 of L=256 65.6 / 48.2, d=64 57.6 / 40.6 (55.9 / 40.5),
//                400 of L=256 30.0 / 22.0, 512 of L=512 89.4 / 78.9 (78.5 / 65.5), 96 of L=1300 91.7 / 88.8 (70.3 / 65.6),
//                12 of L=5000 131.6 / 128.5 (95.8 / 70.2), 148 of L=2048 264 / 250 (175 / 161), 128 of L=4096 894 / 827
//   grid:        8 of L=512 d=64 12.3 / 18.6, 40 of L=2048 86.4 / 103.5 (57.9 / 67.7), 20 of L=4000 158 / 198 (97.5 / 111),
//                52 of L=1280 42.4 / 68.4 (38.0 / 50.6), 100 of L=700 41.8 / 49.6 (31.4 / 41.8), 60 of L=2700 202 / 225
//                (127 / 133), 200 of L=768 71.5 / 73.4 (57.1 / 65.0), 100 of L=1792 143.8 / 151.4
//   misses:      96 of Lq=512 Lkv=4096 107.5 / 121.4 and 256 of L=1024 causal 100.6 / 105.3, where the rule takes the
//                persistent form; d=64 96 of Lq=512 Lkv=4096 causal 99 / 95, where it takes the grid
struct FaFormCost {
  double grid, persistent;
};

inline FaFormCost fa_form_cost(long long slices, int Lq, int Lkv, bool causal, int sms) {
  const long long nqb = (Lq + 255ll) / 256, nblk = (Lkv + 127ll) / 128, shift = static_cast<long long>(Lkv) - Lq;
  auto blocks = [&](long long item) -> double {  // KV blocks its last row sees
    if (!causal) return static_cast<double>(nblk);
    const long long keys = 256 * (item + 1) + shift, n = keys > 0 ? (keys + 127) / 128 : 0;
    return static_cast<double>(n < nblk ? n : nblk);
  };
  const double first = blocks(0), last = blocks(nqb - 1), mean = 0.5 * (first + last);
  const long long items = slices * nqb, rounds = (items + sms - 1) / sms;
  const double even = static_cast<double>(rounds) * (first + 2.6), heavy = static_cast<double>(rounds) * (last + 2.6),
               spread = static_cast<double>(items) / sms * (mean + 2.6) + 0.6 * (last + 2.6);
  const double uneven = heavy < spread ? heavy : spread;

  const long long npair = (nqb + 1) / 2, units = (slices * npair + sms - 1) / sms;
  long long a = sms, b = npair;  // greatest common divisor
  while (b != 0) {
    const long long r = a % b;
    a = b;
    b = r;
  }
  const long long middles = (nqb % 2 != 0 && a == 1) ? units / npair : 0;
  return FaFormCost{even > uneven ? even : uneven,
                    static_cast<double>(units - middles) * (first + last + 2.0) + static_cast<double>(middles) * (mean + 1.0) + 2.0};
}

// Long items (more than 40 KV blocks on average) take the grid form whatever the count: a static work list loses more to the
// slowest SM than the boundaries cost. Grid / persistent, without a mask (causal): 16 slices of L=16384 1570 / 1887 (937 / 974),
// 64 of L=8192 1535 / 1704, 32 of Lq=1024 Lkv=9000 122 / 252.
inline bool fa_form_persistent(long long slices, int Lq, int Lkv, bool causal, int sms) {
  const int nblk = (Lkv + 127) / 128;
  if ((causal ? (nblk + 1) / 2 : nblk) > 40) return false;
  const FaFormCost c = fa_form_cost(slices, Lq, Lkv, causal, sms);
  return c.persistent < c.grid;
}

}  // namespace ab200
