// sweep_times.h -- what one sweep of a layer's tets takes on each launch path
// (B200, us), by material and precision: the choice between them.
//
// Measured on beams of 28 k to 3.5 M tets (25 to 33 colours) and batches of
// 64 to 4,096 blocks of 192 to 10,368 tets, whole recorded steps of 20
// iterations, with bodies' or monitored loops one iteration per launch.  One
// mesh, us per sweep in a fixed loop, dataflow / through L2 / colour launches:
//   Neo-Hookean FP32       28 k 33/67/61    98 k 43/63/68   166 k 55/67/82
//                         263 k 86/70/90   393 k 138/75/96  831 k 340/78/107
//                         1.3 M -/117/118  2.4 M -/203/186  3.5 M -/290/218
//   Neo-Hookean FP64       28 k 38/111/73   98 k 57/106/92  166 k 83/111/112
//                         263 k 126/121/122 393 k 201/147/128 831 k -/170/145
//   StVK, damped, FP64     28 k 78/149/114  98 k 110/148/142 166 k 176/155/157
// and with one iteration per launch (a monitored loop, the monitor's 7 to
// 20 us included):
//   Neo-Hookean FP32       28 k 50/80/67    98 k 63/82/71   166 k 86/84/75
//                         393 k 172/97/96  831 k 520/105/138
//   Neo-Hookean FP64       28 k 57/123/77   98 k 90/125/83  166 k 130/128/90
//   64 blocks of 10,368    FP32 92/100/121   FP64 123/202/166
// The sweep through L2 loses in FP64 at every size (its records are three
// words); above 1.3 M tets its records and rest data leave L2 and it loses in FP32.
// Estimates within a tenth of one another can pick the longer path: nine
// damped FP64 blocks of 83 k tets in a fixed loop take 204 here, 186 by colours.
#pragma once

#include <algorithm>
#include <cmath>

namespace mlx {

struct SweepTimes {
  double chain;    // dataflow: a colour, while the warps wait for records
  double chunk;    // dataflow: a chunk of the largest part, while they share the SM (a sum of squares)
  double contact;  // dataflow: the same with every 3rd to 13th vertex in contact
  double colour;   // a colour launch
  double tet;      // colour launches: a tet's traffic
  double l2;       // the sweep through L2: a tet of a vertex's chain
};

enum SweepMat : int { SWEEP_NH, SWEEP_BLOCKS, SWEEP_BLOCKS_DAMPED, SWEEP_LAME, SWEEP_LAME_DAMPED };

inline const SweepTimes& sweep_times(bool fp64, SweepMat m) {
  static const SweepTimes t[2][5] = {{{0.98, 0.137, 0.27, 1.80, 5.0e-5, 2.85},
                                      {0.98, 0.137, 0.33, 1.92, 7.5e-5, 2.85},
                                      {1.50, 0.21, 0.36, 2.30, 6.5e-5, 3.8},
                                      {1.07, 0.145, 0.33, 2.27, 5.5e-5, 3.0},
                                      {1.30, 0.17, 0.33, 2.50, 5.5e-5, 3.45}},
                                     {{1.10, 0.215, 0.26, 2.10, 1.15e-4, 4.8},
                                      {1.56, 0.28, 0.45, 2.65, 1.4e-4, 5.4},
                                      {2.30, 0.37, 0.56, 3.35, 1.2e-4, 6.6},
                                      {1.58, 0.27, 0.45, 2.90, 1.1e-4, 5.7},
                                      {1.88, 0.34, 0.48, 3.25, 9.0e-5, 6.4}}};
  return t[fp64 ? 1 : 0][m];
}

// The dataflow sweep of `colours` colours whose largest part has `chunks`
// chunks, on `ctas` CTAs.  A chunk takes longer where most SMs are busy: 83 k
// tets per 16 CTAs, 1 / 4 clusters 40 / 45 us FP32, 92 / 131 damped FP64; with
// resting contacts 0.25 / 0.36 us a chunk on 16 / 72 CTAs (FP32 Neo-Hookean).
// once: one iteration per launch, which reads positions and multipliers anew
// (FP64, 20 / 140 / 875 chunks of 148 CTAs: 18 of 50, 32 of 97, 419 of 717).
inline double flow_us(const SweepTimes& t, bool fp64, SweepMat m, double colours, double chunks, int ctas, bool once,
                      bool contacts) {
  const double busy = std::min(1.0, ctas / 148.0);
  const double shared = 1.0 + 0.9 * std::max(0.0, busy - 0.25);
  const double chain = t.chain * colours + (contacts ? 17.0 : 0.0);
  const double issue = chunks * (contacts ? t.contact * (1.0 + 1.3 * std::clamp(busy - 0.1, 0.0, 0.35)) : t.chunk * shared);
  const double q = std::max(0.0, chunks - 0.5 * colours);  // (half a chunk per colour is rounding)
  const double again = fp64 ? 6.0 + q * (0.12 + busy * (0.15 + 0.00035 * q))
                            : m == SWEEP_NH ? 5.0 + q * (0.04 + 0.08 * busy) : 8.0 + q * (0.07 + 0.08 * busy);
  return std::sqrt(chain * chain + issue * issue) + (once ? again : 0.0);
}
inline double colours_us(const SweepTimes& t, double colours, double tets) { return t.colour * colours + t.tet * tets; }
// The sweep through L2; chain: tets at a vertex, on average (22 of the beams'
// 33 colours; layers with bodies 13 to 15, where it is 11 us shorter than the
// colour launches at 120 to 220 k tets).
inline double l2_us(const SweepTimes& t, double chain, double tets, bool once) {
  return t.l2 * chain + 2e-5 * tets + 8e-5 * std::max(0.0, tets - 8.5e5) + (once ? 6.0 : 0.0);
}

}  // namespace mlx
