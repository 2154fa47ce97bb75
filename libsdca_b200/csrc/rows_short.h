// Dispatch to the kernels of rows_short.cu: one thread per row.
#pragma once

#include "prox_core.cuh"

namespace sdcab {

// Thresholds in double: with float thresholds what a caller gets depends on the order of the float
// sums, and those launches keep the route they have always had.
template <typename Data>
int launch_short_rows(int prox, const Data* a, Data* out, int m, long long n, const ProxParams& q,
                      cudaStream_t stream);

// The longest rows that one thread per row takes, float and double data.  us at 262 144 rows (k = 8 for
// the top-k operators), thread / warp, at the limit and one size past it:
//   knapsack            f32 48:  88 / 125,  64: 144 / 130      f64 32:  76 / 113,  40:  92 / 116
//   knapsack_le         f32 48:  93 / 171,  64: 150 / 178      f64 40:  96 / 140,  48: 131 / 141
//   knapsack_le_biased  f32 48: 104 / 188,  64: 160 / 177      f64 40: 110 / 176,  48: 147 / 161
//   topk_simplex        f32 48: 184 / 247,  64: 267 / 247      f64 48: 247 / 370,  64: 382 / 370
//   topk_simplex_biased f32 40: 470 / 828,  48: 539 / 575      f64 40: 490 / 959,  48: 617 / 669
//   topk_cone           f32 64: 202 / 305,  80: 224 / 242      f64 64: 253 / 415,  80: 331 / 372
//   topk_cone_biased    f32 32: 298 / 1465, 40: 370 / 491      f64 32: 297 / 1421, 40: 379 / 506
//   entropy             f32 48:  76 /  96,  64:  96 /  95      f64 64: 185 / 207,  80: 283 / 277
//   topk_entropy        f32 32: 146 / 501,  40: 153 / 171      f64 64: 331 / 325,  80: 489 / 378
// The lines were drawn where the thread stopped being faster before its searches took their cuts and
// lost a comparison per entry: some could lie one size further out now.
// The Lambert operators' rows differ too much in cost to share a warp.
inline int short_row_limit(int prox, bool is_double) {
  switch (prox) {
    case kKnapsackEq: return is_double ? 32 : 48;
    case kKnapsackLe: case kKnapsackLeBiased: return is_double ? 40 : 48;
    case kTopkSimplex: return 48;
    case kTopkSimplexBiased: return 40;
    case kTopkCone: return 64;
    case kTopkConeBiased: return 32;
    case kEntropy: return is_double ? 64 : 48;
    case kTopkEntropy: return is_double ? 64 : 32;
    default: return 0;
  }
}

// A thread's time grows with the row and does not shrink with the launch, so the fewer rows there
// are, the shorter they have to be: knapsack of 32 floats took 19 us against a warp's 18 us at 16 384
// rows, 36 against 51 us at 98 304 and 59 against 115 us at 262 144.
inline bool short_rows_usable(int prox, int m, long long n, bool is_double) {
  return m <= short_row_limit(prox, is_double) && n >= 3000LL * m;
}

}  // namespace sdcab
