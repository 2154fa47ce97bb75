// Pieces shared by the kernels that walk through a block of SDCA steps (fit_steps.cuh, fit_entropy.cuh)
// and by their launches (fit.cu).
#pragma once

#include "update_core.cuh"

namespace sdcab {

constexpr int kHelperThreads = 256;   // keep the score rows current while a step is worked out
constexpr int kFitThreads = 32 + kHelperThreads;   // warp 0 steps
constexpr int kBlockSteps = 64;   // steps whose score products are formed together

// ---- the chain ---------------------------------------------------------------
// One thread block walks through the `count` steps of a block of examples
// i_0, i_1, ...  It starts from S[b] = scores of example i_b under the variables
// the block began with; after step b changed a_{i_b} by delta, the scores of
// every later example of the block move by delta * G[b][b''], with
// G[b][b''] = K[i_b, i_b''] (kernel input) or -<x_{i_b}, x_{i_b''}> with
// delta = a_old - a_new (features, update.h:77-84), so S[b''] += delta * G[b][b'']
// keeps the rows current.  Rows are corrected in step order, which fixes the
// order of the floating-point sums.
struct ChainArgs {
  ObjectiveParams o;
  const int64_t* order;    // the block's examples: order[0 .. count)
  const int64_t* labels;
  const int64_t* offsets;  // multilabel objectives: the labels of example i are labels[offsets[i] .. offsets[i+1])
  double* S;               // count x m, scores at the start of the block (updated in place
                           // when they do not fit on chip)
  const double* G;         // kBlockSteps x kBlockSteps (row b = example i_b)
  void* A;                 // dual variables, n x m
  void* D;                 // features: count x m, a_old - a_new of every step (0 if skipped)
  double* t_keep;          // n: every example's threshold from its last step
  int m, count, kernel_input, s_on_chip;
};

struct ChainKernel {
  void (*kernel)(ChainArgs) = nullptr;
  int threads = 0;
};
// Chosen in fit_steps.cuh, which is compiled for each pair of types in a translation unit of its own.
template <typename Data, typename R>
ChainKernel pick_chain_kernel(const ObjectiveParams& o, long long m, bool s_on_chip);

// The general routine, out of line so that the chain's registers are set by the
// common path.
template <typename R, typename Data>
__device__ __noinline__ void general_update(const ObjectiveParams* o, Data norm2, const Data* scores,
                                            Data* a, Data* v, int m, int y) {
  update_dual_variables_multiclass<R, Data>(*o, norm2, scores, a, v, m, y);
}

template <typename R, typename Data>
__device__ __noinline__ void general_update_multilabel(const ObjectiveParams* o, Data norm2,
                                                       const Data* scores, Data* a, Data* v, int m,
                                                       const unsigned* mask, int num_labels) {
  update_dual_variables_multilabel_hinge<R, Data>(*o, norm2, scores, a, v, m, mask, num_labels);
}

// dst[0 .. n) = src[0 .. n) by `threads` threads, n doubles on 16-byte boundaries, eight loads in
// flight per thread: the chain cannot start before its 80 KB are in.
__device__ __forceinline__ void fill_shared(double* dst, const double* __restrict__ src, int n, int tid, int threads) {
  const double2* s2 = reinterpret_cast<const double2*>(src);
  double2* d2 = reinterpret_cast<double2*>(dst);
#pragma unroll 8
  for (int t = tid; t < n / 2; t += threads) d2[t] = s2[t];
  if (tid == 0 && (n & 1)) dst[n - 1] = src[n - 1];
}

// Rows b + 1 .. of S move by the change of step b - 1 times G[b - 1][row]; h numbers the
// kHelperThreads threads that do it.
__device__ __forceinline__ void move_later_rows(double* S, const double* G, const double* d_prev, int b,
                                                int count, int m, int h) {
  const double* Gp = G + (b - 1) * kBlockSteps;
  constexpr int kRowGroups = kHelperThreads >> 7, kFlight = 8;
  for (int j = h & 127; j < m; j += 128) {
    const double dj = d_prev[j];
    for (int first = b + 1 + (h >> 7); first < count; first += kFlight * kRowGroups) {
      double sv[kFlight], gv[kFlight];
#pragma unroll
      for (int r = 0; r < kFlight; ++r) {
        const int bb = first + r * kRowGroups;
        if (bb < count) {
          gv[r] = Gp[bb];
          sv[r] = S[static_cast<size_t>(bb) * m + j];
        }
      }
#pragma unroll
      for (int r = 0; r < kFlight; ++r) {
        const int bb = first + r * kRowGroups;
        if (bb < count) S[static_cast<size_t>(bb) * m + j] = fma(dj, gv[r], sv[r]);
      }
    }
  }
}

}  // namespace sdcab
