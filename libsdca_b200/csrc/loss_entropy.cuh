// Loss stage of the softmax objective with the score row in registers: rows of up to 1024 classes,
// float or double, training and held-out sets.
//
// The general kernel reduces every term of every example over the warp and works out each example's
// closed forms on 32 lanes for one lane's worth of result: 17 000 cycles an example, most of them
// latency at four blocks of 128 registers per SM.  Here only what an example needs before it can go
// on is reduced at once -- its largest score and its sum of exponentials; every lane keeps its own
// shares of the other sums over all the examples of its warp, and the logarithms of the sums of
// exponentials are taken for 32 examples at a time.  A whole evaluation of 30 000 x 101 doubles with
// 300 features: 192 us, 272 us with the general kernel (113 us of it).  Bound: the double-precision
// pipe (an exponential and, with A, a logarithm per entry).
#pragma once

#include "loss_rows.cuh"

namespace sdcab {

// the largest of the lanes' values (no NaN among them)
__device__ __forceinline__ float largest_of_lanes(float v) { return warp_max_fast(v); }
// doubles through the integer reduction unit: the halves of the order-preserving integer
__device__ __forceinline__ double largest_of_lanes(double v) {
  const long long bits = __double_as_longlong(v);
  const long long key = bits ^ static_cast<long long>(static_cast<unsigned long long>(bits >> 63) >> 1);
  const int hi = static_cast<int>(key >> 32);
  const int top_hi = __reduce_max_sync(kFullMask, hi);
  const unsigned top_lo = __reduce_max_sync(kFullMask, hi == top_hi ? static_cast<unsigned>(key) : 0u);
  const long long top = (static_cast<long long>(top_hi) << 32) | top_lo;
  return __longlong_as_double(top ^ static_cast<long long>(static_cast<unsigned long long>(top >> 63) >> 1));
}

// NE: entries per lane, entry j of the row with lane j mod 32.
template <typename Data, typename R, int NE>
__global__ void __launch_bounds__(kLossThreads)
eval_softmax_loss_kernel(LossArgs g, const Data* __restrict__ scores, const Data* __restrict__ A,
                         double* __restrict__ block_partials, unsigned long long* __restrict__ hist) {
  __shared__ double warp_sums[kLossThreads / 32][3];
  __shared__ unsigned int local_hist[kHistLocal];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = kLossThreads / 32;
  for (int i = threadIdx.x; i < kHistLocal; i += kLossThreads) local_hist[i] = 0;
  __syncthreads();
  const int m = g.m;
  const R c = static_cast<R>(g.obj.c);
  const R entropy_c = x_log_x(c);
  double primal = 0, dual = 0, reg = 0;   // this lane's shares
  R kept_sum = 0, kept_base = 0;          // lane r: example r of the last 32
  int kept = 0;
  auto settle = [&]() {
    // include/sdca/math/log_exp.h:88-103 with l2_entropy.h:77-91
    if (lane < kept) primal += static_cast<double>(kept_base + log1p_(kept_sum));
    kept = 0;
  };
  for (long long e = static_cast<long long>(blockIdx.x) * warps + warp; e < g.n;
       e += static_cast<long long>(gridDim.x) * warps) {
    const Data* s_g = scores + e * m;
    const long long ex = g.first + e;
    const Data* a_g = (g.is_train && A) ? A + (g.a_row_offset + ex) * m : nullptr;
    const int y = static_cast<int>(g.labels[ex]);
    Data s[NE];
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      const int j = lane + 32 * i;
      s[i] = j < m ? __ldcs(s_g + j) : -num<Data>::inf();
    }
    Data top = s[0], own = s[0];
#pragma unroll
    for (int i = 1; i < NE; ++i) {
      top = max_(top, s[i]);
      own = (y >> 5) == i ? s[i] : own;
    }
    own = __shfl_sync(kFullMask, own, y & 31);
    top = largest_of_lanes(top);
    // the other classes scoring at least as high as the label (eval/primal.h:42-52), the sum of
    // exp(s_j - top) without one instance of the largest score.  The entries past the row's end, -inf,
    // are left out of all three: a label's score of -inf is no higher than they are.
    int rank = 0, ties = 0;
    R sum = 0;
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      const int j = lane + 32 * i;
      if (j < m) {
        rank += (j != y && s[i] >= own) ? 1 : 0;
        if (s[i] == top) ++ties;
        else sum += exp_(static_cast<R>(s[i]) - static_cast<R>(top));
      }
    }
    sum = warp_sum(sum);
    const int counts = warp_sum((ties << 16) + rank);
    rank = counts & 0xffff; ties = counts >> 16;
    // The one that is left out never enters the sum: next to it a small remainder would be lost.  Every
    // other tie adds exp(0) (and makes the loss of several infinite scores NaN, as the general kernel's).
    if (ties != 1) sum += static_cast<R>(ties - 1) * exp_(static_cast<R>(top) - static_cast<R>(top));
    if (lane == 0) {
      if (rank < kHistLocal) atomicAdd(&local_hist[rank], 1u);
      else atomicAdd(&hist[rank], 1ull);
    }
    if (lane == kept) {
      kept_sum = sum;
      kept_base = static_cast<R>(top) - static_cast<R>(own);
    }
    if (++kept == 32) settle();
    if (a_g) {
      // l2_entropy.h:94-114 with one label: the entropies of the other classes' variables and of
      // c - a_y
      R acc = 0, dot = 0;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int j = lane + 32 * i;
        if (j < m) {
          const R v = static_cast<R>(__ldcs(a_g + j));
          acc += x_log_x(j == y ? c - v : -v);
          if (g.kernel_input) dot += v * static_cast<R>(s[i]);   // eval/regularizer.h:82-98
        }
      }
      dual -= static_cast<double>(acc);
      if (lane == 0) dual += static_cast<double>(entropy_c);
      reg += static_cast<double>(dot) * 0.5;
    }
  }
  settle();
  primal = warp_sum(primal); dual = warp_sum(dual); reg = warp_sum(reg);
  if (lane == 0) { warp_sums[warp][0] = primal; warp_sums[warp][1] = dual; warp_sums[warp][2] = reg; }
  __syncthreads();
  if (threadIdx.x < 4) {
    double total = 0;
    if (threadIdx.x < 3)
      for (int w = 0; w < warps; ++w) total += warp_sums[w][threadIdx.x];
    block_partials[static_cast<size_t>(blockIdx.x) * 4 + threadIdx.x] = total;
  }
  for (int i = threadIdx.x; i < kHistLocal && i < m; i += kLossThreads)
    if (local_hist[i]) atomicAdd(&hist[i], static_cast<unsigned long long>(local_hist[i]));
}

inline bool softmax_loss_usable(const LossArgs& g) { return g.obj.id == kObjL2Entropy && g.m <= 1024; }

template <typename Data, typename R>
int launch_softmax_loss(const LossArgs& g, const Data* scores, const Data* A, double* partials,
                        unsigned long long* hist, int blocks, cudaStream_t stream) {
  auto kernel = g.m <= 128 ? eval_softmax_loss_kernel<Data, R, 4>
                           : (g.m <= 256 ? eval_softmax_loss_kernel<Data, R, 8>
                                         : eval_softmax_loss_kernel<Data, R, 32>);
  kernel<<<blocks, kLossThreads, 0, stream>>>(g, scores, A, partials, hist);
  SDCAB_CUDA_TRY(cudaGetLastError());
  return SDCAB_OK;
}

}  // namespace sdcab
