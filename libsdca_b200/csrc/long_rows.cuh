// Rows longer than a warp's registers hold (more than 1024 floats / 512 doubles): one thread block
// per row for the knapsack and top-k operators.
//
// The row is read from HBM once, into shared memory when it fits, and every thread keeps the
// largest entry of its share on the way.  The maxima are folded into 32 group maxima -- each an
// entry of its own -- from which one warp derives a cut below the whole support: the threshold of
// the same projection restricted to those 32 entries is a lower bound of the threshold of the row,
// because leaving entries out only lowers the sum that the threshold balances.  The entries above
// the cut (about twenty of 10 000 normally distributed ones) are compacted, one warp solves on
// them, and the block maps the row and stores it.  The general routine of thresholds.cuh needs
// about fifteen passes of one warp over the whole row instead.
//
// Bound: HBM, one read and one write of the matrix.  Several blocks of 256 threads are resident on
// an SM, so that while one of them reduces or solves the others keep loads and stores in flight.
#pragma once

#include "fast_rows.cuh"

namespace sdcab {

constexpr int kLongMaxThreads = 512;
constexpr int kLongDoubles = 1024;
constexpr int kLongSlots = 1024;       // candidates a block keeps; rows with more take the general routine

// A row cut at 16-byte boundaries: `head` entries before the first one, then whole vectors, then
// the rest.  Entry i sits at position i + shift of the staged copy, which puts the vectors on
// 16-byte boundaries there as well.
template <typename Data>
struct LongRow {
  typedef typename VecOf<Data>::type Vec;
  static constexpr int VN = VecOf<Data>::N;
  static constexpr int kBatch = 4;     // vectors a thread has in flight
  const Data* p;
  int m, head, nvec, shift;

  __device__ __forceinline__ LongRow(const Data* p_, int m_) : p(p_), m(m_) {
    const int off = static_cast<int>((reinterpret_cast<uintptr_t>(p_) & 15) / sizeof(Data));
    head = min(off ? VN - off : 0, m);
    nvec = (m - head) / VN;
    shift = off;                       // off + head is a multiple of VN (or the row ends before it)
  }
  __device__ __forceinline__ const Vec* vectors() const { return reinterpret_cast<const Vec*>(p + head); }

  // f(entries) on this thread's share of the row in global memory, a vector's VN entries or one at a
  // time; with `copy` the entries are left in the staged copy as well
  template <typename F>
  __device__ __forceinline__ void read(Data* copy, F&& f) const {
    const int nt = blockDim.x;
    const Vec* gv = vectors();
    Vec* cv = reinterpret_cast<Vec*>(copy + (copy ? shift + head : 0));
    int i = threadIdx.x;
    for (; i + (kBatch - 1) * nt < nvec; i += kBatch * nt) {
      Vec v[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) v[b] = __ldcg(gv + i + b * nt);
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        if (copy) cv[i + b * nt] = v[b];
        f(reinterpret_cast<const Data(&)[VN]>(v[b]));
      }
    }
    for (; i < nvec; i += nt) {
      const Vec v = __ldcg(gv + i);
      if (copy) cv[i] = v;
      f(reinterpret_cast<const Data(&)[VN]>(v));
    }
    edges([&](int j) {
      const Data x[1] = {p[j]};
      if (copy) copy[j + shift] = x[0];
      f(x);
    });
  }
  // the same from the staged copy (every entry is visited by the thread that copied it)
  template <typename F>
  __device__ __forceinline__ void revisit(const Data* copy, F&& f) const {
    const Vec* cv = reinterpret_cast<const Vec*>(copy + shift + head);
#pragma unroll 4
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      const Vec v = cv[i];
      f(reinterpret_cast<const Data(&)[VN]>(v));
    }
    edges([&](int j) {
      const Data x[1] = {copy[j + shift]};
      f(x);
    });
  }
  // out_i = f(a_i); the rows of `out` may sit differently on the 16-byte grid
  template <typename F>
  __device__ __forceinline__ void map(const Data* copy, Data* out, F&& f) const {
    const bool same_grid = ((reinterpret_cast<uintptr_t>(p) ^ reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (same_grid) {
      const Vec* src = copy ? reinterpret_cast<const Vec*>(copy + shift + head) : vectors();
      Vec* dst = reinterpret_cast<Vec*>(out + head);
#pragma unroll 4
      for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
        Vec v = copy ? src[i] : __ldcs(src + i);
        Data* e = reinterpret_cast<Data*>(&v);
#pragma unroll
        for (int c = 0; c < VN; ++c) e[c] = f(e[c]);
        __stcs(dst + i, v);
      }
      edges([&](int i) { out[i] = f(p[i]); });
    } else {
      for (int i = threadIdx.x; i < m; i += blockDim.x) out[i] = f(copy ? copy[i + shift] : p[i]);
    }
  }

 private:
  template <typename F>
  __device__ __forceinline__ void edges(F&& f) const {
    const int tid = threadIdx.x;
    if (tid < head) f(tid);
    const int rest = head + nvec * VN;
    if (tid >= 32 && tid - 32 < m - rest) f(rest + tid - 32);
  }
};

__device__ __forceinline__ float max_of(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double max_of(double a, double b) { return max_(a, b); }

// What pass 1 needs besides the maximum.
template <int PROX> struct LongKind {
  static constexpr bool kSimplex = (PROX == kTopkSimplex || PROX == kTopkSimplexBiased);
  static constexpr bool kCone = (PROX == kTopkCone);
  static constexpr bool kKnapsack = (PROX == kKnapsackEq || PROX == kKnapsackLe || PROX == kKnapsackLeBiased);
};

// The cut from the 32 group maxima (one per lane, unordered), by warp 0.  Returns false when no
// cut is known to lie below the support.
template <typename R, int PROX, typename Data>
__device__ __forceinline__ bool long_row_cut(Data gmax, const ProxParams& q, const TopkConsts<R>& tc, R rho,
                                             bool equality, R* sorted, int lane, Data& cut) {
  LaneRow<Data> g;
  g.x = gmax; g.valid = true; g.reported = 32;
  const int n = __popc(__ballot_sync(kFullMask, gmax > -num<Data>::inf()));
  if (n < 32) return false;            // rows this long fill every group
  const Sorted<R> c = sort_candidates<R>(g, 32, lane);
  const R top = c.at(0);
  const R slack = (abs_(top) + static_cast<R>(q.rhs)) * num<R>::eps() * 64;
  R bound;
  if (LongKind<PROX>::kKnapsack) {
    // t_j = (sum of the j largest - rhs) / j bounds t from below for every j as long as no entry
    // reaches hi; the same for the root of t = rho sum (a_i - t)_+
    const R hi = static_cast<R>(q.hi), rhs = static_cast<R>(q.rhs);
    bound = warp_max(over_count(c.P - rhs, lane + 1));
    // the clipped row stays below rhs: t = 0 without any candidates
    if (!equality) return false;
    // t >= rho rhs is the equality case; below that the root of t = rho sum (a_i - t)_+ counts
    if (PROX == kKnapsackLeBiased && rho != R(0) && bound < rho * rhs + slack)
      bound = min_(bound, warp_max(rho * c.P / (R(1) + rho * static_cast<R>(lane + 1))));
    // entries add up to rhs at most: no entry is above it
    if (!(hi >= rhs) && !(top - bound <= hi)) return false;
  } else {
    // the k + 1 largest entries are candidates in any case
    const R tau = c.at(q.k);
    bound = tau;
    if (LongKind<PROX>::kSimplex) {
      bound = tau - tc.H;
      Thr<R> sub;
      R sum_U;
      if (sorted_capped_simplex<R>(c, tc.H, static_cast<R>(q.rhs), q.k, lane, sorted, sub, sum_U))
        bound = max_(bound, sub.t);
      bound = min_(bound, tau);
    }
  }
  const R low = bound - slack - abs_(bound) * num<R>::eps() * 16 - num<R>::tiny();
  cut = round_down(low, Data(0));
  return cut > -num<Data>::inf();
}

// Descending bitonic sort of `count` (a power of two) values by the block.
template <typename Data>
__device__ __forceinline__ void block_sort_desc(Data* v, int count) {
  for (int k = 2; k <= count; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < count; i += blockDim.x) {
        const int o = i ^ j;
        if (o > i) {
          const Data x = v[i], y = v[o];
          if (((i & k) == 0) ? (x < y) : (y < x)) { v[i] = y; v[o] = x; }
        }
      }
      __syncthreads();
    }
  }
}

// Descending sort of the first `count` (at most 32) values of a warp, one per lane; the lanes from there
// on hold -inf.  Five candidates take six exchanges instead of the fifteen of a whole warp.
template <typename T>
__device__ __forceinline__ T sort_first_desc(T v, int count, int lane) {
  for (int k = 2; k < 2 * count; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      const T w = __shfl_xor_sync(kFullMask, v, j);
      const bool keep_max = ((lane & j) != 0) != ((lane & k) == 0);
      v = keep_max ? (w > v ? w : v) : (w < v ? w : v);
    }
  }
  return v;
}

// More candidates than a warp holds: out of line, so that the registers are set by the common case.
template <typename R, typename Data>
__device__ __noinline__ bool simplex_of_long_list(const Data* list, int total, int k, R rhs, R rho, Thr<R>* thr) {
  return topk_simplex_without_search<R>(StridedRow<Data>(list, total), k, rhs, rho, false, *thr);
}

// The thresholds from the `total` candidates in `slots`, by warp 0.  `s` is the sum that pass 1
// took: of the positive entries (cone), of the entries clipped to [0, hi] (knapsack_le).
template <typename R, int PROX, typename Data>
__device__ __forceinline__ FastStatus long_row_solve(Data* slots, int total, int m, R s,
                                                     const ProxParams& q, const TopkConsts<R>& tc, R rho,
                                                     R* sorted, int lane, Thr<R>& thr) {
  const R rhs = static_cast<R>(q.rhs);
  if (!LongKind<PROX>::kKnapsack && total <= q.k) return kFastNeedsFullRow;
  if (total < 1) return kFastNeedsFullRow;
  // Slots are handed out in the order in which the block's threads come by.  Lists that one warp holds
  // are sorted here, longer ones by the block: every sum over them is the same from run to run.
  LaneRow<Data> cand;
  cand.valid = lane < total;
  cand.x = lane < total ? slots[lane] : -num<Data>::inf();
  cand.reported = m;
  if (LongKind<PROX>::kKnapsack && total <= 32) {
    cand.x = sort_first_desc(cand.x, total, lane);
    if (cand.valid) slots[lane] = cand.x;
    __syncwarp();
  }
  StridedRow<Data> list(slots, total);
  if (LongKind<PROX>::kSimplex) {
    if (total <= 32)
      return topk_simplex_of_candidates<R>(cand, total, m, q.k, rhs, rho, tc, sorted, lane, thr);
    return simplex_of_long_list<R>(slots, total, q.k, rhs, rho, &thr) ? kFastDone : kFastNeedsFullRow;
  }
  if (LongKind<PROX>::kCone) {
    R top;
    if (total <= 32) {
      const Sorted<R> c = sort_candidates<R>(cand, total, lane);
      if (sorted_special_cases<R>(c, m, q.k, tc.inv_K, thr) != kProjGeneral) return kFastDone;
      top = c.at(0);
    } else {
      if (topk_special_cases<R>(list, q.k, tc.K, thr) != kProjGeneral) return kFastDone;
      top = static_cast<R>(slots[0]);  // sorted
    }
    // U empty: t = 0 and hi = s / k (include/sdca/prox/topk_cone.h:83-98)
    const R hi = s * tc.inv_K;
    if (!(s > 0 && top - 16 * num<R>::eps() <= hi)) return kFastNeedsFullRow;
    thr = make_thr(R(0), R(0), hi, 0, 0, num<R>::inf(), R(0));
    return kFastDone;
  }
  const R hi = static_cast<R>(q.hi);
  thr = (PROX == kKnapsackLeBiased && rho != 0) ? thr_knapsack_le_biased<R>(list, R(0), hi, rhs, rho)
                                                : thr_knapsack_eq<R>(list, R(0), hi, rhs);
  return thr.status == kThrSolved ? kFastDone : kFastNeedsFullRow;
}

template <typename Data, typename R, int PROX>
__global__ void __launch_bounds__(kLongMaxThreads, 2)
long_rows_kernel(const Data* a, Data* out, int m, long long n, ProxParams q, int staged) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ Data s_max[kLongMaxThreads];
  __shared__ R s_part[kLongMaxThreads / 32];
  __shared__ R sorted[64];
  __shared__ Data slots[kLongSlots];
  __shared__ int s_count, s_full;
  __shared__ Data s_cut;
  __shared__ R s_sum, s_t, s_lo, s_hi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  Data* const copy = staged ? reinterpret_cast<Data*>(smem_raw) : nullptr;
  constexpr bool kNeedsSum = LongKind<PROX>::kCone || PROX == kKnapsackLe || PROX == kKnapsackLeBiased;
  const R rho = (PROX == kTopkSimplexBiased || PROX == kKnapsackLeBiased) ? static_cast<R>(q.rho) : R(0);
  const R rhs = static_cast<R>(q.rhs);
  const TopkConsts<R> tc(q.k > 0 ? q.k : 1, rhs, rho);
  for (long long r = blockIdx.x; r < n; r += gridDim.x) {
    const LongRow<Data> row(a + r * m, m);
    Data mx = -num<Data>::inf(), zero = 0;
    R sum = 0;
    row.read(copy, [&](const auto& e) {
#pragma unroll
      for (const Data x : e) {
        mx = max_of(mx, x);
        zero += x * Data(0);           // stays 0 unless an entry is infinite or NaN
        if (LongKind<PROX>::kCone) sum += static_cast<R>(max_of(x, Data(0)));
        else if (kNeedsSum) sum += min_(max_(static_cast<R>(x), R(0)), static_cast<R>(q.hi));
      }
    });
    s_max[tid] = mx;
    if (kNeedsSum) {
      sum = warp_sum(sum);
      if (lane == 0) s_part[warp] = sum;
    }
    // infinities and NaN are left to the general routine
    const bool full_row = __syncthreads_or(!(zero == Data(0)));
    if (warp == 0) {
      Data g = s_max[lane];
      for (int w = 1; w < warps; ++w) g = max_(g, s_max[w * 32 + lane]);
      R total_sum = 0;
      if (kNeedsSum) for (int w = 0; w < warps; ++w) total_sum += s_part[w];
      // knapsack_le (include/sdca/prox/knapsack_le.h:17-44): the clipped sum decides between t = 0
      // and the projection onto <1, x> = rhs
      const bool le = PROX == kKnapsackLe || (PROX == kKnapsackLeBiased && rho == R(0));
      const bool equality = !le || total_sum > rhs + num<R>::eps() * max_(R(1), abs_(rhs));
      Data cut = num<Data>::inf();
      int verdict = full_row ? 1 : 0;  // 1: the general routine, 2: done with t = 0
      if (!verdict && !equality) verdict = 2;
      if (!verdict && !long_row_cut<R, PROX>(g, q, tc, rho, equality, sorted, lane, cut)) verdict = 1;
      if (lane == 0) {
        s_count = 0; s_cut = cut; s_full = verdict; s_sum = total_sum;
        if (verdict == 2) { s_t = R(0); s_lo = R(0); s_hi = static_cast<R>(q.hi); }
      }
    }
    __syncthreads();
    int verdict = s_full;
    if (verdict == 0) {
      const Data cut = s_cut;
      auto collect = [&](const auto& e) {
        bool any = false;
#pragma unroll
        for (const Data x : e) any |= x > cut;
        if (!any) return;              // one branch per vector: hardly any holds a candidate
        for (const Data x : e) {
          if (x > cut) {
            const int pos = atomicAdd(&s_count, 1);
            if (pos < kLongSlots) slots[pos] = x;
          }
        }
      };
      if (copy) row.revisit(copy, collect); else row.read(nullptr, collect);
      __syncthreads();
      const int total = s_count;
      if (total > 32 && total <= kLongSlots) {
        int pow2 = 64;
        while (pow2 < total) pow2 <<= 1;
        for (int i = total + tid; i < pow2; i += blockDim.x) slots[i] = -num<Data>::inf();
        __syncthreads();
        block_sort_desc(slots, pow2);
      }
      if (total > kLongSlots) verdict = 1;
    }
    if (warp == 0 && verdict != 2) {
      Thr<R> thr;
      FastStatus st = kFastNeedsFullRow;
      if (verdict == 0)
        st = long_row_solve<R, PROX>(slots, s_count, m, s_sum, q, tc, rho, sorted, lane, thr);
      if (st != kFastDone) {
        __syncwarp();
        thr = full_row_thresholds<R, Data, PROX>(copy ? copy + row.shift : row.p, m, &q);
      }
      if (lane == 0) { s_t = thr.t; s_lo = thr.lo; s_hi = thr.hi; }
    }
    __syncthreads();
    const Applier<Data> f(make_thr(s_t, s_lo, s_hi, 0, 0, R(0), R(0)), kMapIdentity, 1.0);
    row.map(copy, out + r * m, f);
    __syncthreads();                   // the copy is free for the next row
  }
}

template <typename Data, typename R, int PROX>
int launch_long(const Data* a, Data* out, int m, long long n, const ProxParams& q, cudaStream_t stream) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc) return rc;
  auto kernel = long_rows_kernel<Data, R, PROX>;
  const size_t row_bytes = (static_cast<size_t>(m) + 2 * VecOf<Data>::N) * sizeof(Data);
  // static shared memory: the candidate slots (up to 8 KB), the maxima (4 KB) and small change
  const int staged = row_bytes + 16 * 1024 <= info.smem_optin ? 1 : 0;
  const size_t smem = staged ? row_bytes : 0;
  // Short rows want many small blocks (a block's barriers and its one solving warp are covered by
  // the others), rows that leave room for one or two copies on an SM want as many threads as fit.
  const int threads = row_bytes <= 16 * 1024 ? 128 : (row_bytes <= 56 * 1024 ? 256 : kLongMaxThreads);
  if (smem > 32 * 1024) {
    rc = allow_shared_memory(reinterpret_cast<const void*>(kernel), smem);
    if (rc) return rc;
  }
  int per_sm = 0;
  SDCAB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  if (per_sm < 1) per_sm = 1;
  const int blocks = static_cast<int>(std::min<long long>(n, static_cast<long long>(per_sm) * info.sm_count));
  kernel<<<blocks, threads, smem, stream>>>(a, out, m, n, q, staged);
  SDCAB_CUDA_TRY(cudaGetLastError());
  return SDCAB_OK;
}

// Rows above the register kernels' limit (fast_rows.cuh takes the shorter ones).  Bounded k: the cut comes from
// 32 group maxima.  The knapsack operators with lo = 0 and positive hi and rhs, as in the register rows.
template <typename Data, typename R>
int launch_long_rows(int prox, const Data* a, Data* out, int m, long long n, const ProxParams& q,
                     cudaStream_t stream) {
  if (m <= 32 * 8 * VecOf<Data>::N) return kNoFastPath;
  // Rows of doubles beyond twice that keep the general kernel: the thresholds of its variable fixing
  // carry an error that grows with the row (5e-13 at 4000 entries, 1e-11 at 15 000), and results would
  // move by that much.
  if (sizeof(Data) == 8 && m > kLongDoubles) return kNoFastPath;
  const bool knapsack = q.lo == 0 && q.hi > 0 && q.rhs > 0;
  const bool topk = q.k <= 24;
  switch (prox) {
    case kKnapsackEq: return knapsack ? launch_long<Data, R, kKnapsackEq>(a, out, m, n, q, stream) : kNoFastPath;
    case kKnapsackLe: return knapsack ? launch_long<Data, R, kKnapsackLe>(a, out, m, n, q, stream) : kNoFastPath;
    case kKnapsackLeBiased:
      return knapsack ? launch_long<Data, R, kKnapsackLeBiased>(a, out, m, n, q, stream) : kNoFastPath;
    case kTopkSimplex: return topk ? launch_long<Data, R, kTopkSimplex>(a, out, m, n, q, stream) : kNoFastPath;
    case kTopkSimplexBiased:
      return topk ? launch_long<Data, R, kTopkSimplexBiased>(a, out, m, n, q, stream) : kNoFastPath;
    case kTopkCone: return topk ? launch_long<Data, R, kTopkCone>(a, out, m, n, q, stream) : kNoFastPath;
    default: break;
  }
  return kNoFastPath;
}

}  // namespace sdcab
