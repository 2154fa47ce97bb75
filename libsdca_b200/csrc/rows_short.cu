// Rows of few entries, many of them: one thread per row.
//
// A warp on a row of ten entries has 22 idle lanes and pays the full price of every reduction: 600
// and more warp instructions per row, the same as for a hundred entries.  Here a block brings 128
// rows into shared memory (they are contiguous, so the loads cover whole lines whatever the length),
// every thread runs the searches of thresholds.cuh on its own row with a group of one lane --
// the rows sit an odd number of entries apart, so that the lanes of a warp read 32 different banks
// -- and the block writes the mapped rows back.  Bound: instruction issue, m entries times the
// passes of the slowest of 32 rows.  262 144 rows of 10 floats against one warp
// per row: knapsack 30 / 117 us, top-k cone (k = 5) 71 / 798 us, top-k entropy 69 / 649 us; rows_short.h
// has the limits.
#define SDCAB_LANE_PER_ROW 1
#include <algorithm>

#include "common_host.h"
#include "prox_core.cuh"
#include "rows_short.h"

namespace sdcab {
namespace {

constexpr int kShortThreads = 128;

// The entries of a row above a cut, as a row of their own (NaN is not above any).
template <typename Data>
struct RowAbove {
  typedef Data data_type;
  const Data* p;
  int m, count;
  Data cut;
  __device__ __forceinline__ RowAbove(const Data* p_, int m_, Data cut_) : p(p_), m(m_), count(0), cut(cut_) {
    for (int i = 0; i < m; ++i) count += p[i] > cut ? 1 : 0;
  }
  __device__ __forceinline__ int size() const { return count; }
  template <typename F>
  __device__ __forceinline__ void for_each(F&& f) const {
    for (int i = 0; i < m; ++i) {
      const Data x = p[i];
      if (x > cut) f(x, i);
    }
  }
};
__device__ __forceinline__ float at_most(double v, float) { return __double2float_rd(v); }
__device__ __forceinline__ double at_most(double v, double) { return v; }

template <int PROX> struct ShortKind {
  static constexpr bool kKnapsack = (PROX == kKnapsackEq || PROX == kKnapsackLe || PROX == kKnapsackLeBiased);
  static constexpr bool kSimplex = (PROX == kTopkSimplex || PROX == kTopkSimplexBiased);
  static constexpr bool kCone = (PROX == kTopkCone || PROX == kTopkConeBiased);
  static constexpr bool kTopk = kSimplex || kCone;
};

// The knapsack operators with lo = 0.  As long as no entry reaches hi, the largest alone adds
// max - t <= rhs to the sum: the support lies above max - rhs, and the search takes the entries above
// that cut only.  Its running t so stays as exact as those entries are, whatever else the row holds --
// the classes that a caller has ruled out by -inf or by the lowest number of the type, above all, whose
// sum the search over the whole row would carry along -- as in the kernels of one warp per row.
template <typename Data, int PROX>
__device__ __forceinline__ Thr<double> short_knapsack(const Data* row, int m, const ProxParams& q) {
  const StridedRow<Data> whole(row, m);
  if (!(q.lo == 0 && q.hi > 0 && q.rhs > 0)) return compute_thresholds<double>(PROX, whole, q);
  const double hi = q.hi, rhs = q.rhs, eps = num<double>::eps() * max_(1.0, rhs);
  const bool le = PROX == kKnapsackLe || (PROX == kKnapsackLeBiased && q.rho == 0);
  Data largest = -num<Data>::inf();
  double clipped = 0;
  whole.for_each([&](Data x, int) {
    largest = max_(largest, x);
    if (le) clipped += min_(max_(0.0, static_cast<double>(x)), hi);
  });
  if (le && !(clipped > rhs + eps)) return make_thr(0.0, 0.0, hi, 0, 0, hi, 0.0);
  const double top = static_cast<double>(largest);
  if (abs_(top) < num<double>::inf()) {
    const RowAbove<Data> near_top(row, m, at_most(top - rhs - (abs_(top) + rhs) * num<double>::eps() * 8, Data()));
    const Thr<double> thr = thr_knapsack_eq<double>(near_top, 0.0, hi, rhs);
    if (!(top - thr.t > hi)) {
      if (le || PROX != kKnapsackLeBiased || thr.t >= q.rho * rhs - eps) return thr;
      return thr_knapsack_le_biased_root<double>(whole, 0.0, hi, rhs, q.rho, thr.t);
    }
  }
  return compute_thresholds<double>(PROX, whole, q);
}

// Entries below -wide_limit() or NaN make a row of the top-k operators a wide one.  On the simplex, sums
// with such entries in them would cost the support its digits (no support reaches that far down, a
// thousand times rhs, unless k entries or fewer are above it); on the cone, only sums that overflow.
template <typename Data, int PROX>
__device__ __forceinline__ Data wide_limit(const ProxParams& q) {
  if (ShortKind<PROX>::kSimplex) return q.rhs > 0 ? static_cast<Data>(1024 * q.rhs) : num<Data>::inf();
  return sizeof(Data) == 8 ? static_cast<Data>(1e300) : num<Data>::max();
}
// The projection of a wide row, from its entries above the limit (t >= v_(k+1) - rhs / k on the simplex,
// t >= -(k - 1) max on the cone): the classes that a caller has ruled out do not take part.
template <typename Data, int PROX>
__device__ __noinline__ Thr<double> short_topk_of_wide_row(const Data* row, int m, const ProxParams* q) {
  const Data limit = wide_limit<Data, PROX>(*q);
  const int k = q->k;
  const double rho = (PROX == kTopkSimplexBiased || PROX == kTopkConeBiased) ? q->rho : 0.0;
  if (RowAbove<Data>(row, m, -limit).count > k) {
    if (ShortKind<PROX>::kCone) return thr_topk_cone<double>(RowAbove<Data>(row, m, -limit), k, rho);
    const Data reach = limit + static_cast<Data>(q->rhs);
    Thr<double> thr;
    if (topk_simplex_without_search<double>(RowAbove<Data>(row, m, -reach), k, q->rhs, rho, false, thr)) return thr;
    return thr_topk_cone_search<double>(RowAbove<Data>(row, m, -static_cast<Data>(k) * reach), k, rho);
  }
  return compute_thresholds<double>(PROX, StridedRow<Data>(row, m), *q);
}

template <typename Data, int PROX>
__device__ __forceinline__ Thr<double> short_row_thresholds(const Data* row, int m, const ProxParams& q, bool wide) {
  if constexpr (ShortKind<PROX>::kKnapsack) return short_knapsack<Data, PROX>(row, m, q);
  if constexpr (ShortKind<PROX>::kTopk) {
    if (wide) return short_topk_of_wide_row<Data, PROX>(row, m, &q);
  }
  return compute_thresholds<double>(PROX, StridedRow<Data>(row, m), q);
}

template <typename Data, int PROX>
__global__ void __launch_bounds__(kShortThreads)
short_rows_kernel(const Data* a, Data* out, int m, long long n, ProxParams q, int pitch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ bool wide[kShortThreads];
  Data* tile = reinterpret_cast<Data*>(smem_raw);
  const int tid = threadIdx.x;
  const Data lowest = -wide_limit<Data, PROX>(q);
  wide[tid] = false;
  __syncthreads();
  const int row_step = kShortThreads / m, col_step = kShortThreads % m;
  for (long long first = static_cast<long long>(blockIdx.x) * kShortThreads; first < n;
       first += static_cast<long long>(gridDim.x) * kShortThreads) {
    const int rows = static_cast<int>(min(static_cast<long long>(kShortThreads), n - first));
    const int total = rows * m;
    const Data* src = a + first * m;
    Data* dst = out + first * m;
    {
      int r = tid / m, c = tid % m;
#pragma unroll 4
      for (int i = tid; i < total; i += kShortThreads) {
        const Data x = __ldcs(src + i);
        tile[r * pitch + c] = x;
        if (ShortKind<PROX>::kTopk && !(x >= lowest)) wide[r] = true;
        r += row_step; c += col_step;
        if (c >= m) { c -= m; ++r; }
      }
    }
    __syncthreads();
    if (tid < rows) {
      Data* row = tile + tid * pitch;
      const Thr<double> thr = short_row_thresholds<Data, PROX>(row, m, q, wide[tid]);
      wide[tid] = false;
      const Applier<Data> f(thr, prox_map(PROX), q.alpha);
      for (int i = 0; i < m; ++i) row[i] = f(row[i]);
    }
    __syncthreads();
    {
      int r = tid / m, c = tid % m;
#pragma unroll 4
      for (int i = tid; i < total; i += kShortThreads) {
        __stcs(dst + i, tile[r * pitch + c]);
        r += row_step; c += col_step;
        if (c >= m) { c -= m; ++r; }
      }
    }
    __syncthreads();
  }
}

template <typename Data, int PROX>
int launch_short(const Data* a, Data* out, int m, long long n, const ProxParams& q, cudaStream_t stream) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc) return rc;
  auto kernel = short_rows_kernel<Data, PROX>;
  const int pitch = m | 1;
  const size_t smem = static_cast<size_t>(kShortThreads) * pitch * sizeof(Data);
  if (smem > 48 * 1024) {
    rc = allow_shared_memory(reinterpret_cast<const void*>(kernel), smem);
    if (rc) return rc;
  }
  int per_sm = 0;
  SDCAB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kShortThreads, smem));
  const long long want = (n + kShortThreads - 1) / kShortThreads;
  const int blocks = static_cast<int>(std::min<long long>(
      want, static_cast<long long>(std::max(1, per_sm)) * info.sm_count));
  kernel<<<blocks, kShortThreads, smem, stream>>>(a, out, m, n, q, pitch);
  SDCAB_CUDA_TRY(cudaGetLastError());
  return SDCAB_OK;
}

}  // namespace

template <typename Data>
int launch_short_rows(int prox, const Data* a, Data* out, int m, long long n, const ProxParams& q,
                      cudaStream_t stream) {
  switch (prox) {
#define CASE(ID) case ID: return launch_short<Data, ID>(a, out, m, n, q, stream);
    CASE(kKnapsackEq) CASE(kKnapsackLe) CASE(kKnapsackLeBiased) CASE(kTopkSimplex)
    CASE(kTopkSimplexBiased) CASE(kTopkCone) CASE(kTopkConeBiased) CASE(kEntropy) CASE(kTopkEntropy)
#undef CASE
    default: break;
  }
  return SDCAB_ERR_PROX;
}

template int launch_short_rows<float>(int, const float*, float*, int, long long, const ProxParams&, cudaStream_t);
template int launch_short_rows<double>(int, const double*, double*, int, long long, const ProxParams&, cudaStream_t);

}  // namespace sdcab
