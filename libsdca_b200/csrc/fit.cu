// SDCA fit on the device: solver::solve of the reference
// (include/sdca/solver.h:39-117) with update_variables
// (include/sdca/solver/update.h:52-107) as the step.
//
// The steps of an epoch form a sequential chain -- step s reads the variables
// step s-1 wrote -- but a step changes the dual variables of one example only,
// so the scores of the next 64 examples can be formed together, from the
// variables as they are now, by one product on the whole GPU (64 columns of K
// against A, or 64 examples against W); the chain itself then runs inside a
// single thread block that corrects the remaining score rows after every step
// by the one-example change (a 64 x 64 block of K, or of the examples' Gram
// matrix, is all it needs).  That turns N matrix-vector products per epoch into
// N / 64 matrix products and keeps the sequential part on chip.  For features
// the primal variables receive the block's rank-one changes afterwards, in
// step order.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <ctime>
#include <vector>

#include "common_host.h"
#include "eval_host.h"
#include "fit_chain.cuh"
#include "fit_host.h"
#include "gemm_blocked.cuh"
#include "primal.h"

namespace sdcab {
namespace {

// S[b][j] = sum over the slices of the split product, plus the share of the previous block's
// examples, which the product left out (kernel input) or whose changes W had not received yet
// (features): sum_b' P[b'][j] * Gx[b'][b], P = the variables a_{i'_b'} (kernel input) or the
// changes D[b'] (features).
template <typename Data>
struct PackArgs {
  const Data* s_parts; int slices; long long slice_stride;
  int count, m;
  double* S;
  const Data* P; const int64_t* prev_order;   // row b' of P: prev_order[b'], or b' if null
  int prev_count; const double* Gx;
};

// Latency bound: the steps wait for it.  The terms of each output are dealt to GROUPS threads (term z
// to thread z mod GROUPS, eight loads in flight); the partial sums are added in a fixed order.
template <typename Data, int GROUPS>
__global__ void __launch_bounds__(256) fit_pack_kernel(PackArgs<Data> p) {
  constexpr int kOutputs = 256 / GROUPS;
  __shared__ double part[GROUPS][kOutputs];
  const int lane = threadIdx.x % kOutputs, group = threadIdx.x / kOutputs;
  const long long t = static_cast<long long>(blockIdx.x) * kOutputs + lane;
  const long long s_elems = static_cast<long long>(p.count) * p.m;
  double acc = 0.0;
  if (t < s_elems) {
    const Data* src = p.s_parts + t;
#pragma unroll 8
    for (int z = group; z < p.slices; z += GROUPS) acc += static_cast<double>(src[z * p.slice_stride]);
    const int b = static_cast<int>(t / p.m), j = static_cast<int>(t % p.m);
#pragma unroll 8
    for (int bp = group; bp < p.prev_count; bp += GROUPS) {
      const long long row = p.prev_order ? p.prev_order[bp] : bp;
      acc = fma(static_cast<double>(p.P[row * p.m + j]), p.Gx[bp * kBlockSteps + b], acc);
    }
  }
  part[group][lane] = acc;
  __syncthreads();
  if (group == 0 && t < s_elems) {
    double total = 0.0;
#pragma unroll
    for (int g = 0; g < GROUPS; g += 2) total += part[g][lane] + part[g + 1][lane];
    p.S[t] = total;
  }
}

// Features: G[b][b'] = -<x_{i_b}, x_{i_b'}> within a block and Gx[b'][b] = -<x_{i'_b'}, x_{i_b}> from
// the previous block's examples, from the slices of the split product of the block's examples with
// the previous block's (the first prev_count columns) and its own.  64 outputs per thread block, the
// terms of each dealt to four threads.
template <typename Data>
__global__ void __launch_bounds__(256)
fit_gram_kernel(const Data* __restrict__ parts, int slices, int count, int prev_count,
                double* __restrict__ G, double* __restrict__ Gx) {
  __shared__ double part[4][64];
  const int b = threadIdx.x & 63, group = threadIdx.x >> 6;
  const int col = blockIdx.x;                       // 0 .. prev_count + count - 1
  const int cols = prev_count + count;
  const long long stride = static_cast<long long>(count) * cols;
  double acc = 0.0;
  if (b < count)
    for (int z = group; z < slices; z += 4) acc -= static_cast<double>(parts[z * stride + static_cast<long long>(b) * cols + col]);
  part[group][b] = acc;
  __syncthreads();
  if (group != 0 || b >= count) return;
  const double total = (part[0][b] + part[1][b]) + (part[2][b] + part[3][b]);
  if (col < prev_count) Gx[col * kBlockSteps + b] = total;
  else G[b * kBlockSteps + (col - prev_count)] = total;
}

// owner[i] = the block of 64 steps in which example i is visited this epoch
__global__ void fit_owner_kernel(const int64_t* __restrict__ order, long long n, int* __restrict__ owner) {
  const long long s = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s < n) owner[order[s]] = static_cast<int>(s / kBlockSteps);
}

// G[b][b'] = K[i_b, i_b'] within a block and Gx[b'][b] = K[i'_b', i_b] from the
// previous block's examples to this block's (kernel input).
template <typename Data>
__global__ void fit_gather_kernel(const Data* __restrict__ K, long long n,
                                  const int64_t* __restrict__ order, int count,
                                  const int64_t* __restrict__ prev_order, int prev_count,
                                  double* __restrict__ G, double* __restrict__ Gx) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  const int which = u / (kBlockSteps * kBlockSteps), e = u % (kBlockSteps * kBlockSteps);
  const int r = e / kBlockSteps, c = e % kBlockSteps;
  if (which == 0) {
    G[e] = (r < count && c < count) ? static_cast<double>(K[order[r] + n * order[c]]) : 0.0;
  } else if (which == 1 && prev_count > 0) {
    Gx[e] = (r < prev_count && c < count) ? static_cast<double>(K[prev_order[r] + n * order[c]]) : 0.0;
  }
}

// W_j <- W_j - x_{i_b} * D[b][j] for the steps of one block in step order, every
// product and difference rounded on its own like the reference's ger (update.h:83).
template <typename Data>
__global__ void __launch_bounds__(256)
fit_primal_update_kernel(Data* W, const Data* __restrict__ X, const Data* __restrict__ D,
                         const int64_t* __restrict__ order, int count, int m, long long d) {
  __shared__ Data s_d[kBlockSteps];
  __shared__ long long s_i[kBlockSteps];
  const int j = blockIdx.y;
  if (threadIdx.x < count) {
    s_d[threadIdx.x] = D[static_cast<size_t>(threadIdx.x) * m + j];
    s_i[threadIdx.x] = order[threadIdx.x];
  }
  __syncthreads();
  const long long r = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= d) return;
  Data w = W[d * j + r];
  for (int b = 0; b < count; ++b) {
    const Data dj = s_d[b];
    if (dj != Data(0)) w = sub_rn_(w, mul_rn_(X[d * s_i[b] + r], dj));
  }
  W[d * j + r] = w;
}

template <typename Data> int eval_sums_call(const sdcab_objective*, const sdcab_problem*, double*, void*);
template <> int eval_sums_call<float>(const sdcab_objective* o, const sdcab_problem* p, double* s, void* st) {
  return sdcab_eval_sums_f32_dev(o, p, s, nullptr, 0, st);
}
template <> int eval_sums_call<double>(const sdcab_objective* o, const sdcab_problem* p, double* s, void* st) {
  return sdcab_eval_sums_f64_dev(o, p, s, nullptr, 0, st);
}

struct DeviceBuffers {
  std::vector<void*> owned;     // three for each held-out set, and there may be any number of those
  cudaStream_t stream = nullptr, ahead = nullptr;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  cudaEvent_t ev_product[2] = {nullptr, nullptr}, ev_steps[2] = {nullptr, nullptr}, ev_start = nullptr;
  ~DeviceBuffers() {
    for (void* ptr : owned) cudaFree(ptr);
    for (int i = 0; i < 4; ++i) if (ev[i]) cudaEventDestroy(ev[i]);
    for (int i = 0; i < 2; ++i) {
      if (ev_product[i]) cudaEventDestroy(ev_product[i]);
      if (ev_steps[i]) cudaEventDestroy(ev_steps[i]);
    }
    if (ev_start) cudaEventDestroy(ev_start);
    if (ahead) cudaStreamDestroy(ahead);
    if (stream) cudaStreamDestroy(stream);
  }
  // One allocation for the arrays of a fit instead of one each: allocations and, more so, the
  // releases at the end wait for the device and for the driver's other callers.
  unsigned char* arena = nullptr;
  size_t arena_bytes = 0, arena_used = 0;
  static size_t padded(size_t bytes) { return (std::max<size_t>(bytes, 1) + 255) & ~static_cast<size_t>(255); }
  int reserve(size_t bytes) {
    void* ptr = nullptr;
    SDCAB_CUDA_TRY(cudaMalloc(&ptr, bytes));
    owned.push_back(ptr);
    arena = static_cast<unsigned char*>(ptr);
    arena_bytes = bytes;
    return SDCAB_OK;
  }
  template <typename T>
  int alloc(T** out, size_t elems) {
    const size_t bytes = padded(elems * sizeof(T));
    if (arena_bytes - arena_used >= bytes) {
      *out = reinterpret_cast<T*>(arena + arena_used);
      arena_used += bytes;
      return SDCAB_OK;
    }
    void* ptr = nullptr;
    SDCAB_CUDA_TRY(cudaMalloc(&ptr, bytes));
    owned.push_back(ptr);
    *out = static_cast<T*>(ptr);
    return SDCAB_OK;
  }
};

// The launches of one block of steps.
template <typename Data, typename R>
struct BlockRunner {
  ObjectiveParams o;
  const sdcab_problem* t;
  int sm_count = 0;
  size_t chain_smem = 0;
  ChainKernel chain;
  int s_on_chip = 0;
  int slices = 1, g_slices = 1;
  int64_t* order = nullptr;     // the epoch's order on the device
  double* S = nullptr;          // 64 x m
  double* t_keep = nullptr;     // n
  // two of each: block b + 1's products are formed while block b steps
  Data* s_parts[2] = {nullptr, nullptr};   // slices x 64 x m
  double* G[2] = {nullptr, nullptr};       // 64 x 64
  double* Gx[2] = {nullptr, nullptr};      // 64 x 64
  Data* D[2] = {nullptr, nullptr};         // features: 64 x m
  Data* g_parts = nullptr;                 // features: g_slices x 64 x 128
  int* owner = nullptr;                    // kernel input: n

  static int pick_slices(int tiles, long long k, int bk, int sm_count) {
    long long want = (2LL * sm_count + tiles - 1) / tiles;
    const long long most = std::max<long long>(1, k / (4LL * bk));
    return static_cast<int>(std::max<long long>(1, std::min(want, most)));
  }

  int launch_chain(const ChainArgs& c, cudaStream_t s) const {
    chain.kernel<<<1, chain.threads, chain_smem, s>>>(c);
    SDCAB_CUDA_TRY(cudaGetLastError());
    return SDCAB_OK;
  }

  int prepare(const DeviceInfo& info, DeviceBuffers& buf) {
    typedef SmallGemmTile<Data> GT;
    const long long m = t->m;
    sm_count = info.sm_count;
    const int tiles = static_cast<int>((m + GT::BN - 1) / GT::BN);
    slices = pick_slices(tiles, t->d, GT::BK, sm_count);
    g_slices = pick_slices(1, t->d, GT::BK, sm_count);
    const size_t fixed = (kBlockSteps * kBlockSteps + 2 * m) * sizeof(double) + 5 * m * sizeof(Data) +
                         static_cast<size_t>(2 * ((m + 31) / 32) + 2) * sizeof(unsigned);
    const size_t with_s = fixed + static_cast<size_t>(kBlockSteps) * m * sizeof(double);
    // beside the kernel's own static shared memory (up to 4 KB, by its step)
    cudaFuncAttributes attr;
    for (s_on_chip = 1; s_on_chip >= 0; --s_on_chip) {
      chain = pick_chain_kernel<Data, R>(o, m, s_on_chip != 0);
      chain_smem = s_on_chip ? with_s : fixed;
      SDCAB_CUDA_TRY(cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(chain.kernel)));
      if (chain_smem + attr.sharedSizeBytes <= info.smem_optin) break;
    }
    if (s_on_chip < 0) return SDCAB_ERR_TOO_LARGE;
    int rc = allow_shared_memory(reinterpret_cast<const void*>(chain.kernel), chain_smem);
    if (rc) return rc;
    const bool kernel_input = t->input_kind == SDCAB_INPUT_KERNEL;
    const size_t n = static_cast<size_t>(t->n), block_row = static_cast<size_t>(kBlockSteps) * m,
                 block_block = static_cast<size_t>(kBlockSteps) * kBlockSteps;
    size_t bytes = DeviceBuffers::padded(n * sizeof(int64_t)) + DeviceBuffers::padded(block_row * sizeof(double)) +
                   DeviceBuffers::padded(n * sizeof(double)) +
                   2 * (DeviceBuffers::padded(slices * block_row * sizeof(Data)) +
                        2 * DeviceBuffers::padded(block_block * sizeof(double))) +
                   DeviceBuffers::padded(SDCAB_EVAL_SUMS(m) * sizeof(double));   // the evaluation's sums
    bytes += kernel_input ? DeviceBuffers::padded(n * sizeof(int))
                          : 2 * DeviceBuffers::padded(block_row * sizeof(Data)) +
                                DeviceBuffers::padded(g_slices * 2 * block_block * sizeof(Data));
    rc = buf.reserve(bytes); if (rc) return rc;
    rc = buf.alloc(&order, n); if (rc) return rc;
    for (int h = 0; h < 2; ++h) {
      rc = buf.alloc(&s_parts[h], static_cast<size_t>(slices) * kBlockSteps * m); if (rc) return rc;
      rc = buf.alloc(&G[h], static_cast<size_t>(kBlockSteps) * kBlockSteps); if (rc) return rc;
      rc = buf.alloc(&Gx[h], static_cast<size_t>(kBlockSteps) * kBlockSteps); if (rc) return rc;
      if (!kernel_input) { rc = buf.alloc(&D[h], static_cast<size_t>(kBlockSteps) * m); if (rc) return rc; }
    }
    if (kernel_input) { rc = buf.alloc(&owner, static_cast<size_t>(t->n)); if (rc) return rc; }
    else { rc = buf.alloc(&g_parts, static_cast<size_t>(g_slices) * kBlockSteps * 2 * kBlockSteps); if (rc) return rc; }
    rc = buf.alloc(&S, static_cast<size_t>(kBlockSteps) * m); if (rc) return rc;
    rc = buf.alloc(&t_keep, static_cast<size_t>(t->n)); if (rc) return rc;
    SDCAB_CUDA_TRY(cudaMemsetAsync(t_keep, 0, static_cast<size_t>(t->n) * sizeof(double), buf.stream));
    return SDCAB_OK;
  }

  // W receives the changes of block b's steps.
  int update_primal(long long b, int count, cudaStream_t s) const {
    const dim3 grid(static_cast<unsigned>((t->d + 255) / 256), static_cast<unsigned>(t->m));
    fit_primal_update_kernel<Data><<<grid, 256, 0, s>>>(
        static_cast<Data*>(const_cast<void*>(t->w)), static_cast<const Data*>(t->x), D[b & 1],
        order + b * kBlockSteps, count, static_cast<int>(t->m), t->d);
    SDCAB_CUDA_TRY(cudaGetLastError());
    return SDCAB_OK;
  }

  // The products of block b: the scores of its examples and the matrix products between its
  // examples (G) and from the `prev` ones of the previous block to its own (Gx).
  int products(long long b, int count, int prev, cudaStream_t s) const {
    typedef SmallGemmTile<Data> GT;
    const int m = static_cast<int>(t->m), h = static_cast<int>(b & 1);
    const Data* X = static_cast<const Data*>(t->x);
    const int64_t* ord = order + b * kBlockSteps;
    GemmExtras x;
    x.a_gather = ord;
    x.slices = slices;
    x.c_slice_stride = static_cast<long long>(count) * m;
    int rc;
    if (t->input_kind == SDCAB_INPUT_KERNEL) {
      // S = K[:, block]' A : rows = columns of K (contiguous), A is n x m; block b - 1's examples
      // are left out (owner -1, the first block: nothing is)
      x.k_owner = owner; x.skip_owner = static_cast<int>(b - 1);
      rc = launch_gemm_tile<Data, GT>(X, static_cast<const Data*>(t->a), s_parts[h], count, m,
                                      static_cast<int>(t->n), t->n, m, m, false, s, x);
      if (rc) return rc;
      fit_gather_kernel<Data><<<2 * kBlockSteps * kBlockSteps / 256, 256, 0, s>>>(
          X, t->n, ord, count, b > 0 ? ord - kBlockSteps : nullptr, prev, G[h], Gx[h]);
    } else {
      // S = X[:, block]' W, both with the feature index contiguous
      const int d = static_cast<int>(t->d);
      rc = launch_gemm_tile<Data, GT>(X, static_cast<const Data*>(t->w), s_parts[h], count, m, d, t->d, t->d,
                                      m, true, s, x);
      if (rc) return rc;
      GemmExtras g;
      g.a_gather = ord; g.b_gather = ord - prev; g.slices = g_slices;
      const int cols = prev + count;
      g.c_slice_stride = static_cast<long long>(count) * cols;
      rc = launch_gemm_tile<Data, GT>(X, X, g_parts, count, cols, d, t->d, t->d, cols, true, s, g);
      if (rc) return rc;
      fit_gram_kernel<Data><<<cols, 256, 0, s>>>(g_parts, g_slices, count, prev, G[h], Gx[h]);
    }
    SDCAB_CUDA_TRY(cudaGetLastError());
    return SDCAB_OK;
  }

  // One epoch with the products one block ahead of the steps.  While block b steps on `sc`, block
  // b + 1's products are formed on `sg` from variables that lack block b's changes: its examples are
  // left out of A (kernel input; their rows are being rewritten), or W has received the changes up
  // to block b - 1 (features).  Block b's share is added afterwards, from the products between the
  // examples of the two blocks (fit_pack_kernel).  The serial schedule kept the steps waiting for
  // 35 us per block of 64 (100 classes, 500 float features).
  int run_epoch(long long n, cudaStream_t sc, cudaStream_t sg, cudaEvent_t (&ev_product)[2],
                cudaEvent_t (&ev_steps)[2], cudaEvent_t ev_start) const {
    const int m = static_cast<int>(t->m);
    const bool kernel_input = t->input_kind == SDCAB_INPUT_KERNEL;
    Data* A = static_cast<Data*>(const_cast<void*>(t->a));
    const long long blocks = (n + kBlockSteps - 1) / kBlockSteps;
    auto count_of = [&](long long b) { return static_cast<int>(std::min<long long>(kBlockSteps, n - b * kBlockSteps)); };
    if (kernel_input) {
      fit_owner_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, sc>>>(order, n, owner);
      SDCAB_CUDA_TRY(cudaGetLastError());
    }
    SDCAB_CUDA_TRY(cudaEventRecord(ev_start, sc));
    SDCAB_CUDA_TRY(cudaStreamWaitEvent(sg, ev_start, 0));
    // A fit of the top-k softmax builds on the last bits of its scores (thr_topk_entropy_biased): they
    // are summed as ever, from the W that has all changes.
    const bool keep_rounding = o.id == kObjL2EntropyTopk;
    const bool ahead = kernel_input || !keep_rounding;
    int rc = SDCAB_OK;
    if (ahead) {
      rc = products(0, count_of(0), 0, sg);
      if (rc) return rc;
      SDCAB_CUDA_TRY(cudaEventRecord(ev_product[0], sg));
    }
    for (long long b = 0; b < blocks; ++b) {
      const int h = static_cast<int>(b & 1), count = count_of(b);
      const int64_t* ord = order + b * kBlockSteps;
      if (ahead) SDCAB_CUDA_TRY(cudaStreamWaitEvent(sc, ev_product[h], 0));
      else { rc = products(b, count, 0, sc); if (rc) return rc; }
      PackArgs<Data> pk;
      pk.s_parts = s_parts[h]; pk.slices = slices; pk.slice_stride = static_cast<long long>(count) * m;
      pk.count = count; pk.m = m; pk.S = S;
      pk.P = kernel_input ? A : D[h ^ 1];
      pk.prev_order = kernel_input ? ord - kBlockSteps : nullptr;
      pk.prev_count = ahead && b > 0 ? kBlockSteps : 0;
      pk.Gx = Gx[h];
      const long long outputs = static_cast<long long>(count) * m;
      if (keep_rounding)
        fit_pack_kernel<Data, 4><<<static_cast<unsigned>((outputs + 63) / 64), 256, 0, sc>>>(pk);
      else
        fit_pack_kernel<Data, 8><<<static_cast<unsigned>((outputs + 31) / 32), 256, 0, sc>>>(pk);
      SDCAB_CUDA_TRY(cudaGetLastError());
      SDCAB_CUDA_TRY(cudaEventRecord(ev_steps[h], sc));   // block b - 1 has stepped, block b's scores are packed
      ChainArgs c;
      c.o = o; c.order = ord; c.labels = t->labels; c.offsets = t->offsets; c.S = S; c.G = G[h]; c.A = A;
      c.D = D[h];
      c.t_keep = t_keep; c.m = m; c.count = count; c.kernel_input = kernel_input ? 1 : 0; c.s_on_chip = s_on_chip;
      rc = launch_chain(c, sc);
      if (rc) return rc;
      // The next products may start once block b - 1 has stepped; they are released
      // together with block b's steps (after the pack), on a stream of lower priority,
      // so that the stepping thread block holds its SM before the products' thread
      // blocks spread over the others.
      if (!ahead) {
        rc = update_primal(b, count, sc);
        if (rc) return rc;
      } else if (b + 1 < blocks) {
        SDCAB_CUDA_TRY(cudaStreamWaitEvent(sg, ev_steps[h], 0));
        if (!kernel_input && b > 0) {
          rc = update_primal(b - 1, kBlockSteps, sg);
          if (rc) return rc;
        }
        rc = products(b + 1, count_of(b + 1), kBlockSteps, sg);
        if (rc) return rc;
        SDCAB_CUDA_TRY(cudaEventRecord(ev_product[h ^ 1], sg));
      }
    }
    if (ahead && !kernel_input) {
      // the last two blocks' changes (every earlier one has been waited for through ev_product)
      if (blocks > 1) { rc = update_primal(blocks - 2, kBlockSteps, sc); if (rc) return rc; }
      rc = update_primal(blocks - 1, count_of(blocks - 1), sc);
      if (rc) return rc;
    }
    return SDCAB_OK;
  }
};

bool is_permutation(const int64_t* p, long long n, std::vector<unsigned char>& seen) {
  seen.assign(static_cast<size_t>(n), 0);
  for (long long i = 0; i < n; ++i) {
    const int64_t v = p[i];
    if (v < 0 || v >= n || seen[static_cast<size_t>(v)]) return false;
    seen[static_cast<size_t>(v)] = 1;
  }
  return true;
}

template <typename Data, typename R>
int fit_dev(const sdcab_objective* obj, const sdcab_problem* train, const sdcab_fit_criteria* crit,
            const int64_t* permutations, sdcab_eval_record* evals, int64_t evals_cap,
            sdcab_fit_result* result, cudaStream_t user_stream,
            const sdcab_fit_history* hist = nullptr) {
  const long long n = train->n, m = train->m;
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc) return rc;

  DeviceBuffers buf;
  int prio_low = 0, prio_high = 0;
  SDCAB_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high));
  SDCAB_CUDA_TRY(cudaStreamCreateWithPriority(&buf.stream, cudaStreamNonBlocking, prio_high));
  SDCAB_CUDA_TRY(cudaStreamCreateWithPriority(&buf.ahead, cudaStreamNonBlocking, prio_low));
  for (int e = 0; e < 4; ++e) SDCAB_CUDA_TRY(cudaEventCreate(&buf.ev[e]));
  for (int e = 0; e < 2; ++e) {
    SDCAB_CUDA_TRY(cudaEventCreateWithFlags(&buf.ev_product[e], cudaEventDisableTiming));
    SDCAB_CUDA_TRY(cudaEventCreateWithFlags(&buf.ev_steps[e], cudaEventDisableTiming));
  }
  SDCAB_CUDA_TRY(cudaEventCreateWithFlags(&buf.ev_start, cudaEventDisableTiming));
  cudaStream_t s = buf.stream;
  // everything queued on the caller's stream so far comes first
  SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[0], user_stream));
  SDCAB_CUDA_TRY(cudaStreamWaitEvent(s, buf.ev[0], 0));

  BlockRunner<Data, R> runner;
  runner.o = to_params(obj);
  runner.t = train;
  rc = runner.prepare(info, buf);
  if (rc) return rc;
  double* sums_dev = nullptr;
  rc = buf.alloc(&sums_dev, static_cast<size_t>(SDCAB_EVAL_SUMS(m)));
  if (rc) return rc;

  // the reference's stopwatches run while it solves and evaluates (solver.h:81-131):
  // processor time by std::clock, wall time by a steady clock
  const std::clock_t cpu_begin = std::clock();
  const auto wall_begin = std::chrono::steady_clock::now();
  auto cpu_now = [&]() { return static_cast<double>(std::clock() - cpu_begin) / CLOCKS_PER_SEC; };
  auto wall_now = [&]() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now() - wall_begin).count();
  };
  int64_t epoch_now = 0;

  sdcab_problem ep = *train;
  ep.is_train = 1; ep.a_row_offset = 0; ep.include_primal_regularizer = 1;
  std::vector<double> sums(static_cast<size_t>(SDCAB_EVAL_SUMS(m)));
  std::vector<sdcab_eval_record> history;
  double eval_ms = 0, solve_ms = 0;
  auto evaluate = [&]() -> int {
    SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[2], s));
    int erc = SDCAB_OK;
    if (crit->recompute_primal && train->input_kind == SDCAB_INPUT_FEATURES) {
      // eval_recompute_primal (eval/core.h:148-182): W rebuilt from A, so that the
      // rounding of the steps' rank-one updates does not accumulate in it
      erc = primal_from_dual_dev<Data>(static_cast<const Data*>(train->x), static_cast<const Data*>(train->a),
                                       static_cast<const Data*>(train->w0),
                                       static_cast<Data*>(const_cast<void*>(train->w)), train->d, m, n, s);
      if (erc) return erc;
    }
    erc = eval_sums_call<Data>(obj, &ep, sums_dev, s);
    if (erc) return erc;
    SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[3], s));
    SDCAB_CUDA_TRY(cudaMemcpyAsync(sums.data(), sums_dev, sums.size() * sizeof(double),
                                   cudaMemcpyDeviceToHost, s));
    SDCAB_CUDA_TRY(cudaStreamSynchronize(s));
    float ms = 0;
    SDCAB_CUDA_TRY(cudaEventElapsedTime(&ms, buf.ev[2], buf.ev[3]));
    eval_ms += ms;
    sdcab_eval_record rec;
    const int64_t slot = static_cast<int64_t>(history.size());
    const bool keep = hist && slot < hist->cap;
    erc = eval_finish(obj, m, sums.data(), &rec,
                      (keep && hist->train_accuracy) ? hist->train_accuracy + slot * m : nullptr);
    if (erc) return erc;
    history.push_back(rec);
    if (evals && static_cast<int64_t>(history.size()) <= evals_cap) evals[history.size() - 1] = rec;
    if (keep) {
      if (hist->train) hist->train[slot] = rec;
      if (hist->epoch) hist->epoch[slot] = epoch_now;
      if (hist->wall_seconds) hist->wall_seconds[slot] = wall_now();
    }
    // every held-out set after the training set (solver.h:124-131): scores from the
    // variables of the training problem, primal loss and accuracy / rank loss only
    if (hist && hist->tests) {
      for (int64_t ti = 0; ti < hist->num_tests; ++ti) {
        sdcab_problem tp = hist->tests[ti];
        tp.input_kind = train->input_kind; tp.is_train = 0; tp.d = train->d; tp.m = train->m;
        tp.a = train->a; tp.w = train->w; tp.w0 = nullptr; tp.a_row_offset = 0;
        tp.include_primal_regularizer = 0;
        SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[2], s));
        erc = eval_sums_call<Data>(obj, &tp, sums_dev, s);
        if (erc) return erc;
        SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[3], s));
        SDCAB_CUDA_TRY(cudaMemcpyAsync(sums.data(), sums_dev, sums.size() * sizeof(double),
                                       cudaMemcpyDeviceToHost, s));
        SDCAB_CUDA_TRY(cudaStreamSynchronize(s));
        SDCAB_CUDA_TRY(cudaEventElapsedTime(&ms, buf.ev[2], buf.ev[3]));
        eval_ms += ms;
        sdcab_eval_record trec;
        double* acc = (keep && hist->test_accuracy)
                          ? hist->test_accuracy + (slot * hist->num_tests + ti) * m : nullptr;
        erc = eval_finish(obj, m, sums.data(), &trec, acc);
        if (erc) return erc;
        if (keep && hist->test) hist->test[slot * hist->num_tests + ti] = trec;
      }
    }
    return SDCAB_OK;
  };
  const double eps_floor = std::max(
      static_cast<double>(num<Data>::eps()), static_cast<double>(num<R>::eps()));
  auto check = [&](int status, int64_t epoch) {
    const sdcab_eval_record* last = history.empty() ? nullptr : &history.back();
    const sdcab_eval_record* before = history.size() > 1 ? &history[history.size() - 2] : nullptr;
    return check_stopping(status, last, before, crit->epsilon, epoch, crit->max_epoch, eps_floor,
                          crit->max_cpu_time, cpu_now(), crit->max_wall_time, wall_now());
  };

  // begin_solve (solver.h:59-80)
  int64_t epoch = 0;
  int status = (crit->max_epoch > 0) ? SDCAB_FIT_SOLVING : SDCAB_FIT_MAX_EPOCH;
  bool evaluated = false;
  if (crit->eval_on_start) {
    rc = evaluate(); if (rc) return rc;
    status = check(status, epoch);
  }

  MinstdRand gen;
  std::vector<int64_t> order_host(static_cast<size_t>(n));
  std::vector<unsigned char> seen;
  for (long long i = 0; i < n; ++i) order_host[static_cast<size_t>(i)] = i;

  while (status == SDCAB_FIT_SOLVING) {
    // begin_epoch (solver.h:94-100)
    evaluated = false;
    const int64_t* order_src;
    if (permutations) {
      order_src = permutations + epoch * n;
      if (!is_permutation(order_src, n, seen)) return SDCAB_ERR_ARG_RANGE;
    } else {
      shuffle_like_libstdcxx(order_host, gen);
      order_src = order_host.data();
    }
    SDCAB_CUDA_TRY(cudaMemcpyAsync(runner.order, order_src, static_cast<size_t>(n) * sizeof(int64_t),
                                   cudaMemcpyHostToDevice, s));
    SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[0], s));
    rc = runner.run_epoch(n, s, buf.ahead, buf.ev_product, buf.ev_steps, buf.ev_start);
    if (rc) return rc;
    SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[1], s));
    SDCAB_CUDA_TRY(cudaStreamSynchronize(s));
    float ms = 0;
    SDCAB_CUDA_TRY(cudaEventElapsedTime(&ms, buf.ev[0], buf.ev[1]));
    solve_ms += ms;

    // end_epoch (solver.h:103-117)
    ++epoch;
    epoch_now = epoch;
    if (crit->eval_epoch > 0 && epoch % crit->eval_epoch == 0) {
      rc = evaluate(); if (rc) return rc;
      evaluated = true;
    }
    status = check(status, epoch);
  }
  // end_solve (solver.h:83-91)
  if (!evaluated && !(crit->eval_on_start && epoch == 0)) {
    rc = evaluate(); if (rc) return rc;
  }
  SDCAB_CUDA_TRY(cudaEventRecord(buf.ev[1], s));
  SDCAB_CUDA_TRY(cudaStreamWaitEvent(user_stream, buf.ev[1], 0));
  SDCAB_CUDA_TRY(cudaStreamSynchronize(s));
  if (result) {
    result->status = status; result->reserved = 0;
    result->epoch = epoch;
    result->num_evals = static_cast<int64_t>(history.size());
    result->solve_seconds = solve_ms * 1e-3;
    result->eval_seconds = eval_ms * 1e-3;
    result->cpu_seconds = cpu_now();
    result->wall_seconds = wall_now();
  }
  return SDCAB_OK;
}

int check_fit_args(const sdcab_objective* obj, const sdcab_problem* t, const sdcab_fit_criteria* c) {
  if (!obj || !t || !c) return SDCAB_ERR_ARG;
  if (t->n <= 0 || t->m <= 0 || t->d <= 0) return SDCAB_ERR_NOT_EMPTY;
  if (t->m < 2) return SDCAB_ERR_NUM_DIM;
  if (t->m > 0x7fffffffLL || t->d > 0x7fffffffLL) return SDCAB_ERR_TOO_LARGE;
  int rc = check_objective(obj, t->m);
  if (rc) return rc;
  if (!objective_has_update(obj->id)) return SDCAB_ERR_NOT_IMPLEMENTED;
  if (!t->x || !t->a || !t->labels) return SDCAB_ERR_ARG;
  if (objective_is_multilabel(obj->id) && !t->offsets) return SDCAB_ERR_ARG;
  if (t->input_kind == SDCAB_INPUT_KERNEL) {
    if (t->d != t->n) return SDCAB_ERR_NUM_DIM;
  } else if (t->input_kind == SDCAB_INPUT_FEATURES) {
    if (!t->w) return SDCAB_ERR_ARG;
  } else {
    return SDCAB_ERR_ARG;
  }
  if (!(c->epsilon >= 0) || c->max_epoch < 0 || c->eval_epoch < 0) return SDCAB_ERR_ARG_RANGE;
  if (!(c->max_cpu_time >= 0) || !(c->max_wall_time >= 0)) return SDCAB_ERR_ARG_RANGE;
  return SDCAB_OK;
}

int check_history(const sdcab_fit_history* h) {
  if (!h) return SDCAB_OK;
  if (h->cap < 0 || h->num_tests < 0) return SDCAB_ERR_ARG_RANGE;
  if (h->num_tests > 0 && !h->tests) return SDCAB_ERR_ARG;
  for (int64_t t = 0; t < h->num_tests; ++t) {
    if (h->tests[t].n <= 0) return SDCAB_ERR_NOT_EMPTY;
    if (!h->tests[t].x || !h->tests[t].labels) return SDCAB_ERR_ARG;
  }
  return SDCAB_OK;
}

template <typename Data>
int fit_entry(const sdcab_objective* obj, const sdcab_problem* t, const sdcab_fit_criteria* c,
              const int64_t* perm, sdcab_eval_record* evals, int64_t cap, sdcab_fit_result* res,
              void* stream, const sdcab_fit_history* hist = nullptr) {
  int rc = check_fit_args(obj, t, c);
  if (rc) return rc;
  rc = check_history(hist);
  if (rc) return rc;
  if (hist && objective_is_multilabel(obj->id))
    for (int64_t q = 0; q < hist->num_tests; ++q)
      if (!hist->tests[q].offsets) return SDCAB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (obj->precision == SDCAB_PRECISION_FLOAT)
    return fit_dev<Data, float>(obj, t, c, perm, evals, cap, res, s, hist);
  return fit_dev<Data, double>(obj, t, c, perm, evals, cap, res, s, hist);
}

// Host buffers: copy the problem to the device, fit, copy the variables back.
template <typename Data>
int fit_host(const sdcab_objective* obj, const sdcab_problem* hp, const sdcab_fit_criteria* c,
             const int64_t* perm, sdcab_eval_record* evals, int64_t cap, sdcab_fit_result* res,
             const sdcab_fit_history* hist = nullptr) {
  int rc = check_fit_args(obj, hp, c);
  if (rc) return rc;
  rc = check_history(hist);
  if (rc) return rc;
  const long long n = hp->n, m = hp->m, d = hp->d;
  const bool kernel = (hp->input_kind == SDCAB_INPUT_KERNEL);
  const bool ml = objective_is_multilabel(obj->id);
  // the label checks of include/sdca/solver/data/output.h:169-215 (labels here are 0-based)
  rc = validate_labels(hp->labels, hp->offsets, n, m, ml);
  if (rc) return rc;
  const long long num_labels = ml ? hp->offsets[n] : n;
  DeviceBuffers buf;
  Data *dX = nullptr, *dA = nullptr, *dW = nullptr, *dW0 = nullptr;
  int64_t *dLab = nullptr, *dOff = nullptr;
  const size_t x_elems = static_cast<size_t>(n) * d, a_elems = static_cast<size_t>(n) * m,
               w_elems = static_cast<size_t>(d) * m;
  const bool with_w0 = !kernel && hp->w0;
  rc = buf.reserve(DeviceBuffers::padded(x_elems * sizeof(Data)) + DeviceBuffers::padded(a_elems * sizeof(Data)) +
                   DeviceBuffers::padded(static_cast<size_t>(num_labels) * sizeof(int64_t)) +
                   (kernel ? 0 : (with_w0 ? 2 : 1) * DeviceBuffers::padded(w_elems * sizeof(Data))) +
                   (ml ? DeviceBuffers::padded(static_cast<size_t>(n + 1) * sizeof(int64_t)) : 0));
  if (rc) return rc;
  rc = buf.alloc(&dX, x_elems); if (rc) return rc;
  rc = buf.alloc(&dA, a_elems); if (rc) return rc;
  rc = buf.alloc(&dLab, static_cast<size_t>(num_labels)); if (rc) return rc;
  SDCAB_CUDA_TRY(cudaMemcpy(dX, hp->x, x_elems * sizeof(Data), cudaMemcpyHostToDevice));
  SDCAB_CUDA_TRY(cudaMemcpy(dA, hp->a, a_elems * sizeof(Data), cudaMemcpyHostToDevice));
  SDCAB_CUDA_TRY(cudaMemcpy(dLab, hp->labels, static_cast<size_t>(num_labels) * sizeof(int64_t),
                            cudaMemcpyHostToDevice));
  if (!kernel) {
    rc = buf.alloc(&dW, w_elems); if (rc) return rc;
    SDCAB_CUDA_TRY(cudaMemcpy(dW, hp->w, w_elems * sizeof(Data), cudaMemcpyHostToDevice));
    if (hp->w0) {
      // the proximal centre of a restarted fit (src/matlab/mex_solve.cpp:529-586): it enters
      // the primal regulariser of every evaluation and the rebuilt W
      rc = buf.alloc(&dW0, w_elems); if (rc) return rc;
      SDCAB_CUDA_TRY(cudaMemcpy(dW0, hp->w0, w_elems * sizeof(Data), cudaMemcpyHostToDevice));
    }
  }
  if (ml) {
    rc = buf.alloc(&dOff, static_cast<size_t>(n + 1)); if (rc) return rc;
    SDCAB_CUDA_TRY(cudaMemcpy(dOff, hp->offsets, static_cast<size_t>(n + 1) * sizeof(int64_t),
                              cudaMemcpyHostToDevice));
  }
  sdcab_problem dp = *hp;
  dp.x = dX; dp.a = dA; dp.w = dW; dp.w0 = dW0; dp.labels = dLab; dp.offsets = dOff;
  // held-out sets: checked like the training labels, then copied to the device
  std::vector<sdcab_problem> dtests;
  sdcab_fit_history dh;
  if (hist) {
    dh = *hist;
    for (int64_t q = 0; q < hist->num_tests; ++q) {
      const sdcab_problem& tp = hist->tests[q];
      if (ml && !tp.offsets) return SDCAB_ERR_ARG;
      rc = validate_labels(tp.labels, tp.offsets, tp.n, m, ml);
      if (rc) return rc;
      const long long tl = ml ? tp.offsets[tp.n] : tp.n;
      Data* tx = nullptr; int64_t *tlab = nullptr, *toff = nullptr;
      rc = buf.alloc(&tx, static_cast<size_t>(tp.n) * d); if (rc) return rc;
      rc = buf.alloc(&tlab, static_cast<size_t>(tl)); if (rc) return rc;
      SDCAB_CUDA_TRY(cudaMemcpy(tx, tp.x, static_cast<size_t>(tp.n) * d * sizeof(Data), cudaMemcpyHostToDevice));
      SDCAB_CUDA_TRY(cudaMemcpy(tlab, tp.labels, static_cast<size_t>(tl) * sizeof(int64_t), cudaMemcpyHostToDevice));
      if (ml) {
        rc = buf.alloc(&toff, static_cast<size_t>(tp.n + 1)); if (rc) return rc;
        SDCAB_CUDA_TRY(cudaMemcpy(toff, tp.offsets, static_cast<size_t>(tp.n + 1) * sizeof(int64_t), cudaMemcpyHostToDevice));
      }
      sdcab_problem q_dev = tp;
      q_dev.x = tx; q_dev.labels = tlab; q_dev.offsets = toff;
      dtests.push_back(q_dev);
    }
    dh.tests = dtests.empty() ? nullptr : dtests.data();
  }
  rc = fit_entry<Data>(obj, &dp, c, perm, evals, cap, res, nullptr, hist ? &dh : nullptr);
  if (rc) return rc;
  SDCAB_CUDA_TRY(cudaMemcpy(const_cast<void*>(hp->a), dA, a_elems * sizeof(Data), cudaMemcpyDeviceToHost));
  if (!kernel)
    SDCAB_CUDA_TRY(cudaMemcpy(const_cast<void*>(hp->w), dW, w_elems * sizeof(Data), cudaMemcpyDeviceToHost));
  return SDCAB_OK;
}

// matsdca_fit without Matlab: datasets + options in, model out.
template <typename Data>
int train_host(const sdcab_dataset* sets, int64_t num_sets, const sdcab_train_options* o, sdcab_model* model) {
  if (!sets || num_sets < 1 || !o || !model) return SDCAB_ERR_ARG;
  if (!model->A) return SDCAB_ERR_ARG;
  const sdcab_dataset& trn = sets[0];
  if (trn.n <= 0 || !trn.x || !trn.labels) return SDCAB_ERR_NOT_EMPTY;
  sdcab_objective obj;
  int rc = objective_from_name(o->objective ? o->objective : "msvm_smooth", o->c, o->gamma, o->k, &obj);
  if (rc) return rc;
  if (o->precision != SDCAB_PRECISION_DOUBLE && o->precision != SDCAB_PRECISION_FLOAT)
    return SDCAB_ERR_PRECISION;
  obj.precision = o->precision;
  const bool ml = objective_is_multilabel(obj.id);
  const bool kernel = o->is_dual != 0;
  const int64_t n = trn.n;
  const int64_t d = kernel ? n : o->num_dimensions;
  if (d <= 0) return SDCAB_ERR_NUM_DIM;
  if (!kernel && !model->W) return SDCAB_ERR_ARG;
  if (ml && !trn.offsets) return SDCAB_ERR_ARG;
  // labels: 0-based or 1-based, decided by the smallest training label
  // (validate_labels, include/sdca/solver/data/output.h:169-182); every set is shifted alike
  std::vector<std::vector<int64_t>> labels(static_cast<size_t>(num_sets));
  int64_t shift = 0, max_label = 0;
  for (int64_t q = 0; q < num_sets; ++q) {
    const sdcab_dataset& ds = sets[q];
    if (ds.n <= 0 || !ds.x || !ds.labels) return SDCAB_ERR_NOT_EMPTY;
    if (ml && !ds.offsets) return SDCAB_ERR_ARG;
    const int64_t count = ml ? ds.offsets[ds.n] : ds.n;
    if (count <= 0) return SDCAB_ERR_LABELS_RANGE;
    int64_t lo = ds.labels[0], hi = ds.labels[0];
    for (int64_t i = 1; i < count; ++i) { lo = std::min(lo, ds.labels[i]); hi = std::max(hi, ds.labels[i]); }
    if (q == 0) {
      if (lo != 0 && lo != 1) return SDCAB_ERR_LABELS_RANGE;
      shift = lo;
    }
    if (lo < shift) return SDCAB_ERR_LABELS_RANGE;
    max_label = std::max(max_label, hi - shift);
    labels[static_cast<size_t>(q)].assign(ds.labels, ds.labels + count);
    for (int64_t& v : labels[static_cast<size_t>(q)]) v -= shift;
  }
  const int64_t m = o->num_classes > 0 ? o->num_classes : max_label + 1;
  if (max_label >= m) return SDCAB_ERR_LABELS_RANGE;

  Data* A = static_cast<Data*>(model->A);
  Data* W = static_cast<Data*>(model->W);
  if (!o->warm_start) {
    std::fill(A, A + static_cast<size_t>(n) * m, Data(0));
    if (!kernel) {
      // W = W0 before the first step of a prox-regularised fit (mex_solve.cpp:566-571)
      if (o->W0) std::memcpy(W, o->W0, static_cast<size_t>(d) * m * sizeof(Data));
      else std::fill(W, W + static_cast<size_t>(d) * m, Data(0));
    }
  }
  sdcab_problem p = sdcab_problem();
  p.input_kind = kernel ? SDCAB_INPUT_KERNEL : SDCAB_INPUT_FEATURES;
  p.is_train = 1; p.d = d; p.n = n; p.m = m;
  p.x = trn.x; p.a = A; p.w = kernel ? nullptr : W; p.w0 = kernel ? nullptr : o->W0;
  p.labels = labels[0].data(); p.offsets = trn.offsets; p.include_primal_regularizer = 1;
  std::vector<sdcab_problem> tests;
  for (int64_t q = 1; q < num_sets; ++q) {
    sdcab_problem tp = sdcab_problem();
    tp.input_kind = p.input_kind; tp.d = d; tp.n = sets[q].n; tp.m = m;
    tp.x = sets[q].x; tp.labels = labels[static_cast<size_t>(q)].data(); tp.offsets = sets[q].offsets;
    tests.push_back(tp);
  }
  sdcab_fit_history h = model->history;
  h.num_tests = num_sets - 1;
  h.tests = tests.empty() ? nullptr : tests.data();
  sdcab_fit_result res = sdcab_fit_result();
  rc = fit_host<Data>(&obj, &p, &o->criteria, nullptr, nullptr, 0, &res, &h);
  if (rc) return rc;
  // the model (mex_solve.cpp:153-376)
  model->num_dimensions = d; model->num_examples = n; model->num_classes = m;
  model->is_dual = kernel ? 1 : 0; model->objective_id = obj.id;
  std::snprintf(model->objective, sizeof(model->objective), "%s", o->objective ? o->objective : "msvm_smooth");
  model->c = obj.c; model->gamma = obj.gamma; model->k = obj.k;
  model->criteria = o->criteria;
  model->status = res.status;
  model->data_precision = sizeof(Data) == 4 ? SDCAB_PRECISION_FLOAT : SDCAB_PRECISION_DOUBLE;
  model->precision = obj.precision;
  model->labels_one_based = static_cast<int32_t>(shift);
  model->epoch = res.epoch;
  model->cpu_time = res.cpu_seconds; model->wall_time = res.wall_seconds;
  model->solve_time = res.solve_seconds; model->eval_time = res.eval_seconds;
  model->num_evals = res.num_evals;
  model->history.num_tests = num_sets - 1;
  model->history.tests = nullptr;
  const int64_t last = std::min(res.num_evals, h.cap) - 1;
  model->relative_gap = (h.train && last >= 0) ? h.train[last].relative_gap : 0.0;
  return SDCAB_OK;
}

}  // namespace
}  // namespace sdcab


extern "C" {

int sdcab_epoch_permutations(int64_t n, int64_t num_epochs, int64_t* perm) {
  if (n < 0 || num_epochs < 0 || (!perm && n * num_epochs > 0)) return SDCAB_ERR_ARG;
  sdcab::epoch_permutations(n, num_epochs, perm);
  return SDCAB_OK;
}

int sdcab_fit_f32_dev(const sdcab_objective* obj, const sdcab_problem* train,
                      const sdcab_fit_criteria* criteria, const int64_t* permutations,
                      sdcab_eval_record* evals, int64_t evals_cap, sdcab_fit_result* result,
                      void* stream) {
  return sdcab::fit_entry<float>(obj, train, criteria, permutations, evals, evals_cap, result, stream);
}

int sdcab_fit_f64_dev(const sdcab_objective* obj, const sdcab_problem* train,
                      const sdcab_fit_criteria* criteria, const int64_t* permutations,
                      sdcab_eval_record* evals, int64_t evals_cap, sdcab_fit_result* result,
                      void* stream) {
  return sdcab::fit_entry<double>(obj, train, criteria, permutations, evals, evals_cap, result, stream);
}

int sdcab_fit_history_f32_dev(const sdcab_objective* obj, const sdcab_problem* train,
                              const sdcab_fit_criteria* criteria, const int64_t* permutations,
                              const sdcab_fit_history* history, sdcab_fit_result* result, void* stream) {
  return sdcab::fit_entry<float>(obj, train, criteria, permutations, nullptr, 0, result, stream, history);
}
int sdcab_fit_history_f64_dev(const sdcab_objective* obj, const sdcab_problem* train,
                              const sdcab_fit_criteria* criteria, const int64_t* permutations,
                              const sdcab_fit_history* history, sdcab_fit_result* result, void* stream) {
  return sdcab::fit_entry<double>(obj, train, criteria, permutations, nullptr, 0, result, stream, history);
}
int sdcab_fit_history_f32(const sdcab_objective* obj, const sdcab_problem* host_train,
                          const sdcab_fit_criteria* criteria, const int64_t* permutations,
                          const sdcab_fit_history* history, sdcab_fit_result* result) {
  return sdcab::fit_host<float>(obj, host_train, criteria, permutations, nullptr, 0, result, history);
}
int sdcab_fit_history_f64(const sdcab_objective* obj, const sdcab_problem* host_train,
                          const sdcab_fit_criteria* criteria, const int64_t* permutations,
                          const sdcab_fit_history* history, sdcab_fit_result* result) {
  return sdcab::fit_host<double>(obj, host_train, criteria, permutations, nullptr, 0, result, history);
}

void sdcab_train_options_default(sdcab_train_options* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->objective = nullptr; o->c = 1; o->gamma = 1; o->k = 1;
  o->is_dual = 0; o->precision = SDCAB_PRECISION_DOUBLE;
  // stopping_criteria of the reference (include/sdca/solver/solverdef.h:50-57)
  o->criteria.epsilon = 1e-3; o->criteria.max_epoch = 1000; o->criteria.eval_epoch = 10;
  o->criteria.eval_on_start = 0; o->criteria.recompute_primal = 0;
  o->criteria.max_cpu_time = 0; o->criteria.max_wall_time = 0;
}
int sdcab_train_f32(const sdcab_dataset* datasets, int64_t num_datasets,
                    const sdcab_train_options* options, sdcab_model* model) {
  return sdcab::train_host<float>(datasets, num_datasets, options, model);
}
int sdcab_train_f64(const sdcab_dataset* datasets, int64_t num_datasets,
                    const sdcab_train_options* options, sdcab_model* model) {
  return sdcab::train_host<double>(datasets, num_datasets, options, model);
}

int sdcab_fit_f32(const sdcab_objective* obj, const sdcab_problem* host_train,
                  const sdcab_fit_criteria* criteria, const int64_t* permutations,
                  sdcab_eval_record* evals, int64_t evals_cap, sdcab_fit_result* result) {
  return sdcab::fit_host<float>(obj, host_train, criteria, permutations, evals, evals_cap, result);
}

int sdcab_fit_f64(const sdcab_objective* obj, const sdcab_problem* host_train,
                  const sdcab_fit_criteria* criteria, const int64_t* permutations,
                  sdcab_eval_record* evals, int64_t evals_cap, sdcab_fit_result* result) {
  return sdcab::fit_host<double>(obj, host_train, criteria, permutations, evals, evals_cap, result);
}

}  // extern "C"
