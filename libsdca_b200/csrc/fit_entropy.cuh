// The chain of SDCA steps for the softmax and multilabel softmax objectives.
//
// Such a step spends its time on  sum_j W(exp(u_j - t)) = alpha : a few dozen evaluations of m
// Lambert functions in double precision, which one warp works off as m / 32 serial evaluations per
// lane (52 us per step for m = 100).  Here four warps share the entries, and the root is found
// cheaply first: a Newton iteration on the logarithm of the sum in float arithmetic, kept inside
// the bracket that the largest entry gives, leaves an error of about 1e-6, and one fourth-order
// Householder step with sums in Result precision -- the step of include/sdca/prox/two_entropy.h:12-37
// -- ends at the rounding error of the sum, as the reference's iteration does.
// Latency bound: about four float and one or two double evaluations per step, each followed by one
// reduction over the four warps.
#pragma once

#include "fit_chain.cuh"

namespace sdcab {

constexpr int kSolverThreads = 128;
constexpr int kSolverWarps = kSolverThreads / 32;
constexpr int kEntropyThreads = kSolverThreads + kHelperThreads;

__device__ __forceinline__ void solver_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
static_assert(kSolverThreads == 128, "solver_barrier names the number of threads");

// Sums over the solver warps; every thread receives the totals, in a fixed order of additions.
// Two buffers in turn: a thread can only write a buffer again after a barrier that every thread
// reached with its reads of that buffer done.
struct SolverReduce {
  double (*buf)[kSolverWarps][4];   // two of them
  int turn;

  template <typename T, int N>
  __device__ __forceinline__ void sum(T (&x)[N]) {
    static_assert(N == 1 || N == 2 || N == 4, "one value per lane group");
    const int lane = static_cast<int>(threadIdx.x) & 31, warp = static_cast<int>(threadIdx.x) >> 5;
    T y;
    int which = 0;
    if (N == 4) {
      const bool hi = (lane & 16) != 0, hi2 = (lane & 8) != 0;
      const T s0 = hi ? x[0] : x[2 % N], s1 = hi ? x[1 % N] : x[3 % N];
      const T k0 = (hi ? x[2 % N] : x[0]) + __shfl_xor_sync(kFullMask, s0, 16);
      const T k1 = (hi ? x[3 % N] : x[1 % N]) + __shfl_xor_sync(kFullMask, s1, 16);
      y = (hi2 ? k1 : k0) + __shfl_xor_sync(kFullMask, hi2 ? k0 : k1, 8);
      which = (hi ? 2 : 0) + (hi2 ? 1 : 0);
    } else if (N == 2) {
      const bool hi = (lane & 16) != 0;
      y = (hi ? x[1 % N] : x[0]) + __shfl_xor_sync(kFullMask, hi ? x[0] : x[1 % N], 16);
      y += __shfl_xor_sync(kFullMask, y, 8);
      which = hi ? 1 : 0;
    } else {
      y = x[0] + __shfl_xor_sync(kFullMask, x[0], 16);
      y += __shfl_xor_sync(kFullMask, y, 8);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(kFullMask, y, o);
    T (*out)[4] = reinterpret_cast<T(*)[4]>(buf[turn]);
    if ((lane & (N == 4 ? 7 : (N == 2 ? 15 : 31))) == 0) out[warp][which] = y;
    solver_barrier();
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = (out[0][i] + out[1][i]) + (out[2][i] + out[3][i]);
    turn ^= 1;
  }
  __device__ __forceinline__ float max(float v) {
    const int lane = static_cast<int>(threadIdx.x) & 31, warp = static_cast<int>(threadIdx.x) >> 5;
    asm volatile("redux.sync.max.f32 %0, %0, 0xffffffff;" : "+f"(v));
    float (*out)[4] = reinterpret_cast<float(*)[4]>(buf[turn]);
    if (lane == 0) out[warp][0] = v;
    solver_barrier();
    v = fmaxf(fmaxf(out[0][0], out[1][0]), fmaxf(out[2][0], out[3][0]));
    turn ^= 1;
    return v;
  }
};

// f0 .. f3 of row_sum_w_exp over the m entries u_j = entry(j), by the solver threads (entry j
// belongs to thread j mod 128), and one Householder step for f0 = alpha from t.  Returns f0 - alpha.
template <typename R, typename Entry>
__device__ __forceinline__ R step_sum_w(int m, R alpha, SolverReduce& red, Entry entry, R& t) {
  R f[4] = {0, 0, 0, 0};
  for (int j = threadIdx.x; j < m; j += kSolverThreads) {
    const R v = lambert_w_exp(static_cast<R>(entry(j)) - t);
    const R q = inverse_of_sum(v), vq = v * q, q2 = q * q;
    f[0] += v;
    f[1] += vq;
    f[2] += vq * q2;
    f[3] += vq * (1 - 2 * v) * (q2 * q2);
  }
  red.sum(f);
  const R f0 = f[0] - alpha;
  const R f02 = f0 * f[2], f11 = f[1] * f[1];
  const R D = 6 * f[1] * (f02 - f11) - f0 * (f0 * f[3]);
  if (abs_(D) > 64 * num<R>::tiny()) t -= 3 * f0 * (2 * f11 - f02) / D;
  return f0;
}

// The largest entry, for the float searches; false for values that float cannot hold.
template <typename R, typename Entry>
__device__ __forceinline__ bool largest_entry(int m, R alpha, SolverReduce& red, Entry entry, R& base) {
  constexpr float kHuge = 1e30f;
  float mx = -kHuge;
  for (int j = threadIdx.x; j < m; j += kSolverThreads) {
    const float u = static_cast<float>(entry(j));
    mx = fabsf(u) < kHuge ? fmaxf(mx, u) : num<float>::inf();
  }
  mx = red.max(mx);
  base = static_cast<R>(mx);
  return mx < kHuge && alpha > R(1e-30) && alpha < R(1e30);
}

// Root of sum_j W(exp(u_j - t)) = alpha.  The sum is convex and decreasing; the largest entry mx
// gives the bracket mx - alpha - log alpha <= t <= mx - alpha / m - log(alpha / m), and the
// reference's iteration (include/sdca/prox/two_entropy.h:94-231) is kept inside a bracket as well:
// the root is what it ends at.  tau_near: where t - mx is looked for first, and where it was found.
template <typename R, typename Entry>
__device__ __forceinline__ bool solve_sum_w(int m, R alpha, SolverReduce& red, Entry entry, float& tau_near, R& t_out) {
  const int tid = threadIdx.x;
  R base;
  if (!largest_entry<R>(m, alpha, red, entry, base)) return false;
  // tau = t - base: the differences are formed in Result precision, so that float holds them
  const float al = static_cast<float>(alpha);
  const float la = logf(al), share = al / static_cast<float>(m);
  float lb = -al - la, ub = -share - logf(share);
  const float slack = 1e-5f * (fabsf(lb) + fabsf(ub) + static_cast<float>(abs_(base)) + 1.0f);
  lb -= slack; ub += slack;
  R lbr = base + static_cast<R>(lb), ubr = base + static_cast<R>(ub);
  // t - mx moves little from one example to the next
  float tau = fminf(fmaxf(tau_near, lb), ub);
  for (int it = 0; it < 24; ++it) {
    float s[2] = {0.0f, 0.0f};
    for (int j = tid; j < m; j += kSolverThreads) {
      const float w = lambert_w_exp(static_cast<float>(entry(j) - base) - tau);
      s[0] += w;
      s[1] += __fdividef(w, 1.0f + w);
    }
    red.sum(s);
    if (s[0] > al) lb = tau; else ub = tau;
    // Newton's step for log(sum) = log(alpha): one step where every term is an exponential
    const float step = __fdividef(s[0], s[1]) * __logf(__fdividef(s[0], al));
    const float next = tau + step;
    const bool inside = next >= lb && next <= ub;
    tau = inside ? next : 0.5f * (lb + ub);
    if (inside && fabsf(step) <= 2e-3f) break;
  }
  tau_near = tau;
  R t = base + static_cast<R>(tau);
  for (int it = 0; it < 32; ++it) {
    const R from = t;
    const R f0 = step_sum_w<R>(m, alpha, red, entry, t);
    if (f0 > 0) lbr = max_(lbr, from); else ubr = min_(ubr, from);
    t = max_(lbr, min_(t, ubr));
    if (abs_(t - from) <= last_step<R>()) break;
  }
  if (!finite_(t)) return false;
  t_out = t;
  return true;
}

// Steps b = 0 .. count - 1 as in fit_chain_kernel (fit_steps.cuh): four warps work the step, eight keep
// the later rows of S current and fetch the next step's variables and labels meanwhile.
template <typename Data, typename R, bool ON_CHIP>
__global__ void __launch_bounds__(kEntropyThreads, 1) fit_entropy_chain_kernel(ChainArgs p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = p.m, count = p.count;
  const int tid = threadIdx.x;
  double* G = reinterpret_cast<double*>(smem_raw);                  // 64 x 64
  double* delta = G + kBlockSteps * kBlockSteps;                    // 2 x m: this step's / the previous one's
  double* S = delta + 2 * m;                                        // count x m when on chip
  Data* scores = reinterpret_cast<Data*>(ON_CHIP ? S + static_cast<size_t>(kBlockSteps) * m : S);
  Data* a_s = scores + m;
  Data* v_s = a_s + m;
  Data* a_next = v_s + m;                                           // 2 x m, rows fetched ahead
  const int mask_words = (m + 31) / 32;
  unsigned* label_mask = reinterpret_cast<unsigned*>(a_next + 2 * m);   // 2 x mask_words (multilabel)
  const bool multilabel = p.o.id == kObjL2MultilabelEntropy;
  __shared__ long long s_off[kBlockSteps];
  __shared__ long long s_idx[kBlockSteps];
  __shared__ int s_lab[kBlockSteps];    // the label, or the number of labels
  __shared__ int s_moved;
  __shared__ double s_red[2][kSolverWarps][4];
  Data* A = static_cast<Data*>(p.A);
  Data* D = static_cast<Data*>(p.D);
  const R c = static_cast<R>(p.o.c);

  fill_shared(G, p.G, kBlockSteps * kBlockSteps, tid, kEntropyThreads);
  if (ON_CHIP) fill_shared(S, p.S, count * m, tid, kEntropyThreads);
  for (int t = tid; t < 2 * m; t += kEntropyThreads) delta[t] = 0.0;
  if (tid < count) {
    const long long i = p.order[tid];
    s_idx[tid] = i;
    if (multilabel) {
      s_off[tid] = p.offsets[i];
      s_lab[tid] = static_cast<int>(p.offsets[i + 1] - p.offsets[i]);
    } else {
      s_lab[tid] = static_cast<int>(p.labels[i]);
    }
  }
  if (!ON_CHIP) S = p.S;
  __syncthreads();
  // what a step needs of its example, by one warp: the variables and the labels' bits
  auto fetch = [&](int b, int h) {
    Data* nxt = a_next + (b & 1) * m;
    const Data* src = A + s_idx[b] * m;
    for (int j = h; j < m; j += 32) nxt[j] = src[j];
    if (multilabel) {
      unsigned* mask = label_mask + (b & 1) * mask_words;
      for (int w = h; w < mask_words; w += 32) mask[w] = 0u;
      __syncwarp();
      for (int g = h; g < s_lab[b]; g += 32) {
        const int lab = static_cast<int>(p.labels[s_off[b] + g]);
        atomicOr(&mask[lab >> 5], 1u << (lab & 31));
      }
    }
  };
  if (tid < 32) fetch(0, tid);
  __syncthreads();

  SolverReduce red;
  red.buf = s_red; red.turn = 0;
  float tau_near = -num<float>::max();
  bool pending = false;                 // the previous step changed something
  for (int b = 0; b < count; ++b) {
    const int cur = b & 1, prev = cur ^ 1;
    bool moved = false, solver_active = false;
    const double* d_prev = delta + prev * m;
    if (tid < kSolverThreads) {
      const long long i = s_idx[b];
      const double g_bb = G[b * kBlockSteps + b];
      const Data norm2 = static_cast<Data>(p.kernel_input ? g_bb : -g_bb);
      const bool active = norm2 > Data(0);    // update.h:63,97
      const Data* a_cur = a_next + cur * m;
      const unsigned* mask = label_mask + cur * mask_words;
      double* d_cur = delta + cur * m;
      Data* d_row = p.kernel_input ? nullptr : D + static_cast<size_t>(b) * m;
      const int y = s_lab[b];
      if (active) {
        const double* Sb = S + static_cast<size_t>(b) * m;
        const double g = pending ? G[(b - 1) * kBlockSteps + b] : 0.0;
        auto is_label = [&](int j) { return multilabel ? ((mask[j >> 5] >> (j & 31)) & 1u) != 0 : j == y; };
        // v = scores - norm2 a (l2_entropy.h:53-57, l2_multilabel_entropy.h:48-52)
        for (int j = tid; j < m; j += kSolverThreads) {
          const Data score = static_cast<Data>(fma(d_prev[j], g, Sb[j]));
          scores[j] = score;
          v_s[j] = add_rn_(mul_rn_(-norm2, a_cur[j]), score);
        }
        const R alpha = c * static_cast<R>(norm2);
        // the labels' block at t, the others at t + alpha / (number of labels)
        const R apart = alpha / static_cast<R>(multilabel ? s_lab[b] : 1);
        R t = 0;
        const bool ok = solve_sum_w<R>(
            m, alpha, red, [&](int j) { return static_cast<R>(v_s[j]) - (is_label(j) ? R(0) : apart); }, tau_near, t);
        if (ok) {
          const Applier<Data> others(make_thr(t + apart, R(0), R(1), 0, 0, R(0), R(0)), kMapScaledLambert,
                                     static_cast<double>(alpha));
          const Data td_label = static_cast<Data>(t);
          const Data minus_c = static_cast<Data>(-c);
          const Data share = static_cast<Data>(c / static_cast<R>(multilabel ? s_lab[b] : 1));
          for (int j = tid; j < m; j += kSolverThreads) {
            Applier<Data> f = others;
            const bool label = is_label(j);
            if (label) f.t = td_label;
            const Data x = mul_rn_(minus_c, f(v_s[j]));
            a_s[j] = label ? add_rn_(x, share) : x;
          }
        } else {
          // values out of the float search's range: the general routine, by one warp
          for (int j = tid; j < m; j += kSolverThreads) a_s[j] = a_cur[j];
          solver_barrier();
          if (tid < 32) {
            if (multilabel) general_update_multilabel<R, Data>(&p.o, norm2, scores, a_s, v_s, m, mask, s_lab[b]);
            else general_update<R, Data>(&p.o, norm2, scores, a_s, v_s, m, y);
          }
          solver_barrier();
        }
        for (int j = tid; j < m; j += kSolverThreads) {
          const Data a_new = a_s[j], a_old = a_cur[j];
          A[i * m + j] = a_new;
          if (p.kernel_input) {
            moved = true;
            d_cur[j] = static_cast<double>(a_new) - static_cast<double>(a_old);
          } else {
            const Data dlt = a_old - a_new;   // var_copy of update.h:74-77
            moved |= abs_(dlt) > num<Data>::eps();
            d_cur[j] = static_cast<double>(dlt);
            d_row[j] = dlt;
          }
        }
      } else if (d_row) {
        for (int j = tid; j < m; j += kSolverThreads) d_row[j] = Data(0);
      }
      // one change above eps: so is their sum (update.h:78).  Without one it has to be formed, by
      // everybody, since everybody learns of it at the barrier.
      solver_active = active && !p.kernel_input;
    } else {
      const int h = tid - kSolverThreads;
      if (h < 32 && b + 1 < count) fetch(b + 1, h);
      if (pending) move_later_rows(S, G, d_prev, b, count, m, h);
    }
    pending = __syncthreads_or(moved);
    if (!pending && !p.kernel_input) {
      if (tid < kSolverThreads && solver_active) {
        R change[1] = {0};
        for (int j = tid; j < m; j += kSolverThreads)
          change[0] += static_cast<R>(abs_(static_cast<Data>(delta[cur * m + j])));
        red.sum(change);
        const bool above = change[0] > static_cast<R>(num<Data>::eps());
        if (!above)
          for (int j = tid; j < m; j += kSolverThreads) D[static_cast<size_t>(b) * m + j] = Data(0);
        if (tid == 0) s_moved = above ? 1 : 0;
      } else if (tid == 0) {
        s_moved = 0;
      }
      __syncthreads();
      pending = s_moved != 0;
    }
  }
}

}  // namespace sdcab
