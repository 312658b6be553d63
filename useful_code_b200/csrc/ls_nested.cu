// ls_nested.cu — Longstaff–Schwartz with nested regressions (depth > 1).
//
// Reference behaviour followed:
//   backward loop, nested    generateRegressionCoefficientsViaLSMulti_gold
//   regressions              (gold/MultiLS_regression.cpp:101-417; the
//                            one-sign shortcut at :212-225 of the root tree)
//                            and its GPU orchestration
//                            generateMultiRegressionCoefficientsViaLS_gpu_
//                            flexisolve (LS_main_cula.h:565-837)
//   path selection           RegressionSelector_gold_Fraction::Select
//                            (gold/Regression_Selector_concrete_gold.cpp:58-205)
//   decision chain           updateDeflatedNextStepValuesMulti_gold
//                            (gold/MultiLS_regression.h:42-99),
//                            exercise_updating_LS_multi_kernel (LS_gpu.cu:312)
//
// Per date e the loop is a fixed sequence of launches with no host
// synchronisation: the decision of date e + 1 is applied to the running
// values; the first regression runs over all paths (ls_date_kernel); then
// for each further depth d one cooperative launch (nested_select_kernel)
// takes the net values of regression d - 1 on its paths, searches the
// half-width of the band of paths to regress again, and forms the moments
// of the selected paths; then the regression over them (ls_date_kernel with
// a mask).  When a date stops nesting (one-sign net values, too few paths,
// or a search that did not finish), a flag makes its remaining launches
// return at once.
//
// The reference's search evaluates one count per step on the whole path
// set.  Here each pass evaluates every count the search can ask for next:
// a stretch of the geometric chain of its grow or shrink loop, or the next
// eight levels of its bisection tree, computed with the same floating-point
// operations, so the search reads exact counts and takes the same steps.
#include "lmm_common.cuh"
#include "lmm_device.cuh"
#include "ls_common.cuh"

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

using namespace lmm;

#define TRY(x)           \
  do {                   \
    const int st_ = (x); \
    if (st_) return st_; \
  } while (0)

namespace {

constexpr int kSelBatch = 256;      // thresholds per selection pass
constexpr int kSelChain = 48;       // of them in a chain pass
constexpr int kSelPasses = 16;      // selection passes of a search at most
constexpr int kSelMaxCounts = 512;  // count evaluations per search
constexpr int kSelCapped = 8;       // status: a search stopped at kSelMaxCounts
constexpr int kSelIncomplete = 16;  // status: a search needed more passes
constexpr int kSelWait = 32;        // status: a wait of the grid ran out
constexpr int kNestThreads = 256;   // decision kernel
constexpr int kSelThreads = 512;    // selection kernel, one CTA per SM

// State of the search for one (date, depth), the same in every CTA's shared
// memory.  A pass counts |net| against the ascending thresholds thr[0 .. nb);
// chain passes hold a geometric chain, tree passes the next eight levels of
// the bisection of [lo, hi] in symmetric order.
enum {
  kPhDone = 0,
  kPhBranch,  // n within the targets: the reference keeps every path (cut 1e4)
  kPhInit,    // g at thr[nb - 1] and the shrinking chain g m, g m^2, ... below it
  kPhGrow,    // g / m, g / m^2, ... (the count at g was below the lower target)
  kPhShrink,  // lo m, lo m^2, ... (the count at lo is above the upper target)
  kPhTree     // halvings of [lo, hi]
};
struct SelState {
  int phase, lo_t, hi_t, evals, c, after, nb, status;
  double g, lo, hi, mult, cut;
};

// Thresholds of the phase's next pass, with the floating-point operations of
// the sequential search.  All threads of the CTA; ends with a barrier.
__device__ void sel_thresholds(SelState& S, double* thr) {
  const int tid = threadIdx.x;
  if (S.phase == kPhTree) {
    // node h (heap order, 1-based) of [lo, hi]: left child = [lo, mid] (the
    // count was above the upper target), right child = [mid, hi]; its rank
    // in symmetric order from its level and place
    for (int h = tid + 1; h < kSelBatch; h += blockDim.x) {
      const int lead = 31 - __clz(h);
      double lo = S.lo, hi = S.hi;
      for (int b = lead - 1; b >= 0; --b) {
        const double mid = 0.5 * (lo + hi);
        if ((h >> b) & 1)
          lo = mid;
        else
          hi = mid;
      }
      thr[((2 * (h - (1 << lead)) + 1) << (7 - lead)) - 1] = 0.5 * (lo + hi);
    }
    if (tid == 0) S.nb = kSelBatch - 1;
  } else if (tid == 0) {
    int n = kSelBatch;
    if (S.phase == kPhBranch) {
      thr[0] = 1e4;
      n = 1;
    } else if (S.phase == kPhGrow) {
      double g = S.g;
      n = kSelChain;
      for (int i = 0; i < n; ++i) thr[i] = g = g / S.mult;
    } else {
      n = kSelChain;
      double l = S.phase == kPhInit ? S.g : S.lo * S.mult;
      for (int i = n - 1; i >= 0; --i, l *= S.mult) thr[i] = l;
    }
    S.nb = n;
  }
  __syncthreads();
}

// Advances the search (thread 0 of every CTA alike) from the counts cnt[i] of
// paths with |net| <= thr[i]; the same steps and stopping rules as
// frac_select of the CPU restatement.  Leaves kPhDone, or the phase of the
// pass whose counts it needs next.
__device__ __forceinline__ void sel_step(SelState& S, const double* thr, const int* cnt) {
  auto done = [&](double cut, int after) {
    S.cut = cut;
    S.after = after;
    S.phase = kPhDone;
  };
  auto capped = [&]() {
    if (S.evals < kSelMaxCounts) return false;
    S.status |= kSelCapped;
    return true;
  };
  auto bisect = [&]() {  // from the chain's bracket
    S.hi = S.g;
    S.phase = kPhTree;
  };
  // after a shrink step left the count S.c at S.lo
  auto shrunk = [&]() {
    if (S.c > S.lo_t)
      done(S.lo, S.c);
    else
      bisect();
  };
  // walk down the chain thr[i], thr[i - 1], ... of candidates for lo
  auto shrink = [&](int i) {
    for (;;) {
      if (!(S.c > S.hi_t) || capped()) return shrunk();
      if (i < 0) {
        S.phase = kPhShrink;  // from S.lo
        return;
      }
      S.lo = thr[i];
      S.c = cnt[i--];
      ++S.evals;
    }
  };
  const int top = S.nb - 1;
  switch (S.phase) {
    case kPhBranch:
      return done(1e4, cnt[0]);
    case kPhInit:
      S.c = cnt[top];
      ++S.evals;
      if (S.c < S.lo_t) {
        S.phase = kPhGrow;
        return;
      }
      if (S.c < S.hi_t) return done(S.g, S.c);
      S.lo = thr[top - 1];
      S.c = cnt[top - 1];
      ++S.evals;
      return shrink(top - 2);
    case kPhGrow: {
      int i = 0;
      while (S.c < S.lo_t && !capped()) {
        if (i > top) return;  // more of the chain, from S.g
        S.g = thr[i];
        S.c = cnt[i++];
        ++S.evals;
      }
      if (S.c < S.hi_t) return done(S.g, S.c);
      // lo = g m need not be a threshold of this pass: start the chain below g
      --S.evals;
      S.phase = kPhInit;
      return;
    }
    case kPhShrink:
      return shrink(top);
    default: {
      int h = 1;  // tree node whose midpoint is asked for
      for (;;) {
        if (h >= kSelBatch) return;  // eight levels used: next pass from [lo, hi]
        const int lead = 31 - __clz(h);
        const int i = ((2 * (h - (1 << lead)) + 1) << (7 - lead)) - 1;
        S.g = thr[i];
        S.c = cnt[i];
        ++S.evals;
        if (!((S.c < S.lo_t || S.c > S.hi_t) && (S.hi - S.lo) > 1e-6) || capped())
          return done(S.g, S.c);
        if (S.c < S.lo_t) {
          S.lo = S.g;
          h = 2 * h + 1;
        } else {
          S.hi = S.g;
          h = 2 * h;
        }
      }
    }
  }
}

__device__ void sel_advance(SelState& shared, const double* thr, const int* cnt) {
  SelState S = shared;  // in registers
  sel_step(S, thr, cnt);
  shared = S;
}

// Barrier of a cooperative grid: generation `gen` (1, 2, ... in this launch)
// is over when the counter has reached gen * gridDim.x.  Every CTA arrives
// once per generation.  The wait is bounded: false when it ran out (it cannot
// while all CTAs are resident and arrive).
__device__ bool grid_wait(unsigned int* counter, unsigned gen, int* ok_s) {
  __syncthreads();
  if (threadIdx.x == 0) {
    *ok_s = grid_arrive_wait(counter, gen * gridDim.x);
  }
  __syncthreads();
  return *ok_s != 0;
}

// Ticket of the grid: true in the last CTA to arrive (after its partials
// are visible to it).
__device__ bool last_block(unsigned int* ticket, int* flag_s) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *flag_s = (atomicAdd(ticket, 1u) == gridDim.x - 1u);
    __threadfence();
  }
  __syncthreads();
  return *flag_s != 0;
}

// Sums over the block of NV values per thread, in out_s[0 .. NV) after the
// call (all threads): a shuffle tree per warp, then the warps in order.
// red_s holds NV x warps.
template <int NV>
__device__ void block_sums(const double (&x)[NV], double* red_s, double* out_s) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  double t[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) t[i] = x[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < NV; ++i) t[i] += __shfl_down_sync(0xffffffffu, t[i], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; ++i) red_s[i * nw + w] = t[i];
  __syncthreads();
  if ((int)threadIdx.x < NV) {
    double s = 0.0;
    for (int i = 0; i < nw; ++i) s += red_s[threadIdx.x * nw + i];
    out_s[threadIdx.x] = s;
  }
  __syncthreads();
}

// The same for maxima.
template <int NV>
__device__ void block_maxima(const double (&x)[NV], double* red_s, double* out_s) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  double t[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) t[i] = x[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < NV; ++i) t[i] = fmax(t[i], __shfl_down_sync(0xffffffffu, t[i], o));
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; ++i) red_s[i * nw + w] = t[i];
  __syncthreads();
  if ((int)threadIdx.x < NV) {
    double m = red_s[threadIdx.x * nw];
    for (int i = 1; i < nw; ++i) m = fmax(m, red_s[threadIdx.x * nw + i]);
    out_s[threadIdx.x] = m;
  }
  __syncthreads();
}

// Per-thread sums over CTAs of the NC columns of per-CTA partials (rows
// b = threadIdx.x, + blockDim.x, ...), all columns of a row loaded together
// and rows four at a time, so the loads of a thread overlap.  Fixed order.
template <int NC>
__device__ void thread_partials(const double* part, int stride, int nblocks, double (&t)[NC]) {
#pragma unroll
  for (int c = 0; c < NC; ++c) t[c] = 0.0;
  int b = threadIdx.x;
  for (; b + 3 * (int)blockDim.x < nblocks; b += 4 * blockDim.x) {
    double v[4][NC];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < NC; ++c) v[u][c] = __ldcg(part + (size_t)(b + u * blockDim.x) * stride + c);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < NC; ++c) t[c] += v[u][c];
  }
  for (; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int c = 0; c < NC; ++c) t[c] += __ldcg(part + (size_t)b * stride + c);
}

// Apply date e's frozen decision (depth chain, no shift) to the running
// values and deflate them to date e - 1 when `deflate`
// (updateDeflatedNextStepValuesMulti_gold then
// updateDeflationOfContinuationValues_gold).
__global__ void __launch_bounds__(kNestThreads)
    nested_decide_kernel(const __grid_constant__ LSDate dd, int kind, int e, int deflate,
                         const LsRuleView rule, const float* __restrict__ vars,
                         const float* __restrict__ cf, const float* __restrict__ ex,
                         const float* __restrict__ num, float* __restrict__ y, int paths) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; p0 < paths;
       p0 += 2 * stride) {
    const bool two = p0 + stride < paths;
    const size_t p[2] = {(size_t)p0, (size_t)(two ? p0 + stride : p0)};
    float v[2][kMaxVars], exv[2], t[2], ratio[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int k = 0; k < kMaxVars; ++k)
        v[h][k] = k < dd.nvars ? vars[((size_t)e * kMaxVars + k) * paths + p[h]] : 0.0f;
      exv[h] = ex ? ex[(size_t)e * paths + p[h]] : 0.0f;
      t[h] = (cf ? cf[(size_t)e * paths + p[h]] : 0.0f) + y[p[h]];
      ratio[h] = deflate ? num[(size_t)(e - 1) * paths + p[h]] / num[(size_t)e * paths + p[h]]
                         : 1.0f;
    }
    double est[2];
    ls_chain_estimates<2>(rule, e, kind, dd.nvars, dd.nbasis, dd.mono, v, exv, est);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h && !two) break;
      const float yy = ((double)exv[h] > est[h]) ? exv[h] : t[h];
      y[p[h]] = deflate ? yy * ratio[h] : yy;
    }
  }
}

struct NestArgs {
  LSDate dd;
  int kind;  // ls_basis_kind of the date's table
  int e, d, rows, paths, min_paths;
  double lower_frac, upper_frac, sds, mult;
};

// Barrier counter, ticket and histograms of one selection launch, zero when
// it starts: a regression holds two, and each launch clears the one that the
// next launch uses.
struct NestSync {
  unsigned int barrier, ticket;
  int hist[kSelPasses][kSelBatch];
};

// From regression d to the paths of regression d + 1 of date e, one
// cooperative launch (one CTA per SM, each thread keeps the same paths
// throughout):
//  * the net values est - exercise value of regression d on its paths
//    (d = 0: all; else |net| <= cut of d - 1, net holding d - 1's values),
//    +inf elsewhere, and their FP64 moments; the one-sign shortcut (d = 0);
//  * the half-width search: each pass counts |net| against up to 256
//    thresholds (a shared-memory histogram per CTA, integer atomics into the
//    pass's global one, whose totals do not depend on the order), and every
//    CTA advances the same search from the totals.  More than min_paths
//    paths selected: cuts of regression d and the path count of regression
//    d + 1; otherwise the date stops nesting;
//  * the moments of the basis variables over the selected paths (means /
//    sds row d + 1; GenerateLSRegressionMatrixSelectivelyNormalisingVariables_
//    gold, gold/LS_regression.h:524-600), joined by the last CTA.
// The passes stream 8-32 MB that sit in L2 and are bound by latency: with one
// launch each for the net values, six selection passes and the moments a
// depth paid eight launch gaps, as many serial tails (a ticket, one thread
// sorting and looking up thresholds, state through global memory) and the
// idle passes.  Here a pass ends with a grid barrier of about 2 us, two to
// three passes per search.  The regression (80 dates, depth 4), together with
// the known basis tables in the net values and decisions and the shorter
// tails of ls_date_kernel: 33.8 -> 14.3 ms at 2^18 paths, 46.3 -> 23.6 ms at
// 2^20, 11.9 -> 5.2 ms for 40 dates at 30,001.
__global__ void __launch_bounds__(kSelThreads, 1)
    nested_select_kernel(const __grid_constant__ NestArgs a, const float* __restrict__ vars,
                         const float* __restrict__ ex, const double* __restrict__ beta,
                         float* means, float* sds, double* cuts, int* npaths, double* net,
                         double* part, NestSync* sync, NestSync* next, int* stopped,
                         int* status) {
  constexpr int NW = kSelThreads / 32;
  __shared__ double beta_s[kMaxBasis];
  __shared__ float mom_s[2][kMaxVars];
  __shared__ double red_s[2 * kMaxVars * NW];
  __shared__ double out_s[2 * kMaxVars];
  __shared__ int before_s[NW];
  __shared__ double thr_s[kSelBatch];
  __shared__ int hist_s[kSelBatch];
  __shared__ SelState S;
  __shared__ int flag_s;
  const int e = a.e, d = a.d, paths = a.paths, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  if (blockIdx.x == 0)
    for (int i = tid; i < (int)(sizeof(NestSync) / 4); i += kSelThreads)
      reinterpret_cast<unsigned*>(next)[i] = 0u;
  // uniform over the grid: this launch sets the flag after a barrier only
  if (stopped[e]) return;
  const size_t row = (size_t)e * a.rows + d;
  if (tid < kMaxBasis) beta_s[tid] = beta[row * kMaxBasis + tid];
  if (tid < kMaxVars) {
    mom_s[0][tid] = means ? means[row * kMaxVars + tid] : 0.0f;
    mom_s[1][tid] = means ? sds[row * kMaxVars + tid] : 1.0f;
  }
  __syncthreads();
  const double cut0 = d > 0 ? cuts[(row - 1) * 2 + 1] : 0.0;
  const long long p_begin = (long long)blockIdx.x * kSelThreads + tid;
  const long long stride = (long long)gridDim.x * kSelThreads;
  // the net values of two paths at a time
  const LsRuleView one{1, beta_s, means ? mom_s[0] : nullptr, mom_s[1], nullptr, nullptr};
  double s1 = 0.0, s2 = 0.0, mx = -INFINITY, mn = INFINITY;
  for (long long p0 = p_begin; p0 < paths; p0 += 2 * stride) {
    const bool two = p0 + stride < paths;
    const size_t p[2] = {(size_t)p0, (size_t)(two ? p0 + stride : p0)};
    float v[2][kMaxVars], exv[2];
    bool member[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      member[h] = d == 0 || fabs(net[p[h]]) <= cut0;
#pragma unroll
      for (int k = 0; k < kMaxVars; ++k)
        v[h][k] = k < a.dd.nvars ? vars[((size_t)e * kMaxVars + k) * paths + p[h]] : 0.0f;
      exv[h] = ex ? ex[(size_t)e * paths + p[h]] : 0.0f;
    }
    double est[2];
    ls_chain_estimates<2>(one, 0, a.kind, a.dd.nvars, a.dd.nbasis, a.dd.mono, v, exv, est);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h && !two) break;
      double nv = INFINITY;
      if (member[h]) {
        nv = est[h] - (double)exv[h];
        s1 += nv;
        s2 += nv * nv;
        mx = fmax(mx, nv);
        mn = fmin(mn, nv);
      }
      net[p[h]] = nv;
    }
  }
  {
    const double sums[2] = {s1, s2}, maxima[2] = {mx, -mn};
    block_sums<2>(sums, red_s, out_s);
    block_maxima<2>(maxima, red_s, out_s + 2);
    if (tid < 4) part[(size_t)blockIdx.x * 4 + tid] = out_s[tid];
  }
  unsigned gen = 1;
  bool ok = grid_wait(&sync->barrier, gen, &flag_s);
  // every CTA joins the partials in the same order
  {
    double t[2], m[2] = {-INFINITY, -INFINITY};
    thread_partials<2>(part, 4, gridDim.x, t);
    for (int b = tid; b < (int)gridDim.x; b += kSelThreads) {
      m[0] = fmax(m[0], __ldcg(part + (size_t)b * 4 + 2));
      m[1] = fmax(m[1], __ldcg(part + (size_t)b * 4 + 3));
    }
    block_sums<2>(t, red_s, out_s);
    block_maxima<2>(m, red_s, out_s + 2);
    const double S1 = out_s[0], S2 = out_s[1], MX = out_s[2], MN = -out_s[3];
    if (tid == 0) {
      S = SelState{};
      S.phase = kPhDone;
      if (d > 0 || !(MX <= 0.0 || MN >= 0.0)) {
        const int n_pre = d == 0 ? paths : npaths[row];
        S.lo_t = (int)(n_pre * a.lower_frac);
        S.hi_t = (int)(n_pre * a.upper_frac);
        S.mult = a.mult;
        if (n_pre > S.lo_t && n_pre < S.hi_t) {
          S.phase = kPhBranch;
        } else {
          const double mean = S1 / n_pre;
          S.g = sqrt(S2 / n_pre - mean * mean) * a.sds;
          S.phase = kPhInit;
        }
      }
    }
    __syncthreads();
  }
  for (int pass = 0; pass < kSelPasses && S.phase != kPhDone && ok; ++pass) {
    sel_thresholds(S, thr_s);
    const int nb = S.nb;
    for (int i = tid; i < nb; i += kSelThreads) hist_s[i] = 0;
    __syncthreads();
    const double top = thr_s[nb - 1];
    for (long long p = p_begin; p < paths; p += stride) {
      const double x = fabs(net[p]);
      if (!(x <= top)) continue;
      int lo = 0, hi = nb - 1;  // first i with x <= thr[i]
      while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (x <= thr_s[m])
          hi = m;
        else
          lo = m + 1;
      }
      atomicAdd(&hist_s[lo], 1);
    }
    __syncthreads();
    int* hist_g = sync->hist[pass];
    for (int i = tid; i < nb; i += kSelThreads)
      if (hist_s[i]) atomicAdd(hist_g + i, hist_s[i]);
    ok = grid_wait(&sync->barrier, ++gen, &flag_s);
    // counts = inclusive prefix of the totals (nb <= 256: eight warps)
    static_assert(kSelBatch == 256 && kSelThreads >= kSelBatch, "one thread per bin");
    int c = tid < nb ? __ldcg(hist_g + tid) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += t;
    }
    if (lane == 31) before_s[warp] = c;
    __syncthreads();
    if (tid < nb) {
      int before = 0;
      for (int w = 0; w < warp; ++w) before += before_s[w];
      hist_s[tid] = before + c;
    }
    __syncthreads();
    if (tid == 0) sel_advance(S, thr_s, hist_s);
    __syncthreads();
  }
  const bool nest = ok && S.phase == kPhDone && S.after > a.min_paths;
  if (blockIdx.x == 0 && tid == 0) {
    int st = S.status;
    if (!ok)
      st |= kSelWait;
    else if (S.phase != kPhDone)
      st |= kSelIncomplete;
    if (st) atomicOr(status, st);
    if (nest) {
      cuts[row * 2] = -S.cut;
      cuts[row * 2 + 1] = S.cut;
      npaths[row + 1] = S.after;
    } else {
      stopped[e] = 1;  // every CTA is past its read of the flag (first barrier)
    }
  }
  if (!nest || !means) return;
  const double cut = S.cut;
  double acc[2 * kMaxVars] = {0, 0, 0, 0, 0, 0};
  for (long long p = p_begin; p < paths; p += stride) {
    if (!(fabs(net[p]) <= cut)) continue;
#pragma unroll
    for (int v = 0; v < kMaxVars; ++v) {
      const double x = v < a.dd.nvars ? vars[((size_t)e * kMaxVars + v) * paths + p] : 0.0;
      acc[2 * v] += x;
      acc[2 * v + 1] += x * x;
    }
  }
  // every CTA has read the net partials before the second barrier at the
  // latest (a search takes one pass or more), so their buffer is free
  block_sums<2 * kMaxVars>(acc, red_s, out_s);
  if (tid < 2 * kMaxVars) part[(size_t)blockIdx.x * 8 + tid] = out_s[tid];
  if (!last_block(&sync->ticket, &flag_s)) return;
  double t6[2 * kMaxVars];
  thread_partials<2 * kMaxVars>(part, 8, gridDim.x, t6);
  block_sums<2 * kMaxVars>(t6, red_s, out_s);
  if (tid < kMaxVars) {
    double m = 0.0, sd = 1.0;
    if (tid < a.dd.nvars) {
      const double n = (double)S.after;
      m = out_s[2 * tid] / n;
      const double var = out_s[2 * tid + 1] / n - m * m;
      sd = var > 0.0 ? sqrt(var) : 1.0;
    }
    means[(row + 1) * kMaxVars + tid] = (float)m;
    sds[(row + 1) * kMaxVars + tid] = (float)sd;
  }
}

// Path counts: regression 0 of every date uses all paths; the rest start
// at zero.  Rows of nested moments start as (0, 1).
__global__ void nested_init_kernel(int n_ex, int rows, int paths, int* __restrict__ npaths,
                                   float* __restrict__ means, float* __restrict__ sds) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_ex * rows) return;
  npaths[i] = (i % rows == 0) ? paths : 0;
  if (means && i % rows != 0)
    for (int v = 0; v < kMaxVars; ++v) {
      means[(size_t)i * kMaxVars + v] = 0.0f;
      sds[(size_t)i * kMaxVars + v] = 1.0f;
    }
}

}  // namespace

namespace lmm {
int reduce_launch(const float* d_in, const float* d_div, size_t n, double scale,
                  double* d_partials, double* d_out, cudaStream_t stream);
}

namespace {

constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

struct NestWs {
  float* y;
  double* part;          // date kernel: ls_gram_blocks() x kLsMaxPairs
  unsigned int* counter; // date kernel tickets [E]
  double* mom;           // all-path moments: E x blocks x 6
  double* red;           // final reduction
  double* net;           // [P]
  double* npart;         // net / moments partials: blocks x 8
  NestSync* sync;        // [2]
  int* stopped;          // [E]
  int* npaths;           // [E][kMaxDepth]
};

size_t nested_ws_bytes(int paths, int n_ex, NestWs* w, char* base) {
  const size_t nb = (size_t)ls_gram_blocks();
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  NestWs t;
  t.y = (float*)take((size_t)paths * sizeof(float));
  t.part = (double*)take(nb * kLsMaxPairs * sizeof(double));
  t.counter = (unsigned int*)take((size_t)n_ex * sizeof(unsigned int));
  t.mom = (double*)take((size_t)n_ex * nb * 6 * sizeof(double));
  t.red = (double*)take(512 * sizeof(double));
  t.net = (double*)take((size_t)paths * sizeof(double));
  t.npart = (double*)take(nb * 8 * sizeof(double));
  t.sync = (NestSync*)take(2 * sizeof(NestSync));
  t.stopped = (int*)take((size_t)n_ex * sizeof(int));
  t.npaths = (int*)take((size_t)n_ex * kMaxDepth * sizeof(int));
  if (w) *w = t;
  return off + 256;
}

// The selection kernel as a cooperative launch (its CTAs wait on one
// another); `k` counts the regression's selection launches.
int launch_select(NestArgs a, int grid, const float* vars, const float* ex, const double* beta,
                  float* means, float* sds, double* cuts, int* npaths, const NestWs& w, int k,
                  int* status, cudaStream_t s) {
  double *net = w.net, *part = w.npart;
  NestSync *sync = w.sync + (k & 1), *next = w.sync + ((k + 1) & 1);
  int* stopped = w.stopped;
  void* args[] = {&a,      &vars, &ex,   &beta, &means, &sds,    &cuts,
                  &npaths, &net,  &part, &sync, &next,  &stopped, &status};
  TRY(check_cuda(cudaLaunchCooperativeKernel((const void*)nested_select_kernel, dim3(grid),
                                             dim3(kSelThreads), args, 0, s),
                 "nested_select_kernel"));
  return check_launch("nested_select_kernel");
}

}  // namespace

extern "C" size_t lmm_ls_nested_workspace_bytes(int paths, int n_exercise) {
  if (paths < 1 || n_exercise < 1) return 0;
  return nested_ws_bytes(paths, n_exercise, nullptr, nullptr);
}

extern "C" int lmm_ls_regress_nested(int n_exercise, int paths, const float* d_vars,
                                     const int* h_nvars, const uint8_t* h_monomials,
                                     const int* h_nbasis, const float* d_cf, const float* d_ex,
                                     const float* d_num, int normalise,
                                     const lmm_ls_select* sel, void* d_workspace,
                                     size_t workspace_bytes, double* d_beta, float* d_means,
                                     float* d_sds, double* d_cuts, int* d_npaths,
                                     int* d_status, double* d_price, lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1,
              "lmm_ls_regress_nested: bad sizes");
  LMM_REQUIRE(d_vars && h_nvars && h_monomials && h_nbasis && d_num && d_workspace && d_beta &&
                  d_cuts && d_status && d_price && sel,
              "lmm_ls_regress_nested: null pointer");
  LMM_REQUIRE(!normalise || (d_means && d_sds),
              "lmm_ls_regress_nested: normalise needs means/sds outputs");
  const int D = sel->depth;
  LMM_REQUIRE(D >= 1 && D <= kMaxDepth, "lmm_ls_regress_nested: depth %d outside 1..%d", D,
              kMaxDepth);
  LMM_REQUIRE(sel->lower_frac > 0.0 && sel->upper_frac > sel->lower_frac &&
                  sel->upper_frac <= 1.0,
              "lmm_ls_regress_nested: need 0 < lower_frac < upper_frac <= 1");
  LMM_REQUIRE(sel->sds > 0.0 && sel->multiplier > 0.0 && sel->multiplier < 1.0 &&
                  sel->min_paths >= 0,
              "lmm_ls_regress_nested: need sds > 0, 0 < multiplier < 1, min_paths >= 0");
  const size_t need = nested_ws_bytes(paths, n_exercise, nullptr, nullptr);
  LMM_REQUIRE(workspace_bytes >= need, "lmm_ls_regress_nested: workspace too small (%zu < %zu)",
              workspace_bytes, need);
  cudaStream_t s = (cudaStream_t)stream;
  NestWs w;
  nested_ws_bytes(paths, n_exercise, &w,
                  (char*)(((uintptr_t)d_workspace + 255) & ~(uintptr_t)255));
  LSBasisSpec spec{h_nvars, h_monomials, h_nbasis};
  std::vector<LSDate> dates(n_exercise);
  for (int e = 0; e < n_exercise; ++e) TRY(ls_fill_date(spec, e, &dates[e]));
  int* npaths = d_npaths ? d_npaths : w.npaths;
  const size_t rows = (size_t)n_exercise * D;

  TRY(check_cuda(cudaMemsetAsync(d_status, 0, sizeof(int), s), "nested: status"));
  TRY(check_cuda(cudaMemsetAsync(w.counter, 0, (size_t)n_exercise * sizeof(unsigned int), s),
                 "nested: counters"));
  TRY(check_cuda(cudaMemsetAsync(w.sync, 0, 2 * sizeof(NestSync), s), "nested: histograms"));
  TRY(check_cuda(cudaMemsetAsync(w.stopped, 0, (size_t)n_exercise * sizeof(int), s),
                 "nested: flags"));
  TRY(check_cuda(cudaMemsetAsync(d_cuts, 0, rows * 2 * sizeof(double), s), "nested: cuts"));
  TRY(check_cuda(cudaMemsetAsync(d_beta, 0, rows * kMaxBasis * sizeof(double), s),
                 "nested: coefficients"));
  TRY(check_cuda(cudaMemsetAsync(w.y, 0, (size_t)paths * sizeof(float), s), "nested: values"));
  nested_init_kernel<<<div_up((int)rows, 128), 128, 0, s>>>(
      n_exercise, D, paths, npaths, normalise ? d_means : nullptr, normalise ? d_sds : nullptr);
  TRY(check_launch("nested_init_kernel"));
  const float* means = nullptr;
  const float* sds = nullptr;
  if (normalise) {
    TRY(ls_moments_launch(d_vars, paths, n_exercise, D, d_means, d_sds, w.mom, s));
    means = d_means;
    sds = d_sds;
  }
  const int nblk = ls_gram_blocks();
  const int grid_path = grid_for(paths, kNestThreads, 4);
  // cooperative launches: no more CTAs than the stream's SMs hold at once
  const int grid_sel = std::min(div_up(paths, kSelThreads), std::min(nblk, stream_sm_count(s)));
  int launches = 0;
  const LsRuleView rule{D, d_beta, means, sds, D > 1 ? d_cuts : nullptr, nullptr};
  for (int e = n_exercise - 1; e >= 0; --e) {
    if (e + 1 < n_exercise) {
      nested_decide_kernel<<<grid_path, kNestThreads, 0, s>>>(
          dates[e + 1], ls_basis_kind(dates[e + 1]), e + 1, 1, rule, d_vars, d_cf, d_ex, d_num, w.y, paths);
      TRY(check_launch("nested_decide_kernel"));
    }
    const int slots = dates[e].nbasis + 1;
    const int per_cta = slots <= 11 ? 512 : slots <= 13 ? 256 : 192;
    const int grid_date = std::min(div_up(paths, per_cta), nblk);
    for (int d = 0; d < D; ++d) {
      NestArgs a;
      memset(&a, 0, sizeof(a));
      a.dd = dates[e];
      a.kind = ls_basis_kind(dates[e]);
      a.e = e;
      a.rows = D;
      a.paths = paths;
      a.min_paths = sel->min_paths;
      a.lower_frac = sel->lower_frac;
      a.upper_frac = sel->upper_frac;
      a.sds = sel->sds;
      a.mult = sel->multiplier;
      if (d > 0) {
        // net values of regression d - 1, the search for its cuts, and the
        // moments of regression d's paths
        a.d = d - 1;
        TRY(launch_select(a, grid_sel, d_vars, d_ex, d_beta, normalise ? d_means : nullptr,
                          normalise ? d_sds : nullptr, d_cuts, npaths, w, launches++, d_status,
                          s));
      }
      LSDateParams P;
      memset(&P, 0, sizeof(P));
      P.e = e;
      P.paths = paths;
      P.cur = dates[e];
      P.has_prev = 0;
      P.read_y = 1;
      P.rows = D;
      P.depth = d;
      if (d > 0) {
        P.mask_net = w.net;
        P.mask_cut = d_cuts + ((size_t)e * D + d - 1) * 2 + 1;
        P.mask_count = npaths + (size_t)e * D + d;
        P.skip = w.stopped + e;
      }
      TRY(launch_date(P, grid_date, d_vars, means, sds, d_cf, d_ex, d_num, d_beta, w.y, w.part,
                      w.counter, nullptr, d_status, nullptr, s));
    }
  }
  nested_decide_kernel<<<grid_path, kNestThreads, 0, s>>>(dates[0], ls_basis_kind(dates[0]), 0, 0, rule, d_vars, d_cf,
                                                          d_ex, d_num, w.y, paths);
  TRY(check_launch("nested_decide_kernel"));
  return reduce_launch(w.y, d_num, (size_t)paths, 1.0 / (double)paths, w.red, d_price, s);
}
