// ls.cu — Longstaff–Schwartz backward induction kept on the device.
//
// Reference behaviour followed (regression depth 1):
//   backward loop        gold/MultiLS_regression.cpp:101-417 and the GPU
//                        orchestration LS_main_cula.h:565-837
//   regression matrix    GenerateLSRegressionMatrixSelectively_gold
//                        (gold/LS_regression.h:431-530): G = E[phi phi^T],
//                        b = E[phi (cf + y)], both divided by the path count
//   exercise update      updateDeflatedNextStepValuesMulti_gold
//                        (gold/MultiLS_regression.h:42-99)
//   deflation            updateDeflationOfContinuationValues_gold
//                        (gold/LS_regression.cpp:98-118): y *= N_{e-1}/N_e
//   basis functions      quadraticPolynomialGenerator /
//                        quadraticPolynomialCrossGenerator
//                        (gold/LS_regression.h:123-240) expressed as monomial
//                        exponent tables, one table per exercise date
//   in-sample price      mean_p y_p / N_0(p)  (MultiLS_regression.cpp:407-416)
// The reference solves each normal-equation system on the host by SVD after
// a device-to-host copy (LinearSolverConcrete_main.cu:127-188); here the
// Gram sums stay on the device and are solved there by a warp-parallel FP64
// Cholesky, so the loop is launch-only and can be captured in a graph: one
// cooperative launch for the whole loop (ls_run_kernel), or one launch per
// date (ls_date_kernel; tables of more than 11 slots, nested regressions and
// the sharded protocol).
#include "lmm_common.cuh"
#include "lmm_device.cuh"
#include "ls_common.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

using namespace lmm;

namespace lmm {
int reduce_launch(const float* d_in, const float* d_div, size_t n,
                  double scale, double* d_partials, double* d_out,
                  cudaStream_t stream);

__device__ __forceinline__ double warp_sum_d(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}

}  // namespace lmm

// Apply the frozen decision of date d to one path and deflate to date d-1,
// from the path's values: xin[v] (v < nvars) the basis variables at d, cf_v
// and ex_v the coupon and exercise value at d, num_prev / num_cur the
// numeraires at d-1 and d, y_in the running value.  beta_d: the date's
// coefficients; mean_d / sd_d: its standardisation (or null).
template <int KIND>
__device__ __forceinline__ float decide_values(const LSDate& dd, int deflate, const float* xin,
                                               const float* mean_d, const float* sd_d,
                                               float cf_v, float ex_v, float num_prev,
                                               float num_cur, const double* beta_d,
                                               float y_in) {
  float x[kMaxVars];
#pragma unroll
  for (int v = 0; v < kMaxVars; ++v) {
    float xv = 0.0f;
    if (v < dd.nvars) {
      xv = xin[v];
      if (mean_d) xv = (xv - mean_d[v]) * sd_d[v];  // sd_d holds 1 / sd
    }
    x[v] = xv;
  }
  float pw[kMaxVars][3];
  ls_powers(x, pw);
  // coefficients re-read per path (volatile) rather than held in 32 registers
  const volatile double* bv = beta_d;
  double est = 0.0;
#pragma unroll
  for (int k = 0; k < kMaxBasis; ++k)
    if (k < (KIND ? basis_K(KIND) : dd.nbasis))
      est += (double)ls_basis<KIND>(pw, dd, k) * bv[k];
  const float t = cf_v + y_in;
  float y = ((double)ex_v > est) ? ex_v : t;
  if (deflate) y = y * (num_prev / num_cur);
  return y;
}

// The same from the arrays of the LS inputs, for path p.
template <int KIND>
__device__ __forceinline__ float apply_decision(
    const LSDate& dd, int d, int deflate, const float* __restrict__ vars,
    const float* mean_d, const float* sd_d, const float* __restrict__ cf,
    const float* __restrict__ ex, const float* __restrict__ num,
    const double* beta_d, float y_in, int paths, int p) {
  float xin[kMaxVars];
#pragma unroll
  for (int v = 0; v < kMaxVars; ++v)
    xin[v] = v < dd.nvars ? vars[((size_t)d * kMaxVars + v) * paths + p] : 0.0f;
  const float cf_v = cf ? cf[(size_t)d * paths + p] : 0.0f;
  const float ex_v = ex ? ex[(size_t)d * paths + p] : 0.0f;
  const float np = deflate ? num[(size_t)(d - 1) * paths + p] : 1.0f;
  const float nc = deflate ? num[(size_t)d * paths + p] : 1.0f;
  return decide_values<KIND>(dd, deflate, xin, mean_d, sd_d, cf_v, ex_v, np, nc, beta_d, y_in);
}

// ---------------------------------------------------------------------------
// One backward date e as one kernel.
//
// Each thread walks its paths (grid stride): it applies date e+1's frozen
// decision (updating the running value y), evaluates the KR - 1 basis slots
// of date e (slots at and above nbasis are zero) and the regression target
// cf_e + y in slot KR - 1, and adds the products of the lower triangle
// (i, j), j <= i < KR, into registers: q(i, j) = i (i + 1) / 2 + j.  With
// NSPLIT = 2 the rows are split between the two warps of a warp pair, which
// handle the same 32 paths, so no thread holds more than 78 sums.  Sums
// within a warp (a few paths per thread, then a fixed shuffle tree over
// its 32 threads) are FP32; everything above them is FP64: a fixed-order
// sum over warps, a partial per CTA in part[cta][q] and the sum over CTAs.  The CTA that finishes last (ticket on
// counter[e]) sums the partials in a fixed order and solves the normal
// equations with a one-warp FP64 Cholesky, so the date needs one launch and
// the result is independent of which CTA came last.
//
// Sums over paths of the reference: GenerateLSRegressionMatrixSelectively_gold
// (gold/LS_regression.h:431-530); its host SVD solve
// (LinearSolverConcrete_main.cu:127-188) is replaced by the Cholesky below.
// ---------------------------------------------------------------------------
// 512 threads per CTA; 384 for 17 slots (78 sums per thread need more than
// the 128 registers a 512-thread CTA allows).
template <int KR>
struct LsThreads {
  static constexpr int value = KR > 13 ? 384 : 512;
};


// rows [R0, R1) of the lower triangle
template <int KR, int R0, int R1>
struct RowSplit {
  static constexpr int q0 = R0 * (R0 + 1) / 2;
  static constexpr int n = R1 * (R1 + 1) / 2 - q0;
};

template <int KR, int NSPLIT>
struct SplitOf;
template <int KR>
struct SplitOf<KR, 1> {
  static constexpr int rs = KR;  // one half: all rows
};
// balance R(R+1)/2 against the rest
template <int KR>
struct SplitOf<KR, 2> {
  static constexpr int rs = KR == 17 ? 12 : KR == 13 ? 9 : (KR * 7) / 10;
};

template <int KR, int R0, int R1>
__device__ __forceinline__ void accumulate_rows(const float* phi, float* acc) {
#pragma unroll
  for (int i = R0; i < R1; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j)
      acc[i * (i + 1) / 2 + j - RowSplit<KR, R0, R1>::q0] += phi[i] * phi[j];
}

// Warp-parallel FP64 Cholesky solve of G beta = b (K <= 16): lane i holds
// row i of G.  A relative diagonal jitter is added and the factorisation
// retried when a pivot fails.  Each column takes one reciprocal square root
// r_j = 1 / sqrt(d_jj): L_jj = d_jj r_j and the column below is scaled by
// r_j, and both substitutions multiply by the kept r_j instead of dividing.
// The back substitution runs by columns of L^T from a shared-memory copy of
// L (Ls, kMaxBasis^2 doubles of scratch).  Returns status bits (1: zero
// diagonal, 2: not positive definite after jitter, 4: jitter added); beta
// is zero on failure.  KC > 0: K is known at compile time (a fixed number of
// columns without a branch each).
template <int KC = 0>
__device__ int warp_cholesky_solve(const double* Gs, int K_in, double* beta_out, double* Ls) {
  constexpr int kMaxBasis = KC > 0 ? KC : lmm::kMaxBasis;  // columns
  const int K = KC > 0 ? KC : K_in;
  const int lane = threadIdx.x & 31;
  if (lane < lmm::kMaxBasis) beta_out[lane] = 0.0;
  double maxd = 0.0;
  for (int i = 0; i < K; ++i) maxd = fmax(maxd, fabs(Gs[i * kLsMaxSlots + i]));
  if (!(maxd > 0.0)) return 1;
  double jitter = 0.0;
  int status = 0;
  double a[kMaxBasis];
  double rinv = 0.0;  // this lane's 1 / L_ii
  bool ok = false;
#pragma unroll 1
  for (int attempt = 0; attempt < 6 && !ok; ++attempt) {
#pragma unroll
    for (int k = 0; k < kMaxBasis; ++k)
      a[k] = (lane < K && k <= lane) ? Gs[lane * kLsMaxSlots + k] +
                                          ((k == lane) ? jitter : 0.0)
                                     : 0.0;
    ok = true;
#pragma unroll
    for (int j = 0; j < kMaxBasis; ++j) {
      if (j < K) {
        const double djj = __shfl_sync(0xffffffffu, a[j], j);
        if (!(djj > 1e-300)) {  // with KC the remaining columns run on, unused
          ok = false;
          if (KC == 0) break;
        }
        const double rj = rsqrt(djj);
        if (lane == j) {
          a[j] = djj * rj;
          rinv = rj;
        }
        if (lane > j) a[j] *= rj;
        // trailing update: a[i][k] -= L[i][j] L[k][j] for j < k <= i
#pragma unroll
        for (int k = j + 1; k < kMaxBasis; ++k) {
          if (k < K) {
            const double lkj = __shfl_sync(0xffffffffu, a[j], k);
            if (lane >= k) a[k] -= a[j] * lkj;
          }
        }
      }
    }
    if (!ok) jitter = (jitter == 0.0) ? 1e-14 * maxd : jitter * 100.0;
  }
  if (!ok) return 2;
  if (jitter > 0.0) status |= 4;
  // forward substitution L z = b: z_j = (b_j - sum_{k<j} L_jk z_k) r_j
  double z = (lane < K) ? Gs[lane * kLsMaxSlots + kLsMaxSlots - 1] : 0.0;
#pragma unroll
  for (int j = 0; j < kMaxBasis; ++j) {
    if (j < K) {
      const double zj = __shfl_sync(0xffffffffu, z * rinv, j);
      if (lane == j) z = zj;
      if (lane > j) z -= a[j] * zj;
    }
  }
  // back substitution L^T beta = z by columns: lane k holds column k of L
  // (L_ik, i > k) and subtracts L_ik beta_i once beta_i is known
  if (lane < K) {
#pragma unroll
    for (int k = 0; k < kMaxBasis; ++k) Ls[lane * kMaxBasis + k] = a[k];
  }
  __syncwarp();
  double lcol[kMaxBasis];
#pragma unroll
  for (int i = 0; i < kMaxBasis; ++i)
    lcol[i] = (lane < K && i < K && i > lane) ? Ls[i * kMaxBasis + lane] : 0.0;
  __syncwarp();
  double bet = 0.0;
#pragma unroll
  for (int i = kMaxBasis - 1; i >= 0; --i) {
    if (i < K) {
      const double bi = __shfl_sync(0xffffffffu, z * rinv, i);
      if (lane == i) bet = bi;
      if (lane < i) z -= lcol[i] * bi;
    }
  }
  if (lane < lmm::kMaxBasis) beta_out[lane] = (lane < K) ? bet : 0.0;
  return status;
}

// acc[0 .. N) summed over the warp's lanes by exchanging halves of the
// accumulators (67 shuffles for 66 sums instead of five each): the lane is
// left with the sums q = first .. first + count - 1 in acc[0 .. count).  Every
// sum is the binary tree over lanes l and l + 16, then + 8, ..., + 1.
template <int N, class V>
__device__ __forceinline__ void warp_sums_range(int o, int& first, int& count) {
  constexpr int H = (N + 1) / 2;
  if (threadIdx.x & o) {
    first += H;
    count = max(count - H, 0);
  } else {
    count = min(count, H);
  }
}
template <int N, class V>
__device__ __forceinline__ void warp_sums_step(V* acc, int o, int& first, int& count) {
  constexpr int H = (N + 1) / 2;
  const bool up = (threadIdx.x & o) != 0;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const V hi = H + i < N ? acc[H + i] : V(0);
    const V send = up ? acc[i] : hi, keep = up ? hi : acc[i];
    acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
  }
  warp_sums_range<N, V>(o, first, count);
}
template <int N>
constexpr int warp_sums_left() {  // five halvings
  return ((((((((((N + 1) / 2) + 1) / 2) + 1) / 2) + 1) / 2) + 1) / 2);
}
template <int N>
__device__ __forceinline__ void warp_sums(float* acc, int& first, int& count) {
  first = 0;
  count = N;
  constexpr int N1 = (N + 1) / 2, N2 = (N1 + 1) / 2, N3 = (N2 + 1) / 2, N4 = (N3 + 1) / 2;
  warp_sums_step<N>(acc, 16, first, count);
  warp_sums_step<N1>(acc, 8, first, count);
  warp_sums_step<N2>(acc, 4, first, count);
  warp_sums_step<N3>(acc, 2, first, count);
  warp_sums_step<N4>(acc, 1, first, count);
}
// the same with the sums in FP64 (the lanes' values still FP32)
template <int N>
__device__ __forceinline__ void warp_sums_d(const float* acc, double (&d)[(N + 1) / 2],
                                            int& first, int& count) {
  constexpr int N1 = (N + 1) / 2, N2 = (N1 + 1) / 2, N3 = (N2 + 1) / 2, N4 = (N3 + 1) / 2;
  const bool up = (threadIdx.x & 16) != 0;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    const float hi = N1 + i < N ? acc[N1 + i] : 0.0f;
    const float send = up ? acc[i] : hi, keep = up ? hi : acc[i];
    d[i] = (double)keep + (double)__shfl_xor_sync(0xffffffffu, send, 16);
  }
  first = 0;
  count = N;
  warp_sums_range<N, double>(16, first, count);
  warp_sums_step<N1>(d, 8, first, count);
  warp_sums_step<N2>(d, 4, first, count);
  warp_sums_step<N3>(d, 2, first, count);
  warp_sums_step<N4>(d, 1, first, count);
}

// Staged loop of the date kernel: the inputs of a path, one shared-memory
// row each, in kLsStages slots per thread (masked launches also stage the
// path's membership value).  Rows: basis variables at e (3), coupon at e, running value y,
// basis variables at e+1 (3), coupon and exercise value at e+1, numeraires
// at e and e+1.
constexpr int kLsStages = 4;
constexpr int kLsInputs = 12;
constexpr int kInX = 0, kInCf = 3, kInY = 4, kInXNext = 5, kInCfNext = 8, kInExNext = 9,
              kInNum = 10, kInNumNext = 11;
// masked launches also stage each path's membership value (mask_net, FP64)
// after the input rows: [kLsStages][threads] doubles
template <int KR, int NSPLIT, bool MASKED>
constexpr size_t ls_stage_bytes() {
  return (size_t)kLsStages * LsThreads<KR>::value *
         (kLsInputs * sizeof(float) + (MASKED ? sizeof(double) : 0));
}

// With rows split over a warp pair only the first warp writes a path's running
// value, in the place both read it from: the pair meets in every iteration,
// so that the second warp's copy of the stage is in before the write.
template <int NSPLIT>
__device__ __forceinline__ void pair_sync(int warp) {
  if (NSPLIT == 2) asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
}

template <int KR, int NSPLIT, int KIND, bool MASKED>
__global__ void __launch_bounds__(LsThreads<KR>::value, 1)
    ls_date_kernel(const __grid_constant__ LSDateParams P,
                   const float* __restrict__ vars,
                   const float* __restrict__ means,
                   const float* __restrict__ sds, const float* __restrict__ cf,
                   const float* __restrict__ ex, const float* __restrict__ num,
                   double* __restrict__ beta, float* __restrict__ y,
                   double* __restrict__ part, unsigned int* __restrict__ counter,
                   double* __restrict__ gram_out, int* __restrict__ status,
                   double* __restrict__ sums_out) {
  constexpr int RS = SplitOf<KR, NSPLIT>::rs;
  constexpr int NA0 = RowSplit<KR, 0, RS>::n;
  constexpr int NA1 = RowSplit<KR, RS, KR>::n;
  constexpr int NA = NA0 > NA1 ? NA0 : NA1;
  constexpr int NPAIRS = KR * (KR + 1) / 2;
  constexpr int kLsThreads = LsThreads<KR>::value;
  constexpr int NW = kLsThreads / 32;
  __shared__ double beta_prev[kMaxBasis];
  __shared__ float mom_s[4][kMaxVars];  // mean, 1/sd of date e, then of e+1
  __shared__ double red_s[NW][NA];
  __shared__ double share_s[kLsThreads];
  __shared__ double sums_s[NPAIRS];
  __shared__ double G_s[kLsMaxSlots * kLsMaxSlots];
  __shared__ int last_s;
  __shared__ const float* src_s[kLsInputs];  // input rows of the staged loop
  extern __shared__ float ls_stage[];        // [kLsStages][kLsInputs][threads]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e = P.e, paths = P.paths;
  if (P.skip && *P.skip) return;
  const int rows = P.rows > 0 ? P.rows : 1;
  const size_t row = (size_t)e * rows + P.depth, prev_row = (size_t)(e + 1) * rows;
  const double cut = MASKED ? *P.mask_cut : 0.0;
  if (tid < kMaxBasis)
    beta_prev[tid] = P.has_prev ? beta[prev_row * kMaxBasis + tid] : 0.0;
  if (tid < kLsInputs) {
    const size_t cur = (size_t)e * paths, nxt = cur + paths;
    const float* sp = nullptr;
    if (tid < kInCf) {
      if (tid < P.cur.nvars) sp = vars + ((size_t)e * kMaxVars + tid) * paths;
    } else if (tid == kInCf) {
      sp = cf ? cf + cur : nullptr;
    } else if (tid == kInY) {
      sp = (P.has_prev || P.read_y) ? y : nullptr;
    } else if (P.has_prev) {
      if (tid < kInCfNext) {
        const int v = tid - kInXNext;
        if (v < P.prev.nvars) sp = vars + ((size_t)(e + 1) * kMaxVars + v) * paths;
      } else if (tid == kInCfNext) {
        sp = cf ? cf + nxt : nullptr;
      } else if (tid == kInExNext) {
        sp = ex ? ex + nxt : nullptr;
      } else if (tid == kInNum) {
        sp = num + cur;
      } else {
        sp = num + nxt;
      }
    }
    src_s[tid] = sp;
  }
  if (tid < kMaxVars && means) {
    mom_s[0][tid] = means[row * kMaxVars + tid];
    mom_s[1][tid] = 1.0f / sds[row * kMaxVars + tid];
    if (P.has_prev) {
      mom_s[2][tid] = means[prev_row * kMaxVars + tid];
      mom_s[3][tid] = 1.0f / sds[prev_row * kMaxVars + tid];
    }
  }
  __syncthreads();
  const int half = (NSPLIT == 2) ? (warp & 1) : 0;
  const int per_cta = kLsThreads / NSPLIT;
  const int K = P.cur.nbasis;
  float acc[NA];
#pragma unroll
  for (int q = 0; q < NA; ++q) acc[q] = 0.0f;
  const int stride = gridDim.x * per_cta;
  // the Gram products of one path from its basis variables at date e, its
  // coupon at e and its running value
  auto accumulate_path = [&](const float* xe, float cfe, float yp) {
    float x[kMaxVars];
#pragma unroll
    for (int v = 0; v < kMaxVars; ++v) {
      float xv = 0.0f;
      if (v < P.cur.nvars) {
        xv = xe[v];
        if (means) xv = (xv - mom_s[0][v]) * mom_s[1][v];
      }
      x[v] = xv;
    }
    float pw[kMaxVars][3];
    ls_powers(x, pw);
    float phi[KR];
#pragma unroll
    for (int k = 0; k < KR - 1; ++k)
      phi[k] = (k < (KIND ? basis_K(KIND) : K)) ? ls_basis<KIND>(pw, P.cur, k) : 0.0f;
    phi[KR - 1] = cfe + yp;
    if (half == 0)
      accumulate_rows<KR, 0, RS>(phi, acc);
    else
      accumulate_rows<KR, RS, KR>(phi, acc);
  };
  {
    // The loop is bound by memory latency: the inputs of each path are
    // copied kLsStages - 1 iterations ahead into shared memory (cp.async, no
    // registers held), one row of the stage per input.  When every input
    // row is 16-byte aligned (paths a multiple of 4) the warp copies its 32
    // paths' rows in 16-byte chunks, lane l taking chunk l % 8 of rows
    // l / 8, l / 8 + 4 and l / 8 + 8; otherwise each thread copies its own
    // path's values.  The loop runs whole warps (a lane past the last path
    // still copies and waits, but adds nothing).  With rows split over a
    // warp pair both warps take the same 32 paths, each staging its own copy.
    const bool vec16 = P.vec16 != 0;
    const int r0 = lane >> 3, c4 = (lane & 7) * 4;
    const float* const rp0 = src_s[r0];
    const float* const rp1 = src_s[r0 + 4];
    const float* const rp2 = src_s[r0 + 8];
    float* const wstage = ls_stage + warp * 32;
    double* const mstage = reinterpret_cast<double*>(ls_stage + kLsStages * kLsInputs * kLsThreads);
    auto issue = [&](int it, int qw) {  // qw: the warp's first path
      float* dst = wstage + (it & (kLsStages - 1)) * kLsInputs * kLsThreads;
      if (MASKED && qw + lane < paths)
        cp_async8(mstage + (it & (kLsStages - 1)) * kLsThreads + tid, P.mask_net + qw + lane);
      if (vec16) {
        const int qb = qw + c4;
        if (qb < paths) {
          if (rp0) cp_async16(dst + r0 * kLsThreads + c4, rp0 + qb);
          if (rp1) cp_async16(dst + (r0 + 4) * kLsThreads + c4, rp1 + qb);
          if (rp2) cp_async16(dst + (r0 + 8) * kLsThreads + c4, rp2 + qb);
        }
      } else if (qw + lane < paths) {
#pragma unroll
        for (int i = 0; i < kLsInputs; ++i)
          if (src_s[i]) cp_async4(dst + i * kLsThreads + lane, src_s[i] + qw + lane);
      }
      cp_async_commit();
    };
    const int w0 = blockIdx.x * per_cta + (warp / NSPLIT) * 32;
#pragma unroll
    for (int k = 0; k < kLsStages - 1; ++k) issue(k, w0 + k * stride);
    int it = 0;
    for (int qw = w0; qw < paths; qw += stride, ++it) {
      issue(it + kLsStages - 1, qw + (kLsStages - 1) * stride);
      cp_async_wait<kLsStages - 1>();
      __syncwarp();
      pair_sync<NSPLIT>(warp);
      const int p = qw + lane;
      const bool member =
          !MASKED || (p < paths && fabs(mstage[(it & (kLsStages - 1)) * kLsThreads + tid]) <= cut);
      if (p < paths && member) {
        const float* in = wstage + (it & (kLsStages - 1)) * kLsInputs * kLsThreads + lane;
        float yp = 0.0f;
        if (P.has_prev) {
          float xp[kMaxVars];
#pragma unroll
          for (int v = 0; v < kMaxVars; ++v)
            xp[v] = v < P.prev.nvars ? in[(kInXNext + v) * kLsThreads] : 0.0f;
          yp = decide_values<KIND>(P.prev, 1, xp, means ? mom_s[2] : nullptr, mom_s[3],
                                   cf ? in[kInCfNext * kLsThreads] : 0.0f,
                                   ex ? in[kInExNext * kLsThreads] : 0.0f,
                                   in[kInNum * kLsThreads], in[kInNumNext * kLsThreads],
                                   beta_prev, in[kInY * kLsThreads]);
        } else if (P.read_y) {
          yp = in[kInY * kLsThreads];
        }
        if (half == 0 && !P.read_y) y[p] = yp;
        float xe[kMaxVars];
#pragma unroll
        for (int v = 0; v < kMaxVars; ++v)
          xe[v] = v < P.cur.nvars ? in[(kInX + v) * kLsThreads] : 0.0f;
        accumulate_path(xe, cf ? in[kInCf * kLsThreads] : 0.0f, yp);
      }
      // every lane's reads of this stage precede its refill, issued by
      // other lanes in a later iteration
      __syncwarp();
    }
    cp_async_wait<0>();
  }
  // warp sums (a fixed tree), then FP64 over warps in a fixed order.
  // All-path launches sum within the warp in FP32 (each thread holds several
  // paths' FP32 sums already).  Masked launches (nested regressions on a
  // subset, about one path per thread) sum in FP64: their Grams are close to
  // singular, and the FP32 tree would be their largest rounding error.
  int first, count;
  if (MASKED) {
    double d[(NA + 1) / 2];
    warp_sums_d<NA>(acc, d, first, count);
#pragma unroll
    for (int i = 0; i < warp_sums_left<NA>(); ++i)
      if (i < count) red_s[warp][first + i] = d[i];
  } else {
    warp_sums<NA>(acc, first, count);
#pragma unroll
    for (int i = 0; i < warp_sums_left<NA>(); ++i)
      if (i < count) red_s[warp][first + i] = (double)acc[i];
  }
  __syncthreads();
  const int nb = gridDim.x;
  for (int q = tid; q < NPAIRS; q += kLsThreads) {
    const int h = (q < RowSplit<KR, 0, RS>::n) ? 0 : 1;
    const int qq = h ? q - RowSplit<KR, 0, RS>::n : q;
    double s = 0.0;
    for (int w = h; w < NW; w += NSPLIT) s += red_s[w][qq];
    part[(size_t)blockIdx.x * NPAIRS + q] = s;
  }
  // last CTA: sum the partials and solve.  The CTA barrier orders every
  // thread's partial writes before thread 0's device-scope fence and ticket
  // (the fence is cumulative), so the other threads do not wait for their
  // own outstanding stores of y here.
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    last_s = (atomicAdd(counter + e, 1u) == (unsigned)nb - 1u);
  }
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  // thread (sub, q) adds every tpq-th CTA's partial of pair q, its loads
  // coalesced and unrolled (one pass of L2 latency, not one per partial), then
  // the shares of a pair follow in a fixed order
  {
    constexpr int tpq = kLsThreads / NPAIRS;
    const int sub = tid / NPAIRS, q = tid - sub * NPAIRS;
    double v = 0.0;
    if (sub < tpq) {
      const double* src = part + q;
#pragma unroll 11
      for (int b = sub; b < nb; b += tpq) v += __ldcg(src + (size_t)b * NPAIRS);
    }
    share_s[tid] = v;
    __syncthreads();
    if (tid < NPAIRS) {
      double t = 0.0;
      for (int k = 0; k < tpq; ++k) t += share_s[k * NPAIRS + tid];
      sums_s[tid] = t;
    }
  }
  __syncthreads();
  if (sums_out) {
    // sharded regression: this GPU's unscaled sums, packed over the slots
    // 0..K (slot K = the target) as (i, j), j <= i, at i (i + 1) / 2 + j
    const int npub = (K + 1) * (K + 2) / 2;
    for (int idx = tid; idx < npub; idx += kLsThreads) {
      int i = 0;
      while ((i + 1) * (i + 2) / 2 <= idx) ++i;
      const int j = idx - i * (i + 1) / 2;
      const int ii = (i == K) ? KR - 1 : i, jj = (j == K) ? KR - 1 : j;
      sums_out[idx] = sums_s[ii * (ii + 1) / 2 + jj];
    }
    if (tid == 0) counter[e] = 0u;
    return;
  }
  const double n_div = MASKED ? (double)*P.mask_count : (double)paths;
  for (int q = tid; q < NPAIRS; q += kLsThreads) sums_s[q] /= n_div;
  __syncthreads();
  // G_s[i][j] (i, j < K) and the right-hand side in column kLsMaxSlots - 1
  for (int idx = tid; idx < kLsMaxSlots * kLsMaxSlots; idx += kLsThreads) {
    const int i = idx / kLsMaxSlots, j = idx - i * kLsMaxSlots;
    double v = 0.0;
    if (i < K && j < K) {
      const int a = i > j ? i : j, b = i > j ? j : i;
      v = sums_s[a * (a + 1) / 2 + b];
    } else if (i < K && j == kLsMaxSlots - 1) {
      v = sums_s[(KR - 1) * KR / 2 + i];
    }
    G_s[idx] = v;
  }
  __syncthreads();
  if (gram_out) {
    double* g = gram_out + (size_t)e * kMaxBasis * (kMaxBasis + 1);
    for (int idx = tid; idx < K * (kMaxBasis + 1); idx += kLsThreads) {
      const int i = idx / (kMaxBasis + 1), j = idx - i * (kMaxBasis + 1);
      double v = 0.0;
      if (j < K)
        v = G_s[i * kLsMaxSlots + j];
      else if (j == K)
        v = G_s[i * kLsMaxSlots + kLsMaxSlots - 1];
      g[idx] = v;
    }
  }
  if (warp == 0) {
    const int st = warp_cholesky_solve(G_s, K, beta + row * kMaxBasis, share_s);
    if (lane == 0) {
      if (st) atomicOr(status, st);
      counter[e] = 0u;
    }
  }
}

// ---------------------------------------------------------------------------
// The whole backward loop (depth 1) as one cooperative launch.
//
// Per date the work is that of ls_date_kernel; what the separate launches
// cost on top is the gap between two launches, the cold start of the input
// pipeline, and the serial tail (CTA partials, their sum, the solve) during
// which nothing else runs.  Here every CTA keeps its paths for all dates: it
// issues the next date's first input copies before it waits for the other
// CTAs, every CTA sums the partials and solves for itself (the same
// arithmetic in the same order, so all hold the same coefficients, with no
// second exchange).
// The dates with few functions (the last ones, with fewer variables) run as
// ls_date_kernel's instantiation for them does, with the same order of the
// partials: their Grams are close to singular, and their coefficients would
// show another order of the sums.  The coefficients are those of one launch
// per date to the last bit.
//
// For tables of at most 11 slots, whose rows one warp holds.  80 dates, 10
// functions: 2.85 -> 2.19 ms at 2^20 paths, 1.97 -> 1.33 at 2^18; 40 dates, 6
// functions: 0.70 -> 0.41 ms at 2^16, 0.62 -> 0.39 at 4,099.  VEC16: rows
// copied in 16-byte chunks (aligned rows, a path count that is a multiple of
// four), else value by value, from row pointers in shared memory: found anew
// for every copy they cost 3.92 ms at 1,000,001 paths against 3.20 with one
// launch per date, so 2.55; both copies in one kernel made aligned
// regressions with generic tables 15% slower.  Larger tables
// keep one launch per date: with their rows split over warp pairs the loop
// gained less (120 dates, 12 functions, 2.65 against 3.0 ms at 150,001 paths),
// and there the compiler contracts other products into the sums than in
// ls_date_kernel, which the third powers' Grams turn into 1e-3 of a
// coefficient.
// ---------------------------------------------------------------------------
struct LSRun {
  int n_ex, paths;
  unsigned char known[kMaxSteps];  // the date's table is the launch's KIND
  LSDate date[kMaxSteps];
};

constexpr int kLsWait = 32;  // status: a wait of the grid ran out

template <int KR, int KIND, bool VEC16>
__global__ void __launch_bounds__(LsThreads<KR>::value, 1)
    ls_run_kernel(const __grid_constant__ LSRun R, const float* __restrict__ vars,
                  const float* __restrict__ means, const float* __restrict__ sds,
                  const float* __restrict__ cf, const float* __restrict__ ex,
                  const float* __restrict__ num, double* __restrict__ beta, float* y,
                  double* part0, double* part1, unsigned int* counter,
                  double* __restrict__ gram_out, int* __restrict__ status) {
  constexpr int NPAIRS = KR * (KR + 1) / 2;  // row of a CTA's partials
  constexpr int T = LsThreads<KR>::value;
  constexpr int NW = T / 32;
  __shared__ double beta_s[kMaxBasis];           // coefficients of the date solved last
  __shared__ float mom_s[kMaxSteps][2][kMaxVars];  // mean and 1 / sd per date
  __shared__ double red_s[NW][NPAIRS];
  __shared__ double share_s[T];
  __shared__ double sums_s[NPAIRS];
  __shared__ double G_s[kLsMaxSlots * kLsMaxSlots];
  __shared__ int ok_s;
  extern __shared__ float ls_stage[];  // [kLsStages][kLsInputs][T]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int paths = R.paths, E = R.n_ex;
  if (means)
    for (int i = tid; i < E * kMaxVars; i += T) {
      mom_s[i / kMaxVars][0][i % kMaxVars] = means[i];
      mom_s[i / kMaxVars][1][i % kMaxVars] = 1.0f / sds[i];
    }
  const int r0 = lane >> 3, c4 = (lane & 7) * 4;
  float* const wstage = ls_stage + warp * 32;
  const int w0 = blockIdx.x * T + warp * 32, stride = gridDim.x * T;
  // input rows of the date in src_s[date & 1] (null: not read), those of the
  // next date written while the loop still reads this one's
  __shared__ const float* src_s[2][kLsInputs];
  auto row_ptr = [&](int e, int i) -> const float* {
    const size_t cur = (size_t)e * paths, nxt = cur + paths;
    if (i < kInCf)
      return i < R.date[e].nvars ? vars + ((size_t)e * kMaxVars + i) * paths : nullptr;
    if (i == kInCf) return cf ? cf + cur : nullptr;
    if (e + 1 >= E) return nullptr;
    if (i == kInY) return y;
    if (i < kInCfNext) {
      const int v = i - kInXNext;
      return v < R.date[e + 1].nvars ? vars + ((size_t)(e + 1) * kMaxVars + v) * paths : nullptr;
    }
    if (i == kInCfNext) return cf ? cf + nxt : nullptr;
    if (i == kInExNext) return ex ? ex + nxt : nullptr;
    return i == kInNum ? num + cur : num + nxt;
  };
  const float *rp0 = nullptr, *rp1 = nullptr, *rp2 = nullptr;
  // copies the inputs of the warp's paths qw .. qw + 31 into stage it
  // (16-byte chunks of rows r0, r0 + 4, r0 + 8 per lane when every row is
  // aligned, else each lane its own path's values)
  auto issue = [&](int e, int it, int qw) {
    float* dst = wstage + (it & (kLsStages - 1)) * kLsInputs * T;
    if (VEC16) {
      const int qb = qw + c4;
      if (qb < paths) {
        if (rp0) cp_async16(dst + r0 * T + c4, rp0 + qb);
        if (rp1) cp_async16(dst + (r0 + 4) * T + c4, rp1 + qb);
        if (rp2) cp_async16(dst + (r0 + 8) * T + c4, rp2 + qb);
      }
    } else if (qw + lane < paths) {
#pragma unroll
      for (int i = 0; i < kLsInputs; ++i)
        if (src_s[e & 1][i]) cp_async4(dst + i * T + lane, src_s[e & 1][i] + qw + lane);
    }
    cp_async_commit();
  };
  auto start_date = [&](int e) {
    rp0 = src_s[e & 1][r0];
    rp1 = src_s[e & 1][r0 + 4];
    rp2 = src_s[e & 1][r0 + 8];
#pragma unroll
    for (int k = 0; k < kLsStages - 1; ++k) issue(e, k, w0 + k * stride);
  };
  // date e with KRD slots: false when a wait ran out
  auto run_date = [&](auto kr_tag, auto kind_tag, const int e) -> bool {
    constexpr int KRD = decltype(kr_tag)::value, KD = decltype(kind_tag)::value;
    constexpr int NP = KRD * (KRD + 1) / 2;
    const LSDate& cur = R.date[e];
    const LSDate& prev = R.date[e + 1 < E ? e + 1 : e];
    const bool has_prev = e + 1 < E;
    const bool prev_known = has_prev && R.known[e + 1];
    const int K = cur.nbasis, nb = gridDim.x;
    float acc[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) acc[q] = 0.0f;
    int it = 0;
    for (int qw = w0; qw < paths; qw += stride, ++it) {
      issue(e, it + kLsStages - 1, qw + (kLsStages - 1) * stride);
      cp_async_wait<kLsStages - 1>();
      __syncwarp();
      const int p = qw + lane;
      if (p < paths) {
        const float* in = wstage + (it & (kLsStages - 1)) * kLsInputs * T + lane;
        float yp = 0.0f;
        if (has_prev) {
          float xp[kMaxVars];
#pragma unroll
          for (int v = 0; v < kMaxVars; ++v)
            xp[v] = v < prev.nvars ? in[(kInXNext + v) * T] : 0.0f;
          const float* mean_p = means ? mom_s[e + 1][0] : nullptr;
          const float cfn = cf ? in[kInCfNext * T] : 0.0f, exn = ex ? in[kInExNext * T] : 0.0f;
          if (KIND != kBasisGeneric && prev_known)
            yp = decide_values<KIND>(prev, 1, xp, mean_p, mom_s[e + 1][1], cfn, exn,
                                     in[kInNum * T], in[kInNumNext * T], beta_s, in[kInY * T]);
          else
            yp = decide_values<kBasisGeneric>(prev, 1, xp, mean_p, mom_s[e + 1][1], cfn, exn,
                                              in[kInNum * T], in[kInNumNext * T], beta_s,
                                              in[kInY * T]);
        }
        y[p] = yp;
        float x[kMaxVars];
#pragma unroll
        for (int v = 0; v < kMaxVars; ++v) {
          float xv = 0.0f;
          if (v < cur.nvars) {
            xv = in[(kInX + v) * T];
            if (means) xv = (xv - mom_s[e][0][v]) * mom_s[e][1][v];
          }
          x[v] = xv;
        }
        float pw[kMaxVars][3];
        ls_powers(x, pw);
        float phi[KRD];
#pragma unroll
        for (int k = 0; k < KRD - 1; ++k)
          phi[k] = (k < (KD ? basis_K(KD) : K)) ? ls_basis<KD>(pw, cur, k) : 0.0f;
        phi[KRD - 1] = (cf ? in[kInCf * T] : 0.0f) + yp;
        accumulate_rows<KRD, 0, KRD>(phi, acc);
      }
      // every lane's reads of this stage precede its refill, issued by
      // other lanes in a later iteration
      __syncwarp();
    }
    cp_async_wait<0>();
    int first, count;
    warp_sums<NP>(acc, first, count);
#pragma unroll
    for (int i = 0; i < warp_sums_left<NP>(); ++i)
      if (i < count) red_s[warp][first + i] = (double)acc[i];
    if (e > 0 && tid < kLsInputs) src_s[(e - 1) & 1][tid] = row_ptr(e - 1, tid);
    __syncthreads();
    double* part = ((E - 1 - e) & 1) ? part1 : part0;
    for (int q = tid; q < NP; q += T) {
      double s = 0.0;
      for (int w = 0; w < NW; ++w) s += red_s[w][q];
      part[(size_t)blockIdx.x * NPAIRS + q] = s;
    }
    // the next date's first inputs (all warps' stores of y precede the
    // barrier above) while the other CTAs finish
    if (e > 0) start_date(e - 1);
    __syncthreads();
    if (tid == 0) {
      const unsigned want = (unsigned)(E - e) * gridDim.x;
      ok_s = grid_arrive_wait(counter, want);
    }
    __syncthreads();
    if (!ok_s) return false;  // never while every CTA is resident
    // thread (sub, q) adds every tpq-th CTA's partial of pair q; the shares of
    // a pair follow in a fixed order
    {
      constexpr int tpq = T / NP;
      const int sub = tid / NP, q = tid - sub * NP;
      double v = 0.0;
      if (sub < tpq) {
        const double* src = part + q;
#pragma unroll 11
        for (int b = sub; b < nb; b += tpq) v += __ldcg(src + (size_t)b * NPAIRS);
      }
      share_s[tid] = v;
      __syncthreads();
      if (tid < NP) {
        double t = 0.0;
        for (int k = 0; k < tpq; ++k) t += share_s[k * NP + tid];
        sums_s[tid] = t / (double)paths;
      }
      __syncthreads();
    }
    // G_s[i][j] (i, j < K) and the right-hand side in column kLsMaxSlots - 1
    for (int idx = tid; idx < kLsMaxSlots * kLsMaxSlots; idx += T) {
      const int i = idx / kLsMaxSlots, j = idx - i * kLsMaxSlots;
      double v = 0.0;
      if (i < K && j < K) {
        const int a = i > j ? i : j, b = i > j ? j : i;
        v = sums_s[a * (a + 1) / 2 + b];
      } else if (i < K && j == kLsMaxSlots - 1) {
        v = sums_s[(KRD - 1) * KRD / 2 + i];
      }
      G_s[idx] = v;
    }
    __syncthreads();
    if (warp == 0) {
      const int st = warp_cholesky_solve<basis_K(KD)>(G_s, K, beta_s, share_s);
      if (lane == 0 && st && blockIdx.x == 0) atomicOr(status, st);
    }
    __syncthreads();
    if (blockIdx.x == 0) {
      if (tid < kMaxBasis) beta[(size_t)e * kMaxBasis + tid] = beta_s[tid];
      if (gram_out) {
        double* g = gram_out + (size_t)e * kMaxBasis * (kMaxBasis + 1);
        for (int idx = tid; idx < K * (kMaxBasis + 1); idx += T) {
          const int i = idx / (kMaxBasis + 1), j = idx - i * (kMaxBasis + 1);
          double v = 0.0;
          if (j < K)
            v = G_s[i * kLsMaxSlots + j];
          else if (j == K)
            v = G_s[i * kLsMaxSlots + kLsMaxSlots - 1];
          g[idx] = v;
        }
        __syncthreads();  // before the next date's G_s
      }
    }
    return true;
  };
  if (tid < kLsInputs) src_s[(E - 1) & 1][tid] = row_ptr(E - 1, tid);
  __syncthreads();
  start_date(E - 1);
  for (int e = E - 1; e >= 0; --e) {
    bool ok;
    // the compile-time table where the date and the next (whose decision it
    // applies) both have it, as launch_date chooses
    if (KIND != kBasisGeneric && R.known[e] && (e + 1 == E || R.known[e + 1]))
      ok = run_date(std::integral_constant<int, KR>(), std::integral_constant<int, KIND>(), e);
    else if (KR > 7 && R.date[e].nbasis < 7)
      ok = run_date(std::integral_constant<int, 7>(),
                    std::integral_constant<int, kBasisGeneric>(), e);
    else
      ok = run_date(std::integral_constant<int, KR>(),
                    std::integral_constant<int, kBasisGeneric>(), e);
    if (!ok) {
      if (tid == 0) atomicOr(status, kLsWait);
      cp_async_wait<0>();
      return;
    }
  }
}

// Final decision at date 0 (no deflation): y holds the value at date 0.
__global__ void ls_final_kernel(const __grid_constant__ LSDateParams P,
                                const float* __restrict__ vars,
                                const float* __restrict__ means,
                                const float* __restrict__ sds,
                                const float* __restrict__ cf,
                                const float* __restrict__ ex,
                                const float* __restrict__ num,
                                const double* __restrict__ beta,
                                float* __restrict__ y) {
  __shared__ double beta0[kMaxBasis];
  __shared__ float mom0[2][kMaxVars];
  if (threadIdx.x < kMaxBasis) beta0[threadIdx.x] = beta[threadIdx.x];
  if (threadIdx.x < kMaxVars && means) {
    mom0[0][threadIdx.x] = means[threadIdx.x];
    mom0[1][threadIdx.x] = 1.0f / sds[threadIdx.x];
  }
  __syncthreads();
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P.paths;
       p += gridDim.x * blockDim.x)
    y[p] = apply_decision<kBasisGeneric>(P.prev, 0, 0, vars, means ? mom0[0] : nullptr,
                          mom0[1], cf, ex, num, beta0, y[p], P.paths, p);
}

// Per-date moments of the basis variables (population mean and sd).
__global__ void __launch_bounds__(256)
    ls_moments_kernel(const float* __restrict__ vars, int paths,
                      double* __restrict__ part) {
  __shared__ double sh[6][8];
  const int e = blockIdx.y;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < paths;
       p += gridDim.x * blockDim.x) {
#pragma unroll
    for (int v = 0; v < kMaxVars; ++v) {
      const double x = vars[((size_t)e * kMaxVars + v) * paths + p];
      acc[2 * v] += x;
      acc[2 * v + 1] += x * x;
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double x = warp_sum_d(acc[i]);
    if (lane == 0) sh[i][w] = x;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double s = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += sh[threadIdx.x][i];
    part[((size_t)e * gridDim.x + blockIdx.x) * 6 + threadIdx.x] = s;
  }
}

__global__ void ls_moments_final_kernel(const double* __restrict__ part,
                                        int nblocks, int n_ex, int paths,
                                        float* __restrict__ means,
                                        float* __restrict__ sds, int rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // e*3 + v
  if (i >= n_ex * kMaxVars) return;
  const int e = i / kMaxVars, v = i % kMaxVars;
  double s = 0.0, s2 = 0.0;
#pragma unroll 8
  for (int b = 0; b < nblocks; ++b) {
    s += part[((size_t)e * nblocks + b) * 6 + 2 * v];
    s2 += part[((size_t)e * nblocks + b) * 6 + 2 * v + 1];
  }
  const double m = s / paths;
  double var = s2 / paths - m * m;
  double sd = var > 0.0 ? sqrt(var) : 0.0;
  if (!(sd > 0.0)) sd = 1.0;
  // depth-0 row of date e when each date holds `rows` rows
  const size_t o = ((size_t)e * rows) * kMaxVars + v;
  means[o] = (float)m;
  sds[o] = (float)sd;
}

namespace lmm {

int ls_fill_date(const LSBasisSpec& spec, int e, LSDate* d) {
  d->nvars = spec.nvars[e];
  d->nbasis = spec.nbasis[e];
  LMM_REQUIRE(d->nvars >= 0 && d->nvars <= kMaxVars,
              "LS: nvars out of range at date %d", e);
  LMM_REQUIRE(d->nbasis >= 1 && d->nbasis <= kMaxBasis,
              "LS: nbasis out of range at date %d", e);
  for (int k = 0; k < d->nbasis; ++k)
    for (int v = 0; v < kMaxVars; ++v) {
      const int x = spec.mono[(e * kMaxBasis + k) * kMaxVars + v];
      LMM_REQUIRE(x >= 0 && x <= 3, "LS: exponent out of range");
      LMM_REQUIRE(x == 0 || v < d->nvars,
                  "LS: monomial uses an absent variable at date %d", e);
      d->mono[k][v] = (unsigned char)x;
    }
  return LMM_OK;
}

// One CTA per SM for the date kernels and the moments.
int ls_gram_blocks() { return sm_count(); }

// CTAs per date of the moments: four paths per thread or more.
static int moment_blocks(int paths) {
  return std::min(ls_gram_blocks(), div_up(paths, 1024));
}

// Moments of every date's basis variables over all paths into row e * rows
// of means / sds; part: n_ex * ls_gram_blocks() * 6 doubles.
int ls_moments_launch(const float* vars, int paths, int n_ex, int rows, float* means,
                      float* sds, double* part, cudaStream_t s) {
  const int nblk = moment_blocks(paths);
  ls_moments_kernel<<<dim3(nblk, n_ex), 256, 0, s>>>(vars, paths, part);
  int st = check_launch("ls_moments");
  if (st) return st;
  ls_moments_final_kernel<<<div_up(n_ex * kMaxVars, 128), 128, 0, s>>>(part, nblk, n_ex,
                                                                       paths, means, sds, rows);
  return check_launch("ls_moments_final");
}

size_t ls_workspace_bytes(int paths, int n_ex) {
  const size_t y = ((size_t)paths * sizeof(float) + 255) & ~(size_t)255;
  const size_t part = (size_t)ls_gram_blocks() * kLsMaxPairs * sizeof(double);
  const size_t cnt = ((size_t)n_ex * sizeof(unsigned int) + 255) & ~(size_t)255;
  const size_t mom = (size_t)n_ex * ls_gram_blocks() * 6 * sizeof(double);
  const size_t red = 512 * sizeof(double);
  return y + part + cnt + mom + red + 256;
}

// allow_smem once per kernel and device: a date launch always asks for the
// same, and the sharded protocol's host work shows every driver call (1.2 us
// of 32 us a date).
template <class Kern>
int ls_stage_attr(Kern kern, size_t bytes) {
  static std::mutex mu;
  static std::vector<std::pair<const void*, int>> done;
  int dev = 0;
  int st = check_cuda(cudaGetDevice(&dev), "ls_date_kernel: cudaGetDevice");
  if (st) return st;
  std::lock_guard<std::mutex> lock(mu);
  for (const auto& d : done)
    if (d.first == (const void*)kern && d.second == dev) return LMM_OK;
  st = allow_smem((const void*)kern, bytes, "ls_date_kernel: shared memory attribute");
  if (st) return st;
  done.emplace_back((const void*)kern, dev);
  return LMM_OK;
}

// Launch the date kernel instantiated for the smallest slot count KR >=
// nbasis + 1 (rows split over warp pairs above 11 slots).
int launch_date(const LSDateParams& P_in, int grid, const float* vars,
                const float* means, const float* sds, const float* cf,
                const float* ex, const float* num, double* beta, float* y,
                double* part, unsigned int* counter, double* gram,
                int* status, double* sums_out, cudaStream_t s) {
  // 16-byte staged copies need every input row 16-byte aligned: aligned
  // bases and a path count that is a multiple of 4
  auto al16 = [](const void* q) { return ((uintptr_t)q & 15u) == 0; };
  LSDateParams P = P_in;
  P.vec16 = (P.paths % 4 == 0) && al16(vars) && al16(cf) && al16(ex) && al16(num) && al16(y);
  const int slots = P.cur.nbasis + 1;
  // straight-line basis code when this date and the next (whose decision
  // the kernel applies) share a known table
  const int kind = ls_basis_kind(P.cur);
  const bool known = kind != kBasisGeneric && (!P.has_prev || ls_basis_kind(P.prev) == kind);
#define LMM_LS_DATE(KR, NS, KIND)                                                    \
  do {                                                                               \
    constexpr size_t sb = ls_stage_bytes<KR, NS, false>();                           \
    const int at = ls_stage_attr(ls_date_kernel<KR, NS, KIND, false>, sb);           \
    if (at) return at;                                                               \
    ls_date_kernel<KR, NS, KIND, false><<<grid, LsThreads<KR>::value, sb, s>>>(      \
        P, vars, means, sds, cf, ex, num, beta, y, part, counter, gram, status, sums_out); \
  } while (0)
#define LMM_LS_DATE_MASKED(KR, NS, KIND)                                             \
  do {                                                                               \
    constexpr size_t sb = ls_stage_bytes<KR, NS, true>();                            \
    const int at = ls_stage_attr(ls_date_kernel<KR, NS, KIND, true>, sb);            \
    if (at) return at;                                                               \
    ls_date_kernel<KR, NS, KIND, true><<<grid, LsThreads<KR>::value, sb, s>>>(       \
        P, vars, means, sds, cf, ex, num, beta, y, part, counter, gram, status, sums_out); \
  } while (0)
  if (P.mask_net) {
    if (kind == kBasisC2)
      LMM_LS_DATE_MASKED(7, 1, kBasisC2);
    else if (kind == kBasisQuad)
      LMM_LS_DATE_MASKED(11, 1, kBasisQuad);
    else if (kind == kBasisCross)
      LMM_LS_DATE_MASKED(11, 1, kBasisCross);
    else if (kind == kBasisC5)
      LMM_LS_DATE_MASKED(13, 2, kBasisC5);
    else if (slots <= 7)
      LMM_LS_DATE_MASKED(7, 1, kBasisGeneric);
    else if (slots <= 11)
      LMM_LS_DATE_MASKED(11, 1, kBasisGeneric);
    else if (slots <= 13)
      LMM_LS_DATE_MASKED(13, 2, kBasisGeneric);
    else
      LMM_LS_DATE_MASKED(17, 2, kBasisGeneric);
    return check_launch("ls_date_kernel (masked)");
  }
  if (known && kind == kBasisC2)
    LMM_LS_DATE(7, 1, kBasisC2);
  else if (known && kind == kBasisQuad)
    LMM_LS_DATE(11, 1, kBasisQuad);
  else if (known && kind == kBasisCross)
    LMM_LS_DATE(11, 1, kBasisCross);
  else if (known && kind == kBasisC5)
    LMM_LS_DATE(13, 2, kBasisC5);
  else if (slots <= 7)
    LMM_LS_DATE(7, 1, kBasisGeneric);
  else if (slots <= 11)
    LMM_LS_DATE(11, 1, kBasisGeneric);
  else if (slots <= 13)
    LMM_LS_DATE(13, 2, kBasisGeneric);
  else
    LMM_LS_DATE(17, 2, kBasisGeneric);
#undef LMM_LS_DATE
#undef LMM_LS_DATE_MASKED
  return check_launch("ls_date_kernel");
}

// The whole backward loop (ls_run_kernel), instantiated for the most slots
// of any date and for the table that most dates share; -1 (nothing launched)
// for tables of more than 11 slots, and on a stream that owns too few SMs to
// hold all CTAs at once (a green context's): the loop of one launch per date
// waits for nobody and gives the same bits.  `part` holds nblk x kLsMaxPairs doubles,
// room for two buffers of 66.
int launch_run(LSRun& R, int nblk, const float* vars, const float* means, const float* sds,
               const float* cf, const float* ex, const float* num, double* beta, float* y,
               double* part, unsigned int* counter, double* gram, int* status,
               cudaStream_t s) {
  auto al16 = [](const void* q) { return ((uintptr_t)q & 15u) == 0; };
  const bool vec16 = (R.paths % 4 == 0) && al16(vars) && al16(cf) && al16(ex) && al16(num) && al16(y);
  int slots = 0, votes[5] = {0, 0, 0, 0, 0}, kind = kBasisGeneric;
  for (int e = 0; e < R.n_ex; ++e) {
    slots = std::max(slots, R.date[e].nbasis + 1);
    ++votes[ls_basis_kind(R.date[e])];
  }
  if (slots > 11) return -1;
  for (int k : {kBasisC2, kBasisQuad, kBasisCross})
    if (votes[k] && (kind == kBasisGeneric || votes[k] > votes[kind])) kind = k;
  if (kind == kBasisC2 && slots > 7) kind = kBasisGeneric;
  for (int e = 0; e < R.n_ex; ++e)
    R.known[e] = kind != kBasisGeneric && ls_basis_kind(R.date[e]) == kind;
  auto go = [&](auto kern, int pairs, size_t stage, int threads) -> int {
    double* part1 = part + (size_t)nblk * pairs;
    const int grid = std::min(div_up(R.paths, threads), nblk);
    if (grid > stream_sm_count(s)) return -1;
    int st = ls_stage_attr(kern, stage);
    if (st) return st;
    void* args[] = {&R, &vars, &means, &sds, &cf, &ex, &num, &beta, &y, &part, &part1,
                    &counter, &gram, &status};
    st = check_cuda(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(threads),
                                                args, stage, s),
                    "ls_run_kernel");
    return st ? st : check_launch("ls_run_kernel");
  };
#define LMM_LS_RUN(KR, KIND)                                                            \
  (vec16 ? go(ls_run_kernel<KR, KIND, true>, KR*(KR + 1) / 2,                           \
              ls_stage_bytes<KR, 1, false>(), LsThreads<KR>::value)                     \
         : go(ls_run_kernel<KR, KIND, false>, KR*(KR + 1) / 2,                          \
              ls_stage_bytes<KR, 1, false>(), LsThreads<KR>::value))
  switch (kind) {
    case kBasisC2: return LMM_LS_RUN(7, kBasisC2);
    case kBasisQuad: return LMM_LS_RUN(11, kBasisQuad);
    case kBasisCross: return LMM_LS_RUN(11, kBasisCross);
    default: break;
  }
  return slots <= 7 ? LMM_LS_RUN(7, kBasisGeneric) : LMM_LS_RUN(11, kBasisGeneric);
#undef LMM_LS_RUN
}

}  // namespace lmm

extern "C" size_t lmm_ls_workspace_bytes(int paths, int n_exercise) {
  return lmm::ls_workspace_bytes(paths, n_exercise);
}

extern "C" int lmm_ls_regress(int n_exercise, int paths, const float* d_vars,
                              const int* h_nvars, const uint8_t* h_monomials,
                              const int* h_nbasis, const float* d_cf,
                              const float* d_ex, const float* d_num,
                              int normalise, void* d_workspace,
                              size_t workspace_bytes, double* d_beta,
                              float* d_means, float* d_sds, double* d_gram,
                              int* d_status, double* d_price,
                              lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1,
              "lmm_ls_regress: bad sizes");
  LMM_REQUIRE(d_vars && h_nvars && h_monomials && h_nbasis && d_num &&
                  d_workspace && d_beta && d_status && d_price,
              "lmm_ls_regress: null pointer");
  LMM_REQUIRE(!normalise || (d_means && d_sds),
              "lmm_ls_regress: normalise needs means/sds outputs");
  LMM_REQUIRE(workspace_bytes >= ls_workspace_bytes(paths, n_exercise),
              "lmm_ls_regress: workspace too small (%zu < %zu)",
              workspace_bytes, ls_workspace_bytes(paths, n_exercise));
  cudaStream_t s = (cudaStream_t)stream;
  LSBasisSpec spec{h_nvars, h_monomials, h_nbasis};
  char* ws = (char*)d_workspace;
  float* y = (float*)ws;
  ws += ((size_t)paths * sizeof(float) + 255) & ~(size_t)255;
  double* part = (double*)ws;
  ws += (size_t)ls_gram_blocks() * kLsMaxPairs * sizeof(double);
  unsigned int* counter = (unsigned int*)ws;
  ws += ((size_t)n_exercise * sizeof(unsigned int) + 255) & ~(size_t)255;
  double* mom = (double*)ws;
  ws += (size_t)n_exercise * ls_gram_blocks() * 6 * sizeof(double);
  double* red = (double*)ws;

  const float* means = nullptr;
  const float* sds = nullptr;
  const int nblk = ls_gram_blocks();
  if (normalise) {
    const int st = ls_moments_launch(d_vars, paths, n_exercise, 1, d_means, d_sds, mom, s);
    if (st) return st;
    means = d_means;
    sds = d_sds;
  }
  int st = check_cuda(cudaMemsetAsync(d_status, 0, sizeof(int), s),
                      "lmm_ls_regress: status reset");
  if (st) return st;
  st = check_cuda(cudaMemsetAsync(counter, 0, (size_t)n_exercise * sizeof(unsigned int), s),
                  "lmm_ls_regress: counter reset");
  if (st) return st;
  LSRun run;
  memset(&run, 0, sizeof(run));
  run.n_ex = n_exercise;
  run.paths = paths;
  for (int e = 0; e < n_exercise; ++e) {
    st = ls_fill_date(spec, e, &run.date[e]);
    if (st) return st;
  }
  st = launch_run(run, nblk, d_vars, means, sds, d_cf, d_ex, d_num, d_beta, y, part, counter,
                  d_gram, d_status, s);
  if (st > 0) return st;
  // otherwise one launch per date
  for (int e = n_exercise - 1; st < 0 && e >= 0; --e) {
    LSDateParams P;
    memset(&P, 0, sizeof(P));
    P.e = e;
    P.paths = paths;
    P.cur = run.date[e];
    P.has_prev = (e + 1 < n_exercise);
    if (P.has_prev) P.prev = run.date[e + 1];
    const int slots = P.cur.nbasis + 1;
    const int per_cta = slots <= 11 ? 512 : slots <= 13 ? 256 : 192;
    int grid = div_up(paths, per_cta);
    if (grid > nblk) grid = nblk;
    const int one = launch_date(P, grid, d_vars, means, sds, d_cf, d_ex, d_num, d_beta, y,
                                part, counter, d_gram, d_status, nullptr, s);
    if (one) return one;
  }
  LSDateParams P;
  memset(&P, 0, sizeof(P));
  P.paths = paths;
  st = ls_fill_date(spec, 0, &P.prev);
  if (st) return st;
  ls_final_kernel<<<grid_for(paths, 256, 4), 256, 0, s>>>(
      P, d_vars, means, sds, d_cf, d_ex, d_num, d_beta, y);
  st = check_launch("ls_final");
  if (st) return st;
  return reduce_launch(y, d_num, (size_t)paths, 1.0 / (double)paths, red,
                       d_price, s);
}

// ---------------------------------------------------------------------------
// Regression with library-owned scratch, for callers that cannot allocate
// device memory (their device memory is owned by an outside pool allocator,
// or allocation is forbidden in their pricing loop because it can
// synchronise the device).  The scratch is the file-scope array below,
// LMM_LS_STATIC_SCRATCH_BYTES bytes, which every GPU that loads this
// library holds until the process exits.  Host code must not pass the
// array's name to a kernel (in host code it is only a host-side stand-in),
// so the first call on each device looks up the device address with
// cudaGetSymbolAddress, with that device current, and caches it; make that
// first call before any stream capture.  All calls share the array and it
// keeps the last call's contents: every scratch region is written before it
// is read, so nothing needs clearing, but calls that overlap on the GPU
// (on different streams, or from different host threads) race on it.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char
    g_ls_static_scratch[LMM_LS_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_mu;
void* g_static_ptr[64] = {};

int static_scratch_address(void** out) {
  int dev = 0;
  int st = check_cuda(cudaGetDevice(&dev), "lmm_ls_regress_static: cudaGetDevice");
  if (st) return st;
  LMM_REQUIRE(dev >= 0 && dev < 64, "lmm_ls_regress_static: device ordinal %d", dev);
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    st = check_cuda(cudaGetSymbolAddress(&p, g_ls_static_scratch),
                    "lmm_ls_regress_static: cudaGetSymbolAddress");
    if (st) return st;
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return LMM_OK;
}
}  // namespace

extern "C" int lmm_ls_regress_static(int n_exercise, int paths,
                                     const float* d_vars, const int* h_nvars,
                                     const uint8_t* h_monomials,
                                     const int* h_nbasis, const float* d_cf,
                                     const float* d_ex, const float* d_num,
                                     int normalise, double* d_beta,
                                     float* d_means, float* d_sds,
                                     double* d_gram, int* d_status,
                                     double* d_price, lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1,
              "lmm_ls_regress_static: bad sizes");
  const size_t need = ls_workspace_bytes(paths, n_exercise);
  LMM_REQUIRE(need <= (size_t)LMM_LS_STATIC_SCRATCH_BYTES,
              "lmm_ls_regress_static: %d paths x %d dates need %zu bytes of "
              "scratch but the static scratch holds %zu bytes; use "
              "lmm_ls_regress with a caller workspace",
              paths, n_exercise, need, (size_t)LMM_LS_STATIC_SCRATCH_BYTES);
  void* ws = nullptr;
  int st = static_scratch_address(&ws);
  if (st) return st;
  return lmm_ls_regress(n_exercise, paths, d_vars, h_nvars, h_monomials,
                        h_nbasis, d_cf, d_ex, d_num, normalise, ws,
                        (size_t)LMM_LS_STATIC_SCRATCH_BYTES, d_beta, d_means,
                        d_sds, d_gram, d_status, d_price, stream);
}

// ---------------------------------------------------------------------------
// Regression over paths sharded across GPUs.  Each GPU runs the backward
// loop on its own paths; per exercise date the sums over paths (the Gram
// and X^T y, unscaled) are summed over the GPUs by the caller (an
// all-reduce), and every GPU solves the same system, so all apply one rule.
// The moments of the basis variables and the in-sample price are summed the
// same way.  The workspace (lmm_ls_workspace_bytes) carries the running
// path values from one date to the next and must be kept between calls.
// ---------------------------------------------------------------------------
__global__ void ls_solve_sums_kernel(int e, int K, const double* __restrict__ sums,
                                     double total, double* __restrict__ beta,
                                     double* __restrict__ gram_out,
                                     int* __restrict__ status) {
  __shared__ double G_s[kLsMaxSlots * kLsMaxSlots];
  __shared__ double L_s[kMaxBasis * kMaxBasis];
  const int tid = threadIdx.x;
  for (int idx = tid; idx < kLsMaxSlots * kLsMaxSlots; idx += blockDim.x) {
    const int i = idx / kLsMaxSlots, j = idx - i * kLsMaxSlots;
    double v = 0.0;
    if (i < K && j < K) {
      const int a = i > j ? i : j, b = i > j ? j : i;
      v = sums[a * (a + 1) / 2 + b] / total;
    } else if (i < K && j == kLsMaxSlots - 1) {
      v = sums[K * (K + 1) / 2 + i] / total;
    }
    G_s[idx] = v;
  }
  __syncthreads();
  if (gram_out) {
    double* g = gram_out + (size_t)e * kMaxBasis * (kMaxBasis + 1);
    for (int idx = tid; idx < K * (kMaxBasis + 1); idx += blockDim.x) {
      const int i = idx / (kMaxBasis + 1), j = idx - i * (kMaxBasis + 1);
      g[idx] = j < K ? G_s[i * kLsMaxSlots + j]
                     : (j == K ? G_s[i * kLsMaxSlots + kLsMaxSlots - 1] : 0.0);
    }
  }
  if (tid < 32) {
    const int st = warp_cholesky_solve(G_s, K, beta + (size_t)e * kMaxBasis, L_s);
    if (tid == 0 && st) atomicOr(status, st);
  }
}

// Unscaled sums of x and x^2 per date and variable from the block partials
// of ls_moments_kernel, in a fixed order: sums[e][2v] and sums[e][2v+1].
__global__ void ls_moment_sums_kernel(const double* __restrict__ part, int nblocks,
                                      int n_ex, double* __restrict__ sums) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // e*6 + c
  if (i >= n_ex * 6) return;
  const int e = i / 6, c = i - e * 6;
  double s = 0.0;
  for (int b = 0; b < nblocks; ++b) s += part[((size_t)e * nblocks + b) * 6 + c];
  sums[i] = s;
}

__global__ void ls_moments_from_sums_kernel(const double* __restrict__ sums, int n_ex,
                                            double total, float* __restrict__ means,
                                            float* __restrict__ sds) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // e*3 + v
  if (i >= n_ex * kMaxVars) return;
  const int e = i / kMaxVars, v = i % kMaxVars;
  const double m = sums[e * 6 + 2 * v] / total;
  const double var = sums[e * 6 + 2 * v + 1] / total - m * m;
  double sd = var > 0.0 ? sqrt(var) : 0.0;
  if (!(sd > 0.0)) sd = 1.0;
  means[i] = (float)m;
  sds[i] = (float)sd;
}

namespace {
struct LsWs {
  float* y;
  double* part;
  unsigned int* counter;
  double* mom;
  double* red;
};

LsWs carve_ls(void* d_workspace, int paths, int n_exercise) {
  char* ws = (char*)d_workspace;
  LsWs w;
  w.y = (float*)ws;
  ws += ((size_t)paths * sizeof(float) + 255) & ~(size_t)255;
  w.part = (double*)ws;
  ws += (size_t)ls_gram_blocks() * kLsMaxPairs * sizeof(double);
  w.counter = (unsigned int*)ws;
  ws += ((size_t)n_exercise * sizeof(unsigned int) + 255) & ~(size_t)255;
  w.mom = (double*)ws;
  ws += (size_t)n_exercise * ls_gram_blocks() * 6 * sizeof(double);
  w.red = (double*)ws;
  return w;
}
}  // namespace

extern "C" int lmm_ls_moment_sums(int n_exercise, int paths, const float* d_vars,
                                  void* d_workspace, size_t workspace_bytes,
                                  double* d_sums, lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1,
              "lmm_ls_moment_sums: bad sizes");
  LMM_REQUIRE(d_vars && d_workspace && d_sums, "lmm_ls_moment_sums: null pointer");
  LMM_REQUIRE(workspace_bytes >= ls_workspace_bytes(paths, n_exercise),
              "lmm_ls_moment_sums: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  LsWs w = carve_ls(d_workspace, paths, n_exercise);
  const int nblk = moment_blocks(paths);
  ls_moments_kernel<<<dim3(nblk, n_exercise), 256, 0, s>>>(d_vars, paths, w.mom);
  int st = check_launch("ls_moments");
  if (st) return st;
  ls_moment_sums_kernel<<<div_up(n_exercise * 6, 128), 128, 0, s>>>(w.mom, nblk, n_exercise,
                                                                    d_sums);
  return check_launch("ls_moment_sums");
}

extern "C" int lmm_ls_moments_from_sums(int n_exercise, double total_paths,
                                        const double* d_sums, float* d_means,
                                        float* d_sds, lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && total_paths >= 1.0,
              "lmm_ls_moments_from_sums: bad sizes");
  LMM_REQUIRE(d_sums && d_means && d_sds, "lmm_ls_moments_from_sums: null pointer");
  ls_moments_from_sums_kernel<<<div_up(n_exercise * kMaxVars, 128), 128, 0,
                                (cudaStream_t)stream>>>(d_sums, n_exercise, total_paths,
                                                        d_means, d_sds);
  return check_launch("ls_moments_from_sums");
}

extern "C" int lmm_ls_date_sums(int e, int n_exercise, int paths, const float* d_vars,
                                const int* h_nvars, const uint8_t* h_monomials,
                                const int* h_nbasis, const float* d_cf,
                                const float* d_ex, const float* d_num,
                                const float* d_means, const float* d_sds,
                                const double* d_beta, void* d_workspace,
                                size_t workspace_bytes, double* d_sums,
                                lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1 && e >= 0 &&
                  e < n_exercise,
              "lmm_ls_date_sums: bad sizes");
  LMM_REQUIRE(d_vars && h_nvars && h_monomials && h_nbasis && d_num && d_beta &&
                  d_workspace && d_sums,
              "lmm_ls_date_sums: null pointer");
  LMM_REQUIRE(!d_means == !d_sds, "lmm_ls_date_sums: means/sds mismatch");
  LMM_REQUIRE(workspace_bytes >= ls_workspace_bytes(paths, n_exercise),
              "lmm_ls_date_sums: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  LsWs w = carve_ls(d_workspace, paths, n_exercise);
  LSBasisSpec spec{h_nvars, h_monomials, h_nbasis};
  LSDateParams P;
  memset(&P, 0, sizeof(P));
  P.e = e;
  P.paths = paths;
  int st = ls_fill_date(spec, e, &P.cur);
  if (st) return st;
  P.has_prev = (e + 1 < n_exercise);
  if (P.has_prev) {
    st = ls_fill_date(spec, e + 1, &P.prev);
    if (st) return st;
  }
  st = check_cuda(cudaMemsetAsync(w.counter + e, 0, sizeof(unsigned int), s),
                  "lmm_ls_date_sums: counter reset");
  if (st) return st;
  const int slots = P.cur.nbasis + 1;
  const int per_cta = slots <= 11 ? 512 : slots <= 13 ? 256 : 192;
  int grid = div_up(paths, per_cta);
  if (grid > ls_gram_blocks()) grid = ls_gram_blocks();
  return launch_date(P, grid, d_vars, d_means, d_sds, d_cf, d_ex, d_num,
                     const_cast<double*>(d_beta), w.y, w.part, w.counter, nullptr,
                     nullptr, d_sums, s);
}

extern "C" int lmm_ls_date_solve(int e, int nbasis, const double* d_sums,
                                 double total_paths, double* d_beta, double* d_gram,
                                 int* d_status, lmm_stream_t stream) {
  LMM_REQUIRE(e >= 0 && e < kMaxSteps && nbasis >= 1 && nbasis <= kMaxBasis &&
                  total_paths >= 1.0,
              "lmm_ls_date_solve: bad sizes");
  LMM_REQUIRE(d_sums && d_beta && d_status, "lmm_ls_date_solve: null pointer");
  ls_solve_sums_kernel<<<1, 128, 0, (cudaStream_t)stream>>>(e, nbasis, d_sums, total_paths,
                                                            d_beta, d_gram, d_status);
  return check_launch("ls_solve_sums_kernel");
}

extern "C" int lmm_ls_final_sum(int n_exercise, int paths, const float* d_vars,
                                const int* h_nvars, const uint8_t* h_monomials,
                                const int* h_nbasis, const float* d_cf,
                                const float* d_ex, const float* d_num,
                                const float* d_means, const float* d_sds,
                                const double* d_beta, void* d_workspace,
                                size_t workspace_bytes, double* d_sum,
                                lmm_stream_t stream) {
  LMM_REQUIRE(n_exercise >= 1 && n_exercise <= kMaxSteps && paths >= 1,
              "lmm_ls_final_sum: bad sizes");
  LMM_REQUIRE(d_vars && h_nvars && h_monomials && h_nbasis && d_num && d_beta &&
                  d_workspace && d_sum,
              "lmm_ls_final_sum: null pointer");
  LMM_REQUIRE(workspace_bytes >= ls_workspace_bytes(paths, n_exercise),
              "lmm_ls_final_sum: workspace too small");
  cudaStream_t s = (cudaStream_t)stream;
  LsWs w = carve_ls(d_workspace, paths, n_exercise);
  LSBasisSpec spec{h_nvars, h_monomials, h_nbasis};
  LSDateParams P;
  memset(&P, 0, sizeof(P));
  P.paths = paths;
  int st = ls_fill_date(spec, 0, &P.prev);
  if (st) return st;
  ls_final_kernel<<<grid_for(paths, 256, 4), 256, 0, s>>>(P, d_vars, d_means, d_sds, d_cf,
                                                         d_ex, d_num, d_beta, w.y);
  st = check_launch("ls_final");
  if (st) return st;
  return reduce_launch(w.y, d_num, (size_t)paths, 1.0, w.red, d_sum, s);
}
