// ab_kernels.cuh — device code of the Andersen–Broadie upper bound
// (included by pipeline.cu).
//
// The reference computes the duality gap on the CPU only: its gold LMM
// example (gold/gold_example/LMM_bermudan_gold.cpp:1132-1382) runs, for every
// outer path and exercise date, a sub-simulation from the outer state
// (LMMEvolverPartial_gold::conditionallyGenerate) priced with the frozen
// exercise strategy, and ABDualityGapEstimate*Rebate
// (gold/Andersen_Broadie_gold.cpp:59-187) turns the continuation estimates
// into the gap.  Here the outer paths come from the fused kernel (outer mode:
// LS inputs at every date and the log-rates at the start of every step), the
// inner paths from ab_inner_kernel: 128 inner paths per (outer
// path, date, chunk), started from the outer state in shared memory, with
// counter-based normals generated in registers (no variates in HBM), and
// the frozen rule applied at the later dates.
#pragma once
#include "fused_pairs.cuh"

namespace lmm {

constexpr int kAbThreads = 128;  // inner paths per unit

// Philox4x32-10 (Salmon, Moraes, Dror and Shaw, SC 2011): ten rounds of two
// 32x32 -> 64-bit products with a Weyl-sequence key schedule.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    if (round) {
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
  }
  return c;
}

struct AbArgs {
  int K;        // outer paths
  int chunks;   // groups of 128 inner paths per (outer path, date)
  int e0;       // first exercise date of the launch
  uint32_t k0, k1;  // Philox key
  int ex_step[kMaxSteps];  // date -> step
};

// Inner paths of a unit = (date e, outer path p, chunk of 128 inner paths):
// from the state at the start of step s0 = ex_step[e] + 1 (ckpt [n][n][K],
// ckptN [n][K]), evolve to the end with the normals of inner path i (Philox
// counter (i, p, 4 s + j, e), words 4j..4j+3 = factors), stop at the first
// later date whose exercise value exceeds the rule's estimate.  A CTA of
// kPairThreads threads runs two units of one date, two paths per thread, as
// fused_pairs_kernel does (log-rates in shared and tensor memory, each
// step's rows copied a step ahead): lane l of warp w holds inner paths
// 64 (w & 1) + l and + 32 of unit 2 b + (w >> 1) of the date's K x chunks.
// Writes each unit's sum and sum of squares of the deflated payoffs to
// part[unit][2], joined over groups of 32 consecutive paths in a fixed order.
// Bermudan payer swaption.  Bound as fused_pairs_kernel, plus the normals
// (a fifth of the instructions): 96 outer paths, 79 dates, 256 inner paths of
// 80 rates and 10 factors 9.45 ms with one path per thread, 8.75 with two and
// the log-rates in shared memory alone, 6.87 so.
template <int FT>
__global__ void __launch_bounds__(kPairThreads, PairShape<FT>::kCtas)
    ab_inner_kernel(const __grid_constant__ AbArgs a, const float* __restrict__ A,
                    const float* __restrict__ fixed, const __grid_constant__ ModelConst mc,
                    const __grid_constant__ ProductConst pc,
                    const __grid_constant__ RuleConst rc, const LsRuleView rule,
                    const float* __restrict__ ckpt, const float* __restrict__ ckptN,
                    double* __restrict__ part, int nt0) {
  constexpr int FM = FPad<FT>::FM;
  constexpr int FP = FPad<FT>::FP;
  constexpr int T = kPairThreads;
  const int F = FT > 0 ? FT : mc.F;
  const int n = mc.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per_date = a.K * a.chunks, ctas = (per_date + 1) / 2;
  const int e = a.e0 + blockIdx.x / ctas;
  const int in_date = (blockIdx.x % ctas) * 2 + (warp >> 1);
  const bool valid = in_date < per_date;  // the same for a warp pair
  const int p = valid ? in_date / a.chunks : 0, chunk = valid ? in_date % a.chunks : 0;
  const int s0 = a.ex_step[e] + 1;
  extern __shared__ __align__(16) float sm[];
  float* const As = sm;               // [2][n][FP]: row r - s of step s
  float* const fx = As + 2 * n * FP;  // [2][n (+ pad)]
  const int fx_rows = (n + 3) & ~3;
  __shared__ double red_s[2][2 * T / 32];
  __shared__ uint32_t tmem_slot;
  LogRates<T> lr;
  lr.row = reinterpret_cast<float2*>(fx + 2 * fx_rows) + tid;  // [nt0][T]
  lr.s_begin = 0;
  lr.nt0 = nt0;
  lr.tmem = 0u;
  const uint32_t tmem_cols = tmem_columns(n - nt0);
  if (warp == 0) tmem_alloc(&tmem_slot, tmem_cols);
  if (tmem_cols) {
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    lr.tmem = tmem_slot + ((uint32_t)(warp * 32) << 16);
  }
  zero_row_pads<FP, T>(As, 2 * n, F);
  auto stage = [&](int s, int b) {
    stage_rows<FT, FP, T>(As + b * n * FP, fx + b * fx_rows, A, fixed, s, n, F);
  };
  stage(s0, 0);
  const uint32_t inner = (uint32_t)(chunk * kAbThreads + (warp & 1) * 64 + lane);
  auto start_rate = [&](int r) {
    return r >= s0 ? dup2(__ldg(ckpt + ((size_t)s0 * n + r) * a.K + p)) : dup2(0.0f);
  };
  for (int r = s0; r < nt0; ++r) lr.row[r * T] = start_rate(r);
  for (int r = nt0; r < n; r += 4) {
    float2 x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = start_rate(r + j);
    __syncwarp();
    tmem_st8(lr.tmem + 2 * (r - nt0), x);
  }
  const float N0 = __ldg(ckptN + (size_t)s0 * a.K + p);
  float N[2] = {N0, N0}, f_first[2] = {0.0f, 0.0f};
  double payoff[2] = {0.0, 0.0};
  bool done[2] = {!valid, !valid};
  for (int s = s0; s < n; ++s) {
    cp_async_wait<0>();
    __syncthreads();  // this step's rows are in; the other buffer is free
    const int buf = (s - s0) & 1;
    if (s + 1 < n) stage(s + 1, buf ^ 1);
    // whole warps only past here (tensor memory is read by whole warps)
    if (__all_sync(0xffffffffu, done[0] && done[1])) continue;
    float2 w[FM], v[FM];
#pragma unroll
    for (int j = 0; j < FP / 4; ++j) {
      if (4 * j < F) {
        const uint4 c0 = philox4x32_10(
            make_uint4(inner, (uint32_t)p, (uint32_t)(4 * s + j), (uint32_t)e), a.k0, a.k1);
        const uint4 c1 = philox4x32_10(
            make_uint4(inner + 32u, (uint32_t)p, (uint32_t)(4 * s + j), (uint32_t)e), a.k0,
            a.k1);
        // the pricing variates' inverse normal (hardware log and
        // reciprocal on the exact tail probability)
        const uint32_t u0[4] = {c0.x, c0.y, c0.z, c0.w}, u1[4] = {c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (4 * j + k < FM)
            w[4 * j + k] = 4 * j + k < F ? icdf_sb_fast2(u0[k], u1[k]) : dup2(0.0f);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (4 * j + k < FM) w[4 * j + k] = dup2(0.0f);
      }
    }
#pragma unroll
    for (int f = 0; f < FM; ++f) v[f] = dup2(0.0f);
    if (s > s0)
#pragma unroll
      for (int h = 0; h < 2; ++h) N[h] = N[h] * (1.0f + mc.tau[s - 1] * f_first[h]);
    const int ed = pc.ex_index[s];
    float2 Prun = dup2(1.0f), ann = dup2(0.0f);
    const float* As_s = As + buf * n * FP;
    const float* fx_s = fx + buf * fx_rows;
    auto curve = [&](int r, float2, float2, float2, float2 ln) {
      const float2 c = cap2(ln, mc.cutoff);
      const float2 fn = __fadd2_rn(make_float2(exp_ftz(c.x), exp_ftz(c.y)), dup2(-mc.disp[r]));
      const float2 t = __ffma2_rn(dup2(mc.tau[r]), fn, dup2(1.0f));
      Prun = __fmul2_rn(Prun, make_float2(rcp_ftz(t.x), rcp_ftz(t.y)));
      ann = __ffma2_rn(dup2(mc.tau[r]), Prun, ann);
    };
    const float2 lf0 =
        ed >= 0 ? pc_step2<FM, FP, T>(lr, s, n, mc, As_s, fx_s, w, v, curve)
                : pc_step2<FM, FP, T>(lr, s, n, mc, As_s, fx_s, w, v,
                                      [](int, float2, float2, float2, float2) {});
    f_first[0] = exp_ftz(lf0.x) - mc.disp[s];
    f_first[1] = exp_ftz(lf0.y) - mc.disp[s];
    if (ed > e) {
      const float Pn[2] = {Prun.x, Prun.y}, an[2] = {ann.x, ann.y};
      float vv[2][kMaxVars], exv[2];
      double est[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float sr = (1.0f - Pn[h]) / an[h];
        exv[h] = fmaxf((sr - pc.strike) * an[h], 0.0f);
        vv[h][0] = f_first[h];
        vv[h][1] = sr;
        vv[h][2] = an[h];
      }
      ls_chain_estimates<2>(rule, ed, rc.kind[ed], rc.nvars[ed], rc.nbasis[ed], rc.mono[ed], vv,
                         exv, est);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (!done[h] && (double)exv[h] > est[h]) {
          payoff[h] = (double)exv[h] / (double)N[h];
          done[h] = true;
        }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double s1 = payoff[h], s2 = payoff[h] * payoff[h];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s1 += __shfl_down_sync(0xffffffffu, s1, o);
      s2 += __shfl_down_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
      red_s[0][2 * warp + h] = s1;
      red_s[1][2 * warp + h] = s2;
    }
  }
  tmem_free(lr.tmem, tmem_cols);  // and red_s is complete
  if ((tid & 63) == 0 && valid) {
    double t1 = 0.0, t2 = 0.0;
    for (int w = 0; w < kAbThreads / 32; ++w) {
      t1 += red_s[0][2 * warp + w];
      t2 += red_s[1][2 * warp + w];
    }
    const size_t unit = (size_t)(e - a.e0) * per_date + in_date;
    part[unit * 2] = t1;
    part[unit * 2 + 1] = t2;
  }
}

// Continuation estimate Q[e][p] (mean over the inner paths, fixed order
// over the CTAs) and its standard error; the last date has none (0).
__global__ void ab_continuation_kernel(int E, int K, int chunks, int inner,
                                       const double* __restrict__ part,
                                       double* __restrict__ Q, double* __restrict__ Qse) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // e * K + p
  if (i >= E * K) return;
  const int e = i / K;
  double m = 0.0, se = 0.0;
  if (e + 1 < E) {
    double t1 = 0.0, t2 = 0.0;
    const double* src = part + (size_t)(e * K + i % K) * chunks * 2;
    for (int c = 0; c < chunks; ++c) {
      t1 += src[2 * c];
      t2 += src[2 * c + 1];
    }
    m = t1 / inner;
    se = sqrt(fmax(t2 / inner - m * m, 0.0) / inner);
  }
  Q[i] = m;
  if (Qse) Qse[i] = se;
}

// The frozen rule's decision at every date of the outer paths (exercise
// value above the estimate, exerciseAllDeterminerEESimple_gold) and the
// deflated exercise values, from their LS inputs.
__global__ void ab_decide_kernel(int E, int K, const __grid_constant__ RuleConst rc,
                                 const LsRuleView rule, const float* __restrict__ vars,
                                 const float* __restrict__ ex, const float* __restrict__ num,
                                 int* __restrict__ X, double* __restrict__ Z) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // e * K + p
  if (i >= E * K) return;
  const int e = i / K, p = i % K;
  float v[kMaxVars];
#pragma unroll
  for (int k = 0; k < kMaxVars; ++k) v[k] = vars[((size_t)e * kMaxVars + k) * K + p];
  const float exv = ex[i];
  const double est = rule_estimate(rc, e, v, exv, rule);
  X[i] = ((double)exv > est) ? 1 : 0;
  Z[i] = (double)exv / (double)num[i];
}

// Duality gap per path (ABDualityGapEstimateNonZeroRebate,
// gold/Andersen_Broadie_gold.cpp:121-187; payoffs null: the zero-rebate form
// of :59-119) and, when lower != null, the value of the frozen rule on the
// outer path (the first date with ex = 1).  ex / payoffs [steps][paths],
// means[p * m_p + s * m_s]; is_ex in the bit mask words is_ex[s / 32].
// Per-CTA FP64 partials: part[b][4] = sum, sum of squares of the gap; sum,
// sum of squares of the lower value.
struct AbGapArgs {
  int steps, paths;
  long long m_p, m_s;
  unsigned is_ex[(kMaxSteps + 32) / 32];
};

__global__ void __launch_bounds__(256)
    ab_gap_kernel(const __grid_constant__ AbGapArgs g, const int* __restrict__ ex,
                  const double* __restrict__ payoffs, const double* __restrict__ means,
                  double* __restrict__ part) {
  __shared__ double red_s[4][8];
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (p < g.paths) {
    double best = 0.0, balance = 0.0, lower = 0.0;
    bool exercised = false;
    const int last = payoffs ? g.steps - 1 : g.steps;
    for (int s = 0; s < last; ++s) {
      if (!((g.is_ex[s >> 5] >> (s & 31)) & 1u)) continue;
      const double z = payoffs ? payoffs[(size_t)s * g.paths + p] : 0.0;
      const double m = means[(size_t)p * g.m_p + (size_t)s * g.m_s];
      double x;
      if (ex[(size_t)s * g.paths + p] == 1) {
        x = -balance;
        balance += z - m;
        if (!exercised) lower = z;
        exercised = true;
      } else {
        x = z - m - balance;
      }
      best = fmax(best, x);
    }
    best = fmax(best, -balance);
    v[0] = best;
    v[1] = best * best;
    v[2] = lower;
    v[3] = lower * lower;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double t = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) red_s[k][w] = t;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red_s[threadIdx.x][i];
    part[(size_t)blockIdx.x * 4 + threadIdx.x] = t;
  }
}

// Means and standard errors from the partials of ab_gap_kernel (fixed
// order): out = {gap mean, gap se, lower mean, lower se}.
__global__ void ab_gap_final_kernel(int nblocks, int paths, const double* __restrict__ part,
                                    double* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = 0; b < nblocks; ++b)
    for (int k = 0; k < 4; ++k) t[k] += part[(size_t)b * 4 + k];
  for (int k = 0; k < 2; ++k) {
    const double m = t[2 * k] / paths;
    out[2 * k] = m;
    out[2 * k + 1] = sqrt(fmax(t[2 * k + 1] / paths - m * m, 0.0) / paths);
  }
}

}  // namespace lmm
