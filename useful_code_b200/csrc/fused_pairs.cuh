// fused_pairs.cuh — the fused evolution with two paths per thread (included
// by pipeline.cu): fused_evolve_kernel's passes for launches with enough
// paths to fill the GPU's SMs with pairs.
#pragma once
#include "fused_kernels.cuh"

namespace lmm {

constexpr int kPairThreads = 128;
constexpr int kPairBlock = 2 * kPairThreads;  // paths per CTA (slots in SegState)

// CTAs per SM that the registers allow, and their __launch_bounds__.
template <int FT>
struct PairShape {
  static constexpr int kCtas = FT > 0 && FT <= 5 ? 4 : 3;
};

// ---------------------------------------------------------------------------
// Fused evolution, two paths per thread (pc_rate2): CTA of 128 threads over
// a tile of kPairBlock = 256 paths; lane l of warp w holds the tile's paths
// 64 w + l and 64 w + 32 + l (coalesced loads and stores of either), as the
// two halves of packed FP32x2 values.  The same arithmetic per path as
// fused_evolve_kernel, so its outputs are bit-identical.
//
// Bound by the FP32 pipe and the latency of the rate step's chain of products,
// exponentials and reciprocals, so by the warps an SM holds; and those by
// the log-rates, 4 bytes per path and rate.  Shared memory alone holds 640
// paths of 80 rates.  The last rates' rows therefore live in tensor memory
// (256 KB per SM that this kernel has no other use for): rates nt0 .. n - 1
// as columns of the CTA's allocation, lane = thread, read and written four
// rates (eight columns) at a time; the rates below nt0 in shared memory.
// That makes room for as many CTAs per SM as the registers allow, three (768
// paths) at 80 rates and 10 factors; up to 52 rates of 3 or 5 factors, or 66
// of more, fit shared memory whole (pair_tmem_rows).
//
// One path per thread with all log-rates in shared memory, two paths per
// thread with them there, and this form: 80 rates, 10 factors, 2^20 paths 9.79,
// 8.83, 7.69 ms (FMA pipe 50, 57, 65% busy), its frozen-rule chain 8.93, 7.68
// (with the known basis tables), 7.1; 120 rates, 15 factors, 2^18 paths 8.07,
// 7.40, 5.70; 40 rates, 5 factors, 2^18 paths (all in shared memory; 128 threads
// per CTA and the row copies make the last difference) 0.61, 0.47, 0.44.  A software-
// pipelined rate loop (three consecutive blocks of rates in three stages) was
// slower: 9.55 ms with 26% more instructions.  At 10 factors three CTAs of 168
// registers beat four of 128 (7.69 against 7.83 ms).
//
// The alive rows of a step's pseudo-root (padded to a multiple of 4 factors
// for 16-byte loads) and fixed drift are copied one step ahead into the other
// of two buffers with cp.async, so a step has one barrier and no exposed load
// of them; the next step's normals are prefetched into L2.
// FT = number of factors (compile time), 0 = generic <= 16.
// ---------------------------------------------------------------------------
template <int FT, int MODE>
__global__ void __launch_bounds__(kPairThreads, PairShape<FT>::kCtas)
    fused_pairs_kernel(int paths, const float* __restrict__ Z,
                        const float* __restrict__ A,
                        const float* __restrict__ fixed,
                        const __grid_constant__ ModelConst mc,
                        const __grid_constant__ ProductConst pc,
                        const __grid_constant__ RuleConst rc,
                        const LsRuleView rule, int total, int col0,
                        float* __restrict__ o_vars, float* __restrict__ o_ex,
                        float* __restrict__ o_cf, float* __restrict__ o_num,
                        float* __restrict__ o_payoff, const RecordOut rec,
                        const SegIO seg, int nt0) {
  constexpr int FM = FPad<FT>::FM;
  constexpr int FP = FPad<FT>::FP;
  constexpr int T = kPairThreads;
  constexpr bool kInputs = MODE == kModeInputs || MODE == kModeOuter;
  // the frozen-rule modes stop a path at its exercise and run in segments
  constexpr bool kSeg = MODE == kModeRule || MODE == kModeRecord;
  const int F = FT > 0 ? FT : mc.F;
  const int n = mc.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool resume = kSeg && seg.in_prefix != nullptr;
  const int s_begin = resume ? seg.s_begin : 0;
  const int s_end = kSeg ? seg.s_end : n;
  const int rows = n - s_begin;  // rates alive in this launch
  extern __shared__ __align__(16) float sm[];
  float* const As = sm;                         // [2][rows][FP]: row r - s of step s
  float* const fx = As + 2 * rows * FP;         // [2][rows (+ pad)]
  const int fx_rows = (rows + 3) & ~3;
  __shared__ uint32_t tmem_slot;
  // this thread's log-rates
  LogRates<T> lr;
  lr.row = reinterpret_cast<float2*>(fx + 2 * fx_rows) + tid;  // [nt0 - s_begin][T]
  lr.s_begin = s_begin;
  lr.nt0 = nt0;
  lr.tmem = 0u;
  const uint32_t tmem_cols = tmem_columns(n - nt0);
  int p[2], src[2] = {0, 0};
  bool valid[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    p[h] = blockIdx.x * kPairBlock + warp * 64 + h * 32 + lane;
    valid[h] = p[h] < paths;
  }
  if (resume) {
    // survivor slot j of the previous segment, found in its CTA's block
    const int live = __ldg(seg.in_prefix + seg.in_blocks);
    if (blockIdx.x * kPairBlock >= live) {  // no survivor slot here: uniform over the CTA
      if (tid == 0 && seg.out.rates != nullptr) seg.out_count[blockIdx.x] = 0;
      return;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = blockIdx.x * kPairBlock + warp * 64 + h * 32 + lane;
      valid[h] = j < live;
      p[h] = 0;
      if (valid[h]) {
        int lo = 0, hi = seg.in_blocks;  // in_prefix[lo] <= j < in_prefix[hi]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (__ldg(seg.in_prefix + mid) <= j) lo = mid; else hi = mid;
        }
        src[h] = lo * kPairBlock + (j - __ldg(seg.in_prefix + lo));
        p[h] = seg.in.path[src[h]];
        if ((unsigned)p[h] >= (unsigned)paths) {  // never for a consistent chain
          valid[h] = false;
          p[h] = 0;
        }
      }
    }
  }
  if (warp == 0) tmem_alloc(&tmem_slot, tmem_cols);
  if (tmem_cols) {
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    lr.tmem = tmem_slot + ((uint32_t)(warp * 32) << 16);
  }
  zero_row_pads<FP, T>(As, 2 * rows, F);
  // copies step s's alive rows into buffer b
  auto stage = [&](int s, int b) {
    stage_rows<FT, FP, T>(As + b * rows * FP, fx + b * fx_rows, A, fixed, s, n, F);
  };
  stage(s_begin, 0);
  float N[2] = {1.0f, 1.0f}, f_first[2] = {0.0f, 0.0f};
  float cf_acc[2] = {0.0f, 0.0f}, N_bucket[2] = {1.0f, 1.0f};
  int bucket = -1, ex_at[2] = {n, n};
  double payoff[2] = {0.0, 0.0};
  float tarn_paid[2] = {0.0f, 0.0f};
  bool tarn_over[2] = {false, false};
  bool done[2] = {!valid[0], !valid[1]};
  // swaption-plus-cap portfolio: after the swaption's exercise the path runs
  // on for the cap strip, with no further exercise dates
  bool exercised[2] = {false, false};
  // An exercise date's discount curve P(T_s, T_{r+1}), r >= s, is completed
  // in the next step's rate loop, which forms 1 / (1 + tau_r f_r) of every
  // later rate for its drift factors anyway (pc_rate2's q); the date's
  // epilogue therefore runs one step later, from this pending state.  Which
  // date is pending (pend_e, at step s - 1) is the same for all paths; pend
  // marks the paths that still take it.
  int pend_e = -1;
  bool pend[2] = {false, false};
  float pend_N[2] = {1.0f, 1.0f}, pend_f[2] = {0.0f, 0.0f}, pend_P1[2] = {1.0f, 1.0f};
  float pend_coupon[2] = {0.0f, 0.0f};
  // the log-rate pair of rate r at the start of the launch
  auto start_rate = [&](int r) {
    if (!resume) return dup2(mc.logf0[r]);
    const float* row = seg.in.rates + (size_t)r * seg.cap;
    return make_float2(valid[0] ? row[src[0]] : 0.0f, valid[1] ? row[src[1]] : 0.0f);
  };
  for (int r = s_begin; r < nt0; ++r) lr.row[(r - s_begin) * T] = start_rate(r);
  for (int r = nt0; r < n; r += 4) {
    float2 x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = start_rate(r + j);
    __syncwarp();
    tmem_st8(lr.tmem + 2 * (r - nt0), x);
  }
  if (resume) {
    const int e = pc.ex_index[s_begin - 1];
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (valid[h]) {
        N[h] = seg.in.N[src[h]];
        f_first[h] = seg.in.f_first[src[h]];
        payoff[h] = seg.in.payoff[src[h]];
        if (e >= 0) {  // the date of step s_begin - 1 waits for this step's curve
          pend[h] = true;
          pend_N[h] = N[h];
          pend_f[h] = f_first[h];
          pend_P1[h] = seg.in.pend_P1[src[h]];
          pend_coupon[h] = seg.in.pend_coupon[src[h]];
        }
      }
    pend_e = e;
  }
  // the exercise date e of step ps, with its curve completed, on the paths
  // that take it
  auto date_epilogue = [&](int e, int ps, const float (&Pn)[2], const float (&ann)[2]) {
    float v[2][kMaxVars], exv[2] = {0.0f, 0.0f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[h][0] = pend_f[h];
      if (pc.kind == LMM_PRODUCT_SWAPTION || pc.kind == LMM_PRODUCT_BERMUDAN_CAP) {
        const float sr = (1.0f - Pn[h]) / ann[h];
        v[h][1] = sr;
        v[h][2] = ann[h];
        exv[h] = fmaxf((sr - pc.strike) * ann[h], 0.0f);
      } else {
        if (ps + 1 < n) {
          const float ann2 = ann[h] - mc.tau[ps] * pend_P1[h];
          v[h][1] = (pend_P1[h] - Pn[h]) / ann2;
        } else {
          v[h][1] = (1.0f - Pn[h]) / ann[h];
        }
        v[h][2] = mc.tau[n - 1] * Pn[h];
      }
    }
    double est[2] = {0.0, 0.0};
    if (!kInputs)
      ls_chain_estimates<2>(rule, e, rc.kind[e], rc.nvars[e], rc.nbasis[e], rc.mono[e], v, exv,
                         est);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!pend[h]) continue;
      pend[h] = false;
      if (kInputs) {
        const int col = col0 + p[h];
        if (bucket >= 0) o_cf[(size_t)bucket * total + col] = cf_acc[h];
        cf_acc[h] = pend_coupon[h];
#pragma unroll
        for (int k = 0; k < kMaxVars; ++k)
          o_vars[((size_t)e * kMaxVars + k) * total + col] = v[h][k];
        o_ex[(size_t)e * total + col] = exv[h];
        o_num[(size_t)e * total + col] = pend_N[h];
      } else if ((double)exv[h] > est[h]) {
        payoff[h] += (double)exv[h] / (double)pend_N[h];
        if (MODE == kModeRecord) ex_at[h] = ps;
        if (pc.kind == LMM_PRODUCT_BERMUDAN_CAP)
          exercised[h] = true;
        else
          done[h] = true;
        continue;
      } else {
        payoff[h] += (double)pend_coupon[h] / (double)pend_N[h];
      }
      N_bucket[h] = pend_N[h];
    }
  };
  for (int s = s_begin; s < s_end; ++s) {
    // the step's normals are loaded first, so that their latency overlaps
    // the staging of the step's pseudo-root rows and the barriers
    float2 w[FM];
    {
      const float* zs = Z + (size_t)s * F * paths;
#pragma unroll
      for (int f = 0; f < FM; ++f) {
        const float* zf = zs + (size_t)f * paths;
        w[f] = make_float2((f < F && !done[0]) ? __ldg(zf + p[0]) : 0.0f,
                           (f < F && !done[1]) ? __ldg(zf + p[1]) : 0.0f);
      }
    }
    cp_async_wait<0>();
    __syncthreads();  // this step's rows are in; the other buffer is free
    const int buf = (s - s_begin) & 1;
    if (s + 1 < s_end) {
      stage(s + 1, buf ^ 1);
      // the next step's normals into L2: whole lines of consecutive paths, or
      // each survivor's own
      if (!resume) {
        if (lane < 2 * F) {
          const int f = lane >= F ? lane - F : lane;
          const int q =
              min(blockIdx.x * kPairBlock + warp * 64 + (lane >= F ? 32 : 0), paths - 1);
          prefetch_l2(Z + ((size_t)(s + 1) * F + f) * paths + q);
        }
      } else {
        const float* zn = Z + (size_t)(s + 1) * F * paths;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (!done[h])
            for (int f = 0; f < F; ++f) prefetch_l2(zn + (size_t)f * paths + p[h]);
      }
    }
    // whole warps only past here (tensor memory is read by whole warps)
    if (__all_sync(0xffffffffu, done[0] && done[1])) continue;
    if (s > 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) N[h] = N[h] * (1.0f + mc.tau[s - 1] * f_first[h]);
    }
    if ((MODE == kModeRecord || MODE == kModeOuter) && s % rec.every == 0) {
      const int c = s / rec.every;
      auto put = [&](int r, float2 x) {
        float* row = rec.ckpt + ((size_t)c * n + r) * paths;
        if (!done[0]) row[p[0]] = x.x;
        if (!done[1]) row[p[1]] = x.y;
      };
      lr.for_each(s, n, put);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (!done[h]) rec.ckptN[(size_t)c * paths + p[h]] = N[h];
    }
    const bool curve = pend_e >= 0;  // uniform over the CTA
    float2 Pd = make_float2(pend_P1[0], pend_P1[1]);
    float2 annd = dup2(0.0f);
    if (curve) annd = make_float2(mc.tau[s - 1] * pend_P1[0], mc.tau[s - 1] * pend_P1[1]);
    float2 v[FM];
#pragma unroll
    for (int f = 0; f < FM; ++f) v[f] = dup2(0.0f);
    // the rate loop, unswitched on whether a date's curve is pending
    const float* As_s = As + buf * rows * FP;
    const float* fx_s = fx + buf * fx_rows;
    const float2 lf0 =
        curve ? pc_step2<FM, FP, T>(lr, s, n, mc, As_s, fx_s, w, v,
                                    [&](int r, float2, float2, float2 q, float2) {
                                      Pd = __fmul2_rn(Pd, q);
                                      annd = __ffma2_rn(dup2(mc.tau[r]), Pd, annd);
                                    })
              : pc_step2<FM, FP, T>(lr, s, n, mc, As_s, fx_s, w, v,
                                    [](int, float2, float2, float2, float2) {});
    const int e = pc.ex_index[s];
    // ---- the previous step's exercise date, then the epilogue at T_s ----
    if (pend[0] || pend[1]) {
      const float Pn[2] = {Pd.x, Pd.y}, ann[2] = {annd.x, annd.y};
      date_epilogue(pend_e, s - 1, Pn, ann);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      f_first[h] = __expf(h ? lf0.y : lf0.x) - mc.disp[s];
      if (done[h]) continue;
      const float P1 = __fdividef(1.0f, 1.0f + mc.tau[s] * f_first[h]);
      if (pc.kind == LMM_PRODUCT_TARN) {
        payoff[h] += (double)(tarn_flow(pc, s, n, mc.tau[s], f_first[h], tarn_paid[h],
                                        tarn_over[h]) *
                              P1) /
                     (double)N[h];
        continue;
      }
      if (pc.kind == LMM_PRODUCT_EUROPEAN) {
        const float tau = mc.tau[s];
        const float cap = tau * fmaxf(f_first[h] - pc.cap_strike, 0.0f);
        const float swp = tau * (f_first[h] - pc.strike) * pc.pay_receive;
        payoff[h] += (double)((cap + swp) * P1) / (double)N[h];
        continue;
      }
      if (pc.kind == LMM_PRODUCT_BERMUDAN_CAP && kSeg) {
        // the portfolio's caplet on f_s, paid at T_{s+1} whether or not the
        // swaption has been exercised
        const float cap = mc.tau[s] * fmaxf(f_first[h] - pc.cap_strike, 0.0f);
        payoff[h] += (double)(cap * P1) / (double)N[h];
      }
      float coupon = 0.0f;
      if (pc.kind == LMM_PRODUCT_CANCELLABLE_SWAP)
        coupon = mc.tau[s] * (f_first[h] - pc.strike) * pc.pay_receive * P1;
      if (e >= 0 && !exercised[h]) {
        pend[h] = true;
        pend_N[h] = N[h];
        pend_f[h] = f_first[h];
        pend_P1[h] = P1;
        pend_coupon[h] = coupon;
      } else if (coupon != 0.0f) {
        if (kInputs) {
          if ((pend_e >= 0 ? pend_e : bucket) >= 0)
            cf_acc[h] += coupon * (N_bucket[h] / N[h]);
        } else {
          payoff[h] += (double)coupon / (double)N[h];
        }
      }
    }
    if (pend_e >= 0) bucket = pend_e;
    pend_e = e;
  }
  if (kSeg && seg.out.rates != nullptr) {
    // end of a segment: pack the survivors of this CTA in path order (the
    // per-warp counts go to the pseudo-root rows, free once every warp is
    // past its last step)
    int* warp_live = reinterpret_cast<int*>(As);
    const bool live[2] = {valid[0] && !done[0], valid[1] && !done[1]};
    const unsigned bal[2] = {__ballot_sync(0xffffffffu, live[0]),
                             __ballot_sync(0xffffffffu, live[1])};
    __syncthreads();
    if (lane == 0) warp_live[warp] = __popc(bal[0]) + __popc(bal[1]);
    __syncthreads();
    int off = 0, tot = 0;
    for (int w = 0; w < T / 32; ++w) {
      const int c = warp_live[w];
      off += w < warp ? c : 0;
      tot += c;
    }
    const unsigned below = (1u << lane) - 1u;
    const int slot0 = blockIdx.x * kPairBlock + off;
    const int slot[2] = {slot0 + __popc(bal[0] & below),
                         slot0 + __popc(bal[0]) + __popc(bal[1] & below)};
    lr.for_each(s_end, n, [&](int r, float2 x) {
      float* row = seg.out.rates + (size_t)r * seg.cap;
      if (live[0]) row[slot[0]] = x.x;
      if (live[1]) row[slot[1]] = x.y;
    });
    tmem_free(lr.tmem, tmem_cols);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (live[h]) {
        seg.out.N[slot[h]] = N[h];
        seg.out.f_first[slot[h]] = f_first[h];
        seg.out.pend_P1[slot[h]] = pend_P1[h];
        seg.out.pend_coupon[slot[h]] = pend_coupon[h];
        seg.out.payoff[slot[h]] = payoff[h];
        seg.out.path[slot[h]] = p[h];
      }
      if (valid[h] && done[h]) {
        o_payoff[p[h]] = (float)payoff[h];
        if (MODE == kModeRecord) rec.ex_step[p[h]] = ex_at[h];
      }
    }
    if (tid == 0) seg.out_count[blockIdx.x] = tot;
    return;
  }
  tmem_free(lr.tmem, tmem_cols);
  // an exercise date at the last step: its curve is the one period
  if (pend[0] || pend[1]) {
    const float ann[2] = {mc.tau[n - 1] * pend_P1[0], mc.tau[n - 1] * pend_P1[1]};
    date_epilogue(pend_e, n - 1, pend_P1, ann);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!valid[h]) continue;
    if (kInputs) {
      const int last = pend_e >= 0 ? pend_e : bucket;
      if (pc.kind != LMM_PRODUCT_EUROPEAN && last >= 0)
        o_cf[(size_t)last * total + col0 + p[h]] = cf_acc[h];
      if ((pc.kind == LMM_PRODUCT_EUROPEAN || pc.kind == LMM_PRODUCT_TARN) && o_payoff)
        o_payoff[p[h]] = (float)payoff[h];
    } else {
      o_payoff[p[h]] = (float)payoff[h];
      if (MODE == kModeRecord) rec.ex_step[p[h]] = ex_at[h];
    }
  }
}

// Tensor-memory rows of a launch whose first step has `rows` alive rates:
// as many (a multiple of four, at most 64) as it takes for PairShape::kCtas
// CTAs to fit the SM's shared memory; none where they fit anyway.
inline int pair_ctas(int F) { return (F == 3 || F == 5) ? 4 : 3; }
inline size_t pair_smem_bytes(int rows, int F, int smem_rows) {
  const size_t stage = (size_t)rows * launched_row_pad(F) + ((rows + 3) & ~3);
  return (2 * stage + (size_t)smem_rows * kPairBlock) * sizeof(float);
}
inline int pair_tmem_rows(int rows, int F) {
  constexpr size_t kSmPerSm = 228 * 1024, kReserved = 1024 + 64;  // per CTA
  const size_t cta = kSmPerSm / pair_ctas(F) - kReserved;
  int t = 0;
  while (t < rows && t < 64 && pair_smem_bytes(rows, F, rows - t) > cta) t += 4;
  return t < rows ? t : rows & ~3;
}

}  // namespace lmm
