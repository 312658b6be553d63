// pc_step.cuh — the predictor-corrector rate step shared by every kernel
// that evolves forward rates path by path: the fused pricing passes
// (fused_kernels.cuh), the adjoint's recompute, the Andersen–Broadie inner
// paths and the full-tensor evolution of lmm_evolve_pc_all.  Keeping one
// definition makes all of them follow exactly the same arithmetic.
#pragma once
#include "lmm_common.cuh"
#include "lmm_device.cuh"

namespace lmm {

// Model constants passed by value as a kernel parameter.
struct ModelConst {
  int n, F, scr_dims;
  float cutoff;
  float tau[kMaxRates], disp[kMaxRates], logf0[kMaxRates];
  float c0[kMaxRates];  // 1 - d_r tau_r: g = F tau / (c0 + F tau)
  float l2tau[kMaxRates];  // log2 tau_r: F tau = 2^(log F log2 e + log2 tau)
};

// Padding of the per-step pseudo-root rows held in shared memory: FT =
// number of factors (compile time), 0 = generic <= kMaxFactors.
template <int FT>
struct FPad {
  static constexpr int FM = FT > 0 ? FT : kMaxFactors;
  static constexpr int FP = (FM + 3) & ~3;
};

// One rate r of one predictor-corrector step.  The spot drift of rate r over
// the rates s..r of the step is mu_r = A_r . e_{r-1} + g_r |A_r|^2 with the
// prefix e_{r-1} = sum_{j<r} g_j A_j and |A_r|^2 = -2 x the fixed drift; the
// corrector's drift uses the predicted rates' prefix ep the same way.  The
// predictor-corrector step of the reference (LMM_evolver_all.cu:615-744,
// gold/LMM_evolver_gold.h:315-387)
//   lp = lf + mu_r + A_r . z + fixed_r,   lf' = lp + (mp_r - mu_r) / 2
// needs three products of A_r with factor vectors (e, z, ep).  Here two
// running vectors are kept instead,
//   w = z + e_{r-1},   v = ep_{r-1} - e_{r-1},
// so that lp = lf + A_r . w + g_r |A_r|^2 + fixed_r and
// lf' = lp + (A_r . v + (gp_r - g_r) |A_r|^2) / 2: two dot products and two
// updates per rate (w += g_r A_r, v += (gp_r - g_r) A_r) in place of three
// and two, the same quantities with other FP32 roundings.  Both dot
// products depend only on the earlier rates, so they overlap this rate's
// exp and reciprocal.  Factors are held in pairs (f = 2k, 2k + 1) and every
// product-sum runs as one packed FP32x2 FMA per pair: the even and odd
// factors accumulate in the two halves, each with the rounding of a scalar
// FMA.  exp(x) tau is formed as 2^(x log2 e + log2 tau) (l2tau = log2 tau).
// Returns the new (capped) log-rate; g and gp are the drift factors
// F tau / (1 + f tau) of the start and predicted rates (F = f + d, c0 =
// 1 - d tau), q = 1 / (1 + tau f) of the start rate (its factor in the
// discount ratios of the previous date), capped whether the cap applied.
// Shared by the pricing kernels, the adjoint's recompute, the
// Andersen–Broadie inner paths and lmm_evolve_pc_all, so all follow exactly
// the same path.
template <int FM, int FP>
__device__ __forceinline__ float pc_rate(float lf, float l2tau, float c0, float fxr,
                                         const float* Arow, float2 (&w)[FP / 2],
                                         float2 (&v)[FP / 2], float cutoff, float& g, float& gp,
                                         float& q, bool& capped) {
  constexpr int NP = (FM + 1) / 2;  // pairs that hold factors
  constexpr float kLog2e = 1.44269504088896341f;
  const float4* a4 = reinterpret_cast<const float4*>(Arow);
  float2 a2[FP / 2];
#pragma unroll
  for (int k = 0; k < FP / 4; ++k) {
    const float4 a = a4[k];
    a2[2 * k] = make_float2(a.x, a.y);
    a2[2 * k + 1] = make_float2(a.z, a.w);
  }
  float2 dw = make_float2(0.0f, 0.0f), dv = dw;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    dw = __ffma2_rn(a2[k], w[k], dw);
    dv = __ffma2_rn(a2[k], v[k], dv);
  }
  const float nA2 = -2.0f * fxr;
  const float Fr = ex2_ftz(fmaf(lf, kLog2e, l2tau));
  q = rcp_ftz(c0 + Fr);
  g = Fr * q;
  lf += fmaf(g, nA2, dw.x + dw.y) + fxr;
  const float Fp = ex2_ftz(fmaf(lf, kLog2e, l2tau));
  gp = Fp * rcp_ftz(c0 + Fp);
  const float dg = gp - g;
  lf += 0.5f * fmaf(dg, nA2, dv.x + dv.y);
  const float2 g2 = make_float2(g, g), dg2 = make_float2(dg, dg);
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    w[k] = __ffma2_rn(a2[k], g2, w[k]);
    v[k] = __ffma2_rn(a2[k], dg2, v[k]);
  }
  capped = lf > cutoff;
  return fminf(lf, cutoff);
}

template <int FM, int FP>
__device__ __forceinline__ float pc_rate(float lf, float l2tau, float c0, float fxr,
                                         const float* Arow, float2 (&w)[FP / 2],
                                         float2 (&v)[FP / 2], float cutoff, float& g, float& gp,
                                         bool& capped) {
  float q;
  return pc_rate<FM, FP>(lf, l2tau, c0, fxr, Arow, w, v, cutoff, g, gp, q, capped);
}

// Running vectors of pc_rate at the start of a step: w = the step's normals
// (in factor pairs), v = 0.
template <int FP>
__device__ __forceinline__ void step_start(const float (&z)[FP], float2 (&w)[FP / 2],
                                           float2 (&v)[FP / 2]) {
#pragma unroll
  for (int k = 0; k < FP / 2; ++k) {
    w[k] = make_float2(z[2 * k], z[2 * k + 1]);
    v[k] = make_float2(0.0f, 0.0f);
  }
}

// pc_rate for two paths per thread: the pair's values in the two halves of a
// float2 and the factor vectors w, v as one float2 per factor, so that every
// operation of the rate step (not only the factor sums) is one packed
// instruction for both paths and the pseudo-root row, the constants and the
// loop control are read once per pair.  Each half runs pc_rate's own sequence
// of roundings (even and odd factors in two accumulators, added last), so a
// path's values are bit-identical to pc_rate's.
__device__ __forceinline__ float2 cap2(float2 lf, float cutoff) {
  return make_float2(fminf(lf.x, cutoff), fminf(lf.y, cutoff));
}

template <int FM, int FP>
__device__ __forceinline__ float2 pc_rate2(float2 lf, float l2tau, float c0, float fxr,
                                           const float* Arow, float2 (&w)[FM], float2 (&v)[FM],
                                           float2& g, float2& gp, float2& q) {
  constexpr float kLog2e = 1.44269504088896341f;
  const float4* a4 = reinterpret_cast<const float4*>(Arow);
  float a[FP];
#pragma unroll
  for (int k = 0; k < FP / 4; ++k) {
    const float4 t = a4[k];
    a[4 * k] = t.x;
    a[4 * k + 1] = t.y;
    a[4 * k + 2] = t.z;
    a[4 * k + 3] = t.w;
  }
  float2 dw[2] = {dup2(0.0f), dup2(0.0f)}, dv[2] = {dup2(0.0f), dup2(0.0f)};
#pragma unroll
  for (int f = 0; f < FM; ++f) {
    dw[f & 1] = __ffma2_rn(dup2(a[f]), w[f], dw[f & 1]);
    dv[f & 1] = __ffma2_rn(dup2(a[f]), v[f], dv[f & 1]);
  }
  const float2 nA2 = dup2(-2.0f * fxr);
  float2 t = __ffma2_rn(lf, dup2(kLog2e), dup2(l2tau));
  const float2 Fr = make_float2(ex2_ftz(t.x), ex2_ftz(t.y));
  t = __fadd2_rn(dup2(c0), Fr);
  q = make_float2(rcp_ftz(t.x), rcp_ftz(t.y));
  g = __fmul2_rn(Fr, q);
  lf = __fadd2_rn(lf, __fadd2_rn(__ffma2_rn(g, nA2, __fadd2_rn(dw[0], dw[1])), dup2(fxr)));
  t = __ffma2_rn(lf, dup2(kLog2e), dup2(l2tau));
  const float2 Fp = make_float2(ex2_ftz(t.x), ex2_ftz(t.y));
  t = __fadd2_rn(dup2(c0), Fp);
  const float2 qp = make_float2(rcp_ftz(t.x), rcp_ftz(t.y));
  gp = __fmul2_rn(Fp, qp);
  const float2 dg = __ffma2_rn(Fp, qp, make_float2(-g.x, -g.y));
  lf = __ffma2_rn(dup2(0.5f), __ffma2_rn(dg, nA2, __fadd2_rn(dv[0], dv[1])), lf);
#pragma unroll
  for (int f = 0; f < FM; ++f) {
    w[f] = __ffma2_rn(dup2(a[f]), g, w[f]);
    v[f] = __ffma2_rn(dup2(a[f]), dg, v[f]);
  }
  return lf;
}

// Tensor memory as storage: allocation of `cols` columns (a power of two) by
// one warp, eight columns of the calling warp's lanes at a time.
__host__ __device__ __forceinline__ uint32_t tmem_columns(int rows) {
  uint32_t c = rows > 0 ? 32u : 0u;
  while (c < 2u * (uint32_t)rows) c *= 2u;
  return c;
}
// `cols` may be 0.  The CTA gives up its right to allocate in either case:
// until a CTA of a kernel with tensor-memory instructions has done so, its SM
// starts no further CTA of the kernel (1 instead of 4 CTAs per SM measured
// without it, 0.92 against 0.44 ms for 2^18 paths of 40 rates).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  __syncwarp();  // whole warps only, after whatever per-path branches came before
  if (cols)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(slot)),
                 "r"(cols)
                 : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Frees the CTA's columns (`cols` may be 0); contains a CTA barrier, all
// threads.  The last step's stores have no load behind them that would wait
// for them, so every warp waits for its own here: once the columns are free,
// another CTA of the SM may be given them.
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
  if (cols) {
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tmem_fence_before();
  }
  __syncthreads();
  if (cols && threadIdx.x < 32) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols)
                 : "memory");
  }
}
__device__ __forceinline__ void tmem_st8(uint32_t a, const float2 (&x)[4]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a),
      "f"(x[0].x), "f"(x[0].y), "f"(x[1].x), "f"(x[1].y), "f"(x[2].x), "f"(x[2].y),
      "f"(x[3].x), "f"(x[3].y)
      : "memory");
}
// waits for this thread's earlier stores, loads, and waits for the load
__device__ __forceinline__ void tmem_ld8(uint32_t a, float2 (&x)[4]) {
  asm volatile(
      "tcgen05.wait::st.sync.aligned;\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(x[0].x), "=f"(x[0].y), "=f"(x[1].x), "=f"(x[1].y), "=f"(x[2].x), "=f"(x[2].y),
        "=f"(x[3].x), "=f"(x[3].y)
      : "r"(a)
      : "memory");
}

// A thread's log-rates of its two paths: rates s_begin .. nt0 - 1 in shared
// memory, row r at row[(r - s_begin) * T]; rates nt0 .. n - 1 (a multiple of
// four of them) in tensor memory, two columns each from column `tmem` of the
// warp's lanes.
template <int T>
struct LogRates {
  float2* row;
  uint32_t tmem;
  int s_begin, nt0;
  // fn(r, pair) for the rates r = s .. n - 1 (whole warps)
  template <class Fn>
  __device__ __forceinline__ void for_each(int s, int n, Fn&& fn) const {
    for (int r = s; r < nt0; ++r) fn(r, row[(r - s_begin) * T]);
    for (int r0 = nt0 + (max(s - nt0, 0) & ~3); r0 < n; r0 += 4) {
      float2 x[4];
      __syncwarp();  // fn may branch per path
      tmem_ld8(tmem + 2 * (r0 - nt0), x);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (r0 + j >= s) fn(r0 + j, x[j]);
    }
  }
};

// One step: pc_rate2 over the rates s .. n - 1 of the log-rates lr (whole
// warps).  As, fx: the step's rows, rate r at row r - s.  hook(r, g, gp, q,
// ln): called per rate with pc_rate2's outputs and the new log-rates before
// the cap; it leaves the warp whole (tensor memory is accessed by whole
// warps).  Returns the new log-rates of rate s.
template <int FM, int FP, int T, class Hook>
__device__ __forceinline__ float2 pc_step2(const LogRates<T>& lr, int s, int n,
                                           const ModelConst& mc, const float* As,
                                           const float* fx, float2 (&w)[FM], float2 (&v)[FM],
                                           Hook&& hook) {
  auto rate = [&](int r, float2 lf) {
    float2 g, gp, q;
    const int i = r - s;
    lf = pc_rate2<FM, FP>(lf, mc.l2tau[r], mc.c0[r], fx[i], As + i * FP, w, v, g, gp, q);
    hook(r, g, gp, q, lf);
    return cap2(lf, mc.cutoff);
  };
  __syncwarp();  // per-path branches of the caller end here
  float2 lf0 = dup2(0.0f);
  float2* row = lr.row + (s - lr.s_begin) * T;
#pragma unroll 4
  for (int r = s; r < lr.nt0; ++r) row[(r - s) * T] = rate(r, row[(r - s) * T]);
  int r0 = lr.nt0;
  if (s < lr.nt0) {
    lf0 = row[0];
  } else {  // the step starts inside the tensor-memory rows, maybe inside a block
    r0 += (s - lr.nt0) & ~3;
    float2 x[4];
    const uint32_t a = lr.tmem + 2 * (r0 - lr.nt0);
    tmem_ld8(a, x);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (r0 + j >= s) {
        x[j] = rate(r0 + j, x[j]);
        if (r0 + j == s) lf0 = x[j];
      }
    tmem_st8(a, x);
    r0 += 4;
  }
#pragma unroll 1
  for (; r0 < n; r0 += 4) {
    float2 x[4];
    const uint32_t a = lr.tmem + 2 * (r0 - lr.nt0);
    tmem_ld8(a, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = rate(r0 + j, x[j]);
    tmem_st8(a, x);
  }
  return lf0;
}

}  // namespace lmm
