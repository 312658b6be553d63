// fused_kernels.cuh — device code of the fused form (included by
// pipeline.cu): the variates kernel (Sobol -> scramble -> inverse normal ->
// bridge) and the per-path evolution kernel with the product epilogue.
//
// Both kernels use the fast hardware approximations of exp, log and
// reciprocal with denormals flushed (ex2/lg2/rcp.approx.ftz, lmm_device.cuh;
// relative error ~1e-7, i.e. a few FP32 ulp); the staged kernels keep the
// IEEE-accurate library forms and serve as the plain-FP32 reference of the
// same arithmetic.
#pragma once
#include <algorithm>
#include <type_traits>
#include "lmm_common.cuh"
#include "lmm_device.cuh"
#include "bridge_plan.h"
#include "ls_common.cuh"
#include "pc_step.cuh"

namespace lmm {

struct ProductConst {
  int kind, n_ex;
  float strike, cap_strike, pay_receive;
  float tarn_total, tarn_mult;
  int ex_index[kMaxSteps];  // step -> exercise index, -1 if none
};

// Basis tables of every exercise date for the in-kernel rule (passed by
// value as a kernel parameter, about 7 KB).
struct RuleConst {
  int nvars[kMaxSteps];
  int nbasis[kMaxSteps];
  unsigned char kind[kMaxSteps];  // ls_basis_kind of the date's table
  unsigned char mono[kMaxSteps][kMaxBasis][kMaxVars];
};

// kModeInputs: write the regression inputs; kModeRule: apply the frozen rule
// and write the payoff; kModeRecord: as kModeRule, and also record what the
// adjoint needs (log-rate checkpoints, numeraires, exercise steps).
// kModeOuter: as kModeInputs (every date, no stopping), and also record the
// log-rates and numeraire at the start of every `every`-th step (the outer
// paths of the Andersen–Broadie estimate).
enum { kModeInputs = 0, kModeRule = 1, kModeRecord = 2, kModeOuter = 3 };

// Paths per CTA of the evolution kernel, and steps per launch of the
// segmented second pass (SegIO below) unless the caller asks otherwise.
constexpr int kFusedBlock = 128;
constexpr int kSegSteps = 8;

// Outputs of kModeRecord.  Every `every` steps (s = c * every) the log-rates
// at the start of the step go to ckpt[c][r][p] (r >= s) and the numeraire to
// ckptN[c][p]; ex_step[p] is the exercise step (rates when never exercised).
struct RecordOut {
  float* ckpt;
  float* ckptN;
  int* ex_step;
  int every;
};

// Segmented rule-mode evolution.  A path stops at its exercise, so its
// lane idles for the rest of the launch; the second pass therefore runs as
// a chain of launches over segments of steps, and the paths still alive at
// the end of a segment are packed into survivor slots that the next
// segment's CTAs take densely.  SegState holds the survivors of one segment
// boundary s1 (after step s1 - 1): log-rates of rows >= s1, the numeraire
// and reset rate of step s1 - 1, the pending exercise date's P(T_s, T_{s+1})
// and coupon (the date is completed in step s1's rate loop), the payoff so
// far and the path's index in the batch.  Slots [b * T, b * T + count[b])
// belong to CTA b of the launch that wrote them (kept in path order).
struct SegState {
  float* rates;     // [rates][cap]
  float* N;         // [cap]
  float* f_first;   // [cap]
  float* pend_P1;   // [cap]
  float* pend_coupon;  // [cap]
  double* payoff;   // [cap]
  int* path;        // [cap]
};

// One launch of the chain: steps [s_begin, s_end).  in_prefix (null for the
// first segment) is the exclusive prefix of the previous launch's per-CTA
// survivor counts over in_blocks CTAs (in_prefix[in_blocks] = survivors);
// out.rates null marks the last segment, else the launch writes its
// survivors to `out` and their count per CTA to out_count.
struct SegIO {
  int s_begin, s_end, cap, in_blocks;
  const int* in_prefix;
  SegState in, out;
  int* out_count;
};

// Continuation estimate of the frozen rule at exercise date e (depth chain
// and Andersen shift of ls_chain_estimates).
__device__ __forceinline__ double rule_estimate(const RuleConst& rc, int e, const float* v,
                                                float exv, const LsRuleView& rule) {
  const float v1[1][kMaxVars] = {{v[0], v[1], v[2]}}, ex1[1] = {exv};
  double est[1];
  ls_chain_estimates<1>(rule, e, rc.kind[e], rc.nvars[e], rc.nbasis[e], rc.mono[e], v1, ex1,
                        est);
  return est[0];
}

// Shaw–Brickman inverse normal on the exact tail probability
// (icdf_sb_tails) with the hardware log and reciprocal approximations, for two
// points per thread: the numerator and denominator recurrences run on the
// packed pair, each half with the roundings of the scalar FMAs, and the sign,
// +1 for integers from 2^31, is set as a bit.
__device__ __forceinline__ float2 icdf_sb_fast2(uint32_t va, uint32_t vb) {
  auto tail = [](uint32_t v) {
    return fmaxf(__uint2float_rn(min(v, 0u - v)) * 4.656612873077392578125e-10f,
                 2.3283064365386963e-10f);
  };
  const float2 z = make_float2(-log_ftz(tail(va)), -log_ftz(tail(vb)));
  float2 p = __ffma2_rn(dup2(4.744820732427972462e-6f), z, dup2(0.0020751409553756572917f));
  float2 q = __ffma2_rn(dup2(0.00010590620919921025259f), z, dup2(0.0120098270559197768f));
  p = __ffma2_rn(p, z, dup2(0.087403248265958578062f));
  q = __ffma2_rn(q, z, dup2(0.23668431621373705623f));
  p = __ffma2_rn(p, z, dup2(0.80002295072483916762f));
  q = __ffma2_rn(q, z, dup2(1.2499328117341603014f));
  p = __ffma2_rn(p, z, dup2(1.9797154223229267471f));
  q = __ffma2_rn(q, z, dup2(2.0795584360534589311f));
  p = __ffma2_rn(p, z, dup2(1.2533136835212087879f));
  q = __ffma2_rn(q, z, dup2(1.0f));
  const float2 x = __fmul2_rn(__fmul2_rn(z, p), make_float2(rcp_ftz(q.x), rcp_ftz(q.y)));
  return make_float2(__uint_as_float(__float_as_uint(x.x) ^ (~va & 0x80000000u)),
                     __uint_as_float(__float_as_uint(x.y) ^ (~vb & 0x80000000u)));
}

__device__ __forceinline__ float icdf_sb_fast(uint32_t v) { return icdf_sb_fast2(v, v).x; }

// ---------------------------------------------------------------------------
// Fused variates: Sobol point -> XOR scramble -> inverse normal -> bridge.
// One thread per factor and pair of paths (p, p + 128), one CTA per factor
// and `tiles` consecutive tiles of 256 paths.  With n = first_index + p and
// gray(n) = n ^ (n >> 1), the bits of gray(n) at and above 7 are
// gray(n >> 7): the first paths of a tile share at most two values h0, h0 + 1
// of n >> 7, so the XOR of the upper direction numbers (with the scrambler
// word folded in) is kept per CTA and Sobol dimension.  The seven low Gray
// bits select from two small XOR tables per dimension, lo4_s (bits 0-3, 16
// entries) and hi3_s (bits 4-6, 8 entries).  The pair's second point n + 128
// has the same low bits of n, so it differs by Gray bit 6 and the one upper
// bit in which gray(h + 1) differs from gray(h): one more XOR with a word
// that is stored beside the upper XOR.  A pair of points costs three
// shared-memory reads, with no data-dependent branch.
//
// The bridge runs depth first over its tree of intervals instead of level by
// level: a point's two neighbours are then its ancestors, and the points come
// out from left to right, each increment as soon as its point's left subtree
// is done.  Only the ancestors of the current point are held, one row per
// depth (at most ten rows for 128 steps, against one per step), so an SM's
// shared memory holds as many CTAs as the registers allow instead of two.
// The host lists the points in that order (make_var_plan); every point is the
// same combination of the same values.  Both paths of a thread run in one
// packed FP32x2 value, so the point's weights and offsets, the addressing and
// the loop control are read once per pair; normals are generated kVarBatch
// points at a time (independent work for the scheduler).  Output
// [step][factor][path] increments.
//
// Bound by instruction issue and the shared-memory reads (the 3.4 GB of
// output at 2^20 paths, 80 steps and 10 factors take 0.5 ms).  One path per
// thread level by level, two paths so, and this form: 1.79, 1.68, 1.17 ms
// there; 200,003 paths, 120 steps, 15 factors 1.18, 1.16, 0.59 ms (one CTA per
// SM level by level); 300,001 paths, 40 steps, 5 factors 141, 117, 114 us.
// ---------------------------------------------------------------------------
constexpr int kVarBlock = 128;
constexpr int kVarTile = 2 * kVarBlock;  // paths per tile
constexpr int kVarBatch = 8;
constexpr int kVarTiles = 8;  // most tiles per CTA

// The bridge's points in depth-first order: weights, rows of the neighbours
// and the point itself (row `rows` - 1 stays zero: the neighbour of a point
// that has none), how many points come out after it, and the Sobol dimension
// of its normal per factor.  out_row: the row of each point in the order of
// the steps.
struct VarPlan {
  int steps, factors, rows;
  float lw[kMaxSteps], rw[kMaxSteps], sd[kMaxSteps];
  unsigned char left[kMaxSteps], right[kMaxSteps], target[kMaxSteps];
  unsigned char emits[kMaxSteps], out_row[kMaxSteps];
  unsigned short dim[kMaxFactors * kMaxSteps];  // [factor][point]
};

inline void make_var_plan(const BridgePlan& b, VarPlan* v) {
  const int S = b.steps;
  int stage_of[kMaxSteps];
  for (int i = 0; i < S; ++i) stage_of[b.bidx[i]] = i;
  v->steps = S;
  v->factors = b.factors;
  int count = 0, depth_max = 0, row_of[kMaxSteps] = {};
  // point p at `depth`, neighbours' points l and r (-1: none)
  auto put = [&](int p, int depth, int l, int r) {
    const int i = stage_of[p], k = count++;
    v->lw[k] = l >= 0 ? b.lw[i] : 0.0f;
    v->rw[k] = r >= 0 ? b.rw[i] : 0.0f;
    v->sd[k] = b.sd[i];
    v->left[k] = l >= 0 ? (unsigned char)row_of[l] : 255;
    v->right[k] = r >= 0 ? (unsigned char)row_of[r] : 255;
    v->target[k] = (unsigned char)depth;
    v->emits[k] = 0;
    for (int f = 0; f < b.factors; ++f)
      v->dim[f * kMaxSteps + k] = (unsigned short)b.alloc[f * S + i];
    row_of[p] = depth;
    depth_max = std::max(depth_max, depth);
    return k;
  };
  int out = 0, last = put(S - 1, 0, -1, -1);  // the terminal point
  // the points strictly between l and r
  auto fill = [&](auto&& self, int l, int r, int depth) -> void {
    if (r - l < 2) return;
    const int m = l + 1 + ((r - 2 - l) >> 1);
    last = put(m, depth, l, r);
    self(self, l, m, depth + 1);
    ++v->emits[last];
    v->out_row[out++] = (unsigned char)depth;
    self(self, m, r, depth + 1);
  };
  fill(fill, -1, S - 1, 1);
  ++v->emits[last];
  v->out_row[out] = 0;
  v->rows = depth_max + 2;
  for (int k = 0; k < S; ++k) {
    if (v->left[k] == 255) v->left[k] = (unsigned char)(v->rows - 1);
    if (v->right[k] == 255) v->right[k] = (unsigned char)(v->rows - 1);
  }
}

// The Sobol tables of one dimension (direction numbers v): returns the XOR of
// the direction numbers over the set Gray bits of the upper index h, and fills
// the two low tables (in vl: v[0 .. 6]), each entry the previous one with its
// lowest set bit cleared, XOR that bit's direction number.
__device__ __forceinline__ uint32_t sobol_tables(const uint32_t* __restrict__ v, uint32_t h,
                                                 uint32_t* l4, uint32_t* h3,
                                                 uint32_t (&vl)[7]) {
  uint32_t g = h ^ (h >> 1), x = 0;
  while (g) {
    x ^= __ldg(v + 7 + (__ffs(g) - 1));
    g &= g - 1u;
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) vl[k] = __ldg(v + k);
  uint32_t t4[16], t3[8];
  t4[0] = 0u;
  t3[0] = 0u;
#pragma unroll
  for (int e = 1; e < 16; ++e) t4[e] = t4[e & (e - 1)] ^ vl[__ffs(e) - 1];
#pragma unroll
  for (int e = 1; e < 8; ++e) t3[e] = t3[e & (e - 1)] ^ vl[4 + __ffs(e) - 1];
#pragma unroll
  for (int e = 0; e < 16; ++e) l4[e] = t4[e];
#pragma unroll
  for (int e = 0; e < 8; ++e) h3[e] = t3[e];
  return x;
}

__global__ void __launch_bounds__(kVarBlock)
    variates_kernel(int paths, uint32_t first_index, int tiles,
                    const uint32_t* __restrict__ dirs,
                    const uint32_t* __restrict__ scr, int scr_dims,
                    float* __restrict__ out,
                    const __grid_constant__ VarPlan plan) {
  constexpr int T = kVarBlock;
  constexpr int kRow = T * (int)sizeof(float2);  // bytes of a bridge row
  const int S = plan.steps, F = plan.factors;
  // shared memory (variates_smem_bytes): the rows of bridge points W[rows][T],
  // the plan per point as {lw, rw, sd} weights with the points to put out and
  // {left row, right row, target row} byte offsets into W, the rows of the
  // points in the order of the steps, and the Sobol tables up[2][S],
  // lo4[S][17], hi3[S][9] (rows padded by one word, so that the
  // one-thread-per-dimension stores hit distinct banks)
  extern __shared__ __align__(16) float var_sm[];
  float2* W = reinterpret_cast<float2*>(var_sm);
  float4* bw_s = reinterpret_cast<float4*>(W + (size_t)plan.rows * T);
  int4* bo_s = reinterpret_cast<int4*>(bw_s + S);
  uint2* up_s = reinterpret_cast<uint2*>(bo_s + S);  // {upper XOR, second point's XOR}
  uint32_t* lo4_s = reinterpret_cast<uint32_t*>(up_s + 2 * S);
  uint32_t* hi3_s = lo4_s + 17 * S;
  int* out_s = reinterpret_cast<int*>(hi3_s + 9 * S);  // byte offsets
  const int tid = threadIdx.x;
  const int f = blockIdx.y;
  const unsigned short* dim = plan.dim + f * kMaxSteps;
  int p0 = blockIdx.x * tiles * kVarTile;
  uint32_t h0 = (first_index + (uint32_t)p0) >> 7;
  // the second points' word for upper index h: Gray bit 6 and the bit that
  // gray(h + 1) = gray(h) ^ 2^ctz(h + 1) flips (indices below 2^31 + 256, so
  // ctz(h + 1) <= 24 and the direction number exists)
  auto second = [](const uint32_t* v, uint32_t h) {
    return __ldg(v + 6) ^ __ldg(v + 7 + (__ffs(h + 1u) - 1));
  };
  // one thread per Sobol dimension of the factor (the upper XORs with the
  // scrambler word)
  for (int i = tid; i < S; i += T) {
    const int d = dim[i];
    const uint32_t* v = dirs + 32 * d;
    uint32_t vl[7];
    uint32_t x = sobol_tables(v, h0, lo4_s + 17 * i, hi3_s + 9 * i, vl);
    if (d < scr_dims) x ^= __ldg(scr + d);
    const uint32_t d0 = second(v, h0), d1 = second(v, h0 + 1u);
    up_s[i] = make_uint2(x, d0);
    up_s[S + i] = make_uint2(x ^ d0 ^ vl[6], d1);
    bw_s[i] = make_float4(plan.lw[i], plan.rw[i], plan.sd[i], __int_as_float(plan.emits[i]));
    bo_s[i] = make_int4(plan.left[i] * kRow, plan.right[i] * kRow, plan.target[i] * kRow, 0);
    out_s[i] = plan.out_row[i] * kRow;
  }
  W[(size_t)(plan.rows - 1) * T + tid] = dup2(0.0f);
  __syncthreads();
  char* wb = reinterpret_cast<char*>(W + tid);
  for (int t = 0; t < tiles && p0 < paths; ++t) {
    const int p = p0 + tid;
    const uint32_t n = first_index + (uint32_t)p;
    const uint32_t glo = (n ^ (n >> 1)) & 127u;
    // this thread's entries of the Sobol tables, stage by stage
    const uint2* up_t = up_s + ((n >> 7) - h0) * S;
    const uint32_t* lo_t = lo4_s + (glo & 15u);
    const uint32_t* h3_t = hi3_s + (glo >> 4);
    const bool both = p + T < paths;
    float2 prev = dup2(0.0f);
    float* o = out + (size_t)f * paths + p;
    const size_t o_step = (size_t)F * paths;
    const int* next_out = out_s;
    // one batch of kVarBatch points from i0; FULL: all of them exist (no
    // clamp of the index, no guard on the bridge step)
    auto batch = [&](int i0, auto full_tag) {
      constexpr bool FULL = decltype(full_tag)::value;
      float2 z[kVarBatch];
#pragma unroll
      for (int k = 0; k < kVarBatch; ++k) {
        const int i = FULL ? i0 + k : min(i0 + k, S - 1);
        const uint2 u = up_t[i];
        const uint32_t x = u.x ^ lo_t[17 * i] ^ h3_t[9 * i];
        z[k] = icdf_sb_fast2(x, x ^ u.y);
      }
#pragma unroll
      for (int k = 0; k < kVarBatch; ++k) {
        const int i = i0 + k;
        if (FULL || i < S) {
          const float4 bw = bw_s[i];
          const int4 bo = bo_s[i];
          // bo: byte offsets of the rows (no index scaling per access)
          float2 y = __fmul2_rn(dup2(bw.x), *reinterpret_cast<const float2*>(wb + bo.x));
          y = __ffma2_rn(dup2(bw.y), *reinterpret_cast<const float2*>(wb + bo.y), y);
          y = __ffma2_rn(dup2(bw.z), z[k], y);
          *reinterpret_cast<float2*>(wb + bo.z) = y;
          // the points whose left subtree this one completes
          for (int c = __float_as_int(bw.w); c > 0; --c, ++next_out, o += o_step) {
            const float2 cur = *reinterpret_cast<const float2*>(wb + *next_out);
            o[0] = cur.x - prev.x;
            if (both) o[T] = cur.y - prev.y;
            prev = cur;
          }
        }
      }
    };
    if (p < paths) {
      int i0 = 0;
      for (; i0 + kVarBatch <= S; i0 += kVarBatch) batch(i0, std::true_type());
      if (i0 < S) batch(i0, std::false_type());
    }
    p0 += kVarTile;
    h0 += 2u;
    if (t + 1 < tiles && p0 < paths) {  // the next tile's upper XORs
      __syncthreads();
      for (int i = tid; i < S; i += T) {
        const uint32_t* v = dirs + 32 * dim[i];
        const uint2 last = up_s[S + i];  // of h0 - 1
        const uint32_t v6 = __ldg(v + 6);
        const uint32_t x = last.x ^ last.y ^ v6;
        const uint32_t d0 = second(v, h0), d1 = second(v, h0 + 1u);
        up_s[i] = make_uint2(x, d0);
        up_s[S + i] = make_uint2(x ^ d0 ^ v6, d1);
      }
      __syncthreads();
    }
  }
}

// Shared memory of variates_kernel.
inline size_t variates_smem_bytes(const VarPlan& p) {
  return (size_t)p.rows * kVarBlock * sizeof(float2) +
         (size_t)p.steps * (sizeof(float4) + sizeof(int4) + 2 * sizeof(uint2) +
                            (17 + 9 + 1) * sizeof(uint32_t));
}

// The same variates level by level, one path per thread and one tile of 128
// paths per CTA, with a row of shared memory per point: for launches whose
// CTAs leave the SMs nearly empty, which last as long as one thread's chain.
// Depth first every point waits for the point before it, and the increments
// come out in between; level by level the points of a level are independent.
// On the device, depth first and so: 80 steps, 10 factors 16.7 -> 8.7 us at
// 1,000 paths, 18.7 -> 13.8 at 4,099; 128 steps, 16 factors 24.2 -> 12.5 us at
// 1,000; 40 steps, 5 factors 9.7 -> 7.0 us at 4,099.
__global__ void __launch_bounds__(kVarBlock)
    variates_levels_kernel(int paths, uint32_t first_index, const uint32_t* __restrict__ dirs,
                           const uint32_t* __restrict__ scr, int scr_dims,
                           float* __restrict__ out, const __grid_constant__ BridgePlan plan) {
  constexpr int T = kVarBlock;
  const int S = plan.steps, F = plan.factors;
  // shared memory (variates_levels_smem_bytes): the bridge points W[S + 1][T]
  // (row S stays zero: the neighbour of a point that has none), the plan per
  // stage as {lw, rw, sd} weights and {left row, right row, target row} byte
  // offsets into W, and the Sobol tables hi[2][S], lo4[S][17], hi3[S][9]
  extern __shared__ __align__(16) float var_sm[];
  float* const W = var_sm;
  float4* bw_s = reinterpret_cast<float4*>(W + (size_t)(S + 1) * T);
  int4* bo_s = reinterpret_cast<int4*>(bw_s + S);
  uint32_t* hi_s = reinterpret_cast<uint32_t*>(bo_s + S);
  uint32_t* lo4_s = hi_s + 2 * S;
  uint32_t* hi3_s = lo4_s + 17 * S;
  const int f = blockIdx.y, tid = threadIdx.x;
  const int* alloc = plan.alloc + f * S;
  const int p0 = blockIdx.x * T;
  const uint32_t h0 = (first_index + (uint32_t)p0) >> 7;
  for (int i = tid; i < S; i += T) {
    const int d = alloc[i];
    const uint32_t* v = dirs + 32 * d;
    uint32_t vl[7];
    uint32_t x = sobol_tables(v, h0, lo4_s + 17 * i, hi3_s + 9 * i, vl);
    if (d < scr_dims) x ^= __ldg(scr + d);
    hi_s[i] = x;
    // that of h0 + 1, which differs in one Gray bit (no entry past bit 31:
    // h0 + 1 = 2^25 has no path)
    const int c = __ffs(h0 + 1u) - 1;
    hi_s[S + i] = (c >= 0 && c < 25) ? x ^ __ldg(v + 7 + c) : x;
    // stage 0 is the terminal point W_S = sd_0 z (row S - 1)
    const int jl = i == 0 ? 0 : plan.left[i];
    bw_s[i] = make_float4(jl != 0 ? plan.lw[i] : 0.0f, i == 0 ? 0.0f : plan.rw[i], plan.sd[i],
                          0.0f);
    bo_s[i] = make_int4((jl != 0 ? jl - 1 : S) * T * 4, (i == 0 ? S : plan.right[i]) * T * 4,
                        (i == 0 ? S - 1 : plan.bidx[i]) * T * 4, 0);
  }
  W[(size_t)S * T + tid] = 0.0f;
  __syncthreads();
  const int p = p0 + tid;
  if (p >= paths) return;
  const uint32_t n = first_index + (uint32_t)p;
  const uint32_t glo = (n ^ (n >> 1)) & 127u;
  char* const wb = reinterpret_cast<char*>(W + tid);
  // this thread's entries of the Sobol tables, stage by stage
  const uint32_t* hi_t = hi_s + ((n >> 7) - h0) * S;
  const uint32_t* lo_t = lo4_s + (glo & 15u);
  const uint32_t* h3_t = hi3_s + (glo >> 4);
  // one batch of kVarBatch stages from i0; FULL: all of them exist
  auto batch = [&](int i0, auto full_tag) {
    constexpr bool FULL = decltype(full_tag)::value;
    float z[kVarBatch];
#pragma unroll
    for (int k = 0; k < kVarBatch; ++k) {
      const int i = FULL ? i0 + k : min(i0 + k, S - 1);
      z[k] = icdf_sb_fast(hi_t[i] ^ lo_t[17 * i] ^ h3_t[9 * i]);
    }
#pragma unroll
    for (int k = 0; k < kVarBatch; ++k) {
      const int i = i0 + k;
      if (FULL || i < S) {
        const float4 bw = bw_s[i];
        const int4 bo = bo_s[i];
        float y = bw.x * *reinterpret_cast<const float*>(wb + bo.x);
        y = fmaf(bw.y, *reinterpret_cast<const float*>(wb + bo.y), y);
        y = fmaf(bw.z, z[k], y);
        *reinterpret_cast<float*>(wb + bo.z) = y;
      }
    }
  };
  int i0 = 0;
  for (; i0 + kVarBatch <= S; i0 += kVarBatch) batch(i0, std::true_type());
  if (i0 < S) batch(i0, std::false_type());
  float prev = 0.0f;
  float* o = out + (size_t)f * paths + p;
  for (int s = 0; s < S; ++s, o += (size_t)F * paths) {
    const float cur = W[s * T + tid];
    *o = cur - prev;
    prev = cur;
  }
}

// Shared memory of variates_levels_kernel.
inline size_t variates_levels_smem_bytes(int S) {
  return (size_t)(S + 1) * kVarBlock * sizeof(float) +
         (size_t)S * (sizeof(float4) + sizeof(int4) + (2 + 17 + 9) * sizeof(uint32_t));
}

}  // namespace lmm

namespace lmm {

// One period of the target redemption note for a path (the reference's
// TARN::getCashFlows, cashFlowGeneration_product_gpu.h:57-98, accruals =
// tau): returns the period's net flow (floating received plus coupon paid,
// at T_{s+1}); `paid` and `over` carry the path's state.
__device__ __forceinline__ float tarn_flow(const ProductConst& pc, int s, int n, float tau,
                                           float f, float& paid, bool& over) {
  if (over) return 0.0f;
  const float flow2 = tau * f;
  float flow1;
  if (s + 1 == n) {
    flow1 = paid - pc.tarn_total;
    over = true;
  } else {
    const float c = fmaxf((pc.strike - pc.tarn_mult * f) * tau, 0.0f);
    const float total = paid + c;
    if (total >= pc.tarn_total) {
      flow1 = paid - pc.tarn_total;
      over = true;
    } else {
      flow1 = -c;
      paid = total;
    }
  }
  return flow1 + flow2;
}

// Pseudo-root columns past the factors stay zero.
template <int FP, int T>
__device__ __forceinline__ void zero_row_pads(float* As, int rows, int F) {
  if (F < FP)
    for (int i = threadIdx.x; i < rows * (FP - F); i += T) {
      const int r = i / (FP - F);
      As[r * FP + F + (i - r * (FP - F))] = 0.0f;
    }
}

// Starts the copy of step s's alive pseudo-root rows and fixed drifts
// (cp.async, one group).
template <int FT, int FP, int T>
__device__ __forceinline__ void stage_rows(float* As, float* fx, const float* __restrict__ A,
                                           const float* __restrict__ fixed, int s, int n,
                                           int F_) {
  const int F = FT > 0 ? FT : F_;
  const float* src = A + ((size_t)s * n + s) * F;
  const int alive = n - s;
  if (F % 2 == 0 && ((uintptr_t)A & 7u) == 0) {
    for (int i = threadIdx.x; i < alive * (F / 2); i += T) {
      const int r = i / (F / 2);
      cp_async8(As + r * FP + 2 * (i - r * (F / 2)), src + 2 * i);
    }
  } else {
    for (int i = threadIdx.x; i < alive * F; i += T) {
      const int r = i / F;
      cp_async4(As + r * FP + (i - r * F), src + i);
    }
  }
  for (int i = threadIdx.x; i < alive; i += T)
    cp_async4(fx + i, fixed + (size_t)s * n + s + i);
  cp_async_commit();
}

// ---------------------------------------------------------------------------
// Fused evolution.  One thread per path, CTA of 128 paths; shared memory
// holds the CTA's log-rates [rate][thread] and the alive rows of the step's
// pseudo-root (padded to a multiple of 4 factors for 16-byte loads) and
// fixed drift.  Launches too small for two paths per thread (fused_pairs.cuh)
// run it, with a few warps per SM or fewer, so a step must not wait for
// memory: its rows are copied one step ahead into the other of two buffers
// (cp.async; one barrier per step) and its normals loaded one step ahead.
// With both and the exercise rule's known tables (launches bound by latency):
// 20 rates, 3 factors, 16,384 paths 52 -> 46 us with the variates; 80 rates,
// 10 factors, 16,384 paths 0.470 -> 0.366 ms, the frozen-rule chain 0.80 ->
// 0.60 ms; 120 rates, 15 factors, 10,000 paths, the chain 1.72 -> 1.23 ms.
// Per rate and step: predictor drift from the rates at the start of
// the step, predicted log-rate, corrector drift, corrected and capped
// log-rate (LMM_evolver_all.cu:615-744, gold/LMM_evolver_gold.h:315-387);
// the spot drift factor is g = F tau / (1 + f tau) with F = f + d the
// displaced rate.  At exercise steps the discount ratios P(T_s, T_{r+1}),
// the coterminal annuity and swap rate are accumulated on the fly.
// FT = number of factors (compile time), 0 = generic <= 16.
//
// AHEAD costs registers and a second row buffer, so CTAs per SM.  Where not all
// CTAs fit the SMs at once the other CTAs hide the loads, and the form without
// it (rows and normals at the start of the step) holds more: 128 rates, 10
// factors, 40,001 paths 1.85 against 1.40 ms (two against three CTAs per SM); 12
// rates, 2 factors, 75,776 paths 61 against 50 us; 20 rates, 3 factors, the
// European strip of 110,001 paths 87 against 70 us.
// ---------------------------------------------------------------------------
template <int FT, bool AHEAD>
struct FusedShape {  // CTAs per SM that the registers have to allow
  static constexpr int kCtas = AHEAD ? (FT == 3 || FT == 5 ? 5 : 3)
                                     : FT == 3 ? 7 : FT == 5 ? 6 : 5;
};

template <int FT, int MODE, bool AHEAD>
__global__ void __launch_bounds__(kFusedBlock, FusedShape<FT, AHEAD>::kCtas)
    fused_evolve_kernel(int paths, const float* __restrict__ Z,
                        const float* __restrict__ A,
                        const float* __restrict__ fixed,
                        const __grid_constant__ ModelConst mc,
                        const __grid_constant__ ProductConst pc,
                        const __grid_constant__ RuleConst rc,
                        const LsRuleView rule, int total, int col0,
                        float* __restrict__ o_vars, float* __restrict__ o_ex,
                        float* __restrict__ o_cf, float* __restrict__ o_num,
                        float* __restrict__ o_payoff, const RecordOut rec,
                        const SegIO seg) {
  constexpr int FM = FPad<FT>::FM;
  constexpr int FP = FPad<FT>::FP;
  const int F = FT > 0 ? FT : mc.F;
  const int n = mc.n;
  constexpr int T = kFusedBlock;
  const int tid = threadIdx.x;
  // the frozen-rule modes stop a path at its exercise and run in segments
  constexpr bool kSeg = MODE == kModeRule || MODE == kModeRecord;
  const bool resume = kSeg && seg.in_prefix != nullptr;
  const int s_begin = resume ? seg.s_begin : 0;
  const int s_end = kSeg ? seg.s_end : n;
  const int rows = n - s_begin;  // rates alive in this launch
  extern __shared__ __align__(16) float sm[];
  constexpr int kBufs = AHEAD ? 2 : 1;
  float* const As_b = sm;                        // [kBufs][rows][FP]: row r - s of step s
  float* const fx_b = As_b + kBufs * rows * FP;  // [kBufs][rows (+ pad)]
  const int fx_rows = (rows + 3) & ~3;
  // [rows][T], indexed by rate from s_begin on
  float* const lfs = fx_b + kBufs * fx_rows - s_begin * T;
  int p = blockIdx.x * T + tid, src = 0;
  bool valid = p < paths;
  if (resume) {
    // survivor slot j of the previous segment, found in its CTA's block
    const int live = __ldg(seg.in_prefix + seg.in_blocks);
    if (blockIdx.x * T >= live) {  // no survivor slot here: uniform over the CTA
      if (tid == 0 && seg.out.rates != nullptr) seg.out_count[blockIdx.x] = 0;
      return;
    }
    const int j = blockIdx.x * T + tid;
    valid = j < live;
    p = 0;
    if (valid) {
      int lo = 0, hi = seg.in_blocks;  // in_prefix[lo] <= j < in_prefix[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(seg.in_prefix + mid) <= j) lo = mid; else hi = mid;
      }
      src = lo * T + (j - __ldg(seg.in_prefix + lo));
      p = seg.in.path[src];
      if ((unsigned)p >= (unsigned)paths) {  // never for a consistent chain
        valid = false;
        p = 0;
      }
    }
  }
  zero_row_pads<FP, T>(As_b, kBufs * rows, F);
  // copies step s's alive rows into buffer b
  auto stage = [&](int s, int b) {
    stage_rows<FT, FP, T>(As_b + b * rows * FP, fx_b + b * fx_rows, A, fixed, s, n, F);
  };
  if (AHEAD) stage(s_begin, 0);
  float N = 1.0f, f_first = 0.0f, cf_acc = 0.0f, N_bucket = 1.0f;
  int bucket = -1, ex_at = n;
  double payoff = 0.0;
  float tarn_paid = 0.0f;
  bool tarn_over = false;
  bool done = !valid;
  // swaption-plus-cap portfolio: after the swaption's exercise the path runs
  // on for the cap strip, with no further exercise dates
  bool exercised = false;
  const int col = col0 + p;
  // An exercise date's discount curve P(T_s, T_{r+1}), r >= s, is completed
  // in the next step's rate loop, which forms 1 / (1 + tau_r f_r) of every
  // later rate for its drift factors anyway (pc_rate's q); the date's
  // epilogue therefore runs one step later, from this pending state.
  int pend_e = -1, pend_s = 0;
  float pend_N = 1.0f, pend_f = 0.0f, pend_P1 = 1.0f, pend_coupon = 0.0f;
  if (!resume) {
    for (int r = 0; r < n; ++r) lfs[r * T + tid] = mc.logf0[r];
  } else {
    for (int r = s_begin; r < n; ++r)
      lfs[r * T + tid] = valid ? seg.in.rates[(size_t)r * seg.cap + src] : 0.0f;
    if (valid) {
      N = seg.in.N[src];
      f_first = seg.in.f_first[src];
      payoff = seg.in.payoff[src];
      const int e = pc.ex_index[s_begin - 1];
      if (e >= 0) {  // the date of step s_begin - 1 waits for this step's curve
        pend_e = e;
        pend_s = s_begin - 1;
        pend_N = N;
        pend_f = f_first;
        pend_P1 = seg.in.pend_P1[src];
        pend_coupon = seg.in.pend_coupon[src];
      }
    }
  }
  auto date_epilogue = [&](float Pn, float ann) {
    const int e = pend_e;
    float v[kMaxVars], exv = 0.0f;
    if (pc.kind == LMM_PRODUCT_SWAPTION || pc.kind == LMM_PRODUCT_BERMUDAN_CAP) {
      const float sr = (1.0f - Pn) / ann;
      v[0] = pend_f;
      v[1] = sr;
      v[2] = ann;
      exv = fmaxf((sr - pc.strike) * ann, 0.0f);
    } else {
      float sr;
      if (pend_s + 1 < n) {
        const float ann2 = ann - mc.tau[pend_s] * pend_P1;
        sr = (pend_P1 - Pn) / ann2;
      } else {
        sr = (1.0f - Pn) / ann;
      }
      v[0] = pend_f;
      v[1] = sr;
      v[2] = mc.tau[n - 1] * Pn;
    }
    pend_e = -1;
    if (MODE == kModeInputs || MODE == kModeOuter) {
      if (bucket >= 0) o_cf[(size_t)bucket * total + col] = cf_acc;
      bucket = e;
      cf_acc = pend_coupon;
#pragma unroll
      for (int k = 0; k < kMaxVars; ++k)
        o_vars[((size_t)e * kMaxVars + k) * total + col] = v[k];
      o_ex[(size_t)e * total + col] = exv;
      o_num[(size_t)e * total + col] = pend_N;
    } else {
      const double est = rule_estimate(rc, e, v, exv, rule);
      if ((double)exv > est) {
        payoff += (double)exv / (double)pend_N;
        if (MODE == kModeRecord) ex_at = pend_s;
        if (pc.kind == LMM_PRODUCT_BERMUDAN_CAP)
          exercised = true;
        else
          done = true;
        return;
      }
      payoff += (double)pend_coupon / (double)pend_N;
    }
    N_bucket = pend_N;
  };
  float z_next[FP];
  auto load_normals = [&](int s) {
#pragma unroll
    for (int f = 0; f < FP; ++f)
      z_next[f] = (f < F && !done) ? __ldg(Z + ((size_t)s * F + f) * paths + p) : 0.0f;
  };
  if (AHEAD) load_normals(s_begin);
  for (int s = s_begin; s < s_end; ++s) {
    if (!AHEAD) {
      load_normals(s);
      __syncthreads();  // every warp is past the step before's rows
      stage(s, 0);
    }
    cp_async_wait<0>();
    __syncthreads();  // this step's rows are in; the other buffer is free
    const int buf = AHEAD ? (s - s_begin) & 1 : 0;
    float z[FP];
#pragma unroll
    for (int f = 0; f < FP; ++f) z[f] = z_next[f];
    if (AHEAD && s + 1 < s_end) {
      stage(s + 1, buf ^ 1);
      load_normals(s + 1);
    }
    if (done) continue;
    const float* As = As_b + buf * rows * FP;
    const float* fx = fx_b + buf * fx_rows;
    if (s > 0) N = N * (1.0f + mc.tau[s - 1] * f_first);
    if ((MODE == kModeRecord || MODE == kModeOuter) && s % rec.every == 0) {
      const int c = s / rec.every;
      for (int r = s; r < n; ++r)
        rec.ckpt[((size_t)c * n + r) * paths + p] = lfs[r * T + tid];
      rec.ckptN[(size_t)c * paths + p] = N;
    }
    const bool pend = pend_e >= 0;
    float Pd = pend_P1, annd = pend ? mc.tau[s - 1] * pend_P1 : 0.0f;
    float2 w[FP / 2], v[FP / 2];
    step_start<FP>(z, w, v);
    // the rate loop, unswitched on whether a date's curve is pending
    auto rate_loop = [&](auto with_curve) {
#pragma unroll 4
      for (int r = s; r < n; ++r) {
        const float tau = mc.tau[r];
        float g, gp, q;
        bool capped;
        const float lf = pc_rate<FM, FP>(lfs[r * T + tid], mc.l2tau[r], mc.c0[r], fx[r - s],
                                         As + (r - s) * FP, w, v, mc.cutoff, g, gp, q, capped);
        lfs[r * T + tid] = lf;
        if (decltype(with_curve)::value) {
          Pd *= q;
          annd += tau * Pd;
        }
      }
    };
    if (pend)
      rate_loop(std::true_type{});
    else
      rate_loop(std::false_type{});
    f_first = __expf(lfs[s * T + tid]) - mc.disp[s];
    const float P1 = __fdividef(1.0f, 1.0f + mc.tau[s] * f_first);
    // ---- the previous step's exercise date, then the epilogue at T_s ----
    if (pend) {
      date_epilogue(Pd, annd);
      if (done) continue;
    }
    if (pc.kind == LMM_PRODUCT_TARN) {
      payoff += (double)(tarn_flow(pc, s, n, mc.tau[s], f_first, tarn_paid, tarn_over) * P1) /
                (double)N;
      continue;
    }
    if (pc.kind == LMM_PRODUCT_EUROPEAN) {
      const float tau = mc.tau[s];
      const float cap = tau * fmaxf(f_first - pc.cap_strike, 0.0f);
      const float swp = tau * (f_first - pc.strike) * pc.pay_receive;
      payoff += (double)((cap + swp) * P1) / (double)N;
      continue;
    }
    if (pc.kind == LMM_PRODUCT_BERMUDAN_CAP && (MODE == kModeRule || MODE == kModeRecord)) {
      // the portfolio's caplet on f_s, paid at T_{s+1} whether or not the
      // swaption has been exercised
      const float cap = mc.tau[s] * fmaxf(f_first - pc.cap_strike, 0.0f);
      payoff += (double)(cap * P1) / (double)N;
    }
    float coupon = 0.0f;
    if (pc.kind == LMM_PRODUCT_CANCELLABLE_SWAP)
      coupon = mc.tau[s] * (f_first - pc.strike) * pc.pay_receive * P1;
    const int e = exercised ? -1 : pc.ex_index[s];
    if (e >= 0) {
      pend_e = e;
      pend_s = s;
      pend_N = N;
      pend_f = f_first;
      pend_P1 = P1;
      pend_coupon = coupon;
    } else if (coupon != 0.0f) {
      if (MODE == kModeInputs || MODE == kModeOuter) {
        if (bucket >= 0) cf_acc += coupon * (N_bucket / N);
      } else {
        payoff += (double)coupon / (double)N;
      }
    }
  }
  if (kSeg && seg.out.rates != nullptr) {
    // end of a segment: pack the survivors of this CTA in path order (the
    // per-warp counts go to the pseudo-root rows, free once every warp is
    // past its last step)
    int* warp_live = reinterpret_cast<int*>(As_b);
    const bool live = valid && !done;
    const unsigned bal = __ballot_sync(0xffffffffu, live);
    const int warp = tid >> 5, lane = tid & 31;
    __syncthreads();
    if (lane == 0) warp_live[warp] = __popc(bal);
    __syncthreads();
    int off = 0, tot = 0;
    for (int w = 0; w < (T >> 5); ++w) {
      const int c = warp_live[w];
      off += w < warp ? c : 0;
      tot += c;
    }
    if (live) {
      const int slot = blockIdx.x * T + off + __popc(bal & ((1u << lane) - 1u));
      for (int r = s_end; r < n; ++r)
        seg.out.rates[(size_t)r * seg.cap + slot] = lfs[r * T + tid];
      seg.out.N[slot] = N;
      seg.out.f_first[slot] = f_first;
      seg.out.pend_P1[slot] = pend_P1;
      seg.out.pend_coupon[slot] = pend_coupon;
      seg.out.payoff[slot] = payoff;
      seg.out.path[slot] = p;
    }
    if (tid == 0) seg.out_count[blockIdx.x] = tot;
    if (valid && done) {
      o_payoff[p] = (float)payoff;
      if (MODE == kModeRecord) rec.ex_step[p] = ex_at;
    }
    return;
  }
  // an exercise date at the last step: its curve is the one period
  if (!done && pend_e >= 0) date_epilogue(pend_P1, mc.tau[n - 1] * pend_P1);
  if (!valid) return;
  if (MODE == kModeInputs || MODE == kModeOuter) {
    if (pc.kind != LMM_PRODUCT_EUROPEAN && bucket >= 0)
      o_cf[(size_t)bucket * total + col] = cf_acc;
    if ((pc.kind == LMM_PRODUCT_EUROPEAN || pc.kind == LMM_PRODUCT_TARN) && o_payoff)
      o_payoff[p] = (float)payoff;
  } else {
    o_payoff[p] = (float)payoff;
    if (MODE == kModeRecord) rec.ex_step[p] = ex_at;
  }
}

// Exclusive prefix of the per-CTA survivor counts of a segment launch
// (prefix[blocks] = survivors), one CTA: each thread sums a contiguous run
// of counts, the runs' sums are scanned across warps, then written back.
__global__ void __launch_bounds__(1024)
    seg_scan_kernel(const int* __restrict__ count, int blocks, int* __restrict__ prefix) {
  __shared__ int warp_sum[32];
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = (blocks + T - 1) / T;
  const int b0 = min(tid * chunk, blocks), b1 = min(b0 + chunk, blocks);
  int local = 0;
  for (int b = b0; b < b1; ++b) local += count[b];
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int w = lane < (T >> 5) ? warp_sum[lane] : 0;
    int x = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += t;
    }
    if (lane < (T >> 5)) warp_sum[lane] = x - w;
  }
  __syncthreads();
  int run = warp_sum[warp] + incl - local;
  for (int b = b0; b < b1; ++b) {
    prefix[b] = run;
    run += count[b];
  }
  if (tid == T - 1) prefix[blocks] = run;
}

// Padded pseudo-root row (floats) of the instantiation launched for F
// factors: 3, 5, 10 and 15 have their own instantiations; every other count
// runs the generic one, whose rows are padded for kMaxFactors.  Shared
// memory must be sized by this, not by F.
inline int launched_fm(int F) {
  return (F == 3 || F == 5 || F == 10 || F == 15) ? F : kMaxFactors;
}
inline int launched_row_pad(int F) { return (launched_fm(F) + 3) & ~3; }

// Shared memory of the fused evolution kernel for `rows` alive rates.
inline size_t fused_smem_bytes(int rows, int F, bool ahead) {
  const size_t stage = (size_t)rows * launched_row_pad(F) + ((rows + 3) & ~3);
  return ((ahead ? 2 : 1) * stage + (size_t)rows * kFusedBlock) * sizeof(float);
}
// The same with one buffer (greeks_segment_kernel).
inline size_t segment_smem_bytes(int rows, int F, int block) {
  const size_t stage = (size_t)rows * launched_row_pad(F) + ((rows + 3) & ~3);
  return (stage + (size_t)rows * block) * sizeof(float);
}

}  // namespace lmm
