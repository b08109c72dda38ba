// Device code of the GLM likelihood shared by its kernels (glm.cu: one
// launch per evaluation or per block of independent chains; glm_loop.cu:
// whole blocks of integrator steps): the link functions, the row tile
// arithmetic and the sums behind U and var(lk).  Kernels that cut a minibatch
// into the same slices, warps and row tiles give the same bits.
#pragma once

#include "common.cuh"
#include "internal.h"

namespace gbsgmc {


enum Mode { kValueGrad = 0, kSgldStep = 1 };

struct GlmArgs {
  int family, d, dq;
  int y_inline;
  int64_t n_obs, n_rows, ld;
  const float* X;
  const float* y;
  float inv_s2;     // 1/sigma^2 (linear-Gaussian)
  float log_norm;   // log sigma + 0.5 log 2 pi (linear-Gaussian)
  float inv_p2;     // 1/prior_scale^2, 0 for a flat prior
  double prior_const;  // d * (log s + 0.5 log 2 pi), 0 for a flat prior
  float inv_temp;
  float scale;      // N / n
  int chains, n, slices, rows_per_slice;
  const int32_t* idx;
  int64_t idx_stride;
  int steps;                // SGLD steps per launch (> 1: one CTA per chain)
  int64_t idx_step_stride;  // elements between the index sets of two steps
  const float* mask;
  int mode;
  float* w;
  float* v;
  float alpha, lmbd;
  Sched sched;
  Noise noise;
  double* U;
  float* grad;
  float* lk;
  double* lk_var;
  float* samples;
  double* sample_lik;
  float4* ws_part;
  double* ws_sums;
  unsigned* ws_ticket;
  void* ws_base;
  size_t ws_size;
  int slices_fixed;   // > 0: slices per chain chosen by the caller
  int rw_fixed;       // > 0: rows per warp chosen by the caller
  int warps_fixed;    // > 0: warps per CTA chosen by the caller
  int pf_fixed;       // 1: prefetching variant, -1: not, 0: library choice
  int dyn_fixed;      // 1: dynamically scheduled kernel, -1: not, 0: library choice
  int* status;
  int vec4;   // rows are 16-byte aligned: 128-bit loads
  // Replica exchange: chain c's index row and noise stream belong to chain
  // ident[c] (the states that moved into c with an exchange); NULL: c itself.
  const int32_t* ident;
};

// Checks a model and its minibatches and fills the arguments common to every
// GLM kernel.
int glm_fill_args(GlmArgs& a, const gbsgmc_glm* m, int chains, int n, const int32_t* idx,
                  int64_t idx_stride, const float* mask, void* ws, size_t ws_size, int* status,
                  GlmTune tune);

// The chain whose index row and noise stream chain (slot) c uses.
__device__ __forceinline__ int ident_of(const GlmArgs& a, int c) {
  return a.ident != nullptr ? __ldg(a.ident + c) : c;
}

// Bernoulli-logit log-likelihood y z - softplus(z) and its derivative
// y - sigmoid(z), from one exponential: e = exp(-|z|),
// softplus(z) = max(z, 0) + log1p(e), sigmoid(z) = 1/(1+e) or e/(1+e).
// Without `want` lk is only a number that is finite where the likelihood is.
__device__ __forceinline__ void logistic_link(float z, float y, bool want, float& lk,
                                              float& dz) {
  const float e = expf(-fabsf(z));
  const float r = 1.0f / (1.0f + e);
  lk = want ? y * z - (fmaxf(z, 0.0f) + log1pf(e)) : z * 1e-6f;
  dz = y - (z >= 0.0f ? r : e * r);
}

// 128-bit read-only load that does not allocate in L1 (rows are read once).
__device__ __forceinline__ float4 ld_row4(const float* p) {
  float4 v;
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(p));
  return v;
}

__device__ __forceinline__ float ld_row1(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// 4-byte asynchronous copy global -> shared (completes in the background;
// cp_async_wait_all waits for the calling thread's copies).
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int RW>
struct Log2;
template <>
struct Log2<1> { static constexpr int v = 0; };
template <>
struct Log2<2> { static constexpr int v = 1; };
template <>
struct Log2<4> { static constexpr int v = 2; };
template <>
struct Log2<8> { static constexpr int v = 3; };
template <>
struct Log2<16> { static constexpr int v = 4; };

// Sum of p[r] over the 32 lanes for RW rows at once.  Returns, in every lane
// of group g = lane >> (5 - log2 RW), the full sum of row g.
template <int RW>
__device__ __forceinline__ float transposed_warp_sum(float (&p)[RW], int lane) {
  constexpr int LOG = Log2<RW>::v;
#pragma unroll
  for (int t = 0; t < LOG; ++t) {
    const int o = 16 >> t;
    const int half = RW >> (t + 1);
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? p[i] : p[i + half];
      const float keep = upper ? p[i + half] : p[i];
      p[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  float z = p[0];
#pragma unroll
  for (int o = 16 >> LOG; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
  return z;
}

// Per-lane accumulators of one CTA row stream.  The likelihood sums stay in
// fp32 per lane (a lane sees a few dozen rows); reduce_lane_sums makes fp64
// totals of them.  GB300's fp64 pipe runs at a small fraction of the fp32 rate,
// so per-row fp64 arithmetic would throttle the kernel.
//
// The sum of the (masked) likelihoods that makes U is compensated: each
// addition's rounding error is carried in mlk_c (Neumaier's variant of
// Kahan summation, A. Neumaier 1974), so a lane's sum is good to about one
// rounding of its total whatever its row count.  Once the sum overflows the
// correction is dropped, so an infinite likelihood sum stays infinite (the
// MH tests reject such a proposal) instead of turning into inf - inf.
//
// The variance needs E[lk^2] - E[lk]^2, which cancels badly when |lk| is
// large, so each lane sums around its first value K: s1 = sum(lk - K),
// s2 = sum((lk - K)^2); the widening to fp64 restores sum(lk) and sum(lk^2).
template <int QPL>
struct Accum {
  float4 acc[QPL];
  float mlk, mlk_c, K, s1, s2;
  int cnt;
};

__device__ __forceinline__ void neumaier_add(float& sum, float& comp, float x) {
  const float t = sum + x;
  const float e = fabsf(sum) >= fabsf(x) ? (sum - t) + x : (x - t) + sum;
  comp += isfinite(t) ? e : 0.0f;
  sum = t;
}

// Likelihood, adjoint and accumulation for a loaded tile (see load_tile).
// Without `want` (no U or var(lk) asked of this gradient) only what the
// adjoint needs is computed, and A.mlk turns non-finite where a likelihood
// would: about a third of the logistic link is its log1p and the
// compensated sums.
template <int QPL, int RW>
__device__ __forceinline__ void consume_tile(const GlmArgs& a, const float* m_s,
                                             float* lk_out, int r0, int lane,
                                             int g, bool leader, bool want,
                                             const float4 (&wq)[QPL],
                                             const float4 (&xv)[RW][QPL],
                                             float yv, int og, Accum<QPL>& A) {
  constexpr int GROUP = 32 / RW;
  float p[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    float z = 0.0f;
#pragma unroll
    for (int k = 0; k < QPL; ++k) {
      z = fmaf(xv[r][k].x, wq[k].x, z);
      z = fmaf(xv[r][k].y, wq[k].y, z);
      z = fmaf(xv[r][k].z, wq[k].z, z);
      z = fmaf(xv[r][k].w, wq[k].w, z);
    }
    p[r] = z;
  }
  const float z = transposed_warp_sum<RW>(p, lane);
  const bool ok = og >= 0;
  const int row = r0 + g;
  const float mw = (ok && a.mask != nullptr) ? m_s[row] : 1.0f;
  float lkv, dz;
  if (a.family == GBSGMC_GLM_LOGISTIC) {
    logistic_link(z, yv, want, lkv, dz);
  } else if (a.family == GBSGMC_GLM_LINEAR) {
    lkv = z;
    dz = 1.0f;
  } else {
    const float res = yv - z;
    lkv = -0.5f * res * res * a.inv_s2 - a.log_norm;
    dz = res * a.inv_s2;
  }
  const float coef = ok ? mw * dz : 0.0f;
  if (ok && leader) {
    if (want) {
      neumaier_add(A.mlk, A.mlk_c, mw * lkv);
      if (A.cnt == 0) A.K = lkv;
      const float dk = lkv - A.K;
      A.s1 += dk;
      A.s2 = fmaf(dk, dk, A.s2);
      A.cnt += 1;
      if (lk_out != nullptr) lk_out[row] = lkv;
    } else {
      A.mlk += mw * lkv;
    }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const float cr = __shfl_sync(0xffffffffu, coef, r * GROUP);
#pragma unroll
    for (int k = 0; k < QPL; ++k) {
      A.acc[k].x = fmaf(cr, xv[r][k].x, A.acc[k].x);
      A.acc[k].y = fmaf(cr, xv[r][k].y, A.acc[k].y);
      A.acc[k].z = fmaf(cr, xv[r][k].z, A.acc[k].z);
      A.acc[k].w = fmaf(cr, xv[r][k].w, A.acc[k].w);
    }
  }
}

// The likelihood sums of one lane that owned rows (a tile group's leader), as
// the kernels hand them to the warp that reduces them.
struct LaneSums {
  float mlk, mlk_c, K, s1, s2;
  int cnt;
};

template <int QPL>
__device__ __forceinline__ LaneSums lane_sums(const Accum<QPL>& A) {
  return LaneSums{A.mlk, A.mlk_c, A.K, A.s1, A.s2, A.cnt};
}

// Totals of `count` lanes' sums by one warp: t[0] = sum m lk, t[1] = sum lk,
// t[2] = sum lk^2 (every lane gets them).  The widening restores sum(lk) =
// s1 + n K and sum(lk^2) = s2 + 2 K s1 + n K^2.  A warp's FP64 instruction
// takes some 64 cycles here, so the lanes add floats in three parts, to more
// bits than FP64 has, and only the totals become FP64, a lane each (16 tiles of
// 4 rows: 3,280 cycles in FP64); sums that are not finite take the FP64 path,
// which keeps infinities what they are.
__device__ __forceinline__ void reduce_lane_sums(const LaneSums* v, int count, int lane,
                                                 double (&t)[3]) {
  Float3Sum f[3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  bool fine = true;
  for (int i = lane; i < count; i += 32) {
    const LaneSums s = v[i];
    const float n_l = static_cast<float>(s.cnt);   // exact: a lane's rows are few
    const Float2Sum nk = two_prod(n_l, s.K), ks = two_prod(2.0f * s.K, s.s1);
    const Float2Sum nkk = two_prod(nk.hi, s.K), rest = two_prod(nk.lo, s.K);
    f[0].add(Float2Sum{s.mlk, s.mlk_c});
    f[1].add(nk);
    f[1].add(s.s1);
    f[2].add(nkk);
    f[2].add(ks);
    f[2].add(s.s2);
    f[2].add_mid(rest.hi);
    f[2].lo = __fadd_rn(f[2].lo, rest.lo);
    // Far from overflow: |values| below 2^96.
    fine = fine && fabsf(s.mlk) < 7.9e28f && fabsf(nkk.hi) < 7.9e28f && fabsf(s.s2) < 7.9e28f &&
           fabsf(ks.hi) < 7.9e28f;
  }
  if (__all_sync(0xffffffffu, fine)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k] = warp_sum(f[k]);
    const double mine = widen(lane == 1 ? f[1] : lane == 2 ? f[2] : f[0]);
#pragma unroll
    for (int k = 0; k < 3; ++k) t[k] = __shfl_sync(0xffffffffu, mine, k);
    return;
  }
  t[0] = t[1] = t[2] = 0.0;
  for (int i = lane; i < count; i += 32) {
    const LaneSums s = v[i];
    const double K = s.K, n_l = s.cnt;
    t[0] += static_cast<double>(s.mlk) + s.mlk_c;
    t[1] += static_cast<double>(s.s1) + n_l * K;
    t[2] += static_cast<double>(s.s2) + 2.0 * K * s.s1 + n_l * K * K;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) t[k] = warp_sum(t[k]);
}

// FP64 totals of a chain's slices ([slices, 4], three used) by one warp.
__device__ __forceinline__ void sum_slices(const double* ps, int slices, int lane,
                                           double (&t)[3]) {
  t[0] = t[1] = t[2] = 0.0;
  for (int s = lane; s < slices; s += 32) {
#pragma unroll
    for (int k = 0; k < 3; ++k) t[k] += __ldcg(ps + s * 4 + k);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) t[k] = warp_sum(t[k]);
}

// sum(w^2) of one warp's lanes holding w in float4 columns q = lane + 32 k
// (zero past d), before the warp sum.
template <int QPL>
__device__ __forceinline__ double lane_sum_squares(const float4 (&wq)[QPL]) {
  double ww = 0.0;
#pragma unroll
  for (int k = 0; k < QPL; ++k) {
    const double e[4] = {wq[k].x, wq[k].y, wq[k].z, wq[k].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) ww += e[i] * e[i];
  }
  return ww;
}

// U = (-N mean(lk) - log p(w)) / T, or (-(N/n) sum m lk - log p(w)) / T with
// a mask, as written in potential.py:183-185 (the unmasked form is exact for
// integer sums), and the biased variance of lk.
__device__ __forceinline__ double glm_potential_mean(const GlmArgs& a, double mean_lk,
                                                     double ww) {
  const double log_prior = -0.5 * ww * a.inv_p2 - a.prior_const;
  const double lik = -static_cast<double>(a.n_obs) * mean_lk;
  return (lik - log_prior) * a.inv_temp;
}
__device__ __forceinline__ double glm_potential(const GlmArgs& a, double sum_mlk, double ww) {
  if (a.mask == nullptr) return glm_potential_mean(a, sum_mlk / a.n, ww);
  const double log_prior = -0.5 * ww * a.inv_p2 - a.prior_const;
  const double lik = -(static_cast<double>(a.n_obs) / a.n) * sum_mlk;
  return (lik - log_prior) * a.inv_temp;
}
__device__ __forceinline__ double glm_variance_mean(double mean_lk, double mean_lk2) {
  return fmax(mean_lk2 - mean_lk * mean_lk, 0.0);
}
__device__ __forceinline__ double glm_variance(const GlmArgs& a, double sum_lk,
                                               double sum_lk2) {
  return glm_variance_mean(sum_lk / a.n, sum_lk2 / a.n);
}

}  // namespace gbsgmc
