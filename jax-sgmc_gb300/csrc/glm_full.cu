// The full-data potential of many chains on the GLM families,
//   U_c = (-sum_i lk_i(w_c) - log p(w_c)) / T over every observation
// (potential.py:219-293), and the Metropolis-Hastings samplers built on it:
// AMAGOLD and SGGMC (solver.py:301-577) with the proposals' trajectories as
// glm_loop launches, or as launches per gradient and update beyond its line.
//
// glm_full_kernel is a tall matrix product (rows x chains over d) whose
// outputs never leave the registers: a CTA takes 256 rows for 2 CB chains, each
// of its halves CB of the chains, thread t of a half the rows t and t + 128.  X
// passes through shared memory in panels of 16 features (cp.async, double
// buffered, rows padded to an odd number of 16-byte words so that a warp's 32
// rows touch every bank), and the chains' weights are broadcast reads.  Each x
// is read from memory once per 2 CB chains; evaluating the chains one by one
// through the minibatch kernel read all rows once per chain and computed
// gradients that no caller used.
//
// A dot product may be no further from the exact one than the minibatch
// kernel's (chains of four to 32 products a lane, then a tree over the lanes):
// chains of four, a tree over a panel, and the panels added with their
// rounding carried along.  One chain of FMAs over d had 2.1 times that kernel's
// rms error at 64 features and 4.7 times at 1,000; this has 0.9 and 0.5 times
// (equal up to 32).  It takes 26.0 us for 100,000 rows of 64 features and 16
// chains where that took 24.2 (1,000,000 rows: 137 and 112; 20,000: 15.9 and
// 18.0, the chains now being split over more warps).
//
// Likelihoods are added compensated per thread and chain, reduced as floats in
// three parts, and the CTAs' FP64 partials summed in a fixed order, so a
// chain's U does not depend on the other chains of the call.
#include <algorithm>
#include <cmath>
#include <new>

#include "common.cuh"
#include "glm.cuh"
#include "internal.h"
#include "plan.cuh"

namespace gbsgmc {
namespace {

constexpr int kHalf = 128;                 // threads of a half: two rows each
constexpr int kFullThreads = 2 * kHalf;
constexpr int kFullRows = 2 * kHalf;       // rows of a tile
constexpr int kPanel = 4;                     // float4 columns of a panel
constexpr int kPanelStride = kPanel + 1;

size_t full_smem(int dq, int cb) {   // cb: chains of a half
  return sizeof(float4) * (2ull * kFullRows * kPanelStride + 2ull * cb * dq);
}

// Row CTAs of a launch: as many as run at once, two per SM (twice as many, for
// 100,000 rows of 64 features and 16 chains: 31.5 us against 26.0).  Depends on
// the data alone (see above).
int full_ctas(int64_t n_rows) {
  const int64_t tiles = (n_rows + kFullRows - 1) / kFullRows;
  return static_cast<int>(std::min<int64_t>(tiles, 2 * glm_sm_count()));
}

__device__ __forceinline__ void full_copy(const GlmArgs& a, float4* buf, int64_t row0, int q0,
                                          int tid) {
  const int cols = min(kPanel, a.dq - q0);
  if (a.vec4) {
    for (int i = tid; i < kFullRows * kPanel; i += kFullThreads) {
      const int r = i / kPanel, v = i % kPanel;
      if (v < cols && row0 + r < a.n_rows)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         smem_addr(buf + r * kPanelStride + v)),
                     "l"(a.X + (row0 + r) * a.ld + 4 * (q0 + v))
                     : "memory");
    }
  } else {
    for (int i = tid; i < kFullRows * 4 * kPanel; i += kFullThreads) {
      const int r = i / (4 * kPanel), j = i % (4 * kPanel), col = 4 * q0 + j;
      if (j < 4 * cols && row0 + r < a.n_rows) {
        const bool ok = col < a.d;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                         smem_addr(reinterpret_cast<float*>(buf + r * kPanelStride) + j)),
                     "l"(a.X + (row0 + r) * a.ld + (ok ? col : 0)), "r"(ok ? 4 : 0)
                     : "memory");
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ float dot4(const float4& x, const float4& k) {
  return fmaf(x.w, k.w, fmaf(x.z, k.z, fmaf(x.y, k.y, x.x * k.x)));
}

// Grid (full_ctas, chain groups of 2 CB).  part[cta][chain] gets the CTA's sum
// of the chain's likelihoods.
template <int CB>
__global__ void __launch_bounds__(kFullThreads, 2) glm_full_kernel(const GlmArgs a, double* part) {
  extern __shared__ __align__(128) unsigned char smem[];
  float4* xs = reinterpret_cast<float4*>(smem);
  float4* ws = xs + 2 * kFullRows * kPanelStride;
  const int tid = threadIdx.x, lane = tid & 31, half = tid / kHalf, row = tid % kHalf;
  const int warp = row >> 5, c0 = blockIdx.y * 2 * CB, dq = a.dq;
  const bool active = c0 + half * CB < a.chains;   // this half has a chain
  // Weights of the group, zero past d and past the last chain.
  for (int i = tid; i < 2 * CB * 4 * dq; i += kFullThreads) {
    const int c = i / (4 * dq), j = i % (4 * dq);
    reinterpret_cast<float*>(ws)[i] =
        c0 + c < a.chains && j < a.d ? a.w[static_cast<int64_t>(c0 + c) * a.d + j] : 0.0f;
  }
  const int panels = (dq + kPanel - 1) / kPanel;
  const int64_t tiles = (a.n_rows + kFullRows - 1) / kFullRows;
  float sum[CB], comp[CB];
#pragma unroll
  for (int c = 0; c < CB; ++c) sum[c] = comp[c] = 0.0f;
  const int64_t first = blockIdx.x;
  if (first < tiles) full_copy(a, xs, first * kFullRows, 0, tid);
  int buf = 0;
  for (int64_t t = first; t < tiles; t += gridDim.x) {
    const int64_t row0 = t * kFullRows + row;
    float y[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int64_t r = row0 + i * kHalf;
      y[i] = 0.0f;
      if (r < a.n_rows)
        y[i] = a.y_inline ? __ldg(a.X + r * a.ld + a.d) : (a.y != nullptr ? __ldg(a.y + r) : 0.0f);
    }
    float z[2][CB], z_lo[2][CB];
#pragma unroll
    for (int c = 0; c < CB; ++c) z[0][c] = z[1][c] = z_lo[0][c] = z_lo[1][c] = 0.0f;
    for (int p = 0; p < panels; ++p) {
      // The next panel: of this tile, or the first of the CTA's next tile.
      const int64_t tn = p + 1 < panels ? t : t + gridDim.x;
      if (tn < tiles)
        full_copy(a, xs + (buf ^ 1) * kFullRows * kPanelStride, tn * kFullRows,
                  p + 1 < panels ? (p + 1) * kPanel : 0, tid);
      else
        asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const float4* xa = xs + (buf * kFullRows + row) * kPanelStride;
      const float4* xb = xa + kHalf * kPanelStride;
      const float4* wp = ws + half * CB * dq + p * kPanel;
      const int cols = min(kPanel, dq - p * kPanel);
      // A panel's 16 products: chains of four, added pairwise.
      float pa[2][CB];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (active && 2 * h < cols) {
          const bool two = 2 * h + 1 < cols;
          const float4 u0 = xa[2 * h], w0 = xb[2 * h];
          const float4 u1 = two ? xa[2 * h + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 w1 = two ? xb[2 * h + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            const float4 k0 = wp[c * dq + 2 * h];
            float a0 = dot4(u0, k0), a1 = dot4(w0, k0);
            if (two) {
              const float4 k1 = wp[c * dq + 2 * h + 1];
              a0 += dot4(u1, k1);
              a1 += dot4(w1, k1);
            }
            pa[0][c] = h ? pa[0][c] + a0 : a0;
            pa[1][c] = h ? pa[1][c] + a1 : a1;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < CB; ++c)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if (!active) continue;
          const Float2Sum s = two_sum(z[r][c], pa[r][c]);
          z[r][c] = s.hi;
          z_lo[r][c] = __fadd_rn(z_lo[r][c], s.lo);
        }
      __syncthreads();  // the buffer is free for the panel after the next
      buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (!active || row0 + i * kHalf >= a.n_rows) continue;
#pragma unroll
      for (int c = 0; c < CB; ++c) {
        // z_lo is no number once z has overflowed.
        const float zi = z[i][c] + (isfinite(z_lo[i][c]) ? z_lo[i][c] : 0.0f);
        float lk, dz;
        if (a.family == GBSGMC_GLM_LOGISTIC) {
          logistic_link(zi, y[i], true, lk, dz);
        } else if (a.family == GBSGMC_GLM_LINEAR) {
          lk = zi;
        } else {
          const float res = y[i] - zi;
          lk = -0.5f * res * res * a.inv_s2 - a.log_norm;
        }
        // (comp is of no account once sum has overflowed.)
        const Float2Sum s = two_sum(sum[c], lk);
        sum[c] = s.hi;
        comp[c] = __fadd_rn(comp[c], s.lo);
      }
    }
  }
  // Sums of the CTA's threads, chain by chain.
  __shared__ double red[2][kHalf / 32][CB];
#pragma unroll
  for (int c = 0; c < CB; ++c) {
    double s;
    if (__all_sync(0xffffffffu, fabsf(sum[c]) < 7.9e28f)) {
      s = widen(warp_sum(Float3Sum{sum[c], comp[c], 0.0f}));
    } else {  // keeps infinities what they are
      s = warp_sum(static_cast<double>(sum[c]));
    }
    if (lane == 0) red[half][warp][c] = s;
  }
  __syncthreads();
  if (tid < 2 * CB && c0 + tid < a.chains) {
    const int g = tid / CB, c = tid % CB;
    double s = red[g][0][c];
#pragma unroll
    for (int w = 1; w < kHalf / 32; ++w) s += red[g][w][c];
    part[static_cast<int64_t>(blockIdx.x) * a.chains + c0 + tid] = s;
  }
}

// U of chain c from its CTA partials and its weights, by one warp.
__device__ double full_value(const GlmArgs& a, const double* part, int ctas, const float* w,
                             int c, double temperature, int lane) {
  double s = 0.0, ww = 0.0;
  for (int i = lane; i < ctas; i += 32) s += part[static_cast<int64_t>(i) * a.chains + c];
  if (a.inv_p2 > 0.0f)
    for (int j = lane; j < a.d; j += 32) ww += static_cast<double>(w[j]) * w[j];
  s = warp_sum(s);
  ww = warp_sum(ww);
  const double log_prior = -0.5 * ww * a.inv_p2 - a.prior_const;
  return (-s - log_prior) / temperature;
}

__global__ void glm_full_value_kernel(const GlmArgs a, const double* part, int ctas,
                                      double temperature) {
  const int c = blockIdx.x, lane = threadIdx.x;
  const double U = full_value(a, part, ctas, a.w + static_cast<int64_t>(c) * a.d, c, temperature,
                              lane);
  if (lane == 0) {
    a.U[c] = U;
    if (!isfinite(U)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
  }
}

struct MhArgs {
  int kind;      // GBSGMC_MH_AMAGOLD / _SGGMC
  int steps;     // integrator steps per iteration
  float *x, *p, *x_old, *p_old;
  double *U_old, *energy, *ke, *U_mean;
  uint64_t seed;
  int chain_base;
  const double* part;
  int ctas;
  double temperature;
  float* samples;
  double* stat;
  const int32_t* keep;   // per iteration
};

// One CTA per chain, after a trajectory and its full-data pass: U of the
// proposal, the decision of mh_accept_kernel, the state kept (accepted, or
// the old positions with the momentum times -1 (AMAGOLD) or 1), the sample of
// a kept iteration, and the accumulators zeroed for the next trajectory.
__global__ void __launch_bounds__(128) glm_mh_finish_kernel(const GlmArgs a, const MhArgs m) {
  __shared__ int accepted;
  const int c = blockIdx.x, tid = threadIdx.x;
  const int64_t it = a.sched.step() / m.steps;   // a.sched is at the trajectory's first step
  const int64_t off = static_cast<int64_t>(c) * a.d;
  const int slot = m.keep != nullptr ? __ldg(m.keep + it) : -1;
  if (tid < 32) {
    const double U_new = full_value(a, m.part, m.ctas, m.x + off, c, m.temperature, tid);
    if (tid == 0) {
      if (!isfinite(U_new)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
      double la;
      if (m.kind == GBSGMC_MH_AMAGOLD) {
        la = m.U_old[c] - U_new + m.energy[c];
        la = la > 0.0 ? 0.0 : la;
      } else {
        const double T = static_cast<double>(a.sched.temperature(a.sched.step(), c));
        la = -1.0 / T * (U_new - m.U_old[c] + m.ke[a.chains + c] - m.ke[c]);
        la = la <= 0.0 ? la : 0.0;
      }
      const int acc = log(mh_uniform(m.seed, static_cast<uint32_t>(m.chain_base + c),
                                     static_cast<uint32_t>(it))) < la
                          ? 1
                          : 0;
      accepted = acc;
      if (acc) m.U_old[c] = U_new;
      if (slot >= 0)
        m.stat[static_cast<int64_t>(slot) * a.chains + c] =
            m.kind == GBSGMC_MH_AMAGOLD ? m.energy[c] : m.U_mean[c];
      if (m.energy != nullptr) m.energy[c] = 0.0;
      if (m.ke != nullptr) m.ke[c] = m.ke[a.chains + c] = 0.0;
    }
  }
  __syncthreads();
  const float sign = m.kind == GBSGMC_MH_AMAGOLD ? -1.0f : 1.0f;
  for (int j = tid; j < a.d; j += blockDim.x) {
    float x = m.x[off + j], p = m.p[off + j];
    if (!accepted) {
      m.x[off + j] = x = m.x_old[off + j];
      m.p[off + j] = p = sign * m.p_old[off + j];
    }
    m.x_old[off + j] = x;
    m.p_old[off + j] = p;
    if (slot >= 0) m.samples[(static_cast<int64_t>(slot) * a.chains + c) * a.d + j] = x;
  }
}

template <int CB>
int launch_full_cb(const GlmArgs& a, double* part, cudaStream_t st) {
  static int done = 0;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(
        glm_full_kernel<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "glm_full: cudaFuncSetAttribute: %s",
                       cudaGetErrorString(e));
    done = 1;
  }
  const dim3 grid(static_cast<unsigned>(full_ctas(a.n_rows)),
                  static_cast<unsigned>(ceil_div(a.chains, 2 * CB)));
  glm_full_kernel<CB><<<grid, kFullThreads, full_smem(a.dq, CB), st>>>(a, part);
  return check_launch("glm_full");
}

int launch_full(const GlmArgs& a, double* part, cudaStream_t st) {
  // Groups of 16 chains (eight a half) when there are more than four: x is read
  // once per group.
  return a.chains > 4 ? launch_full_cb<8>(a, part, st) : launch_full_cb<2>(a, part, st);
}

size_t full_ws_bytes(const gbsgmc_glm* m, int chains) {
  const int64_t rows = m->n_rows > 0 ? m->n_rows : m->n_obs;
  return sizeof(double) * static_cast<size_t>(full_ctas(rows)) * chains;
}

// The arguments of a full-data pass (the index stream is not used).
int full_args(GlmArgs& a, const gbsgmc_glm* m, int chains, const float* w, int* status) {
  GlmTune t;
  t.rows_per_warp = 4;   // no tuned shape is looked up
  static const int32_t unused = 0;
  int rc = glm_fill_args(a, m, chains, 1, &unused, 1, nullptr, nullptr, 0, status, t);
  if (rc != GBSGMC_OK) return rc;
  if (w == nullptr) return set_error(GBSGMC_ERR_ARG, "glm_full: null w");
  a.mode = kValueGrad;
  a.w = const_cast<float*>(w);
  return GBSGMC_OK;
}

struct GlmMhPlan final : gbsgmc_plan {
  gbsgmc_glm model, full;
  int chains = 0, n = 0, steps = 0, ctas = 1;
  bool loop = true;
  gbsgmc_integrator integ{};
  gbsgmc_sched sched{};
  gbsgmc_noise noise{};
  gbsgmc_index_src isrc{};
  MhArgs mh{};
  int* status = nullptr;
  int32_t* idx = nullptr;   // owned [G, chains, draws * n]
  float* old = nullptr;     // owned [2, chains, d]
  double* acc = nullptr;    // owned: energy [C], ke [2 C], U [C], lk_var [C]
  double* part = nullptr;   // owned
  // Trajectories by launches: gradient [chains, d], the second minibatch's
  // potential, workspace of the gradient calls (all owned).
  float* grad = nullptr;
  double* U2 = nullptr;
  void* ws = nullptr;
  size_t ws_size = 0;

  bool amagold() const { return mh.kind == GBSGMC_MH_AMAGOLD; }
  int draws() const { return amagold() ? 1 : 2; }
  ~GlmMhPlan() override {
    if (stream != nullptr) cudaStreamSynchronize(stream);
    plan_free(this, idx);
    plan_free(this, old);
    plan_free(this, acc);
    plan_free(this, part);
    plan_free(this, grad);
    plan_free(this, U2);
    plan_free(this, ws);
  }
  int step_multiple() const override { return steps; }
  // Index draw and step counter, and per iteration the trajectory, the
  // full-data pass and the decision.
  int64_t launches_per_block(int g) const override {
    const int64_t traj = loop ? 1 : amagold() ? 3 * int64_t{steps} + 1 : 4 * int64_t{steps} + 1;
    return 2 + (traj + 2) * (g / steps);
  }

  int gradient(const int32_t* ix, int64_t stride, double* U, cudaStream_t s) const {
    return gbsgmc_glm_value_and_grad(&model, chains, n, ix, stride, nullptr, mh.x, U, grad,
                                     nullptr, nullptr, ws, ws_size, status, s);
  }

  // The trajectory of the iteration whose first step is j, a launch at a time:
  // the reversible leapfrog (integrator.py:349-560; half a position step at
  // both ends) or OBABO (integrator.py:138-346).
  int trajectory(int j, int64_t cn, int per, cudaStream_t s) const {
    const int d = model.d;
    const float f = integ.friction;
    gbsgmc_sched sj = sched;
    sj.base_dev = base;
    sj.keep_slot_dev = nullptr;
    int rc;
    for (int i = 0; i < steps; ++i) {
      const int32_t* ix = idx + (j + i) * cn;
      sj.offset = j + i;
      if (amagold()) {
        if ((rc = gbsgmc_leapfrog_position(chains, d, mh.x, mh.p, nullptr, i == 0 ? 0.5f : 1.0f,
                                           &sj, s)) ||
            (rc = gradient(ix, per, mh.U_mean, s)) ||
            (rc = gbsgmc_amagold_momentum(chains, d, mh.p, grad, nullptr, f, mh.energy, &sj, &noise,
                                          s)))
          return rc;
      } else {
        if ((rc = gradient(ix, per, mh.U_mean, s)) ||
            (rc = gbsgmc_obabo_first(chains, d, mh.x, mh.p, grad, nullptr, f, mh.ke, &sj, &noise,
                                     s)) ||
            (rc = gradient(ix + n, per, U2, s)) ||
            (rc = gbsgmc_obabo_second(chains, d, mh.p, grad, nullptr, f, mh.ke + chains, &sj,
                                      &noise, s)))
          return rc;
      }
    }
    if (amagold()) return gbsgmc_leapfrog_position(chains, d, mh.x, mh.p, nullptr, 0.5f, &sj, s);
    return mean_pair(chains, mh.U_mean, U2, s);
  }

  int enqueue(int g, cudaStream_t s) override {
    const int per = draws() * n;
    const int64_t cn = static_cast<int64_t>(chains) * per;
    const int64_t rows = model.n_rows > 0 ? model.n_rows : model.n_obs;
    int rc = gbsgmc_index_draw_pcg64(isrc.pcg_dev, chains, rows, static_cast<int64_t>(g) * per,
                                     per, idx, per, cn, status, s);
    if (rc != GBSGMC_OK) return rc;
    GlmArgs a;
    if ((rc = full_args(a, &full, chains, mh.x, status))) return rc;
    for (int j = 0; j < g; j += steps) {
      gbsgmc_sched sj = sched;
      sj.base_dev = base;
      sj.offset = j;
      sj.keep_slot_dev = nullptr;
      GlmLoopCall c;
      c.model = &model;
      c.kind = amagold() ? kLoopLeapfrog : kLoopObabo;
      c.chains = chains;
      c.n = n;
      c.steps = steps;
      c.ctas = ctas;
      c.idx = idx + j * cn;
      c.idx_stride = per;
      c.idx_step_stride = cn;
      c.x = mh.x;
      c.aux = mh.p;
      c.friction = integ.friction;
      c.sched = &sj;
      c.noise = &noise;
      c.U = mh.U_mean;
      c.lk_var = mh.U_mean + chains;
      c.ke = mh.ke;
      c.energy = mh.energy;
      c.status = status;
      if ((rc = loop ? glm_loop(c, s) : trajectory(j, cn, per, s))) return rc;
      if ((rc = launch_full(a, part, s))) return rc;
      a.sched = to_sched(&sj);
      glm_mh_finish_kernel<<<chains, 128, 0, s>>>(a, mh);
      if ((rc = check_launch("glm_mh_finish"))) return rc;
    }
    return plan_advance(this, g, s);
  }
};

}  // namespace
}  // namespace gbsgmc

using namespace gbsgmc;

extern "C" size_t gbsgmc_glm_full_workspace_bytes(const gbsgmc_glm* model, int chains) {
  if (model == nullptr || chains <= 0 || model->n_obs < 1) return 0;
  return full_ws_bytes(model, chains);
}

extern "C" int gbsgmc_glm_full_potential(const gbsgmc_glm* model, int chains, const float* w_dev,
                                         double* U_dev, void* ws, size_t ws_bytes,
                                         int* status_dev, gbsgmc_stream_t stream) {
  if (model == nullptr || U_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "glm_full_potential: null argument");
  GlmArgs a;
  int rc = full_args(a, model, chains, w_dev, status_dev);
  if (rc != GBSGMC_OK) return rc;
  if (chains == 0) return GBSGMC_OK;
  if (ws == nullptr || ws_bytes < full_ws_bytes(model, chains))
    return set_error(GBSGMC_ERR_ARG, "glm_full_potential: workspace missing or too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  a.U = U_dev;
  double* part = static_cast<double*>(ws);
  if ((rc = launch_full(a, part, st))) return rc;
  glm_full_value_kernel<<<chains, 32, 0, st>>>(a, part, full_ctas(a.n_rows),
                                               static_cast<double>(model->temperature));
  return check_launch("glm_full_value");
}

extern "C" int gbsgmc_glm_mh_plan_create(
    gbsgmc_plan** out, const gbsgmc_glm* model, const gbsgmc_glm* full, int kind, int chains,
    int n, const gbsgmc_integrator* integ, float* x_dev, float* p_dev, double* U_dev,
    const gbsgmc_sched* sched, const gbsgmc_noise* noise, const gbsgmc_index_src* isrc,
    uint64_t mh_seed, const int32_t* keep_dev, float* samples_dev, double* stat_dev,
    int block_iterations, int* status_dev) {
  if (out == nullptr) return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: null plan");
  *out = nullptr;
  if (model == nullptr || full == nullptr || integ == nullptr || x_dev == nullptr ||
      p_dev == nullptr || U_dev == nullptr || sched == nullptr || noise == nullptr ||
      isrc == nullptr || status_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: null argument");
  if (kind != GBSGMC_MH_AMAGOLD && kind != GBSGMC_MH_SGGMC)
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: unknown kind %d", kind);
  if (chains <= 0 || n <= 0 || integ->leapfrog_steps < 1 || block_iterations < 1 ||
      static_cast<int64_t>(block_iterations) * integ->leapfrog_steps > 100000)
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: bad chains/n/steps");
  if (isrc->pcg_dev == nullptr || isrc->external)
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: needs PCG64 index streams");
  if (integ->mass_dev != nullptr)
    return set_error(GBSGMC_ERR_UNSUPPORTED, "glm_mh_plan_create: unit mass only");
  if (keep_dev != nullptr && (samples_dev == nullptr || stat_dev == nullptr))
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: keep table without sample buffers");
  if (model->d != full->d)
    return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: the models differ in d");
  GlmMhPlan* p = new (std::nothrow) GlmMhPlan();
  if (p == nullptr) return set_error(GBSGMC_ERR_ARG, "glm_mh_plan_create: out of memory");
  p->model = *model;
  p->full = *full;
  p->chains = chains;
  p->n = n;
  p->steps = integ->leapfrog_steps;
  p->integ = *integ;
  p->sched = *sched;
  p->noise = *noise;
  p->isrc = *isrc;
  p->status = status_dev;
  MhArgs& m = p->mh;
  m.kind = kind;
  m.steps = p->steps;
  m.x = x_dev;
  m.p = p_dev;
  m.U_old = U_dev;
  m.seed = mh_seed;
  m.chain_base = noise->chain_base;
  m.temperature = full->temperature;
  m.samples = samples_dev;
  m.stat = stat_dev;
  m.keep = keep_dev;
  int rc;
  do {
    const int G = block_iterations * p->steps;
    const size_t xbytes = sizeof(float) * static_cast<size_t>(chains) * model->d;
    if ((rc = plan_init(p, G))) break;
    if ((rc = plan_alloc(p, &p->idx,
                         sizeof(int32_t) * static_cast<size_t>(G) * chains * p->draws() * n,
                         "glm_mh_plan_create: index buffer")))
      break;
    if ((rc = plan_alloc(p, &p->old, 2 * xbytes, "glm_mh_plan_create: state"))) break;
    if ((rc = plan_alloc(p, &p->acc, 5 * sizeof(double) * chains, "glm_mh_plan_create: sums")))
      break;
    if ((rc = plan_alloc(p, &p->part, full_ws_bytes(full, chains),
                         "glm_mh_plan_create: partials")))
      break;
    m.x_old = p->old;
    m.p_old = p->old + static_cast<size_t>(chains) * model->d;
    m.energy = p->amagold() ? p->acc : nullptr;
    m.ke = p->amagold() ? nullptr : p->acc + chains;
    m.U_mean = p->acc + 3 * chains;
    m.part = p->part;
    m.ctas = full_ctas(full->n_rows > 0 ? full->n_rows : full->n_obs);
    // The state the first proposal is compared with.
    if ((rc = cuda_err(cudaMemcpyAsync(m.x_old, x_dev, xbytes, cudaMemcpyDeviceToDevice,
                                       p->stream), "glm_mh_plan_create: copy")))
      break;
    if ((rc = cuda_err(cudaMemcpyAsync(m.p_old, p_dev, xbytes, cudaMemcpyDeviceToDevice,
                                       p->stream), "glm_mh_plan_create: copy")))
      break;
    if ((rc = glm_prepare())) break;
    p->loop = glm_loop_pays(chains, 1, n, model->d);
    if (p->loop) {
      p->ctas = glm_loop_ctas(chains, 1, n);
    } else {
      p->ws_size = glm_ws_bytes(chains, n, model->d);
      if ((rc = plan_alloc(p, &p->grad, xbytes, "glm_mh_plan_create: gradient"))) break;
      if ((rc = plan_alloc(p, &p->U2, sizeof(double) * chains, "glm_mh_plan_create: U"))) break;
      if ((rc = plan_alloc(p, &p->ws, p->ws_size, "glm_mh_plan_create: workspace"))) break;
    }
    rc = plan_capture(p);
  } while (false);
  if (rc != GBSGMC_OK) {
    delete p;
    return rc;
  }
  *out = p;
  return GBSGMC_OK;
}
