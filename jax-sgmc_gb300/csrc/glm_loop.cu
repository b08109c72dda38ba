// Whole blocks of integrator steps on the GLM potentials in one launch: SGLD
// (+RMSprop), OBABO, SGHMC, the reversible leapfrog of AMAGOLD, and reSGLD
// (normal, hot) pairs with their exchange.
//
// What bounds a step of a small chain is not its bytes (a minibatch of 128
// rows of 32 features is 16 KB) but the chain of dependent latencies: index
// load, row load, dot products, block reduction, update, next step; and, with
// a launch per gradient and per update, the launches between them.  Here a
// cluster of S CTAs owns a chain for the whole block:
//   * CTA s holds rows [s R, (s + 1) R) of every minibatch.  The minibatches
//     of a block are known before it starts, so indices and rows of the next
//     chunks are copied to shared memory (cp.async, a ring of `depth` chunk
//     buffers) while the current one is consumed: a step never waits for the
//     row loads unless the memory system is the bound.
//   * warps 0..7 take row tiles of the chunk exactly as glm_kernel does (same
//     slices, warps, tiles and summation orders: the same bits), and the
//     threads that own four parameters each keep x and v (or p) in registers.
//   * every CTA writes its partial gradient into all CTAs of the cluster
//     (distributed shared memory), one cluster barrier, and every CTA adds
//     the partials in slice order and updates its own copy of x: no second
//     exchange is needed.
//   * warp 8 (the clerk) draws the update's Philox noise, reads the schedule
//     and does the FP64 sums (U, var(lk), kinetic energies, the exchange
//     decision) while the other warps stream rows.
// reSGLD pairs: both chains of a pair share a cluster (2 S CTAs).  An
// exchange swaps the chains' roles (temperature, slot) instead of their
// states; the rows are written to the slots they ended in when the block
// ends.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "glm.cuh"
#include "internal.h"

namespace gbsgmc {
namespace {

namespace cg = cooperative_groups;

constexpr int kRowWarps = 8;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kLoopThreads = kRowThreads + 32;  // + the clerk warp
constexpr int kMaxCtas = 8;                     // portable cluster size
constexpr int kMaxDepth = 4;

struct LoopArgs {
  GlmArgs g;
  int kind;        // GlmLoopKind
  int draws;       // minibatches per step (OBABO: 2)
  int leapfrog;    // SGHMC: steps per momentum resample
  float friction;
  const float* mass;
  float* aux;      // RMSprop state (or null), or the momentum
  double* ke;      // OBABO: kinetic energies [2, chains] to add to, or null
  double* energy;  // leapfrog: energies [chains] to add to
  int ctas;        // CTAs per chain
  int chunk_rows, chunks, depth, idx_slots;
  int row_shift;   // log2 of the lanes that copy one row
  // pairs
  int pairs;
  double F;
  uint64_t swap_seed;
  const int32_t* pair_chain;
  int32_t* ident;
  double* ssq;
  int64_t* kc;
  int32_t* counts;
  // shared-memory offsets
  unsigned o_y, o_idx, o_red, o_part, o_w, o_xi, o_xr, o_ke, o_lane, o_sums, o_step;
};

// What the clerk hands the updating threads for one gradient.
struct StepInfo {
  float h, T, h_next;
  int slot, want_u, role;
};

__device__ __forceinline__ void cp16(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(ok ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most `pending` of this thread's newest groups are in flight.
__device__ __forceinline__ void cp_wait(int pending) {
  if (pending <= 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
  else if (pending == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 2;" ::: "memory");
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The OBABO halves of one parameter, rounded as update.cu's kernels do.
struct ObaboStep {
  float h, keep, inject, half;
  __device__ __forceinline__ ObaboStep(float step, float T, float friction) {
    h = step;
    const float permanence = expf(-friction * h);
    keep = sqrtf(permanence);
    inject = sqrtf((1.0f - permanence) * T);
    half = 0.5f * h;
  }
  __device__ __forceinline__ void first(float mi, float ms, float g, float xi, float& p, float& x,
                                        float& ke) const {
    float pj = __fmaf_rn(keep, p, __fmul_rn(inject, __fmul_rn(ms, xi)));
    ke = __fmaf_rn(__fmul_rn(0.5f, pj), __fmul_rn(mi, pj), ke);
    pj = __fmaf_rn(-half, g, pj);
    p = pj;
    x = __fmaf_rn(h, __fmul_rn(mi, pj), x);
  }
  __device__ __forceinline__ void second(float mi, float ms, float g, float xi, float& p,
                                         float& ke) const {
    const float pj = __fmaf_rn(-half, g, p);
    ke = __fmaf_rn(__fmul_rn(0.5f, pj), __fmul_rn(mi, pj), ke);
    p = __fmaf_rn(keep, pj, __fmul_rn(inject, __fmul_rn(ms, xi)));
  }
};

// A slice's sums, as one CTA publishes them: sum m lk, sum lk, sum lk^2, and
// its chain's sum(w^2).
struct SliceSums {
  double v[4];
};

// Total of one sum over a chain's slices, in the order of sum_slices (a
// pairwise tree: lane s of 32 holding slice s).
__device__ __forceinline__ double slice_total(const SliceSums* s, int ctas, int k) {
  double t[kMaxCtas];
#pragma unroll
  for (int i = 0; i < kMaxCtas; ++i) t[i] = i < ctas ? s[i].v[k] : 0.0;
#pragma unroll
  for (int o = kMaxCtas / 2; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) t[i] += t[i + o];
  return t[0];
}

template <int QPL, int RW>
__global__ void __launch_bounds__(kLoopThreads, QPL <= 2 ? 2 : 1)
    glm_loop_kernel(const LoopArgs L) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int LOG = Log2<RW>::v;
  constexpr int GROUP = 32 >> LOG;
  constexpr int kStride = kRowWarps * RW;
  const GlmArgs& a = L.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool clerk = warp == kRowWarps;
  const int g = lane >> (5 - LOG);
  const bool leader = (lane & (GROUP - 1)) == 0;
  const int dq = a.dq, d = a.d, S = L.ctas, CH = L.chunk_rows, depth = L.depth;
  const bool pairs = L.kind == kLoopPairs;
  const bool moves = L.kind == kLoopSgld || pairs;  // aux is the RMSprop state

  // This CTA's chain, slice and cluster rank (1-D grid, 1-D clusters).
  const int ncta = pairs ? 2 * S : S;
  const int rank = blockIdx.x % ncta, unit = blockIdx.x / ncta;
  const int slice = rank % S, rank0 = rank - slice;
  const int half = rank / S;  // pairs: the slot this chain starts the block in
  const int row_in = pairs ? (half ? L.pairs + unit : unit) : unit;
  const int who = pairs ? L.ident[row_in] : row_in;  // index stream, noise chain
  const int row0 = slice * a.rows_per_slice;
  const int R = max(0, min(a.rows_per_slice, a.n - row0));
  const int events = a.steps * L.draws;
  const int total = events * L.chunks;

  float4* rows_s = reinterpret_cast<float4*>(smem);
  float* y_s = reinterpret_cast<float*>(smem + L.o_y);
  int32_t* idx_s = reinterpret_cast<int32_t*>(smem + L.o_idx);
  float4* red = reinterpret_cast<float4*>(smem + L.o_red);
  float4* part = reinterpret_cast<float4*>(smem + L.o_part);   // [2][S][dq]
  float4* w_s = reinterpret_cast<float4*>(smem + L.o_w);
  float4* xi_s = reinterpret_cast<float4*>(smem + L.o_xi);
  float4* xr_s = reinterpret_cast<float4*>(smem + L.o_xr);     // SGHMC resample
  float* ke_s = reinterpret_cast<float*>(smem + L.o_ke);
  LaneSums* lsum = reinterpret_cast<LaneSums*>(smem + L.o_lane);
  SliceSums* sums = reinterpret_cast<SliceSums*>(smem + L.o_sums);  // [2][ncta]
  StepInfo* info = reinterpret_cast<StepInfo*>(smem + L.o_step);

  // ---- copies ----------------------------------------------------------------
  auto issue_idx = [&](int e, int q, int slot) {
    const int cnt = min(CH, R - q * CH);
    const int32_t* src = a.idx + (e / L.draws) * a.idx_step_stride +
                         static_cast<int64_t>(who) * a.idx_stride + (e % L.draws) * a.n + row0 +
                         q * CH;
    for (int r = tid; r < cnt; r += kRowThreads) cp4(idx_s + slot * CH + r, src + r, true);
  };
  auto issue_rows = [&](int q, int slot, int buf) {
    const int cnt = min(CH, R - q * CH);
    const int32_t* ix = idx_s + slot * CH;
    float4* dst = rows_s + static_cast<int64_t>(buf) * CH * dq;
    const int per = 32 >> L.row_shift, sub = lane >> L.row_shift;
    const int ql = lane & ((1 << L.row_shift) - 1);
    for (int r = warp * per + sub; r < cnt; r += kRowWarps * per) {
      const int o = ix[r];
      const bool ok = o >= 0 && o < a.n_rows;
      if (!ok && ql == 0) raise_status(a.status, GBSGMC_ERR_INDEX);
      const float* src = a.X + (ok ? static_cast<int64_t>(o) * a.ld : 0);
      if (a.vec4) {
        for (int v = ql; v < dq; v += 32) cp16(dst + r * dq + v, src + 4 * v, ok);
      } else {
        float* out = reinterpret_cast<float*>(dst + r * dq);
        for (int j = ql; j < 4 * dq; j += 1 << L.row_shift)
          cp4(out + j, src + (j < d ? j : 0), ok && j < d);
      }
    }
    if (a.y_inline || a.y != nullptr) {
      for (int r = tid; r < cnt; r += kRowThreads) {
        const int o = ix[r];
        const bool ok = o >= 0 && o < a.n_rows;
        const float* src = a.y_inline ? a.X + (ok ? static_cast<int64_t>(o) * a.ld + d : 0)
                                      : a.y + (ok ? o : 0);
        cp4(y_s + buf * CH + r, src, ok);
      }
    }
  };

  // Sequence numbers of the next index and row chunks to request.
  int ie = 0, iq = 0, islot = 0;             // index chunk
  int rs = 0, rq = 0, rslot = 0, rbuf = 0;   // row chunk
  auto next_idx = [&]() {
    if (ie < events && !clerk) issue_idx(ie, iq, islot);
    if (++iq == L.chunks) iq = 0, ++ie;
    if (++islot == L.idx_slots) islot = 0;
  };
  auto next_rows = [&]() {
    if (rs < total && !clerk) issue_rows(rq, rslot, rbuf);
    ++rs;
    if (++rq == L.chunks) rq = 0;
    if (++rslot == L.idx_slots) rslot = 0;
    if (++rbuf == depth) rbuf = 0;
  };

  for (int i = 0; i < 2 * (depth - 1); ++i) next_idx();
  cp_commit();
  if (ncta > 1) cluster_arrive();  // every CTA runs before any remote write

  // ---- state -----------------------------------------------------------------
  const int64_t k0 = a.sched.step();
  float* x_row = a.w + static_cast<int64_t>(row_in) * d;
  float* aux_row = L.aux != nullptr ? L.aux + static_cast<int64_t>(row_in) * d : nullptr;
  const bool owner = tid < dq;
  float xs[4] = {0.f, 0.f, 0.f, 0.f}, as[4] = {0.f, 0.f, 0.f, 0.f};
  float mi[4] = {1.f, 1.f, 1.f, 1.f}, ms[4] = {1.f, 1.f, 1.f, 1.f};
  if (owner) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = 4 * tid + e;
      if (j >= d) break;
      xs[e] = x_row[j];
      if (aux_row != nullptr) as[e] = aux_row[j];
      if (L.mass != nullptr) {
        const float m = __ldg(L.mass + j);
        mi[e] = 1.0f / m;
        ms[e] = sqrtf(m);
      }
    }
    if (L.kind == kLoopSghmc) {
      // A block starts at a resample (its steps are whole trajectories).
      float xi[4];
      noise4(a.noise, who, 4 * tid, d, k0, GBSGMC_TAG_SGHMC_RESAMPLE, xi);
      const float h = a.sched.step_size(k0);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        as[e] = ms[e] * xi[e];
        const float pj = as[e];
        const float sm = mi[e] * pj;
        xs[e] = xs[e] + h * sm;
        as[e] = pj + (-h * L.friction) * sm;
      }
    } else if (L.kind == kLoopLeapfrog) {
      const float s = 0.5f * a.sched.step_size(k0);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float sm = mi[e] * as[e];
        xs[e] = xs[e] + s * sm;
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * tid + e >= d) xs[e] = as[e] = 0.f;
    w_s[tid] = make_float4(xs[0], xs[1], xs[2], xs[3]);
  }

  // The clerk's running state.
  double ke_acc[2] = {0.0, 0.0};
  double U_first = 0.0;            // OBABO: the step's first minibatch
  double U_mine = 0.0, var_mine = 0.0;
  double ssq = 0.0;
  int64_t kc = 0;
  int exchanges = 0;
  int role = half;                 // pairs: the slot this chain is in now
  double U_pair[2] = {0.0, 0.0}, var_pair[2] = {0.0, 0.0};  // by chain (half)
  if (clerk && pairs) {
    ssq = L.ssq[unit];
    kc = L.kc[unit];
  }

  // FP64 sum of the threads' kinetic-energy (or energy) parts of one update,
  // in the order of update.cu's block sums.
  auto energy_sum = [&]() {
    double t = 0.0;
    for (int w0 = 0; w0 < dq; w0 += 32) {
      const double v = w0 + lane < dq ? static_cast<double>(ke_s[w0 + lane]) : 0.0;
      t += warp_sum(v);
    }
    return t;
  };
  // The pair's decision after step k (gradient sums in buffer par): roles
  // swap when log u >= log s.  Lanes 0 and 1 evaluate chain 0's and 1's U and
  // var side by side.
  auto decide = [&](int64_t k, int par) {
    const int h = lane & 1;
    const SliceSums* sp = sums + par * ncta + h * S;
    const double U = glm_potential(a, slice_total(sp, S, 0), a.inv_p2 > 0.f ? sp[0].v[3] : 0.0);
    const double var = glm_variance(a, slice_total(sp, S, 1), slice_total(sp, S, 2));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      U_pair[i] = __shfl_sync(0xffffffffu, U, i);
      var_pair[i] = __shfl_sync(0xffffffffu, var, i);
    }
    const int n_chain = half ^ role;  // the chain in the normal slot
    const double Un = U_pair[n_chain], Uh = U_pair[n_chain ^ 1];
    kc += 1;
    const double sa = 1.0 / static_cast<double>(kc);
    ssq = (1.0 - sa) * ssq + sa * var_pair[n_chain];
    const double Tn = a.sched.temperature(k, unit);
    const double Th = a.sched.temperature(k, L.pairs + unit);
    const double dbeta = 1.0 / Tn - 1.0 / Th;
    const double log_s = dbeta * (Un - Uh - dbeta * ssq / L.F);
    const uint64_t key = (L.swap_seed << 32) | static_cast<uint32_t>(__ldg(L.pair_chain + unit));
    const double u = swap_uniform(key, 0u, static_cast<uint32_t>(k + 1));
    // The reference keeps the pair when log u < log s (lax.cond true branch).
    if (!(log(u) < log_s)) {
      role ^= 1;
      ++exchanges;
    }
    const int slot = a.sched.keep_slot(k);
    if (slot >= 0 && role == 0 && slice == 0) {
      const int64_t at = static_cast<int64_t>(slot) * L.pairs + unit;
      const float* x = reinterpret_cast<const float*>(w_s);
      for (int j = lane; j < d; j += 32) a.samples[at * d + j] = x[j];
      if (lane == 0 && a.sample_lik != nullptr) a.sample_lik[at] = -U_pair[half];
    }
  };

  float4 wq[QPL];
  Accum<QPL> A;

  cp_wait(0);
  __syncthreads();
  if (ncta > 1) cluster_wait();
  for (int i = 0; i + 1 < depth; ++i) {
    next_rows();
    cp_commit();
  }

  int e = 0, q = 0, slot_c = 0, buf_c = 0;
  for (int s = 0; s < total; ++s) {
    cp_wait(depth - 2);
    __syncthreads();  // chunk s has arrived; the last update of w_s is visible
    next_rows();
    next_idx();
    cp_commit();
    const int j = L.draws == 2 ? e >> 1 : e;
    const int par = e & 1;
    if (q == 0) {
      if (!clerk) {
#pragma unroll
        for (int k = 0; k < QPL; ++k) {
          const int v = lane + 32 * k;
          wq[k] = v < dq ? w_s[v] : make_float4(0.f, 0.f, 0.f, 0.f);
          A.acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        A.mlk = A.mlk_c = A.K = A.s1 = A.s2 = 0.0f;
        A.cnt = 0;
      } else {
        // The clerk: last step's decision and energies, this step's schedule,
        // noise and, where U is wanted, the prior's sum(w^2).
        const int64_t k = k0 + j;
        if (pairs && e > 0) decide(k - 1, par ^ 1);
        if (e > 0 && (L.energy != nullptr || L.ke != nullptr)) ke_acc[L.draws == 2 ? par ^ 1 : 0] += energy_sum();
        const int keep = pairs ? -1 : a.sched.keep_slot(k);
        const bool want = pairs || j + 1 == a.steps || keep >= 0;
        if (lane == 0) {
          StepInfo in;
          in.h = a.sched.step_size(k);
          in.T = a.sched.temperature(k, pairs ? (role ? L.pairs + unit : unit) : unit);
          in.h_next = j + 1 < a.steps ? a.sched.step_size(k + 1) : in.h;
          in.slot = keep;
          in.want_u = want && L.kind != kLoopLeapfrog;
          in.role = role;
          *info = in;
        }
        const uint32_t tag = moves ? GBSGMC_TAG_SGLD
                             : L.kind == kLoopObabo
                                 ? (par == 0 ? GBSGMC_TAG_OBABO_1 : GBSGMC_TAG_OBABO_2)
                                 : L.kind == kLoopSghmc ? GBSGMC_TAG_SGHMC_STEP
                                                        : GBSGMC_TAG_AMAGOLD;
        const bool resample = L.kind == kLoopSghmc && (j + 1) % L.leapfrog == 0 &&
                              j + 1 < a.steps;
        for (int v = lane; v < dq; v += 32) {
          float xi[4];
          noise4(a.noise, who, 4 * v, d, k, tag, xi);
          xi_s[v] = make_float4(xi[0], xi[1], xi[2], xi[3]);
          if (resample) {
            noise4(a.noise, who, 4 * v, d, k + 1, GBSGMC_TAG_SGHMC_RESAMPLE, xi);
            xr_s[v] = make_float4(xi[0], xi[1], xi[2], xi[3]);
          }
        }
        if (want && a.inv_p2 > 0.0f && L.kind != kLoopLeapfrog) {
          float4 own[QPL];
#pragma unroll
          for (int i = 0; i < QPL; ++i) {
            const int v = lane + 32 * i;
            own[i] = v < dq ? w_s[v] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
          const double ww = warp_sum(lane_sum_squares<QPL>(own));
          if (lane == 0) sums[par * ncta + rank].v[3] = ww;
        }
      }
    }
    if (!clerk) {
      const int cnt = min(CH, R - q * CH);
      const float4* rows = rows_s + static_cast<int64_t>(buf_c) * CH * dq;
      const int32_t* ix = idx_s + slot_c * CH;
      for (int r0 = warp * RW; r0 < cnt; r0 += kStride) {
        float4 xv[RW][QPL];
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int k = 0; k < QPL; ++k) {
            const int v = lane + 32 * k;
            xv[r][k] = r0 + r < cnt && v < dq ? rows[(r0 + r) * dq + v]
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        int og = r0 + g < cnt ? ix[r0 + g] : -1;
        if (og >= a.n_rows) og = -1;
        const float yv = og >= 0 ? y_s[buf_c * CH + r0 + g] : 0.0f;
        consume_tile<QPL, RW>(a, nullptr, nullptr, r0, lane, g, leader, wq, xv, yv, og, A);
      }
    }
    if (++slot_c == L.idx_slots) slot_c = 0;
    if (++buf_c == depth) buf_c = 0;
    if (++q < L.chunks) continue;
    q = 0;

    // ---- the gradient's reduction --------------------------------------------
    if (!clerk) {
#pragma unroll
      for (int k = 0; k < QPL; ++k) {
        const int v = lane + 32 * k;
        if (v < dq) red[warp * dq + v] = A.acc[k];
      }
      if (leader) {
        lsum[warp * RW + g] = lane_sums<QPL>(A);
        if (!isfinite(A.mlk)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
      }
    }
    __syncthreads();
    const StepInfo in = *info;
    float4 gs = make_float4(0.f, 0.f, 0.f, 0.f);
    if (owner) {
      gs = red[tid];
#pragma unroll
      for (int w = 1; w < kRowWarps; ++w) {
        const float4 u = red[w * dq + tid];
        gs.x += u.x;
        gs.y += u.y;
        gs.z += u.z;
        gs.w += u.w;
      }
    }
    if (clerk && in.want_u) {
      double t[3];
      reduce_lane_sums(lsum, kRowWarps * RW, lane, t);
      if (lane == 0) {
        SliceSums* mine = sums + par * ncta + rank;
        mine->v[0] = t[0];
        mine->v[1] = t[1];
        mine->v[2] = t[2];
        if (ncta > 1) {
          const SliceSums out = *mine;
          const cg::cluster_group cl = cg::this_cluster();
          for (int r = 0; r < ncta; ++r)
            if (r != rank) *cl.map_shared_rank(mine, r) = out;
        }
      }
    }
    if (ncta > 1) {
      const cg::cluster_group cl = cg::this_cluster();
      if (owner && S > 1) {
        float4* mine = part + (par * S + slice) * dq + tid;
        for (int r = 0; r < S; ++r) *cl.map_shared_rank(mine, rank0 + r) = gs;
      }
      cluster_arrive();
      cluster_wait();
      if (owner && S > 1) {
        const float4* all = part + par * S * dq + tid;
        gs = all[0];
        for (int r = 1; r < S; ++r) {
          const float4 u = all[r * dq];
          gs.x += u.x;
          gs.y += u.y;
          gs.z += u.z;
          gs.w += u.w;
        }
      }
    }

    // ---- the update ------------------------------------------------------------
    if (owner) {
      const float gl[4] = {gs.x, gs.y, gs.z, gs.w};
      const float4 x4 = xi_s[tid];
      const float xi[4] = {x4.x, x4.y, x4.z, x4.w};
      float gv[4];
      bool bad = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        gv[i] = 4 * tid + i < d ? (-a.scale * gl[i] + xs[i] * a.inv_p2) * a.inv_temp : 0.0f;
        bad |= !isfinite(gv[i]);
      }
      if (bad) raise_status(a.status, GBSGMC_ERR_NONFINITE);
      if (moves) {
        const float noise_scale = sqrtf(2.0f * in.T * in.h);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float x = xs[i];
          const float scaled_gradient = -in.h * gv[i];
          const float scaled_noise = noise_scale * xi[i];
          if (aux_row != nullptr) {
            const float vn = a.alpha * as[i] + (1.0f - a.alpha) * (gv[i] * gv[i]);
            const float G = 1.0f / (a.lmbd + sqrtf(vn));
            const float sG = sqrtf(G);
            as[i] = vn;
            xs[i] = x + ((0.0f + G * scaled_gradient) + sG * scaled_noise);
          } else {
            xs[i] = x + (scaled_gradient + scaled_noise);
          }
        }
      } else if (L.kind == kLoopObabo) {
        const ObaboStep ob(in.h, in.T, L.friction);
        float ke = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (4 * tid + i >= d) break;
          if (par == 0) ob.first(mi[i], ms[i], gv[i], xi[i], as[i], xs[i], ke);
          else ob.second(mi[i], ms[i], gv[i], xi[i], as[i], ke);
        }
        ke_s[tid] = ke;
      } else if (L.kind == kLoopSghmc) {
        const float noise_scale = sqrtf(2.0f * in.h);
        const bool more = j + 1 < a.steps;
        const bool resample = more && (j + 1) % L.leapfrog == 0;
        const float4 r4 = xr_s[tid];
        const float xr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float pj = as[i] + (-in.h) * gv[i];
          pj = pj + L.friction * (noise_scale * xi[i]);
          if (resample) pj = ms[i] * xr[i];
          as[i] = pj;
        }
        // A kept step's state is this one, before the next step's position.
        if (in.slot >= 0 && slice == 0) {
          float* smp = a.samples + (static_cast<int64_t>(in.slot) * a.chains + unit) * d + 4 * tid;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (4 * tid + i < d) smp[i] = xs[i];
        }
        if (more) {
          const float h = in.h_next;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float pj = as[i];
            const float sm = mi[i] * pj;
            xs[i] = xs[i] + h * sm;
            as[i] = pj + (-h * L.friction) * sm;
          }
        }
      } else {  // reversible leapfrog
        const float decay = 1.0f - in.h * L.friction;
        const float inv = 1.0f / (1.0f + in.h * L.friction);
        const float ns = sqrtf(4.0f * L.friction * in.h);
        const float s = (j + 1 < a.steps ? 1.0f : 0.5f) * in.h;
        float en = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (4 * tid + i >= d) break;
          const float pj = as[i], gj = gv[i];
          const float noise_j = ns * (ms[i] * xi[i]);
          const float pn = inv * ((decay * pj + (-in.h) * gj) + noise_j);
          as[i] = pn;
          en += (pj + pn) * (mi[i] * gj);
          const float sm = mi[i] * pn;
          xs[i] = xs[i] + s * sm;
        }
        ke_s[tid] = 0.5f * in.h * en;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * tid + i >= d) xs[i] = as[i] = 0.f;
      w_s[tid] = make_float4(xs[0], xs[1], xs[2], xs[3]);
      if (in.slot >= 0 && slice == 0 && L.kind != kLoopSghmc &&
          (L.draws == 1 || par == 1)) {
        float* smp = a.samples + (static_cast<int64_t>(in.slot) * a.chains + unit) * d + 4 * tid;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (4 * tid + i < d) smp[i] = xs[i];
      }
    }
    if (clerk && in.want_u && !pairs) {
      const SliceSums* sp = sums + par * ncta;
      double U = glm_potential(a, slice_total(sp, S, 0), a.inv_p2 > 0.f ? sp[slice].v[3] : 0.0);
      if (!isfinite(U) && lane == 0) raise_status(a.status, GBSGMC_ERR_NONFINITE);
      if (L.kind == kLoopObabo) {
        if (par == 0) U_first = U;
        else U = 0.5 * (U_first + U);
      }
      U_mine = U;
      var_mine = glm_variance(a, slice_total(sp, S, 1), slice_total(sp, S, 2));
      if (in.slot >= 0 && a.sample_lik != nullptr && slice == 0 && lane == 0 &&
          (L.draws == 1 || par == 1))
        a.sample_lik[static_cast<int64_t>(in.slot) * a.chains + unit] = moves ? -U : U;
    }
    ++e;
  }

  // ---- the block's end -----------------------------------------------------------
  cp_wait(0);
  __syncthreads();
  if (clerk) {
    if (pairs) {
      decide(k0 + a.steps - 1, (events - 1) & 1);
      if (lane == 0) info->role = role;
    }
    if (L.energy != nullptr || L.ke != nullptr) ke_acc[L.draws == 2 ? 1 : 0] += energy_sum();
    if (lane == 0 && slice == 0) {
      if (pairs) {
        const int row = role ? L.pairs + unit : unit;
        a.U[row] = U_pair[half];
        a.lk_var[row] = var_pair[half];
        L.ident[row] = who;
        if (half == 0) {
          L.ssq[unit] = ssq;
          L.kc[unit] = kc;
          if (L.counts != nullptr) L.counts[unit] += exchanges;
        }
      } else {
        if (L.kind != kLoopLeapfrog) {
          if (a.U != nullptr) a.U[unit] = U_mine;
          if (a.lk_var != nullptr) a.lk_var[unit] = var_mine;
        }
        if (L.kind == kLoopObabo && L.ke != nullptr) {
          L.ke[unit] += ke_acc[0];
          L.ke[a.chains + unit] += ke_acc[1];
        }
        if (L.kind == kLoopLeapfrog) L.energy[unit] += ke_acc[0];
      }
    }
  }
  __syncthreads();
  if (owner && slice == 0) {
    const int row = pairs ? (info->role ? L.pairs + unit : unit) : row_in;
    float* xo = a.w + static_cast<int64_t>(row) * d;
    float* ao = L.aux != nullptr ? L.aux + static_cast<int64_t>(row) * d : nullptr;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (4 * tid + i >= d) break;
      xo[4 * tid + i] = xs[i];
      if (ao != nullptr) ao[4 * tid + i] = as[i];
    }
  }
}

size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// Fills the chunk sizes and shared-memory offsets of a launch; returns its
// shared memory, or 0 when no chunk fits.  A CTA's whole slice of a minibatch
// is one chunk when three such chunks fit (two minibatches ahead of the one
// being consumed); longer slices stream through up to four smaller chunks.
size_t loop_layout(LoopArgs& L, int rw, int ncta, size_t limit) {
  const int dq = L.g.dq, stride = kRowWarps * rw, R = L.g.rows_per_slice;
  const size_t row = static_cast<size_t>(dq) * 16;
  const auto fixed = [&]() {
    return 16 + kRowWarps * row + (L.ctas > 1 ? 2 * L.ctas * row : 0) + 3 * row +
           align16(4 * kRowThreads) + align16(sizeof(LaneSums) * kRowWarps * rw) +
           sizeof(SliceSums) * 2 * ncta + align16(sizeof(StepInfo)) + 64;
  };
  const auto ring = [&](int depth, int rows) {
    return depth * static_cast<size_t>(rows) * (row + 4) + (2 * depth - 1) * 4ull * rows;
  };
  if (fixed() >= limit) return 0;
  const size_t room = limit - fixed();
  const int whole = ceil_div(R, stride) * stride;
  int depth = 0, rows = 0;
  if (ring(3, whole) <= room) {
    depth = 3;
    rows = whole;
  } else {
    for (int dp = kMaxDepth; dp >= 2 && depth == 0; --dp) {
      const size_t per = ring(dp, stride);
      const int m = static_cast<int>(room / per);
      if (m >= 1) {
        depth = dp;
        rows = std::min(m * stride, whole);
      }
    }
    if (depth == 0) return 0;
  }
  L.depth = depth;
  L.chunk_rows = rows;
  L.chunks = std::max(1, ceil_div(R, rows));
  L.idx_slots = 2 * depth - 1;
  size_t o = static_cast<size_t>(depth) * rows * row;
  const auto take = [&](size_t bytes) {
    const size_t at = o;
    o += align16(bytes);
    return static_cast<unsigned>(at);
  };
  L.o_y = take(4ull * depth * rows);
  L.o_idx = take(4ull * L.idx_slots * rows);
  L.o_red = take(kRowWarps * row);
  L.o_part = take(L.ctas > 1 ? 2 * L.ctas * row : 0);
  L.o_w = take(row);
  L.o_xi = take(row);
  L.o_xr = take(row);
  L.o_ke = take(4 * kRowThreads);
  L.o_lane = take(sizeof(LaneSums) * kRowWarps * rw);
  L.o_sums = take(sizeof(SliceSums) * 2 * ncta);
  L.o_step = take(sizeof(StepInfo));
  return o;
}

constexpr size_t kSmemOne = 220 * 1024;   // one CTA per SM
constexpr size_t kSmemTwo = 110 * 1024;   // two CTAs per SM

template <int QPL, int RW>
struct LoopVariant {
  static int prepare() {
    static int done = 0;
    if (done) return GBSGMC_OK;
    const cudaError_t e =
        cudaFuncSetAttribute(glm_loop_kernel<QPL, RW>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemOne);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "glm_loop: cudaFuncSetAttribute: %s",
                       cudaGetErrorString(e));
    done = 1;
    return GBSGMC_OK;
  }
  static int launch(LoopArgs& L, int units, int ncta, cudaStream_t st) {
    int rc = prepare();
    if (rc != GBSGMC_OK) return rc;
    const bool sparse = static_cast<int64_t>(units) * ncta <= glm_sm_count();
    const size_t smem = loop_layout(L, RW, ncta, sparse || QPL > 2 ? kSmemOne : kSmemTwo);
    if (smem == 0)
      return set_error(GBSGMC_ERR_SHAPE, "glm_loop: shared memory too large");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(units) * ncta);
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ncta;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, glm_loop_kernel<QPL, RW>, L);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "glm_loop: %s", cudaGetErrorString(e));
    return check_launch("glm_loop");
  }
};

}  // namespace

// CTAs per chain: as many as give every row warp a tile (n / (8 RW)) while
// all CTAs of the launch still find an SM of their own, in powers of two up
// to the portable cluster size.
int glm_loop_ctas(int units, int chains_per_unit, int n, int d) {
  const int rw = glm_rows_per_warp((d + 3) / 4);
  const int most = kMaxCtas / chains_per_unit;
  const char* env = std::getenv("GBSGMC_GLM_SLICES");
  const int forced = env != nullptr ? std::atoi(env) : 0;
  int s = 1;
  if (forced > 0) {
    while (2 * s <= std::min(forced, most)) s *= 2;
    return s;
  }
  while (2 * s <= most && n >= 2 * s * kRowWarps * rw &&
         static_cast<int64_t>(units) * chains_per_unit * 2 * s <= glm_sm_count())
    s *= 2;
  return s;
}

int glm_loop_prepare() {
  int rc = LoopVariant<1, 2>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<1, 4>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<1, 8>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<2, 2>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<2, 4>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<2, 8>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<4, 2>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<8, 1>::prepare();
  return rc;
}

int glm_loop(const GlmLoopCall& c, cudaStream_t st) {
  if (c.model == nullptr || c.x == nullptr || c.sched == nullptr || c.noise == nullptr ||
      c.steps < 1 || c.ctas < 1)
    return set_error(GBSGMC_ERR_ARG, "glm_loop: bad argument");
  const bool pairs = c.kind == kLoopPairs;
  if (c.kind != kLoopSgld && !pairs && c.aux == nullptr)
    return set_error(GBSGMC_ERR_ARG, "glm_loop: needs a momentum buffer");
  if (c.sched->keep_slot_dev != nullptr && c.samples == nullptr)
    return set_error(GBSGMC_ERR_ARG, "glm_loop: keep table given without sample buffer");
  if (c.noise->noise_dev != nullptr)
    return set_error(GBSGMC_ERR_ARG, "glm_loop: injected noise needs one step per launch");
  LoopArgs L = {};
  GlmTune t;
  t.slices = c.ctas;
  t.rows_per_warp = 4;
  int rc = glm_fill_args(L.g, c.model, c.chains, c.n, c.idx, c.idx_stride, nullptr, nullptr, 0,
                         c.status, t);
  if (rc != GBSGMC_OK) return rc;
  if (c.chains == 0 || c.n == 0) return GBSGMC_OK;
  L.g.mode = kSgldStep;
  L.g.steps = c.steps;
  L.g.idx_step_stride = c.idx_step_stride;
  L.g.slices = c.ctas;
  L.g.rows_per_slice = ceil_div(c.n, c.ctas);
  L.g.w = c.x;
  L.g.alpha = c.alpha;
  L.g.lmbd = c.lmbd;
  L.g.sched = to_sched(c.sched);
  L.g.noise = to_noise(c.noise);
  L.g.U = c.U;
  L.g.lk_var = c.lk_var;
  L.g.samples = c.samples;
  L.g.sample_lik = c.sample_lik;
  L.kind = c.kind;
  L.draws = c.kind == kLoopObabo ? 2 : 1;
  L.leapfrog = c.leapfrog;
  L.friction = c.friction;
  L.mass = c.mass;
  L.aux = c.aux;
  L.ke = c.kind == kLoopObabo ? c.ke : nullptr;
  L.energy = c.kind == kLoopLeapfrog ? c.energy : nullptr;
  L.ctas = c.ctas;
  L.row_shift = 0;
  while (L.row_shift < 5 && (1 << L.row_shift) < L.g.dq) ++L.row_shift;
  int units = c.chains, ncta = c.ctas;
  if (pairs) {
    units = L.pairs = c.chains / 2;
    ncta = 2 * c.ctas;
    L.F = c.F;
    L.swap_seed = c.swap_seed;
    L.pair_chain = c.pair_chain;
    L.ident = c.ident;
    L.ssq = c.ssq;
    L.kc = c.k;
    L.counts = c.counts;
  }
  if (ncta > kMaxCtas) return set_error(GBSGMC_ERR_SHAPE, "glm_loop: too many CTAs per cluster");
  const int qpl = glm_qpl(L.g.dq);
  const int rw = c.rows_per_warp > 0 ? c.rows_per_warp : glm_rows_per_warp(L.g.dq);
  if (qpl == 1)
    return rw == 8   ? LoopVariant<1, 8>::launch(L, units, ncta, st)
           : rw == 4 ? LoopVariant<1, 4>::launch(L, units, ncta, st)
                     : LoopVariant<1, 2>::launch(L, units, ncta, st);
  if (qpl == 2)
    return rw == 8   ? LoopVariant<2, 8>::launch(L, units, ncta, st)
           : rw == 4 ? LoopVariant<2, 4>::launch(L, units, ncta, st)
                     : LoopVariant<2, 2>::launch(L, units, ncta, st);
  if (qpl == 4) return LoopVariant<4, 2>::launch(L, units, ncta, st);
  return LoopVariant<8, 1>::launch(L, units, ncta, st);
}

}  // namespace gbsgmc
