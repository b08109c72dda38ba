// Whole blocks of integrator steps on the GLM potentials in one launch: SGLD
// (+RMSprop), OBABO, SGHMC, the reversible leapfrog of AMAGOLD, and reSGLD
// (normal, hot) pairs with their exchange.
//
// What bounds a step of a small chain is not its bytes (a minibatch of 128
// rows of 32 features is 16 KB) but the chain of dependent latencies: index
// load, row load, dot products, block reduction, update, next step; and, with
// a launch per gradient and per update, the launches between them.  Here a
// cluster of S CTAs owns a chain for the whole block, and in each CTA
//   * the copy warps run ahead: the minibatches of a block are known before it
//     starts, so they gather the rows of the next chunks into a ring of shared
//     memory buffers (full / empty mbarriers), up to `depth` chunks before
//     they are needed.  Issuing the copies is what bounds a step of more than
//     about 16 rows a CTA: a cp.async per 16 bytes took a copy warp 110 cycles
//     a row of 101 features, a bulk copy per row (each lane its own) is better
//     (24 chains of 500 such rows: 3.8 to 3.0 us a gradient) and a gather of
//     four rows per instruction takes the copies off the critical path (1.9
//     us; 64 chains of 512 rows of 32 features 299 to 136 us a 50 steps, 64
//     of 128 features 307 to 153; never slower);
//   * the row warps do what nothing else can do earlier: row tiles of the
//     chunk by glm_kernel's code, the reduction, the exchange and the update.
//     The slices (glm_loop_ctas) and rows per warp (loop_rows_per_warp) are this
//     kernel's own, so its sums have other orders than glm_kernel's unless these
//     coincide, and a chain's bits depend on how many chains run beside it.  CTA s holds rows [s R, (s + 1) R) of every minibatch; it sends
//     its partial gradient into all CTAs of the cluster (st.async, counted on
//     the receivers' mbarriers), and every CTA adds the partials in slice
//     order and updates its own copy of x, held in registers, so no second
//     exchange is needed;
//   * the noise warp draws the next gradient's Philox normals one gradient
//     ahead, and the clerk warp reads the schedule and does the FP64 work (U,
//     var(lk), kinetic energies, the exchange decision).
// reSGLD pairs: both chains of a pair share a cluster (2 S CTAs).  An
// exchange swaps the chains' roles (temperature, slot) instead of their
// states; the rows are written to the slots they ended in when the block
// ends.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "glm.cuh"
#include "internal.h"
#include "tc.cuh"
#include "tc_gemm.cuh"

namespace gbsgmc {
namespace {

constexpr int kRowWarps = 8;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kCopyWarps = 2;
constexpr int kCopyThreads = kCopyWarps * 32;
constexpr int kClerkWarp = kRowWarps;
constexpr int kNoiseWarp = kRowWarps + 1;
constexpr int kLoopThreads = kRowThreads + 64 + kCopyThreads;  // 168 registers a thread
constexpr int kMaxCtas = 8;                     // portable cluster size
constexpr uint64_t kLingerNs = 1000000;         // copies and sends in flight land in microseconds
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
  int chunk_rows, chunks, depth;
  int row_quads;   // 16-byte words of a row in shared memory
  int cp_y;        // y is copied by itself: rows are not aligned, or it is not in them
  int cp_async;    // some copies are made by cp.async
  int gather;      // rows are copied four at a time
  int row_cols;    // floats of a row that are read (16-byte words)
  uint64_t wait_ns;  // bound of each wait
  int missing;     // arrivals that a chunk waits for and that never come
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
  unsigned o_y, o_idx, o_red, o_part, o_w, o_xi, o_xr, o_ke, o_lane, o_sums, o_step, o_pair, o_bar;
};

// What the clerk hands the row warps for one gradient.
struct StepInfo {
  float h, h_next;
  float c[4];     // the integrator's coefficients (step_coefs)
  int want_next;  // want_u of the next gradient
  int slot;       // sample slot of this step, or -1
  int prev_slot;  // pairs: the previous step's slot if this chain is to store it
  int want_u;     // the clerk waits for this gradient's likelihood sums
};

// Pairs: what a decision needs besides the sums.
struct PairConsts {
  double dbeta, sa, log_u, pad;
};

struct LoopBars {
  uint64_t full[kMaxDepth], empty[kMaxDepth];
  uint64_t part[2], sums[2];
  int stop;  // a wait ran out: the remaining ones give up at once
};

// 4 bytes global -> shared, or zeros when !ok.
__device__ __forceinline__ void cp4(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src),
               "r"(ok ? 4 : 0)
               : "memory");
}
// This thread's cp4 so far count as one arrival on `bar` when they land.
__device__ __forceinline__ void cp_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
// Bytes of bulk copies to come, counted on the barrier's current phase.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// Named barriers (ids below 16): sync waits, arrive does not.
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kBarRows = 1;   // the row warps among themselves
constexpr int kBarStep = 2;   // + parity: partials, noise and the clerk's hand-over are ready
constexpr int kBarSums = 4;   // + parity: rows -> clerk, the likelihood sums
constexpr int kBarDone = 6;   // + parity: rows -> clerk, the update is done
constexpr int kBarFree = 8;   // + parity: rows -> noise warp, the normals have been used
constexpr int kBarEnd = 10;   // clerk -> rows, the last decision
constexpr int kBarInit = 11;  // rows -> clerk, the first x is in shared memory
constexpr int kWithOne = kRowThreads + 32;
constexpr int kWithBoth = kRowThreads + 64;

// Address of `p` (this CTA's shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  return a;
}
// 4 or 16 bytes to another CTA of the cluster, counted on that CTA's mbarrier.
__device__ __forceinline__ void send4(uint32_t dst, uint32_t bar, float v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                   dst),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send16(uint32_t dst, uint32_t bar, uint32_t x, uint32_t y,
                                       uint32_t z, uint32_t w) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
      ::"r"(dst), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}
// Bounded wait for phase `phase` of a barrier; false when it ran out.  The caller
// then takes no further part in any barrier exchange (no copies, sends or
// arrivals: the phases are no longer those that it counts) and runs through to
// the kernel's end, so that the named barriers stay matched.
__device__ __forceinline__ bool wait_phase(const LoopArgs& L, LoopBars* b, uint64_t* bar,
                                           int phase) {
  if (mbar_try_wait(bar, phase & 1)) return true;
  if (mbar_wait_bounded(bar, phase & 1, &b->stop, L.wait_ns)) return true;
  b->stop = 1;
  raise_status(L.g.status, GBSGMC_ERR_TIMEOUT);
  return false;
}
__device__ __forceinline__ bool stopped(const LoopBars* b) {
  return *static_cast<const volatile int*>(&b->stop) != 0;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// What an update needs of the schedule alone: SGLD and SGHMC the noise scale
// (c[0]); OBABO keep, inject and the half step; the leapfrog decay, 1 / (1 + h
// f) and the noise scale.
__device__ __forceinline__ void step_coefs(int kind, float h, float T, float friction,
                                           float (&c)[4]) {
  if (kind == kLoopObabo) {
    const float permanence = expf(-friction * h);
    c[0] = sqrtf(permanence);
    c[1] = sqrtf((1.0f - permanence) * T);
    c[2] = 0.5f * h;
  } else if (kind == kLoopSghmc) {
    c[0] = sqrtf(2.0f * h);
  } else if (kind == kLoopLeapfrog) {
    c[0] = 1.0f - h * friction;
    c[1] = 1.0f / (1.0f + h * friction);
    c[2] = sqrtf(4.0f * friction * h);
  } else {
    c[0] = sqrtf(2.0f * T * h);
  }
}

// The OBABO halves of one parameter, rounded as update.cu's kernels do; each
// returns the factors of the parameter's kinetic energy.
__device__ __forceinline__ float2 obabo_first(const StepInfo& q, float mi, float ms, float g,
                                              float xi, float& p, float& x) {
  float pj = __fmaf_rn(q.c[0], p, __fmul_rn(q.c[1], __fmul_rn(ms, xi)));
  const float2 ke = make_float2(__fmul_rn(0.5f, pj), __fmul_rn(mi, pj));
  pj = __fmaf_rn(-q.c[2], g, pj);
  p = pj;
  x = __fmaf_rn(q.h, __fmul_rn(mi, pj), x);
  return ke;
}
__device__ __forceinline__ float2 obabo_second(const StepInfo& q, float mi, float ms, float g,
                                               float xi, float& p) {
  const float pj = __fmaf_rn(-q.c[2], g, p);
  p = __fmaf_rn(q.c[0], pj, __fmul_rn(q.c[1], __fmul_rn(ms, xi)));
  return make_float2(__fmul_rn(0.5f, pj), __fmul_rn(mi, pj));
}

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
__device__ __forceinline__ void loop_roles(const LoopArgs& L, const CUtensorMap& map,
                                           unsigned char* smem) {
  constexpr int LOG = Log2<RW>::v;
  constexpr int GROUP = 32 >> LOG;
  constexpr int kStride = kRowWarps * RW;
  constexpr int kMaxOwned = QPL <= 2 ? 1 : QPL / 2;   // parameters of a row thread
  const GlmArgs& a = L.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int dq = a.dq, d = a.d, rq = L.row_quads, S = L.ctas, CH = L.chunk_rows, depth = L.depth;
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

  float4* rows_s = reinterpret_cast<float4*>(smem);
  float* y_s = reinterpret_cast<float*>(smem + L.o_y);
  int32_t* idx_s = reinterpret_cast<int32_t*>(smem + L.o_idx);
  float4* red = reinterpret_cast<float4*>(smem + L.o_red);
  float4* part = reinterpret_cast<float4*>(smem + L.o_part);   // [2][S][dq]
  float4* w_s = reinterpret_cast<float4*>(smem + L.o_w);       // [2][dq]
  float4* xi_s = reinterpret_cast<float4*>(smem + L.o_xi);     // [2][dq]
  float4* xr_s = reinterpret_cast<float4*>(smem + L.o_xr);     // [2][dq] (SGHMC resample)
  float2* ke_s = reinterpret_cast<float2*>(smem + L.o_ke);     // [2][4 dq] energy factors
  LaneSums* lsum = reinterpret_cast<LaneSums*>(smem + L.o_lane);    // [2][kRowWarps RW]
  SliceSums* sums = reinterpret_cast<SliceSums*>(smem + L.o_sums);  // [2][ncta]
  StepInfo* info = reinterpret_cast<StepInfo*>(smem + L.o_step);    // [2]
  PairConsts* pair_c = reinterpret_cast<PairConsts*>(smem + L.o_pair);  // [4]
  LoopBars* bars = reinterpret_cast<LoopBars*>(smem + L.o_bar);

  if (tid == 0) {
    for (int i = 0; i < depth; ++i) {
      mbar_init(bars->full + i, kCopyWarps + (L.cp_async ? kCopyThreads : 0) + L.missing);
      mbar_init(bars->empty + i, kRowWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars->part + i, 1);
      mbar_init(bars->sums + i, 1);
    }
    bars->stop = 0;
    mbar_fence_init();
    for (int i = 0; i < 2; ++i) {
      mbar_arrive_expect_tx(bars->part + i, static_cast<uint32_t>(S) * d * 4);
      mbar_arrive_expect_tx(bars->sums + i, static_cast<uint32_t>(ncta) * sizeof(SliceSums));
    }
  }
  __syncthreads();
  if (ncta > 1) {  // every CTA runs, and its barriers exist, before any remote write
    cluster_arrive();
    cluster_wait();
  }

  // ============================== copy warps ====================================
  if (warp > kNoiseWarp) {
    const int cw = warp - kNoiseWarp - 1;
    const int share = (CH + kCopyWarps - 1) / kCopyWarps;   // rows of a chunk per copy warp
    const float* X = a.X;
    const float* yv = a.y;
    const int64_t ld = a.ld, n_rows = a.n_rows;
    const int vec4 = a.vec4, y_inline = a.y_inline, chunks = L.chunks;
    const uint32_t row_bytes = static_cast<uint32_t>(rq) * 16;
    int buf = 0, use = 0;  // ring position, times round the ring
    bool live = true;      // no wait has run out
    for (int e = 0; live && e < events; ++e) {
      const int32_t* src = a.idx + (L.draws == 2 ? e >> 1 : e) * a.idx_step_stride +
                           static_cast<int64_t>(who) * a.idx_stride +
                           (L.draws == 2 ? (e & 1) * a.n : 0) + row0;
      for (int q = 0; q < chunks; ++q) {
        const int cnt = min(CH, R - q * CH);
        const int r_end = min(cnt, (cw + 1) * share);
        float4* dst = rows_s + buf * CH * rq;
        const int32_t* at = src + q * CH;
        int* idx_b = idx_s + buf * CH;
        float* y_b = y_s + buf * CH;
        if (L.gather) {
          // Lane l takes rows 4 l .. 4 l + 3 of each 128.  An index out of
          // range, or past the chunk, is sent to the row after the last one,
          // which the copy reads as zeros.
          int o[4];
          const auto fetch = [&](int r) {
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = r + j < r_end ? __ldg(at + r + j) : -1;
          };
          fetch(cw * share + 4 * lane);
          if (use > 0)
            live = __all_sync(0xffffffffu,
                              wait_phase(L, bars, bars->empty + buf, use - 1));
          if (!live) break;
          for (int r0 = cw * share; r0 < r_end; r0 += 128) {
            const int r = r0 + 4 * lane;
            if (r0 > cw * share) fetch(r);
            if (lane == 0)
              mbar_expect_tx(bars->full + buf, min(32, (r_end - r0 + 3) / 4) * 4 * row_bytes);
            __syncwarp();
            if (r < r_end) {
              int at_row[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (r + j < r_end && (o[j] < 0 || o[j] >= n_rows)) {
                  raise_status(a.status, GBSGMC_ERR_INDEX);
                  o[j] = -1;
                }
                at_row[j] = o[j] < 0 ? static_cast<int>(n_rows) : o[j];
              }
              tc::tma_gather4(dst + r * rq, &map, 0, at_row[0], at_row[1], at_row[2], at_row[3],
                              bars->full + buf);
              *reinterpret_cast<int4*>(idx_b + r) = make_int4(o[0], o[1], o[2], o[3]);
              if (L.cp_y) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  if (o[j] >= 0) cp4(y_b + r + j, yv + o[j], true);
              }
            }
          }
        } else {
          int o = cw * share + lane < r_end ? __ldg(at + cw * share + lane) : -1;
          if (use > 0)
            live = __all_sync(0xffffffffu,
                              wait_phase(L, bars, bars->empty + buf, use - 1));
          if (!live) break;
          for (int r0 = cw * share; r0 < r_end; r0 += 32) {
            const int r = r0 + lane;
            if (r0 > cw * share) o = r < r_end ? __ldg(at + r) : -1;
            if (r < r_end) {
              if (o < 0 || o >= n_rows) {   // left out: its row is zero
                raise_status(a.status, GBSGMC_ERR_INDEX);
                o = -1;
                for (int v = 0; v < rq; ++v) dst[r * rq + v] = make_float4(0.f, 0.f, 0.f, 0.f);
                tc::fence_async_shared();
              }
              idx_b[r] = o;
              if (o >= 0 && L.cp_y) cp4(y_b + r, y_inline ? X + o * ld + d : yv + o, true);
            }
            if (vec4) {   // one copy a row, its y with it
              const unsigned live = __ballot_sync(0xffffffffu, o >= 0);
              if (lane == 0) mbar_expect_tx(bars->full + buf, __popc(live) * row_bytes);
              __syncwarp();
              if (o >= 0) bulk_g2s(dst + r * rq, X + o * ld, row_bytes, bars->full + buf);
            } else {
              for (int i = 0; i < min(32, r_end - r0); ++i) {
                const int oi = __shfl_sync(0xffffffffu, o, i);
                if (oi < 0) continue;
                float* out = reinterpret_cast<float*>(dst + (r0 + i) * rq);
                for (int j = lane; j < 4 * dq; j += 32)
                  cp4(out + j, X + oi * ld + (j < d ? j : 0), j < d);
              }
            }
          }
        }
        if (L.cp_async) cp_arrive(bars->full + buf);
        __syncwarp();
        if (lane == 0) mbar_arrive(bars->full + buf);
        if (++buf == depth) {
          buf = 0;
          ++use;
        }
      }
    }
    // No copy is in flight when the CTA ends, even if a wait has run out (the
    // other copy warp may then have left its part out: a short bound).
    for (int i = 0; i < depth; ++i) {
      const int last = use - (i < buf ? 0 : 1);
      if (last >= 0)
        mbar_wait_bounded(bars->full + i, last & 1, nullptr, live ? kWaitLimitNs : kLingerNs);
    }
    return;
  }

  const int64_t k0 = a.sched.step();

  // ============================== the noise warp ================================
  if (warp == kNoiseWarp) {
    const uint32_t tag0 = moves ? GBSGMC_TAG_SGLD
                          : L.kind == kLoopObabo ? GBSGMC_TAG_OBABO_1
                          : L.kind == kLoopSghmc ? GBSGMC_TAG_SGHMC_STEP
                                                 : GBSGMC_TAG_AMAGOLD;
    const uint64_t key = pairs ? (L.swap_seed << 32) |
                                     static_cast<uint32_t>(__ldg(L.pair_chain + unit))
                               : 0;
    int64_t kc = pairs ? L.kc[unit] : 0;
    for (int e = 0; e < events; ++e) {
      if (e > 1) bar_sync(kBarFree + (e & 1), kWithOne);  // update e - 2 is done
      const int j = L.draws == 2 ? e >> 1 : e;
      const int64_t k = k0 + j;
      const uint32_t tag = L.draws == 2 ? tag0 + (e & 1) : tag0;
      const bool resample =
          L.kind == kLoopSghmc && (j + 1) % L.leapfrog == 0 && j + 1 < a.steps;
      for (int v = lane; v < dq; v += 32) {
        float xi[4];
        noise4(a.noise, who, 4 * v, d, k, tag, xi);
        xi_s[(e & 1) * dq + v] = make_float4(xi[0], xi[1], xi[2], xi[3]);
        if (resample) {
          noise4(a.noise, who, 4 * v, d, k + 1, GBSGMC_TAG_SGHMC_RESAMPLE, xi);
          xr_s[(e & 1) * dq + v] = make_float4(xi[0], xi[1], xi[2], xi[3]);
        }
      }
      if (pairs) {
        const double T = a.sched.temperature(k, (lane & 1) ? L.pairs + unit : unit);
        kc += 1;
        // Lanes 0, 1: 1 / T of the normal and the hot slot; others: 1 / k.
        const double inv = 1.0 / (lane < 2 ? T : static_cast<double>(kc));
        const double b0 = __shfl_sync(0xffffffffu, inv, 0), b1 = __shfl_sync(0xffffffffu, inv, 1);
        if (lane == 2)   // four steps deep: the clerk may lag two behind
          pair_c[e & 3] = PairConsts{
              b0 - b1, inv, log(swap_uniform(key, 0u, static_cast<uint32_t>(k + 1))), 0.0};
        __syncwarp();
      }
      bar_arrive(kBarStep + (e & 1), kWithBoth);
    }
    // Each kBarFree generation that the rows complete is matched here.
    for (int e = max(events - 2, 0); e < events; ++e) bar_sync(kBarFree + (e & 1), kWithOne);
    return;
  }

  // ============================== the clerk =====================================
  if (warp == kClerkWarp) {
    double ke_acc[2] = {0.0, 0.0};
    double U_first = 0.0, U_last = 0.0, var_last = 0.0;
    double ssq = pairs ? L.ssq[unit] : 0.0;
    int exchanges = 0, role = half, wants = 0;
    int done_slot = -1;  // pairs: sample slot of the step last decided
    bool live = true;    // no wait has run out
    const bool energies = L.energy != nullptr || L.ke != nullptr;
    StepInfo in = {};
    auto wanted = [&](int j, int slot) {
      return L.kind != kLoopLeapfrog && (pairs || j + 1 == a.steps || slot >= 0);
    };
    // The schedule of gradient e (its temperature and role come when the
    // previous step's exchange is decided).
    auto prepare = [&](int e) {
      const int j = L.draws == 2 ? e >> 1 : e;
      const int jn = L.draws == 2 ? (e + 1) >> 1 : e + 1;
      const int64_t k = k0 + j;
      in.h = a.sched.step_size(k);
      in.h_next = j + 1 < a.steps ? a.sched.step_size(k + 1) : in.h;
      in.slot = a.sched.keep_slot(k);
      in.want_u = wanted(j, in.slot);
      in.want_next = jn < a.steps && wanted(jn, a.sched.keep_slot(k0 + jn));
    };
    auto hand_over = [&](int e) {
      const int64_t k = k0 + (L.draws == 2 ? e >> 1 : e);
      StepInfo out = in;
      step_coefs(L.kind, in.h,
                 a.sched.temperature(k, pairs ? (role ? L.pairs + unit : unit) : unit),
                 L.friction, out.c);
      out.prev_slot = -1;
      if (pairs) {
        out.prev_slot = role == 0 ? done_slot : -1;
        out.slot = -1;
      }
      if (lane == 0) info[e & 1] = out;
      __syncwarp();
      bar_arrive(kBarStep + (e & 1), kWithBoth);
    };
    // FP64 sum of the energy parts of update e in the order of update.cu's
    // kernels: a part is four parameters' products, added in turn in FP32.
    auto take_energy = [&](int e) {
      if (!energies) return;
      const float2* p = ke_s + (e & 1) * 4 * dq;
      const int64_t k = k0 + (L.draws == 2 ? e >> 1 : e);
      const float half_h = L.kind == kLoopLeapfrog ? 0.5f * a.sched.step_size(k) : 0.f;
      double t = 0.0;
      for (int w0 = 0; w0 < dq; w0 += 32) {
        float part = 0.f;
        if (w0 + lane < dq) {
          for (int i = 0; i < 4 && 4 * (w0 + lane) + i < d; ++i) {
            const float2 f = p[4 * (w0 + lane) + i];
            part = __fmaf_rn(f.x, f.y, part);
          }
          if (L.kind == kLoopLeapfrog) part = half_h * part;
        }
        t += warp_sum(static_cast<double>(part));
      }
      ke_acc[L.draws == 2 ? e & 1 : 0] += t;
    };

    prepare(0);
    hand_over(0);
    bar_sync(kBarInit, kWithOne);
    for (int e = 0; e < events; ++e) {
      const int want = in.want_u, slot = in.slot;
      if (e > 0) {
        bar_sync(kBarDone + ((e - 1) & 1), kWithOne);
        take_energy(e - 1);
      }
      double ww = 0.0;
      if (want && a.inv_p2 > 0.0f) {
        float4 own[QPL];
#pragma unroll
        for (int i = 0; i < QPL; ++i) {
          const int v = lane + 32 * i;
          own[i] = v < dq ? w_s[(e & 1) * dq + v] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        ww = warp_sum(lane_sum_squares<QPL>(own));
      }
      if (e + 1 < events) prepare(e + 1);
      if (want) {
        bar_sync(kBarSums + (e & 1), kWithOne);
        double t[3];
        reduce_lane_sums(lsum + (e & 1) * kRowWarps * RW, kRowWarps * RW, lane, t);
        SliceSums* all = sums + (wants & 1) * ncta;
        if (live && lane < ncta) {
          const uint32_t dst = cluster_addr(all + rank, lane);
          const uint32_t bar = cluster_addr(bars->sums + (wants & 1), lane);
          const double v[4] = {t[0], t[1], t[2], ww};
#pragma unroll
          for (int i = 0; i < 2; ++i)
            send16(dst + 16 * i, bar, __double2loint(v[2 * i]), __double2hiint(v[2 * i]),
                   __double2loint(v[2 * i + 1]), __double2hiint(v[2 * i + 1]));
        }
        live &= __all_sync(0xffffffffu,
                           wait_phase(L, bars, bars->sums + (wants & 1), wants >> 1)) != 0;
        if (live && lane == 0 && e + 1 < events)
          mbar_arrive_expect_tx(bars->sums + (wants & 1),
                                static_cast<uint32_t>(ncta) * sizeof(SliceSums));
        ++wants;
        // Means over the minibatch by chain (lane & 1) and sum (lane >> 1),
        // so that their divisions run side by side.
        const int h = pairs ? lane & 1 : 0, which = (lane >> 1) % 3;
        const double mean = slice_total(all + h * S, S, which) / a.n;
        const double prior = a.inv_p2 > 0.f ? all[h * S].v[3] : 0.0;
        double U = glm_potential_mean(a, __shfl_sync(0xffffffffu, mean, lane & 1), prior);
        double var = glm_variance_mean(__shfl_sync(0xffffffffu, mean, 2 + (lane & 1)),
                                       __shfl_sync(0xffffffffu, mean, 4 + (lane & 1)));
        if (!pairs) {
          U = __shfl_sync(0xffffffffu, U, 0);
          var = __shfl_sync(0xffffffffu, var, 0);
          if (!isfinite(U) && lane == 0) raise_status(a.status, GBSGMC_ERR_NONFINITE);
          if (L.draws == 2) {
            if ((e & 1) == 0) U_first = U;
            else U = 0.5 * (U_first + U);
          }
          U_last = U;
          var_last = var;
          if (slot >= 0 && a.sample_lik != nullptr && slice == 0 && lane == 0 &&
              (L.draws == 1 || (e & 1)))
            a.sample_lik[static_cast<int64_t>(slot) * a.chains + unit] = moves ? -U : U;
        } else {
          // The exchange decision after step k: the roles swap when
          // log u >= log s (the reference keeps the pair when log u < log s,
          // lax.cond's true branch).
          const double dbeta = pair_c[e & 3].dbeta, sa = pair_c[e & 3].sa;
          const double log_u = pair_c[e & 3].log_u;
          const int n_chain = half ^ role;  // the chain in the normal slot
          const double Un = __shfl_sync(0xffffffffu, U, n_chain);
          const double Uh = __shfl_sync(0xffffffffu, U, n_chain ^ 1);
          ssq = (1.0 - sa) * ssq + sa * __shfl_sync(0xffffffffu, var, n_chain);
          const double corr = dbeta * ssq;
          const double log_s = dbeta * (Un - Uh - (L.F == 1.0 ? corr : corr / L.F));
          if (!(log_u < log_s)) {
            role ^= 1;
            ++exchanges;
          }
          U_last = __shfl_sync(0xffffffffu, U, half);
          var_last = __shfl_sync(0xffffffffu, var, half);
          done_slot = slot;
          if (slot >= 0 && role == 0 && slice == 0 && lane == 0 && a.sample_lik != nullptr)
            a.sample_lik[static_cast<int64_t>(slot) * L.pairs + unit] = -U_last;
        }
      }
      if (e + 1 < events) hand_over(e + 1);
    }
    bar_sync(kBarDone + ((events - 1) & 1), kWithOne);
    take_energy(events - 1);
    // The last decision, for the threads that write the rows back.
    if (pairs && lane == 0) {
      info[0].slot = role;
      info[0].prev_slot = role == 0 ? done_slot : -1;
    }
    __syncwarp();
    bar_arrive(kBarEnd, kWithOne);
    if (lane == 0 && slice == 0) {
      if (pairs) {
        const int row = role ? L.pairs + unit : unit;
        a.U[row] = U_last;
        a.lk_var[row] = var_last;
        L.ident[row] = who;
        if (half == 0) {
          L.ssq[unit] = ssq;
          L.kc[unit] += a.steps;
          if (L.counts != nullptr) L.counts[unit] += exchanges;
        }
      } else {
        if (L.kind != kLoopLeapfrog) {
          if (a.U != nullptr) a.U[unit] = U_last;
          if (a.lk_var != nullptr) a.lk_var[unit] = var_last;
        }
        if (L.kind == kLoopObabo && L.ke != nullptr) {
          L.ke[unit] += ke_acc[0];
          L.ke[a.chains + unit] += ke_acc[1];
        }
        if (L.kind == kLoopLeapfrog) L.energy[unit] += ke_acc[0];
      }
    }
    return;
  }

  // ============================== row warps =====================================
  float* x_row = a.w + static_cast<int64_t>(row_in) * d;
  float* aux_row = L.aux != nullptr ? L.aux + static_cast<int64_t>(row_in) * d : nullptr;
  // Thread t owns the parameters t, t + 256, ...: one chain of square roots
  // and divisions per thread where d allows.
  const int owned = tid < d ? (d - tid + kRowThreads - 1) / kRowThreads : 0;
  const int g = lane >> (5 - LOG);
  const bool leader = (lane & (GROUP - 1)) == 0;
  float xs[kMaxOwned], as[kMaxOwned], mi[kMaxOwned], ms[kMaxOwned];
  float* wf = reinterpret_cast<float*>(w_s);
#pragma unroll
  for (int i = 0; i < kMaxOwned; ++i) {
    xs[i] = as[i] = 0.f;
    mi[i] = ms[i] = 1.f;
    if (i >= owned) continue;
    const int p = tid + i * kRowThreads;
    xs[i] = x_row[p];
    if (aux_row != nullptr) as[i] = aux_row[p];
    if (L.mass != nullptr) {
      const float m = __ldg(L.mass + p);
      mi[i] = 1.0f / m;
      ms[i] = sqrtf(m);
    }
    if (L.kind == kLoopSghmc) {
      // A block starts at a resample (its steps are whole trajectories).
      float xi[4];
      noise4(a.noise, who, p & ~3, d, k0, GBSGMC_TAG_SGHMC_RESAMPLE, xi);
      const float h = a.sched.step_size(k0);
      const float z = (p & 2) ? ((p & 1) ? xi[3] : xi[2]) : ((p & 1) ? xi[1] : xi[0]);
      as[i] = ms[i] * z;
      const float pj = as[i];
      const float sm = mi[i] * pj;
      xs[i] = xs[i] + h * sm;
      as[i] = pj + (-h * L.friction) * sm;
    } else if (L.kind == kLoopLeapfrog) {
      const float s = 0.5f * a.sched.step_size(k0);
      const float sm = mi[i] * as[i];
      xs[i] = xs[i] + s * sm;
    }
  }
  // Columns d .. 4 dq stay zero in both copies of w.
  for (int p = tid; p < 8 * dq; p += kRowThreads) wf[p] = 0.f;
  bar_sync(kBarRows, kRowThreads);
#pragma unroll
  for (int i = 0; i < kMaxOwned; ++i)
    if (i < owned) wf[tid + i * kRowThreads] = xs[i];
  bar_arrive(kBarInit, kWithOne);
  bar_sync(kBarRows, kRowThreads);

  // Stores the thread's positions in sample row `at`.
  auto keep_x = [&](int64_t at) {
#pragma unroll
    for (int i = 0; i < kMaxOwned; ++i)
      if (i < owned) a.samples[at * d + tid + i * kRowThreads] = xs[i];
  };

  // The cluster's shared-memory windows: address of `here` in each CTA.
  const uint32_t here = smem_addr(smem);
  uint32_t peer[kMaxCtas];
#pragma unroll
  for (int r = 0; r < kMaxCtas; ++r) peer[r] = r < S ? cluster_addr(smem, rank0 + r) : 0u;

  const bool y_in_row = a.y_inline != 0;
  int want = pairs || (L.kind != kLoopLeapfrog &&
                       (a.steps == 1 || a.sched.keep_slot(k0) >= 0));
  int buf = 0, use = 0;
  bool live = true;   // no wait of this thread has run out
  for (int e = 0; e < events; ++e) {
    const int j = L.draws == 2 ? e >> 1 : e;
    const int par = e & 1;
    float4 wq[QPL];
    Accum<QPL> A;
#pragma unroll
    for (int k = 0; k < QPL; ++k) {
      const int v = lane + 32 * k;
      wq[k] = v < dq ? w_s[par * dq + v] : make_float4(0.f, 0.f, 0.f, 0.f);
      A.acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    A.mlk = A.mlk_c = A.K = A.s1 = A.s2 = 0.0f;
    A.cnt = 0;
    for (int q = 0; q < L.chunks; ++q) {
      live &= wait_phase(L, bars, bars->full + buf, use);
      const int cnt = min(CH, R - q * CH);
      const float4* rows = rows_s + buf * CH * rq;
      const int32_t* ix = idx_s + buf * CH;
      for (int r0 = warp * RW; r0 < cnt; r0 += kStride) {
        const int og = r0 + g < cnt ? ix[r0 + g] : -1;
        const float yv = og < 0     ? 0.0f
                         : L.cp_y   ? y_s[buf * CH + r0 + g]
                         : y_in_row ? reinterpret_cast<const float*>(rows + (r0 + g) * rq)[d]
                                    : 0.0f;
        float4 xv[RW][QPL];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
#pragma unroll
          for (int k = 0; k < QPL; ++k) {
            const int v = lane + 32 * k;
            xv[r][k] = r0 + r < cnt && v < dq ? rows[(r0 + r) * rq + v]
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        consume_tile<QPL, RW>(a, nullptr, nullptr, r0, lane, g, leader, want, wq, xv, yv, og,
                              A);
      }
      __syncwarp();
      if (live && lane == 0) mbar_arrive(bars->empty + buf);
      if (++buf == depth) {
        buf = 0;
        ++use;
      }
    }

    // ---- the gradient's reduction ----------------------------------------------
#pragma unroll
    for (int k = 0; k < QPL; ++k) {
      const int v = lane + 32 * k;
      if (v < dq) red[warp * dq + v] = A.acc[k];
    }
    if (leader) {
      lsum[(par * kRowWarps + warp) * RW + g] = lane_sums<QPL>(A);
      if (!isfinite(A.mlk)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
    }
    bar_sync(kBarStep + par, kWithBoth);
    if (want) bar_arrive(kBarSums + par, kWithOne);
    const StepInfo in = info[par];
    want = in.want_next;
    if (owned > 0) {
      const float* redf = reinterpret_cast<const float*>(red);
      float* partf = reinterpret_cast<float*>(part) + par * S * 4 * dq;
      const float* xif = reinterpret_cast<const float*>(xi_s + par * dq);
      const float* xrf = reinterpret_cast<const float*>(xr_s + par * dq);
      float gl[kMaxOwned];
#pragma unroll
      for (int i = 0; i < kMaxOwned; ++i) {
        gl[i] = 0.f;
        if (i >= owned) continue;
        const int p = tid + i * kRowThreads;
        float t[kRowWarps];
#pragma unroll
        for (int w = 0; w < kRowWarps; ++w) t[w] = redf[w * 4 * dq + p];
        gl[i] = t[0];
#pragma unroll
        for (int w = 1; w < kRowWarps; ++w) gl[i] += t[w];
        if (S > 1 && live) {
          const uint32_t at = smem_addr(partf + slice * 4 * dq + p) - here;
          const uint32_t bar = smem_addr(bars->part + par) - here;
#pragma unroll
          for (int r = 0; r < kMaxCtas; ++r)
            if (r < S) send4(peer[r] + at, peer[r] + bar, gl[i]);
        }
      }
      if (S > 1) {
        live &= wait_phase(L, bars, bars->part + par, e >> 1);
        if (live && tid == 0 && e + 2 < events)
          mbar_arrive_expect_tx(bars->part + par, static_cast<uint32_t>(S) * d * 4);
#pragma unroll
        for (int i = 0; i < kMaxOwned; ++i) {
          if (i >= owned) continue;
          const float* all = partf + tid + i * kRowThreads;
          float t[kMaxCtas];
#pragma unroll
          for (int r = 0; r < kMaxCtas; ++r) t[r] = r < S ? all[r * 4 * dq] : 0.f;
          gl[i] = t[0];
#pragma unroll
          for (int r = 1; r < kMaxCtas; ++r)
            if (r < S) gl[i] += t[r];
        }
      }

      // ---- the update ------------------------------------------------------------
      if (in.prev_slot >= 0 && slice == 0)
        keep_x(static_cast<int64_t>(in.prev_slot) * L.pairs + unit);
#pragma unroll
      for (int i = 0; i < kMaxOwned; ++i) {
        if (i >= owned) continue;
        const int p = tid + i * kRowThreads;
        const float xi = xif[p];
        const float gv = (-a.scale * gl[i] + xs[i] * a.inv_p2) * a.inv_temp;
        if (!isfinite(gv)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
        if (moves) {
          const float noise_scale = in.c[0];
          const float x = xs[i];
          const float scaled_gradient = -in.h * gv;
          const float scaled_noise = noise_scale * xi;
          if (aux_row != nullptr) {
            const float vn = a.alpha * as[i] + (1.0f - a.alpha) * (gv * gv);
            const float G = 1.0f / (a.lmbd + sqrtf(vn));
            const float sG = sqrtf(G);
            as[i] = vn;
            xs[i] = x + ((0.0f + G * scaled_gradient) + sG * scaled_noise);
          } else {
            xs[i] = x + (scaled_gradient + scaled_noise);
          }
        } else if (L.kind == kLoopObabo) {
          if (par == 0) ke_s[p] = obabo_first(in, mi[i], ms[i], gv, xi, as[i], xs[i]);
          else ke_s[4 * dq + p] = obabo_second(in, mi[i], ms[i], gv, xi, as[i]);
        } else if (L.kind == kLoopSghmc) {
          const float noise_scale = in.c[0];
          float pj = as[i] + (-in.h) * gv;
          pj = pj + L.friction * (noise_scale * xi);
          const bool more = j + 1 < a.steps;
          if (more && (j + 1) % L.leapfrog == 0) pj = ms[i] * xrf[p];
          as[i] = pj;
          // A kept step's state is this one, before the next step's position.
          if (in.slot >= 0 && slice == 0)
            a.samples[(static_cast<int64_t>(in.slot) * a.chains + unit) * d + p] = xs[i];
          if (more) {
            const float h = in.h_next;
            const float sm = mi[i] * pj;
            xs[i] = xs[i] + h * sm;
            as[i] = pj + (-h * L.friction) * sm;
          }
        } else {  // reversible leapfrog
          const float decay = in.c[0], inv = in.c[1], ns = in.c[2];
          const float s = (j + 1 < a.steps ? 1.0f : 0.5f) * in.h;
          const float pj = as[i];
          const float noise_j = ns * (ms[i] * xi);
          const float pn = inv * ((decay * pj + (-in.h) * gv) + noise_j);
          as[i] = pn;
          ke_s[par * 4 * dq + p] = make_float2(pj + pn, mi[i] * gv);
          const float sm = mi[i] * pn;
          xs[i] = xs[i] + s * sm;
        }
        wf[(par ^ 1) * 4 * dq + p] = xs[i];
      }
      if (in.slot >= 0 && slice == 0 && L.kind != kLoopSghmc && (L.draws == 1 || par == 1))
        keep_x(static_cast<int64_t>(in.slot) * a.chains + unit);
    }
    bar_arrive(kBarDone + par, kWithOne);
    bar_arrive(kBarFree + par, kWithOne);
    bar_sync(kBarRows, kRowThreads);  // the new w is visible; red is free
  }

  // ---- the block's end -----------------------------------------------------------
  bar_sync(kBarEnd, kWithOne);
  if (owned > 0 && slice == 0) {
    int row = row_in;
    if (pairs) {
      row = info[0].slot ? L.pairs + unit : unit;
      if (info[0].prev_slot >= 0)
        keep_x(static_cast<int64_t>(info[0].prev_slot) * L.pairs + unit);
    }
    float* xo = a.w + static_cast<int64_t>(row) * d;
    float* ao = L.aux != nullptr ? L.aux + static_cast<int64_t>(row) * d : nullptr;
#pragma unroll
    for (int i = 0; i < kMaxOwned; ++i) {
      if (i >= owned) continue;
      xo[tid + i * kRowThreads] = xs[i];
      if (ao != nullptr) ao[tid + i * kRowThreads] = as[i];
    }
  }
}

template <int QPL, int RW>
__global__ void __launch_bounds__(kLoopThreads, 1)
    glm_loop_kernel(const __grid_constant__ LoopArgs L, const __grid_constant__ CUtensorMap map) {
  extern __shared__ __align__(128) unsigned char smem[];
  loop_roles<QPL, RW>(L, map, smem);
  // No CTA ends while another of its cluster may send to it.  In a run without
  // a timeout each CTA's own waits have seen every send land.  After one they
  // have not: the cluster waits for its last sender, tells all of its CTAs of
  // the timeout, and they wait for the sends (and their own copies) to land.
  LoopBars* bars = reinterpret_cast<LoopBars*>(smem + L.o_bar);
  const int ncta = L.kind == kLoopPairs ? 2 * L.ctas : L.ctas;
  if (ncta > 1) {
    if (stopped(bars) && threadIdx.x < ncta)
      asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(cluster_addr(&bars->stop, threadIdx.x))
                   : "memory");
    cluster_arrive();
    cluster_wait();
  }
  if (stopped(bars)) {
    const uint64_t t0 = global_ns();
    while (global_ns() - t0 < kLingerNs) {
    }
  }
}

constexpr size_t kLoopSmem = 220 * 1024;   // one CTA per SM

size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// Fills the chunk sizes and shared-memory offsets of a launch; returns its
// shared memory, or 0 when no chunk fits.  A CTA's whole slice of a minibatch
// is one chunk when three such chunks fit (two minibatches ahead of the one
// being consumed); longer slices stream through up to four smaller chunks.
size_t loop_layout(LoopArgs& L, int rw, int ncta) {
  const int dq = L.g.dq, stride = kRowWarps * rw, R = L.g.rows_per_slice;
  const size_t row = static_cast<size_t>(dq) * 16;
  const size_t n_red = kRowWarps * row, n_part = L.ctas > 1 ? 2 * L.ctas * row : 0;
  const size_t n_ke = 4 * row, n_lane = 2 * sizeof(LaneSums) * kRowWarps * rw;
  const size_t n_sums = 2 * sizeof(SliceSums) * ncta, n_step = 2 * sizeof(StepInfo);
  const size_t n_pair = 4 * sizeof(PairConsts);
  const size_t fixed = n_red + n_part + 6 * row + align16(n_ke) + align16(n_lane) +
                       align16(n_sums) + align16(n_step) + n_pair + align16(sizeof(LoopBars)) + 64;
  const auto ring = [&](int depth, int rows) {
    return depth * static_cast<size_t>(rows) * (16 * L.row_quads + 8);
  };
  if (fixed >= kLoopSmem) return 0;
  const size_t room = kLoopSmem - fixed;
  const int whole = std::max(1, ceil_div(R, stride)) * stride;
  int depth = 0, rows = 0;
  if (ring(3, whole) <= room) {
    depth = 3;
    rows = whole;
  } else {
    for (int dp = kMaxDepth; dp >= 2 && depth == 0; --dp) {
      const int m = static_cast<int>(room / ring(dp, stride));
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
  size_t o = static_cast<size_t>(depth) * rows * 16 * L.row_quads;
  const auto take = [&](size_t bytes) {
    const size_t at = o;
    o += align16(bytes);
    return static_cast<unsigned>(at);
  };
  L.o_y = take(4ull * depth * rows);
  L.o_idx = take(4ull * depth * rows);
  L.o_red = take(n_red);
  L.o_part = take(n_part);
  L.o_w = take(2 * row);
  L.o_xi = take(2 * row);
  L.o_xr = take(2 * row);
  L.o_ke = take(n_ke);
  L.o_lane = take(n_lane);
  L.o_sums = take(n_sums);
  L.o_step = take(n_step);
  L.o_pair = take(n_pair);
  L.o_bar = take(sizeof(LoopBars));
  return o;
}

template <int QPL, int RW>
struct LoopVariant {
  static int prepare() {
    static int done = 0;
    if (done) return GBSGMC_OK;
    const cudaError_t e =
        cudaFuncSetAttribute(glm_loop_kernel<QPL, RW>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kLoopSmem);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "glm_loop: cudaFuncSetAttribute: %s",
                       cudaGetErrorString(e));
    done = 1;
    return GBSGMC_OK;
  }
  static int launch(LoopArgs& L, int units, int ncta, cudaStream_t st) {
    int rc = prepare();
    if (rc != GBSGMC_OK) return rc;
    const size_t smem = loop_layout(L, RW, ncta);
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
    CUtensorMap map = {};
    if (L.gather &&
        (rc = make_tmap_f32_gather(&map, L.g.X, L.row_cols, L.g.n_rows, L.g.ld, 4 * L.row_quads)) !=
            GBSGMC_OK)
      return rc;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, glm_loop_kernel<QPL, RW>, L, map);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "glm_loop: %s", cudaGetErrorString(e));
    return check_launch("glm_loop");
  }
};

}  // namespace

namespace {

// Clusters of `ctas` loop CTAs (one per SM) that the device holds at once: its
// GPCs are not whole multiples of 8 SMs, so fewer than SMs / ctas.  A CTA's
// registers fill an SM in every variant.
int clusters_at_once(int ctas) {
  static std::atomic<int> known[4];
  const int slot = ctas >= 8 ? 3 : ctas >= 4 ? 2 : ctas >= 2 ? 1 : 0;
  int n = known[slot].load(std::memory_order_relaxed);
  if (n > 0) return n;
  n = glm_sm_count() / ctas;
  if (ctas > 1 && LoopVariant<1, 4>::prepare() == GBSGMC_OK) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(kLoopThreads);
    cfg.dynamicSmemBytes = kLoopSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int held = 0;
    if (cudaOccupancyMaxActiveClusters(&held, glm_loop_kernel<1, 4>, &cfg) == cudaSuccess &&
        held > 0)
      n = held;
    else
      cudaGetLastError();
  }
  known[slot].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace

// CTAs per chain: in powers of two up to the portable cluster size, as long
// as each keeps two rows a row warp and all clusters run at once.  16 chains
// of 200 rows of 16 features, OBABO: 3,069, 1,969, 1,413 us with 1, 2, 4 CTAs,
// and 1,898 with 8, where two clusters wait for the others; 8 chains: 1,361 us
// with 4, 1,285 with 8.
int glm_loop_ctas(int units, int chains_per_unit, int n) {
  const int most = kMaxCtas / chains_per_unit;
  const char* env = std::getenv("GBSGMC_GLM_SLICES");
  const int forced = env != nullptr ? std::atoi(env) : 0;
  int s = 1;
  if (forced > 0) {
    while (2 * s <= std::min(forced, most)) s *= 2;
    return s;
  }
  while (2 * s <= most && n >= 2 * s * kRowWarps * 2 &&
         units <= clusters_at_once(2 * s * chains_per_unit))
    s *= 2;
  return s;
}

// A CTA streams its rows at 11 to 47 GB/s (12 ns a row of up to 128 features,
// 21 of 256, 110 of 1,000), so that few CTAs with many rows each take longer
// than launches per gradient, which spread a chain over up to 64 CTAs.  The
// line between them by the rows of a CTA, the width (float4 columns per lane)
// and the share of the SMs that the clusters keep busy over their waves; us
// an OBABO step, this form and the other: one chain of 16,384 rows of 256
// features 90 and 130, of 65,536 353 and 212, of 65,536 x 1,000 1,858 and 413;
// 16 of 8,192 x 256 83 and 97, of 16,384 164 and 155; 100 of 4,096 x 256 150
// and 200, of 16,384 598 and 557; 64 of 2,048 x 1,000 206 and 256, of 8,192
// 797 and 786.  One table serves SGHMC and the pairs too, whose lines lie up to
// a third lower: over some 2,300 shapes of 1 to 600 chains, 256 to 65,536 rows
// and 8 to 1,000 features this form is nowhere taken where it is more than 5 %
// slower, and nowhere left where it is more than a third faster.
bool glm_loop_pays(int units, int chains_per_unit, int n, int d) {
  struct Line {
    double busy;
    int rows[4];   // 1, 2, 4, 8 float4 columns per lane
  };
  constexpr int kAny = 1 << 30;
  constexpr Line kLines[] = {{0.25, {5000, 3000, 1000, 350}},
                             {0.5, {8200, 4000, 1000, 400}},
                             {0.8, {20000, 6000, 2500, 1000}},
                             {0.95, {kAny, 20000, 8000, 1400}},
                             {1.0, {kAny, kAny, kAny, 12000}}};
  const int ctas = glm_loop_ctas(units, chains_per_unit, n);
  const int64_t used = static_cast<int64_t>(units) * chains_per_unit * ctas, sms = glm_sm_count();
  const double busy = static_cast<double>(used) / (sms * ((used + sms - 1) / sms));
  const int qpl = glm_qpl((d + 3) / 4), width = qpl == 1 ? 0 : qpl == 2 ? 1 : qpl == 4 ? 2 : 3;
  for (const Line& l : kLines)
    if (busy <= l.busy) return ceil_div(n, ctas) <= l.rows[width];
  return true;
}

namespace {

// Rows a warp takes at once: its whole share of the slice where the registers
// allow (a tile's latency is one dot product, reduction and link whatever its
// rows: 125 rows of 101 features took 5,060 cycles in tiles of 4).
int loop_rows_per_warp(int qpl, int rows_per_slice) {
  const char* env = std::getenv("GBSGMC_GLM_RW");
  const int forced = env != nullptr ? std::atoi(env) : 0;
  const int least = qpl <= 2 ? 4 : (qpl == 4 ? 2 : 1);
  const int most = qpl == 1 ? 16 : (qpl == 2 ? 8 : (qpl == 4 ? 4 : 1));
  if (qpl <= 2 && (forced == 4 || forced == 8)) return forced;
  int rw = least;
  while (rw < most && rw * kRowWarps < rows_per_slice) rw *= 2;
  return rw;
}

}  // namespace

int glm_loop_prepare() {
  int rc = LoopVariant<1, 4>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<1, 8>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<1, 16>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<2, 4>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<2, 8>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<4, 2>::prepare();
  if (rc == GBSGMC_OK) rc = LoopVariant<4, 4>::prepare();
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
  // The waits' bound.  With 0 they are sure to run out: every chunk waits for
  // one arrival that never comes.
  const char* wait = std::getenv("GBSGMC_LOOP_WAIT_NS");
  L.wait_ns = wait != nullptr ? std::strtoull(wait, nullptr, 10) : kWaitLimitNs;
  L.missing = L.wait_ns == 0 ? 1 : 0;
  const bool y_in_row = L.g.vec4 && L.g.y_inline;
  L.row_quads = (L.g.d + (y_in_row ? 1 : 0) + 3) / 4;
  L.cp_y = !y_in_row && (L.g.y_inline || L.g.y != nullptr) ? 1 : 0;
  L.cp_async = !L.g.vec4 || L.cp_y ? 1 : 0;
  // Rows on 16-byte boundaries are copied four at a time where a box holds a
  // row (256 columns); in shared memory they then start on multiples of 32
  // bytes, so that four rows, the target of one copy, start on 128.  The row
  // after the last one has to be an int32 coordinate.  Wider rows are copied
  // one by one; from about 200 columns the bytes bound a step, not the copies
  // (24 chains of 250 rows of 200 features: 2.1 us a gradient by either).
  L.row_cols = 4 * L.row_quads;
  L.gather = L.g.vec4 && L.row_quads <= 64 && L.g.n_rows < (1ll << 31) - 1 ? 1 : 0;
  if (L.gather) L.row_quads += L.row_quads & 1;
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
  const int rw = loop_rows_per_warp(qpl, L.g.rows_per_slice);
  if (qpl == 1)
    return rw == 16  ? LoopVariant<1, 16>::launch(L, units, ncta, st)
           : rw == 8 ? LoopVariant<1, 8>::launch(L, units, ncta, st)
                     : LoopVariant<1, 4>::launch(L, units, ncta, st);
  if (qpl == 2)
    return rw == 8 ? LoopVariant<2, 8>::launch(L, units, ncta, st)
                   : LoopVariant<2, 4>::launch(L, units, ncta, st);
  if (qpl == 4)
    return rw == 4 ? LoopVariant<4, 4>::launch(L, units, ncta, st)
                   : LoopVariant<4, 2>::launch(L, units, ncta, st);
  return LoopVariant<8, 1>::launch(L, units, ncta, st);
}

}  // namespace gbsgmc
