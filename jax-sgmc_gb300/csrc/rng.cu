// Index and noise streams.
//
// * gbsgmc_index_draw_pcg64 reproduces numpy's Generator.choice(arange(N), n,
//   replace=True) bit for bit.  numpy draws each index as a 32-bit Lemire
//   bounded integer (Lemire 2019, "Fast random integer generation in an
//   interval"): x = next_uint32(); m = x * N; accept when (m mod 2^32) >=
//   2^32 mod N, the index being m >> 32.  next_uint32 hands out the low half
//   of a fresh PCG64 output and keeps the high half for the next call.  The
//   accept test depends only on the 32-bit value, so a CTA expands 4096 PCG64
//   outputs at once (each thread jumps ahead to its own 8 consecutive steps
//   by LCG jump-ahead, Brown 1994, "Random number generation with arbitrary
//   strides"), tests the 8192 halves, and compacts the accepted ones with a
//   block scan.  The chain's stream state (128-bit LCG state,
//   buffered half) is advanced exactly as numpy advances it.
// * gbsgmc_index_draw_philox and gbsgmc_philox_normal use Philox4x32-10.
#include "common.cuh"

namespace gbsgmc {
namespace {

constexpr int kDrawThreads = 512;
constexpr int kDrawPerThread = 8;   // consecutive LCG outputs per thread per round

// The LCG map s -> a s + inc applied k times is s -> a^k s + inc G_k with
// G_k = 1 + a + ... + a^(k - 1) (Brown 1994): a^k and G_k do not depend on
// the stream.  Tables of them, made at compile time, replace the 11 squarings
// and up to 12 compositions that every thread did before its first draw: the
// first steps of 16 neighbouring threads, the strides between such groups,
// and a whole round.
struct Jump {
  unsigned long long a_hi, a_lo, g_hi, g_lo;
};
struct JumpTable {
  Jump low[16];                    // t = 0 .. 15: t kDrawPerThread + 1 steps
  Jump high[kDrawThreads / 16];    // u: 16 u kDrawPerThread steps
  Jump round;                      // kDrawThreads kDrawPerThread steps
};
constexpr Jump jump_of(unsigned k) {
  using u128 = unsigned __int128;
  const u128 a = (static_cast<u128>(0x2360ED051FC65DA4ull) << 64) | 0x4385DF649FCCF645ull;
  u128 A = 1, G = 0, p = a, s = 1;   // (p, s): the map of 2^i steps
  while (k > 0) {
    if (k & 1u) {
      G = p * G + s;
      A = p * A;
    }
    s = s * p + s;
    p = p * p;
    k >>= 1;
  }
  return Jump{static_cast<unsigned long long>(A >> 64), static_cast<unsigned long long>(A),
              static_cast<unsigned long long>(G >> 64), static_cast<unsigned long long>(G)};
}
constexpr JumpTable make_jumps() {
  JumpTable t{};
  for (int i = 0; i < 16; ++i) t.low[i] = jump_of(i * kDrawPerThread + 1);
  for (int i = 0; i < kDrawThreads / 16; ++i) t.high[i] = jump_of(16 * i * kDrawPerThread);
  t.round = jump_of(kDrawThreads * kDrawPerThread);
  return t;
}
__device__ const JumpTable g_jumps = make_jumps();

__device__ __forceinline__ U128 load_hi_lo(const unsigned long long& hi,
                                           const unsigned long long& lo) {
  return U128{__ldg(&hi), __ldg(&lo)};
}
// The map of `j`'s steps on a stream of increment inc.
__device__ __forceinline__ Affine jump_map(const Jump& j, U128 inc) {
  return Affine{load_hi_lo(j.a_hi, j.a_lo), mul128(load_hi_lo(j.g_hi, j.g_lo), inc)};
}

// Block-wide exclusive scan of small non-negative ints; returns the exclusive
// prefix and sets *total.  Contains __syncthreads.
__device__ __forceinline__ int block_excl_scan(int v, int* warp_tot,
                                               int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kDrawThreads / 32; ++w) {
    const int t = warp_tot[w];
    before += (w < warp) ? t : 0;
    all += t;
  }
  *total = all;
  return before + incl - v;
}

__global__ void __launch_bounds__(kDrawThreads)
    pcg64_draw_kernel(gbsgmc_pcg64* states, int64_t n_obs, int64_t draws,
                      int per_step, int32_t* idx, int64_t chain_stride,
                      int64_t step_stride) {
  __shared__ int warp_tot[kDrawThreads / 32];
  // A round's values by rank, position p at p + p / 16: thread t's sixteen
  // values start near 16 t, so that a warp's stores of value i hit 32 banks.
  __shared__ int32_t vals[kDrawThreads * 2 * kDrawPerThread * 17 / 16 + 1];

  const int c = blockIdx.x;
  const int t = threadIdx.x;
  gbsgmc_pcg64* st = states + c;
  int32_t* out = idx + static_cast<int64_t>(c) * chain_stride;
  auto put = [&](int64_t pos, int32_t v) {
    out[(pos / per_step) * step_stride + pos % per_step] = v;
  };

  if (draws <= 0) return;
  if (n_obs == 1) {  // numpy returns the offset without consuming randomness
    for (int64_t j = t; j < draws; j += kDrawThreads) put(j, 0);
    return;
  }

  U128 s{st->state_hi, st->state_lo};
  const U128 inc{st->inc_hi, st->inc_lo};
  uint32_t has = st->has_uint32;
  const uint32_t buffered = st->uinteger;
  const uint64_t N = static_cast<uint64_t>(n_obs);
  const uint32_t threshold = static_cast<uint32_t>((1ull << 32) % N);

  // A round is kDrawThreads * kDrawPerThread LCG steps; this thread's
  // outputs are steps t*K + 1 .. t*K + K of the round (K = kDrawPerThread),
  // so the thread order of the scan is the stream order.
  const Affine jump =
      compose(jump_map(g_jumps.high[t >> 4], inc), jump_map(g_jumps.low[t & 15], inc));
  const Affine step1{pcg_multiplier(), inc};
  const Affine round_jump = jump_map(g_jumps.round, inc);

  int64_t produced = 0;
  if (has) {  // the half buffered by the previous call comes first
    const bool acc = static_cast<uint32_t>(buffered * N) >= threshold;
    if (acc) {
      if (t == 0) put(0, static_cast<int32_t>((buffered * N) >> 32));
      produced = 1;
    }
    has = 0;
    if (produced == draws) {
      __syncthreads();
      if (t == 0) st->has_uint32 = 0u;
      return;
    }
  }

  for (;;) {
    U128 sj[kDrawPerThread];
    uint32_t lo[kDrawPerThread], hi[kDrawPerThread];
    unsigned acc = 0;  // bit 2i: low half i accepted, bit 2i+1: high half i
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < kDrawPerThread; ++i) {
      sj[i] = i == 0 ? apply(jump, s) : apply(step1, sj[i - 1]);
      const uint64_t o = pcg_output(sj[i]);
      lo[i] = static_cast<uint32_t>(o);
      hi[i] = static_cast<uint32_t>(o >> 32);
      const unsigned a0 = static_cast<uint32_t>(lo[i] * N) >= threshold ? 1u : 0u;
      const unsigned a1 = static_cast<uint32_t>(hi[i] * N) >= threshold ? 1u : 0u;
      acc |= (a0 << (2 * i)) | (a1 << (2 * i + 1));
      cnt += static_cast<int>(a0 + a1);
    }
    int total;
    const int excl = block_excl_scan(cnt, warp_tot, &total);
    // Through shared memory, so that the indices leave as whole segments
    // (a thread's own sixteen stores each touched a sector of their own:
    // 50,000 draws took 38 us against 27).
    int rank0 = excl;
#pragma unroll
    for (int i = 0; i < kDrawPerThread; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if ((acc >> (2 * i + h)) & 1u) {
          const uint32_t v = h ? hi[i] : lo[i];
          vals[rank0 + (rank0 >> 4)] = static_cast<int32_t>((v * N) >> 32);
          ++rank0;
        }
      }
    }
    __syncthreads();
    const int64_t left = draws - produced;
    const int out_n = left < total ? static_cast<int>(left) : total;
    if (produced + out_n <= 0xffffffffll) {
      const uint32_t base = static_cast<uint32_t>(produced), per = per_step;
      for (int p = t; p < out_n; p += kDrawThreads) {
        const uint32_t pos = base + p, q = pos / per;
        out[q * step_stride + (pos - q * per)] = vals[p + (p >> 4)];
      }
    } else {
      for (int p = t; p < out_n; p += kDrawThreads) put(produced + p, vals[p + (p >> 4)]);
    }
    if (produced + total >= draws) {
      // The thread holding the last value used stores the stream state after
      // its output, and buffers the high half if the low half was the last.
      const int64_t last = draws - 1 - produced;  // rank of the last value used
      if (cnt > 0 && last >= excl && last < excl + cnt) {
        int64_t rank = excl;
#pragma unroll
        for (int i = 0; i < kDrawPerThread; ++i) {
          if ((acc >> (2 * i)) & 1u) {
            if (rank == last) {
              st->state_hi = sj[i].hi;
              st->state_lo = sj[i].lo;
              st->has_uint32 = 1u;
              st->uinteger = hi[i];
            }
            ++rank;
          }
          if ((acc >> (2 * i + 1)) & 1u) {
            if (rank == last) {
              st->state_hi = sj[i].hi;
              st->state_lo = sj[i].lo;
              st->has_uint32 = 0u;
              st->uinteger = hi[i];
            }
            ++rank;
          }
        }
      }
      return;
    }
    produced += total;
    s = apply(round_jump, s);
  }
}

__global__ void philox_index_kernel(uint64_t seed, int chain_base, int chains,
                                    const int64_t* base, int64_t first_step,
                                    int steps,
                                    int per_step, int64_t n_obs, int32_t* idx,
                                    int64_t chain_stride,
                                    int64_t step_stride) {
  // One thread per pair of draws: a 64-bit uniform per draw keeps the
  // multiply-shift bias below n_obs / 2^64.
  const int pairs = (per_step + 1) / 2;
  const int64_t total = static_cast<int64_t>(chains) * steps * pairs;
  const uint64_t N = static_cast<uint64_t>(n_obs);
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
       g < total; g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int p = static_cast<int>(g % pairs);
    const int64_t cs = g / pairs;
    const int sidx = static_cast<int>(cs % steps);
    const int c = static_cast<int>(cs / steps);
    const int64_t step = (base != nullptr ? *base : 0) + first_step + sidx;
    const U32x4 r = philox4x32_10(
        U32x4{static_cast<uint32_t>(p), static_cast<uint32_t>(step),
              static_cast<uint32_t>(chain_base + c), GBSGMC_TAG_INDEX},
        static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32));
    const uint64_t u0 = (static_cast<uint64_t>(r.y) << 32) | r.x;
    const uint64_t u1 = (static_cast<uint64_t>(r.w) << 32) | r.z;
    int32_t* o = idx + c * chain_stride + sidx * step_stride;
    const int j0 = 2 * p;
    o[j0] = static_cast<int32_t>(__umul64hi(u0, N));
    if (j0 + 1 < per_step) o[j0 + 1] = static_cast<int32_t>(__umul64hi(u1, N));
  }
}

__global__ void philox_normal_kernel(uint64_t seed, int chain_base,
                                     int chains, int64_t step, uint32_t tag,
                                     int64_t count, float* out,
                                     int64_t stride) {
  const int64_t groups = (count + 3) / 4;
  const int64_t total = groups * chains;
  for (int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
       g < total; g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(g / groups);
    const int64_t q = g % groups;
    float z[4];
    philox_normal4(seed, static_cast<uint32_t>(q), static_cast<uint32_t>(step),
                   static_cast<uint32_t>(chain_base + c), tag, z);
    float* o = out + c * stride + 4 * q;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (4 * q + i < count) o[i] = z[i];
  }
}

int grid_for(int64_t work, int threads) {
  int64_t b = (work + threads - 1) / threads;
  if (b > 152 * 32) b = 152 * 32;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace

int launch_philox_index(uint64_t seed, int chain_base, int chains,
                        const int64_t* base, int64_t first_step, int steps,
                        int per_step, int64_t n_obs, int32_t* idx,
                        int64_t chain_stride, int64_t step_stride,
                        cudaStream_t stream) {
  const int64_t work =
      static_cast<int64_t>(chains) * steps * ((per_step + 1) / 2);
  if (work == 0) return GBSGMC_OK;
  philox_index_kernel<<<grid_for(work, 256), 256, 0, stream>>>(
      seed, chain_base, chains, base, first_step, steps, per_step, n_obs, idx,
      chain_stride, step_stride);
  return check_launch("index_draw_philox");
}

}  // namespace gbsgmc

using namespace gbsgmc;

// Fresh numpy PCG64 streams of chains registered with the given seeds: the
// generator numpy.random.default_rng(SeedSequence(seed).spawn(1)[0]) starts
// with.  SeedSequence is M. O'Neill's seed_seq_fe entropy mixer ("Developing
// a seed_seq Alternative", 2015) over a pool of four 32-bit words with its
// published hash and mix constants; the assembled entropy of a chain is its
// seed as four little-endian 32-bit words (zero-padded to the pool size, as
// SeedSequence does when a spawn key follows) and the spawn key word 0.  Four 64-bit words generated from the pool seed
// PCG64 as numpy does: state = 0, inc = 2 initseq + 1, one LCG step,
// state += initstate, one LCG step.
namespace {

struct SeedSeqFe {
  uint32_t hash_a = 0x43B0D7E5u;
  uint32_t hashmix(uint32_t v) {
    v ^= hash_a;
    hash_a *= 0x931E8875u;
    v *= hash_a;
    return v ^ (v >> 16);
  }
  static uint32_t mix(uint32_t x, uint32_t y) {
    const uint32_t r = 0xCA01F9DDu * x - 0x4973F715u * y;
    return r ^ (r >> 16);
  }
};

void pcg64_seed_one(uint64_t lo, uint64_t hi, uint64_t (&out)[5]) {
  // With a spawn key the run entropy is zero-padded to the pool size, so
  // the assembled entropy is always the four seed limbs and the key word.
  const int n = 5;
  const uint32_t ent[5] = {static_cast<uint32_t>(lo), static_cast<uint32_t>(lo >> 32),
                           static_cast<uint32_t>(hi), static_cast<uint32_t>(hi >> 32),
                           0u};  // spawn key (0,)
  SeedSeqFe h;
  uint32_t pool[4];
  for (int i = 0; i < 4; ++i) pool[i] = h.hashmix(ent[i]);
  for (int s = 0; s < 4; ++s)
    for (int d = 0; d < 4; ++d)
      if (s != d) pool[d] = SeedSeqFe::mix(pool[d], h.hashmix(pool[s]));
  for (int i = 4; i < n; ++i)
    for (int d = 0; d < 4; ++d) pool[d] = SeedSeqFe::mix(pool[d], h.hashmix(ent[i]));
  uint32_t hash_b = 0x8B51F9DDu;
  uint32_t w[8];
  for (int i = 0; i < 8; ++i) {
    uint32_t v = pool[i % 4] ^ hash_b;
    hash_b *= 0x58F38DEDu;
    v *= hash_b;
    w[i] = v ^ (v >> 16);
  }
  using u128 = unsigned __int128;
  const auto word64 = [&](int k) {
    return static_cast<uint64_t>(w[2 * k]) | (static_cast<uint64_t>(w[2 * k + 1]) << 32);
  };
  const u128 initstate = (static_cast<u128>(word64(0)) << 64) | word64(1);
  const u128 initseq = (static_cast<u128>(word64(2)) << 64) | word64(3);
  const u128 mult = (static_cast<u128>(0x2360ED051FC65DA4ull) << 64) | 0x4385DF649FCCF645ull;
  const u128 inc = (initseq << 1) | 1u;
  u128 state = inc;                 // 0 * mult + inc
  state += initstate;
  state = state * mult + inc;
  out[0] = static_cast<uint64_t>(state >> 64);
  out[1] = static_cast<uint64_t>(state);
  out[2] = static_cast<uint64_t>(inc >> 64);
  out[3] = static_cast<uint64_t>(inc);
  out[4] = 0;  // no buffered 32-bit half
}

}  // namespace

extern "C" int gbsgmc_pcg64_seed(const uint64_t* seeds_lo, const uint64_t* seeds_hi, int count,
                                 uint64_t* words) {
  if (count < 0) return set_error(GBSGMC_ERR_ARG, "pcg64_seed: negative count");
  if (count > 0 && (seeds_lo == nullptr || words == nullptr))
    return set_error(GBSGMC_ERR_ARG, "pcg64_seed: null pointer");
  for (int c = 0; c < count; ++c) {
    uint64_t out[5];
    pcg64_seed_one(seeds_lo[c], seeds_hi != nullptr ? seeds_hi[c] : 0, out);
    for (int k = 0; k < 5; ++k) words[5 * static_cast<int64_t>(c) + k] = out[k];
  }
  return GBSGMC_OK;
}

extern "C" int gbsgmc_index_draw_pcg64(gbsgmc_pcg64* states_dev, int chains,
                                       int64_t n_obs, int64_t draws,
                                       int per_step, int32_t* idx_dev,
                                       int64_t chain_stride,
                                       int64_t step_stride, int* status_dev,
                                       gbsgmc_stream_t stream) {
  (void)status_dev;
  if (states_dev == nullptr || idx_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "index_draw_pcg64: null pointer");
  if (chains < 0 || draws < 0 || per_step <= 0)
    return set_error(GBSGMC_ERR_ARG, "index_draw_pcg64: negative size");
  if (n_obs < 1 || n_obs >= (1ll << 31))
    return set_error(GBSGMC_ERR_SHAPE,
                     "index_draw_pcg64: n_obs must be in [1, 2^31), got %lld",
                     static_cast<long long>(n_obs));
  if (chains == 0 || draws == 0) return GBSGMC_OK;
  pcg64_draw_kernel<<<chains, kDrawThreads, 0,
                      static_cast<cudaStream_t>(stream)>>>(
      states_dev, n_obs, draws, per_step, idx_dev, chain_stride, step_stride);
  return check_launch("index_draw_pcg64");
}

extern "C" int gbsgmc_index_draw_philox(uint64_t seed, int chain_base,
                                        int chains, int64_t first_step,
                                        int steps, int per_step, int64_t n_obs,
                                        int32_t* idx_dev, int64_t chain_stride,
                                        int64_t step_stride,
                                        gbsgmc_stream_t stream) {
  if (idx_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "index_draw_philox: null pointer");
  if (chains < 0 || steps < 0 || per_step <= 0)
    return set_error(GBSGMC_ERR_ARG, "index_draw_philox: negative size");
  if (n_obs < 1 || n_obs >= (1ll << 31))
    return set_error(GBSGMC_ERR_SHAPE,
                     "index_draw_philox: n_obs must be in [1, 2^31)");
  return launch_philox_index(seed, chain_base, chains, nullptr, first_step,
                             steps, per_step, n_obs, idx_dev, chain_stride,
                             step_stride, static_cast<cudaStream_t>(stream));
}

extern "C" int gbsgmc_philox_normal(uint64_t seed, int chain_base, int chains,
                                    int64_t step, uint32_t tag, int64_t count,
                                    float* out_dev, int64_t stride,
                                    gbsgmc_stream_t stream) {
  if (out_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "philox_normal: null pointer");
  if (chains < 0 || count < 0 || stride < count)
    return set_error(GBSGMC_ERR_ARG, "philox_normal: bad size or stride");
  const int64_t work = static_cast<int64_t>(chains) * ((count + 3) / 4);
  if (work == 0) return GBSGMC_OK;
  philox_normal_kernel<<<grid_for(work, 256), 256, 0,
                         static_cast<cudaStream_t>(stream)>>>(
      seed, chain_base, chains, step, tag, count, out_dev, stride);
  return check_launch("philox_normal");
}
