// Convolutional classifier with a softmax likelihood: U, dU/dw, lk and
// var(lk) for many chains at once, the convolutions as GEMMs on the tcgen05
// tensor cores.
//
// Network (NHWC, SAME padding, stride 1):
//   x [32,32,3] -> conv3x3 32 + b, ReLU, 2x2 max-pool -> [16,16,32]
//               -> conv3x3 64 + b, ReLU, 2x2 max-pool -> [8,8,64]
//               -> conv3x3 128 + b, ReLU, 2x2 max-pool -> [4,4,128]
//               -> flatten (h, w, c) 2048 -> dense 10 -> logits
//   lk = logits[label] - logsumexp(logits)   (the negative softmax cross
//   entropy of the reference's classifier example, examples/cifar.md:203-210)
// Flat parameters: the sorted ravel of {conv1: {b, w}, conv2: {b, w},
// conv3: {b, w}, linear: {b, w}} with w in HWIO / [in, out] layout:
//   b1 32 | W1 [3,3,3,32] | b2 64 | W2 [3,3,32,64] | b3 128 | W3 [3,3,64,128]
//   | bd 10 | Wd [2048,10],   P = 113,738.
//
// Each convolution is a GEMM over the im2col matrix Col [pixels, K] with K
// ordered (kh, kw, ci), which is never formed:
//   forward  Y = ReLU(Col W + b)          A = Col (K-major), B = W
//   weights  dW = dY^T Col                 both MN-major
//   inputs   dX = sum over taps of dY shifted back by the tap times the tap's
//            W^T (the transposed convolution), A = dY (K-major), B = W
//            (K-major), then the pooling's argmax routing and the ReLU mask.
// conv1 and its weight gradient build their operands in shared memory from
// the images; the others' maps are stored in rows of channel octets, so that a
// box of a strip or an image pair with its halo serves all taps (see the
// kernels).  The epilogues apply bias and ReLU and the 2x2 max-pool to the
// fp32 accumulators themselves and write the pooled BF16 map and the argmax
// marks; no pre-pool activation is stored.  A mark byte holds the argmax (bits
// 0-1) and whether the maximum is positive (bit 2), the ReLU mask of the
// element that the backward pass routes the gradient to.
// Everything a GEMM reads is BF16.  The dense layer, softmax and their
// adjoints are small and run on the CUDA cores in fp32.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.h"
#include "tc_gemm.cuh"

namespace gbsgmc {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kImg = 32, kInC = 3, kClasses = 10;
constexpr int kC1 = 32, kC2 = 64, kC3 = 128;
constexpr int kFlat = 4 * 4 * kC3;  // 2048
constexpr int kK1 = 27;  // conv1's K (3 x 3 taps x 3 channels)
constexpr int kX8 = 8;   // slots of a pixel's word: its left neighbour's 3, its own 3, 0, 0
constexpr int kK2 = 9 * kC1;
constexpr int kK3 = 9 * kC2;

// Offsets of the leaves in a chain's flat parameter vector.
constexpr int64_t ob1 = 0, oW1 = ob1 + kC1, ob2 = oW1 + kK1 * kC1, oW2 = ob2 + kC2,
                  ob3 = oW2 + kK2 * kC2, oW3 = ob3 + kC3, obd = oW3 + kK3 * kC3,
                  oWd = obd + kClasses, kP = oWd + kFlat * kClasses;
static_assert(kP == 113738, "parameter count");

struct CnnLayout {
  size_t w2b, w3b;                    // BF16 weights (cnn_prep)
  size_t p1, p2, p3;                  // BF16 GEMM operands
  size_t dy2, dy3;                    // BF16 output gradients of conv2, conv3
  size_t m1, m2, m3;                  // uint8 argmax of each pool window
  size_t dp1;                         // fp32 input gradient of conv2
  size_t labels;                      // int32
  size_t dp3, gl;                     // fp32 dP3 [n, 2048], dlogits [n, 10]
  size_t psq, plk;                    // fp64 partial sums
  size_t part[3], bpart[3];           // split-K weight partials, bias partials by layer
  size_t total;
};

constexpr int kPrepBlocks = 64;  // Σw² partial sums per chain

// Split-K factors of the weight gradients (K = pixels of n images: 16n, 4n and
// n slices of 64 for the three layers; n is even; a factor divides the slice
// count).
inline int wsplit(int layer, int n) {
  return layer == 1 ? 32 : layer == 2 ? (n % 4 == 0 ? 16 : 8) : (n % 4 == 0 ? 4 : 2);
}

CnnLayout cnn_layout(int chains, int n) {
  CnnLayout L;
  size_t off = 0;
  auto take = [&](size_t per_chain) {
    const size_t at = off;
    off += (per_chain * static_cast<size_t>(chains) + 255) & ~static_cast<size_t>(255);
    return at;
  };
  const size_t N = n;
  L.w2b = take(2 * kK2 * kC2);
  L.w3b = take(2 * kK3 * kC3);
  L.p1 = take(2 * N * 256 * kC1);
  L.dy2 = take(2 * N * 256 * kC2);
  L.p2 = take(2 * N * 64 * kC2);
  L.dy3 = take(2 * N * 64 * kC3);
  L.p3 = take(2 * N * 16 * kC3);
  L.m1 = take(N * 256 * kC1);
  L.m2 = take(N * 64 * kC2);
  L.m3 = take(N * 16 * kC3);
  L.dp1 = take(4 * N * 256 * kC1);
  L.labels = take(4 * N);
  L.dp3 = take(4 * N * kFlat);
  L.gl = take(4 * N * kClasses);
  L.psq = take(8 * kPrepBlocks);
  L.plk = take(8 * 4 * N);
  const size_t wc[3] = {size_t(kC1) * kK1, size_t(kC2) * kK2, size_t(kC3) * kK3};
  for (int l = 0; l < 3; ++l) L.part[l] = take(4 * wsplit(l + 1, n) * wc[l]);
  // Bias partials: one per unpool block and channel, 8 pooled elements per
  // thread and 256 threads per block: n*Ho*Wo*C / 2048 * C = 128 n floats
  // for layers 2 and 3 (at least one block), and layer 1's units as many.
  for (int l = 0; l < 3; ++l) L.bpart[l] = take(4 * 128 * (N + 1));
  L.total = off;
  return L;
}

struct CnnArgs {
  int chains, n, want_grad;
  int64_t n_obs, n_rows, ld;
  const float* X;       // image rows: 3072 floats (32x32x3 NHWC) at X + row*ld
  const float* labels;  // label of row r at labels[r * label_ld]
  int64_t label_ld;
  const float* mask;
  const int32_t* idx;
  int64_t idx_stride;
  const float* w;
  float prior_scale, temperature;
  double* U;
  float* grad;
  float* lk;
  double* lk_var;
  int* status;
  bf16 *w2b, *w3b, *p1, *p2, *p3;
  float* dp1;
  bf16 *dy2, *dy3;
  uint8_t *m1, *m2, *m3;
  int32_t* lab;
  float *dp3, *gl;
  double *psq, *plk;
  float *part[3], *bpart[3];
  int split[3], bblocks[3];   // split-K partials, unpool blocks by layer
  float pf;                   // 1 / (s^2 T) of the prior, 0 for a flat one
  double prior_const;         // P (log s + 0.5 log 2 pi), 0 for a flat prior
};

__device__ __forceinline__ float bf(bf16 v) { return __bfloat162float(v); }

// ---------------------------------------------------------------------------
// conv1 straight from the images.
//
// conv1 has 27 inputs per output: as im2col boxes of 16 bytes a pixel its
// GEMMs were bound by the rate at which TMA takes box rows (720 cycles per 64
// pixels), and dY1, three quarters zeros, was the largest array of a
// gradient.  Here a CTA takes a strip (8 pool windows of all 16 window rows of
// an image) at a time and builds the operands in shared memory itself.
//
// X8: pixel (h, w) is one 16-byte word of BF16, the channels of (h, w - 1),
// its own, two zeros.  Tap pair p = 0 of output pixel (h, w) and kernel row
// kh is the word (h + kh - 1, w) (kw = 0, 1), p = 1 the word (.., w + 1) (its
// slots 3-5 are kw = 2; slots 0-2 repeat kw = 1 and have zero weights), so a
// K = 16 slice is a kernel row.  The words lie in planes by column parity (E:
// w = 16 s + 2 j, O: w = 16 s + 2 j + 1; 34 image rows with the zero rows
// above and below, 9 words a row): 8 neighbouring windows' words at one
// position of the window are 128 contiguous bytes, a core matrix of the
// unswizzled layout, and a descriptor's strides reach the other window rows,
// the second tap pair and the other kernel rows.  Nothing is copied per tap.
// Core matrices start on 16-byte boundaries, as that layout allows.
// For 8 x 256 images the forward pass took 128 us as three launches (weights,
// gather, GEMM) and takes 36; the output gradient with the weight GEMM took 137
// and, as a launch of its own, 55.  It now shares cnn_weight_grads_kernel with
// the other layers' (all three and the routing: 85).
// ---------------------------------------------------------------------------
constexpr int kStripThreads = 128;
constexpr int kPlaneRow = 9 * 16, kPlane = 34 * kPlaneRow;   // bytes
constexpr int kStripItems = 32 * 9, kStripIters = (kStripItems + kStripThreads - 1) / kStripThreads;

// Bounded wait that raises the CTA's abort flag and the status.
__device__ __forceinline__ bool conv_wait(uint64_t* bar, uint32_t parity, volatile int* abort,
                                          int* status) {
  if (mbar_wait_bounded(bar, parity, abort)) return true;
  raise_status(status, GBSGMC_ERR_TIMEOUT);
  *abort = 1;
  return false;
}

// Routing of a pooled map's gradient by the marks: o[pos] = the BF16 pairs of
// 8 channels at window position pos (zero where the ReLU was closed), val the
// routed (rounded) values.
__device__ __forceinline__ void route_octet(const float (&g)[8], uint2 mark, uint32_t (&o)[4][4],
                                            float (&val)[8]) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {   // four channels, a word of marks
    uint32_t pk[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(g[4 * half + 2 * e], g[4 * half + 2 * e + 1]);
      pk[e] = *reinterpret_cast<const uint32_t*>(&p);
    }
    const uint32_t m = (half ? mark.y : mark.x) & 0x07070707u;
#pragma unroll
    for (int pos = 0; pos < 4; ++pos) {
      // Bit 7 of a byte: its mark is not 4 + pos; spread over the channel's 16
      // bits by prmt's sign mode.
      const uint32_t off = (m ^ (0x01010101u * (4 + pos))) + 0x7f7f7f7fu;
      uint32_t lo, hi;
      asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(lo) : "r"(off));
      asm("prmt.b32 %0, %1, 0, 0xbbaa;" : "=r"(hi) : "r"(off));
      o[pos][2 * half] = pk[0] & ~lo;
      o[pos][2 * half + 1] = pk[1] & ~hi;
    }
#pragma unroll
    for (int e = 2 * half; e < 2 * half + 2; ++e) {
      const uint32_t v = o[0][e] | o[1][e] | o[2][e] | o[3][e];
      val[2 * e] = __uint_as_float(v << 16);
      val[2 * e + 1] = __uint_as_float(v & 0xffff0000u);
    }
  }
}

// 8 words (a 32-byte sector).
__device__ __forceinline__ void store_sector(void* at, const uint32_t (&l)[4],
                                             const uint32_t (&r)[4]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "r"(l[0]),
               "r"(l[1]), "r"(l[2]), "r"(l[3]), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}

// Pixels w - 1, w, w + 1 (w even) of an image row, px pointing at w; zeros
// when !in, and at w - 1 when !left.  `pair`: rows are 8-byte aligned, so are
// pixel pairs (6 floats).
__device__ __forceinline__ void pair_load(const float* px, bool in, bool left, bool pair,
                                          float (&v)[9]) {
#pragma unroll
  for (int e = 0; e < 9; ++e) v[e] = 0.f;
  if (pair) {
    if (in && left) {
      v[0] = __ldg(px - 3);
      const float2 q = __ldg(reinterpret_cast<const float2*>(px - 2));
      v[1] = q.x;
      v[2] = q.y;
    }
    if (in) {
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const float2 q = __ldg(reinterpret_cast<const float2*>(px) + e);
        v[3 + 2 * e] = q.x;
        v[4 + 2 * e] = q.y;
      }
    }
  } else {
#pragma unroll
    for (int e = 0; e < 9; ++e)
      if (in && (e >= 3 || left)) v[e] = __ldg(px - 3 + e);
  }
}

// Their words: E of pixel w, O of pixel w + 1.
__device__ __forceinline__ void pair_words(const float (&v)[9], uint4& e, uint4& o) {
  uint32_t q[5];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    q[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  const __nv_bfloat162 last = __floats2bfloat162_rn(v[8], 0.f);
  q[4] = *reinterpret_cast<const uint32_t*>(&last);
  e = make_uint4(q[0], q[1], q[2], 0u);
  o = make_uint4(__byte_perm(q[1], q[2], 0x5432), __byte_perm(q[2], q[3], 0x5432),
                 __byte_perm(q[3], q[4], 0x5432), 0u);
}
__device__ __forceinline__ void store_word(uint8_t* at, const uint4& v) {
  tc::sts128(at, v.x, v.y, v.z, v.w);
}

// Index of image `img` (of all chains'), as given.
__device__ __forceinline__ int image_index(const CnnArgs& a, int64_t img) {
  const int c = static_cast<int>(img / a.n), i = static_cast<int>(img - int64_t(c) * a.n);
  return __ldg(a.idx + c * a.idx_stride + i);
}
// Its observation: the first one stands in for an invalid index (which the
// forward pass reports).
__device__ __forceinline__ int64_t valid_row(const CnnArgs& a, int o) {
  return o >= 0 && o < a.n_rows ? o : 0;
}

// One thread's share of a strip, in registers: items (image row h, pair j),
// item = 9 h + j: pixels w - 1, w, w + 1 with w = 16 s + 2 j.
struct StripRegs {
  float v[kStripIters][9];
  float label;   // the last thread's
};

__device__ __forceinline__ void strip_load(const CnnArgs& a, int index, int s, bool pair,
                                           StripRegs& x) {
  const int64_t o = valid_row(a, index);
  if (o != index) raise_status(a.status, GBSGMC_ERR_INDEX);
  const float* row = a.X + o * a.ld;
  if (threadIdx.x == kStripThreads - 1) x.label = __ldg(a.labels + o * a.label_ld);
#pragma unroll
  for (int k = 0; k < kStripIters; ++k) {
    const int item = threadIdx.x + k * kStripThreads;
    const int h = item / 9, w = 16 * s + 2 * (item % 9);
    pair_load(row + (h * kImg + w) * kInC, item < kStripItems && w < kImg, w > 0, pair, x.v[k]);
  }
}

// The strip's words into planes E, O and E again (so that the second tap pair
// of an odd column lies a positive stride from the first).
__device__ __forceinline__ void strip_store(const StripRegs& x, uint8_t* planes) {
#pragma unroll
  for (int k = 0; k < kStripIters; ++k) {
    const int item = threadIdx.x + k * kStripThreads;
    if (item >= kStripItems) break;
    uint8_t* at = planes + kPlaneRow + 16 * item;
    uint4 e, o;
    pair_words(x.v[k], e, o);
    store_word(at, e);
    store_word(at + kPlane, o);
    store_word(at + 2 * kPlane, e);
  }
}

// Zero rows above and below the image in the planes.
__device__ __forceinline__ void strip_borders(uint8_t* smem) {
  for (int e = threadIdx.x; e < 3 * 18; e += kStripThreads) {
    const int p = e / 18, r = e % 18;
    tc::sts128(smem + p * kPlane + (r < 9 ? 16 * r : 33 * kPlaneRow + 16 * (r - 9)), 0u, 0u, 0u,
               0u);
  }
}

// BF16 weights of conv2 ([output octet][tap, input][8], so that outputs and
// inputs both lie in core matrices) and conv3 ([tap][output octet][input][8])
// and part `b` of a chain's sum
// of squares.
__device__ __forceinline__ void cnn_prep(const CnnArgs& a, int c, int b, double* red) {
  constexpr int kCols = 256, kEach = kCols / kStripThreads, kStride = kPrepBlocks * kCols;
  constexpr int kRounds = static_cast<int>((kP + kStride - 1) / kStride);
  const float* w = a.w + static_cast<int64_t>(c) * kP;
  float sq[kEach] = {}, v[kRounds][kEach];
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      const int j = b * kCols + threadIdx.x + r * kStride + u * kStripThreads;
      v[r][u] = j < kP ? __ldg(w + j) : 0.f;
    }
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      const int j = b * kCols + threadIdx.x + r * kStride + u * kStripThreads;
      const float x = v[r][u];
      if (j < kP) sq[u] = fmaf(x, x, sq[u]);
      if (j >= oW2 && j < ob3)
        a.w2b[static_cast<int64_t>(c) * kK2 * kC2 +
              ((j - oW2) % kC2 / 8 * kK2 + (j - oW2) / kC2) * 8 + j % 8] = __float2bfloat16_rn(x);
      else if (j >= oW3 && j < obd)
        a.w3b[static_cast<int64_t>(c) * kK3 * kC3 +
              (((j - oW3) / kC3 / kC2 * (kC3 / 8) + (j - oW3) % kC3 / 8) * kC2 +
               (j - oW3) / kC3 % kC2) * 8 + (j - oW3) % 8] = __float2bfloat16_rn(x);
    }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < kEach; ++u) {
    const double part = warp_sum(static_cast<double>(sq[u]));
    if (lane == 0) red[u * (kStripThreads / 32) + warp] = part;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int i = 0; i < kCols / 32; ++i) tot += red[i];
    a.psq[c * kPrepBlocks + b] = tot;
  }
  __syncthreads();
}

// 16 columns of each of four accumulators 32 columns apart (one wait).
__device__ __forceinline__ void tmem_ld16x4(uint32_t taddr, float (&v)[4][16]) {
  uint32_t r[4][16];
#pragma unroll
  for (int p = 0; p < 4; ++p)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[p][0]), "=r"(r[p][1]), "=r"(r[p][2]), "=r"(r[p][3]), "=r"(r[p][4]),
          "=r"(r[p][5]), "=r"(r[p][6]), "=r"(r[p][7]), "=r"(r[p][8]), "=r"(r[p][9]),
          "=r"(r[p][10]), "=r"(r[p][11]), "=r"(r[p][12]), "=r"(r[p][13]), "=r"(r[p][14]),
          "=r"(r[p][15])
        : "r"(taddr + p * kC1));
#pragma unroll
  for (int p = 0; p < 4; ++p)   // the registers may be used after the wait only
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[p][0]), "+r"(r[p][1]), "+r"(r[p][2]), "+r"(r[p][3]), "+r"(r[p][4]),
                   "+r"(r[p][5]), "+r"(r[p][6]), "+r"(r[p][7]), "+r"(r[p][8]), "+r"(r[p][9]),
                   "+r"(r[p][10]), "+r"(r[p][11]), "+r"(r[p][12]), "+r"(r[p][13]),
                   "+r"(r[p][14]), "+r"(r[p][15])
                 :
                 : "memory");
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int i = 0; i < 16; ++i) v[p][i] = __uint_as_float(r[p][i]);
}

// Forward: P1 and its marks, and beside it what needs no launch of its own:
// the labels, the BF16 weights of the other layers and the sums of squares.
// Four CTAs per SM (128 TMEM columns each), each a run of consecutive strips;
// one CTA's loads and epilogue overlap the others' MMAs.  The four pixels of
// a window are four accumulators (M = 128 windows, N = 32) of the same TMEM
// lane, so the pooling needs no exchange between lanes.
__global__ void __launch_bounds__(kStripThreads, 4) cnn_conv1_kernel(const CnnArgs a, int pair) {
  __shared__ __align__(128) uint8_t planes[3 * kPlane];
  __shared__ __align__(128) bf16 w_s[6 * kC1 * kX8];   // [tap pair 2 kh + p][output][slot]
  __shared__ float b_s[kC1];
  __shared__ double red[32];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(&tmem_slot, 128);
    tc::tmem_relinquish();
  }
  strip_borders(planes);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();
  pdl_wait();

  // CTAs past the strips' prepare weights alone; without such, all do.
  const int64_t strips = 2 * static_cast<int64_t>(a.chains) * a.n;
  const int own = strips < gridDim.x ? static_cast<int>(strips) : gridDim.x;
  const int b = blockIdx.x;
  const int64_t u0 = b < own ? strips * b / own : 0, u1 = b < own ? strips * (b + 1) / own : 0;
  const int preps = gridDim.x > own ? gridDim.x - own : own;
  StripRegs x;
  int next = 0;   // index of the strip after the loaded one
  if (u0 < u1) {
    strip_load(a, image_index(a, u0 >> 1), static_cast<int>(u0 & 1), pair, x);
    if (u0 + 1 < u1) next = image_index(a, (u0 + 1) >> 1);
  }
  for (int e = preps == own ? b : b - own; e >= 0 && e < a.chains * kPrepBlocks; e += preps)
    cnn_prep(a, e / kPrepBlocks, e % kPrepBlocks, red);

  constexpr uint32_t idesc = tc::idesc_bf16_f32(128, kC1);
  int chain = -1;
  uint32_t phase = 0;
  bool ok = true;
  for (int64_t u = u0; u < u1; ++u, phase ^= 1u) {
    const int64_t img = u >> 1;
    const int s = static_cast<int>(u & 1), c = static_cast<int>(img / a.n);
    if (c != chain) {
      chain = c;
      const float* w = a.w + static_cast<int64_t>(c) * kP;
      for (int e = t; e < 6 * kC1 * kX8; e += kStripThreads) {
        const int g = e / (kC1 * kX8), co = (e / kX8) % kC1, sl = e % kX8;
        const int kw = (g & 1) + sl / kInC, ci = sl % kInC;
        const bool real = sl < 2 * kInC && ((g & 1) == 0 || sl >= kInC);
        const float v = real ? __ldg(w + oW1 + (((g >> 1) * 3 + kw) * kInC + ci) * kC1 + co) : 0.f;
        w_s[e] = __float2bfloat16_rn(v);
      }
      if (t < kC1) b_s[t] = __ldg(w + ob1 + t);
    }
    strip_store(x, planes);
    tc::fence_async_shared();
    if (t == kStripThreads - 1 && s == 0) {
      int lab = static_cast<int>(x.label);
      if (!(x.label >= 0.f) || lab >= kClasses) {
        raise_status(a.status, GBSGMC_ERR_INDEX);
        lab = 0;
      }
      a.lab[img] = lab;
    }
    // The next strip's loads are under way while this one is multiplied.
    if (u + 1 < u1) {
      strip_load(a, next, static_cast<int>((u + 1) & 1), pair, x);
      if (u + 2 < u1) next = image_index(a, (u + 2) >> 1);
    }
    __syncthreads();
    if (warp == 0 && tc::elect_one()) {
      tc::fence_after_sync();
      const uint64_t A0 = tc::sdesc_none(planes, kPlane, 2 * kPlaneRow);
      const uint64_t A1 = tc::sdesc_none(planes + kPlane, kPlane + 16, 2 * kPlaneRow);
      const uint64_t B = tc::sdesc_none(w_s, kC1 * 16, 128);
#pragma unroll
      for (int pos = 0; pos < 4; ++pos)
#pragma unroll
        for (int kh = 0; kh < 3; ++kh)
          tc::mma_bf16(tmem + pos * kC1,
                       ((pos & 1) ? A1 : A0) + ((pos >> 1) + kh) * (kPlaneRow / 16),
                       B + kh * (2 * kC1 * kX8 * 2 / 16), idesc, kh != 0);
      tc::mma_commit(&bar);
    }
    ok = mbar_wait_bounded(&bar, phase, nullptr);
    tc::fence_after_sync();
    if (ok) {
      // Lane 8 i + j of warp q is the window (4 q + i, 8 s + j).
      const int64_t pix = img * 256 + (4 * warp + (lane >> 3)) * 16 + 8 * s + (lane & 7);
      bf16* p1 = a.p1 + ((img * 16 + 4 * warp + (lane >> 3)) * 64 + 8 * s + (lane & 7)) * 8;
      const uint32_t acc = tmem + (static_cast<uint32_t>(warp * 32) << 16);
#pragma unroll
      for (int q = 0; q < kC1 / 16; ++q) {
        float v[4][16];
        tmem_ld16x4(acc + 16 * q, v);
        uint32_t pk[8], mk[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) mk[e] = 0u;
        float best[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float b = b_s[16 * q + j];
          const float y0 = v[0][j] + b, y1 = v[1][j] + b, y2 = v[2][j] + b, y3 = v[3][j] + b;
          // The ReLU of the maximum, and the first position that has it (of no
          // account where the ReLU is closed).
          best[j] = fmaxf(fmaxf(fmaxf(y0, y1), fmaxf(y2, y3)), 0.f);
          const uint32_t at = y0 == best[j] ? 4u : y1 == best[j] ? 5u : y2 == best[j] ? 6u : 7u;
          mk[j >> 2] |= (best[j] > 0.f ? at : 0u) << (8 * (j & 3));
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(best[2 * e], best[2 * e + 1]);
          pk[e] = *reinterpret_cast<const uint32_t*>(&pr);
        }
        *reinterpret_cast<uint4*>(p1 + 256 * q) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(p1 + 256 * q + 128) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        *reinterpret_cast<uint4*>(a.m1 + pix * kC1 + 16 * q) =
            make_uint4(mk[0], mk[1], mk[2], mk[3]);
      }
    }
    tc::fence_before_sync();
    if (__syncthreads_or(!ok)) break;   // also: the planes and accumulators are free
  }
  if (!ok) {
    raise_status(a.status, GBSGMC_ERR_TIMEOUT);
    mbar_wait_bounded(&bar, phase, nullptr);   // MMAs still in flight
  }
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 128);
  }
}

// dW1 = dY1^T Col1 and db1, dY1 built from dP1 and the marks in units of 8
// image rows.  A CTA adds its run of 64-pixel slices (4 rows of a 16-column
// half; the order of slices: rows 0-3 and 4-7 of the left half, then of the
// right) in one accumulator (M = 64 output channels, 32 real) and writes one
// split-K partial; a K = 16 slice is the half's 16 pixels of an image row, its
// even columns, then its odd ones.  Here a row's words lie in three runs of
// 16, E, O and E one column on, and the N groups of an MMA are three rows' runs
// (N = 72, the stride of a run): for the even columns E is tap pair 0 and O
// pair 1, for the odd ones (one run further on) O and the shifted E, and the
// third run of each row is dropped.  dY: [image row h][half][column parity]
// [channel octet][8 windows] words of 8 channels; the rows past the octets
// that the MMA reads belong to the next block of dY (or to the words) and end
// in accumulator rows that nothing reads.  The operands are double buffered:
// the MMAs of a unit (issued by a warp of its own) run while the next is
// built.  db1 (another warp): the routed
// (BF16-rounded) values of a unit's 64 windows are added in window order, a
// partial per unit.
constexpr int kDyWarps = 8, kWordWarps = 6, kUnitThreads = 32 * (kDyWarps + kWordWarps + 2);
constexpr int kUnitRow = 3 * 256;   // bytes of a row's E, O and shifted E
constexpr int kUnitDy = 8 * 2 * 1024, kUnitWords = 11 * kUnitRow, kUnitBias = 64 * 36 * 4;
constexpr int kUnitBuf = kUnitDy + kUnitWords + kUnitBias;
static_assert(kUnitBuf % 128 == 0, "buffer alignment");
constexpr int kUnitSmem = 2 * kUnitBuf;

__device__ __forceinline__ void conv1_grad(const CnnArgs& a, int pair, uint8_t* unit_smem, int c,
                                           int split, int S) {
  __shared__ uint64_t full[2], free_[2];   // a buffer is built; its MMAs and sums are done
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(full + i, kDyWarps + kWordWarps);
      mbar_init(free_ + i, 2);
    }
    abort_s = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(&tmem_slot, 128);
    tc::tmem_relinquish();
  }
  // The words' last row stands behind a unit's last for the dropped run.
  for (int e = t; e < 2 * kUnitRow / 16; e += kUnitThreads)
    store_word(unit_smem + (e & 1) * kUnitBuf + kUnitDy + 10 * kUnitRow + (e >> 1) * 16,
               make_uint4(0u, 0u, 0u, 0u));
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  pdl_trigger();
  pdl_wait();

  const int each = 16 * a.n / S, q0 = each * split, q1 = q0 + each;   // slices
  const int u0 = q0 >> 2, u1 = (q1 + 3) >> 2;                              // units
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    return conv_wait(bar, parity, abort_flag, a.status);
  };
  if (warp == kDyWarps + kWordWarps) {   // the MMAs
    constexpr uint32_t idesc = tc::idesc_bf16_f32(64, 72, true, true);
    if (tc::elect_one()) {
      for (int u = u0; u < u1; ++u) {
        const int it = u - u0, b = it & 1;
        if (!wait(full + b, (it >> 1) & 1u)) break;
        tc::fence_after_sync();
        const uint8_t* dy = unit_smem + b * kUnitBuf;
        const uint64_t A = tc::sdesc_none(dy, 512, 128);
        const uint64_t B = tc::sdesc_none(dy + kUnitDy, 256, 256);
#pragma unroll
        for (int q = 0; q < 4; ++q) {   // the unit's slices: half q / 2, rows 4 (q % 2) ..
          if (4 * u + q < q0 || 4 * u + q >= q1) continue;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int h = 4 * (q & 1) + r, half = q >> 1;
            tc::mma_bf16(tmem, A + (2 * h + half) * 64, B + (h * kUnitRow + half * 128) / 16,
                         idesc, 4 * u + q > q0 || r > 0);
          }
        }
        tc::mma_commit(free_ + b);
      }
    }
    __syncwarp();
  } else if (warp > kDyWarps + kWordWarps) {   // the bias
    for (int u = u0; u < u1; ++u) {
      const int it = u - u0, b = it & 1;
      if (!__all_sync(0xffffffffu, wait(full + b, (it >> 1) & 1u))) break;
      const float* bias =
          reinterpret_cast<const float*>(unit_smem + b * kUnitBuf + kUnitDy + kUnitWords);
      float sum = 0.f;
#pragma unroll 16
      for (int w = 0; w < 64; ++w) sum += bias[w * 36 + lane];
      __syncwarp();
      if (lane == 0) mbar_arrive(free_ + b);
      // A unit cut by a split boundary belongs to the split of its first slice.
      if (4 * u >= q0) a.bpart[0][(int64_t(c) * 4 * a.n + u) * kC1 + lane] = sum;
    }
  } else if (warp < kDyWarps) {
    // dY: this thread's window (row wy of the unit's 4, column wx) and octet.
    const int j = lane & 7, oct = lane >> 3, wx = 8 * (warp & 1) + j, wy = warp >> 1;
    struct Part {
      float4 g[2];
      uint2 mark;
    };
    auto load = [&](int u, Part& p) {
      const int64_t row = (int64_t(c) * a.n + (u >> 2)) * 16 + 4 * (u & 3) + wy;
      const float4* d = reinterpret_cast<const float4*>(a.dp1 + (row * 64 + 16 * oct + wx) * 8);
      p.g[0] = __ldg(d);
      p.g[1] = __ldg(d + 1);
      p.mark = __ldg(reinterpret_cast<const uint2*>(a.m1 + (row * 16 + wx) * kC1 + 8 * oct));
    };
    auto unit = [&](int u, Part& p) -> bool {
      const int it = u - u0, b = it & 1;
      uint8_t* dy = unit_smem + b * kUnitBuf;
      float* bias = reinterpret_cast<float*>(dy + kUnitDy + kUnitWords);
      if (it >= 2 && !__all_sync(0xffffffffu, wait(free_ + b, ((it >> 1) - 1) & 1u))) return false;
      const float4 &g0 = p.g[0], &g1 = p.g[1];
      const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      uint32_t o[4][4];
      float val[8];
      route_octet(g, p.mark, o, val);
#pragma unroll
      for (int pos = 0; pos < 4; ++pos)
        tc::sts128(dy + ((2 * wy + (pos >> 1)) * 2 + (warp & 1)) * 1024 + (pos & 1) * 512 +
                       16 * lane,
                   o[pos][0], o[pos][1], o[pos][2], o[pos][3]);
      float4* bd = reinterpret_cast<float4*>(bias + (16 * wy + wx) * 36 + 8 * oct);
      bd[0] = make_float4(val[0], val[1], val[2], val[3]);
      bd[1] = make_float4(val[4], val[5], val[6], val[7]);
      tc::fence_async_shared();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + b);
      if (u + 2 < u1) load(u + 2, p);
      return true;
    };
    Part part[2];   // loads are two units ahead of their use
    load(u0, part[0]);
    if (u0 + 1 < u1) load(u0 + 1, part[1]);
    for (int u = u0; u < u1; u += 2) {
      if (!unit(u, part[0])) break;
      if (u + 1 < u1 && !unit(u + 1, part[1])) break;
    }
  } else {
    // X8: this thread's pixel pair (rows -1 .. 8 of the unit, 17 pairs a row;
    // the last holds the column past the image: zeros, as at w = -1).
    const int e = t - 32 * kDyWarps, xr = e / 17, xj = e % 17;
    struct Pair {
      float x[9];
    };
    auto row_of = [&](int u) { return image_index(a, int64_t(c) * a.n + (u >> 2)); };
    auto load = [&](int u, int index, Pair& p) {
      const int h = 8 * (u & 3) + xr - 1;
      const bool in = xr < 10 && h >= 0 && h < kImg && xj < 16;
      pair_load(a.X + valid_row(a, index) * a.ld + (h * kImg + 2 * xj) * kInC, in, xj > 0, pair,
                p.x);
    };
    Pair part[2];
    load(u0, row_of(u0), part[0]);
    if (u0 + 1 < u1) load(u0 + 1, row_of(u0 + 1), part[1]);
    int next = u0 + 2 < u1 ? row_of(u0 + 2) : 0;   // indices a unit further ahead
    auto unit = [&](int u, Pair& p) -> bool {
      const int it = u - u0, b = it & 1;
      uint8_t* at = unit_smem + b * kUnitBuf + kUnitDy + xr * kUnitRow + 16 * xj;
      if (it >= 2 && !__all_sync(0xffffffffu, wait(free_ + b, ((it >> 1) - 1) & 1u))) return false;
      if (xr < 10) {
        uint4 even, odd;
        pair_words(p.x, even, odd);
        if (xj < 16) {
          store_word(at, even);
          store_word(at + 256, odd);
        }
        if (xj > 0) store_word(at + 512 - 16, even);
      }
      tc::fence_async_shared();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + b);
      if (u + 2 < u1) {
        load(u + 2, next, p);
        if (u + 3 < u1) next = row_of(u + 3);
      }
      return true;
    };
    for (int u = u0; u < u1; u += 2) {
      if (!unit(u, part[0])) break;
      if (u + 1 < u1 && !unit(u + 1, part[1])) break;
    }
  }
  // Every MMA has completed: the last two units' are waited for here.
  const int done = u1 - u0;
  for (int i = done > 1 ? done - 2 : 0; i < done; ++i)
    if (!mbar_wait_bounded(free_ + (i & 1), (i >> 1) & 1u, abort_flag)) {
      raise_status(a.status, GBSGMC_ERR_TIMEOUT);
      *abort_flag = 1;
    }
  __syncthreads();
  if (*abort_flag) {   // MMAs issued complete within microseconds
    const uint64_t t0 = global_ns();
    while (global_ns() - t0 < 2000000ull) {
    }
  }
  tc::fence_after_sync();
  if (warp < 2) {
    // Accumulator row r of an M = 64 tile is TMEM lane 32 (r / 16) + r % 16.
    float* dst = a.part[0] + (static_cast<int64_t>(c) * S + split) * kK1 * kC1 + 16 * warp +
                 lane;
#pragma unroll
    for (int kh = 0; kh < 3; ++kh) {   // columns (kh, run, slot)
      float v[32];
      tc::tmem_ld32(tmem + 24 * kh + (static_cast<uint32_t>(warp * 32) << 16), v);
      if (lane < 16) {
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int sl = p * kInC; sl < 2 * kInC; ++sl)
            dst[((kh * 3 + p + sl / kInC) * kInC + sl % kInC) * kC1] = v[8 * p + sl];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 128);
  }
}

// The 2 x 2 max-pool of 32 channels of a warp's 32 pixels (ReLU applied): the
// window of lane l is lanes (base, base + 1, base + V, base + V + 1), base = l
// & ~(V | 1), in window order.  Lane l ends with the maxima (BF16) and marks
// of 8 channels, chunk `wp` (returned) of the 32.  The window maxima take two
// exchange stages instead of four shuffles per channel: the two pixels of a
// window row swap the halves of the channels they do not keep (16 shuffles)
// and keep the pairwise maximum, then the two rows swap halves again (8
// shuffles); comparisons are strict in window order (left before right, top
// before bottom), which keeps the first maximum of the window as the
// sequential scan does.
template <int V>
__device__ __forceinline__ int pool_windows(const float (&x)[32], uint4& p, uint2& mk) {
  const unsigned full = 0xffffffffu;
  const int lane = epi::lane_id();
  const int wp = ((lane & V) ? 2 : 0) | (lane & 1);
  // Stage 1, the window row's two pixels (lanes l, l ^ 1): keep the
  // chunks {cbit, cbit + 2} of 8 channels (kept channel i: i < 8 in
  // the first, i >= 8 in the second), send the other two.
  const bool cbit = (lane & 1) != 0, rbit = (lane & V) != 0;
  float m1[16];
  uint32_t col_bits = 0;  // bit i: kept channel i's maximum is the right pixel
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int lo = q < 8 ? q : 8 + q, hi = lo + 8;
    const float mine = cbit ? x[hi] : x[lo];
    const float other = __shfl_xor_sync(full, cbit ? x[lo] : x[hi], 1);
    const float left = cbit ? other : mine, right = cbit ? mine : other;
    const bool rt = right > left;
    m1[q] = rt ? right : left;
    col_bits |= (rt ? 1u : 0u) << q;
  }
  // Stage 2, the window's two rows (lanes l, l ^ V): the top row keeps
  // kept channels 0-7 (chunk cbit), the bottom row 8-15 (chunk
  // cbit + 2): chunk wp of the 32 channels.
  const uint32_t other_bits = __shfl_xor_sync(full, col_bits, V);
  float best_mine[8];
  uint32_t mark_mine[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int ki = rbit ? 8 + q : q;
    const float mine = rbit ? m1[8 + q] : m1[q];
    const float other = __shfl_xor_sync(full, rbit ? m1[q] : m1[8 + q], V);
    const uint32_t my_col = (col_bits >> ki) & 1u, ot_col = (other_bits >> ki) & 1u;
    const float top = rbit ? other : mine, bot = rbit ? mine : other;
    const uint32_t top_col = rbit ? ot_col : my_col, bot_col = rbit ? my_col : ot_col;
    const bool b2 = bot > top;
    const float best = b2 ? bot : top;
    best_mine[q] = best;
    mark_mine[q] = (b2 ? 2u + bot_col : top_col) | (best > 0.f ? 4u : 0u);
  }
  uint32_t pk[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __nv_bfloat162 pr = __floats2bfloat162_rn(best_mine[2 * e], best_mine[2 * e + 1]);
    pk[e] = *reinterpret_cast<const uint32_t*>(&pr);
  }
  p = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  mk.x = mark_mine[0] | (mark_mine[1] << 8) | (mark_mine[2] << 16) | (mark_mine[3] << 24);
  mk.y = mark_mine[4] | (mark_mine[5] << 8) | (mark_mine[6] << 16) | (mark_mine[7] << 24);
  return wp;
}

// ---------------------------------------------------------------------------
// conv2 (16 x 16 images), its input gradient and its weight gradient without
// an im2col.
//
// The maps they read are stored in rows of channel octets, [image][h][octet]
// [w][8]: one TMA box of a strip (8 columns of an image, all rows) with its
// halo lands as [h][octet][10 columns] words of 16 bytes, zeros outside the
// image (the SAME padding), and any 8 neighbouring pixels of an octet are a
// core matrix of the unswizzled layout.  A tap is then only another start
// address of the same box: conv2's box of 128 pixels is 72 rows of 160 bytes
// for TMA instead of 9 boxes, or an im2col of 9 times the map, written and read
// back.  2,048 images: 25 us against 147 with the im2col (335 MB), dP1 26
// against 115 with a box per tap, dW2, while it had a launch of its own, 25
// against 95 (now part of cnn_weight_grads_kernel).  W2 lies in shared memory,
// [output octet][tap, input][8], for a run of strips of one chain: MN-major B
// of the forward GEMM, K-major B of the transposed one.
// ---------------------------------------------------------------------------
constexpr int kW2Bytes = kC2 * kK2 * 2, kW2Octet = kK2 * 16;
constexpr int strip_box(int channels) { return 18 * (channels / 8) * 160; }

// Forward (CK = 32 input channels, N = 64 outputs) or transposed (CK = 64, N
// = 32): per strip D (128 pixels x N) = sum over taps and K = 16 slices of
// the box's shifted words times W2, in the order (tap, channel).  Roles: warp
// 0 (a lane) loads boxes into a ring and W2 when the chain changes, warp 1 (a
// lane) issues the MMAs into two accumulators, eight warps run the epilogue
//   epi.tile(image, chain, strip, lane quarter, first column, values)
// on 32 lanes and 32 columns at a time: with N = 64 each accumulator's halves
// go to four warps each, with N = 32 the two accumulators do.  Two CTAs per
// SM, each a run of consecutive strips.
constexpr int kConvStages = 3;   // 23 KB each for 64 channels
constexpr int kConvThreads = 64 + 8 * 32;
template <int CK>
constexpr int conv_smem() {
  return kW2Bytes + kConvStages * strip_box(CK) + 128 + 256;
}

template <int CK, int N, class Epi>
__global__ void __launch_bounds__(kConvThreads, 2)
    cnn_conv2_kernel(const __grid_constant__ CUtensorMap map, const bf16* wts, int chains, int n,
                     int* status, const __grid_constant__ Epi epi) {
  constexpr bool kFwd = N == kC2;
  constexpr int kBox = strip_box(CK), kRow = (CK / 8) * 160;   // bytes of a box, an image row
  constexpr uint32_t kCols = 2 * N;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* w_s = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* ring = w_s + kW2Bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + kConvStages * kBox);
  uint64_t* empty = full + kConvStages;
  uint64_t* wfull = empty + kConvStages;
  uint64_t* tfull = wfull + 1;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kConvStages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(wfull, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull + i, 1);
      mbar_init(tempty + i, kFwd ? 8 : 4);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, kCols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int64_t strips = 2 * static_cast<int64_t>(chains) * n;
  const int64_t u0 = strips * blockIdx.x / gridDim.x, u1 = strips * (blockIdx.x + 1) / gridDim.x;

  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t it = 0, loads = 0;
      int chain = -1;
      for (int64_t u = u0; u < u1; ++u, ++it) {
        const int64_t img = u >> 1;
        const int c = static_cast<int>(img / n), s = it % kConvStages;
        if (c != chain) {
          // W2 is free once the last strip's MMAs are.
          if (it > 0 && !conv_wait(empty + (it - 1) % kConvStages, ((it - 1) / kConvStages) & 1u,
                                   abort_flag, status))
            break;
          chain = c;
          mbar_arrive_expect_tx(wfull, kW2Bytes);
          bulk_g2s(w_s, wts + static_cast<int64_t>(c) * kC2 * kK2, kW2Bytes, wfull);
          ++loads;
        }
        if (!conv_wait(empty + s, ((it / kConvStages) & 1u) ^ 1u, abort_flag, status)) break;
        mbar_arrive_expect_tx(full + s, kBox);
        tc::tma_load_4d(ring + s * kBox, &map, 64 * static_cast<int>(u & 1) - 8, 0, -1,
                        static_cast<int>(img), full + s);
      }
      if (*abort_flag) {   // copies in flight land before the CTA ends
        for (uint32_t i = it > kConvStages ? it - kConvStages : 0; i < it; ++i)
          mbar_wait_bounded(full + i % kConvStages, (i / kConvStages) & 1u, nullptr);
        if (loads > 0) mbar_wait_bounded(wfull, (loads - 1) & 1u, nullptr);
      }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(128, N, false, kFwd);
      const uint64_t B = kFwd ? tc::sdesc_none(w_s, 128, kW2Octet)
                              : tc::sdesc_none(w_s, kW2Octet, 128);
      uint32_t it = 0, loads = 0;
      int chain = -1;
      for (int64_t u = u0; u < u1; ++u, ++it) {
        const int c = static_cast<int>((u >> 1) / n), s = it % kConvStages;
        const uint32_t buf = it & 1u;
        if (c != chain) {
          chain = c;
          if (!conv_wait(wfull, loads & 1u, abort_flag, status)) break;
          ++loads;
        }
        if (!conv_wait(tempty + buf, ((it >> 1) & 1u) ^ 1u, abort_flag, status) ||
            !conv_wait(full + s, (it / kConvStages) & 1u, abort_flag, status))
          break;
        tc::fence_after_sync();
        const uint64_t A = tc::sdesc_none(ring + s * kBox, 160, kRow);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
          const int kh = kFwd ? tap / 3 : 2 - tap / 3, kw = kFwd ? tap % 3 : 2 - tap % 3;
#pragma unroll
          for (int k = 0; k < CK / 16; ++k)
            tc::mma_bf16(tmem + buf * N, A + (kh * kRow + kw * 16 + k * 320) / 16,
                         B + (kFwd ? (tap * CK + 16 * k) : tap * N + k * (2 * kW2Octet / 16)),
                         idesc, (tap | k) != 0);
        }
        tc::mma_commit(empty + s);
        tc::mma_commit(tfull + buf);
      }
      tc::mma_commit(drain);   // every MMA of this CTA has completed once it flips
      mbar_wait_bounded(drain, 0, nullptr);
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint32_t it = 0;
    for (int64_t u = u0; u < u1; ++u, ++it) {
      const uint32_t buf = it & 1u;
      if (!kFwd && static_cast<int>(buf) != half) continue;
      const bool ok = mbar_wait_bounded(tfull + buf, (it >> 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0 && !*abort_flag) {
          raise_status(status, GBSGMC_ERR_TIMEOUT);
          *abort_flag = 1;
        }
        break;
      }
      tc::fence_after_sync();
      const int col0 = kFwd ? 32 * half : 0;
      const tc::TmemRows load{tmem + buf * N + col0 + (static_cast<uint32_t>(q * 32) << 16)};
      float v[32];
      load(0, v);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty + buf);   // the accumulator is in registers
      epi.tile(u >> 1, static_cast<int>((u >> 1) / n), static_cast<int>(u & 1), q, col0, v);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kCols);
  }
}

// conv2's pooling: lane 8 i + j of quarter q is the pixel (4 q + i, 8 s + j).
struct EpiStripPool {
  const float* w;
  bf16* P;      // [pair][h][image of the pair][octet][w][8]
  uint8_t* M;
  __device__ __forceinline__ void tile(int64_t img, int c, int s, int q, int col0,
                                       float (&v)[32]) const {
    const int lane = epi::lane_id();
    const int base = lane & ~9;
    const int h = 2 * q + (base >> 4), x = 4 * s + ((base & 7) >> 1);
    const float bl = __ldg(w + static_cast<int64_t>(c) * kP + ob2 + col0 + lane);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j] + __shfl_sync(0xffffffffu, bl, j), 0.f);
    uint4 p;
    uint2 m;
    const int wp = pool_windows<8>(v, p, m);
    *reinterpret_cast<uint4*>(
        P + ((((img >> 1) * 8 + h) * 2 + (img & 1)) * 8 + col0 / 8 + wp) * 64 + x * 8) = p;
    *reinterpret_cast<uint2*>(M + (img * 64 + h * 8 + x) * kC2 + col0 + 8 * wp) = m;
  }
};

// conv2's input gradient as fp32, [image][h][octet][w][8], a sector per store.
struct EpiStripDX {
  float* dx;
  __device__ __forceinline__ void tile(int64_t img, int, int s, int q, int,
                                       float (&v)[32]) const {
    const int lane = epi::lane_id();
    float* dst = dx + ((img * 16 + 4 * q + (lane >> 3)) * 64 + 8 * s + (lane & 7)) * 8;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const float* e = v + 8 * o;
      asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 128 * o),
                   "f"(e[0]), "f"(e[1]), "f"(e[2]), "f"(e[3]), "f"(e[4]), "f"(e[5]), "f"(e[6]),
                   "f"(e[7])
                   : "memory");
    }
  }
};

// dW2 = dY2^T Col2: per 64-pixel slice (4 image rows) the boxes of dY2 and of
// P1 with its halo, both MN-major with an image row's 16 pixels as K; a
// column shift kw is one MMA of M = 64 outputs x N = 96 (three kernel rows x
// 32 inputs: the box's [h][octet] words lie 288 bytes apart).  The sums of a
// run of a chain's slices stay in TMEM and are written as one split-K partial
// [tap, input][output].  A CTA takes a split and a column shift.
constexpr int kDy2Box = 4 * (kC2 / 8) * 256, kP1Box = 6 * (kC1 / 8) * 288;
constexpr int kDw2Stages = 7, kDw2Threads = 64 + 4 * 32;
constexpr int kDw2Smem = kDw2Stages * (kDy2Box + kP1Box) + 128 + 256;

__device__ __forceinline__ void conv2_dw(const CUtensorMap& mdy, const CUtensorMap& mp1,
                                         float* part, int n, int* status, uint8_t* smem_raw, int c,
                                         int split, int S, int kw) {
  constexpr int kStage = kDy2Box + kP1Box;
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + kDw2Stages * kStage);
  uint64_t* empty = full + kDw2Stages;
  uint64_t* done = empty + kDw2Stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kDw2Stages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, 128);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int each = 4 * n / S, u0 = each * split, u1 = u0 + each;   // slices
  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t it = 0;
      for (int u = u0; u < u1; ++u, ++it) {
        const int s = it % kDw2Stages, img = c * n + (u >> 2), h0 = 4 * (u & 3);
        if (!conv_wait(empty + s, ((it / kDw2Stages) & 1u) ^ 1u, abort_flag, status)) break;
        uint8_t* dst = ring + s * kStage;
        mbar_arrive_expect_tx(full + s, kStage);
        tc::tma_load_4d(dst, &mdy, 0, 0, h0, img, full + s);
        tc::tma_load_4d(dst + kDy2Box, &mp1, -8, 0, h0 - 1, img, full + s);
      }
      if (*abort_flag)
        for (uint32_t i = it > kDw2Stages ? it - kDw2Stages : 0; i < it; ++i)
          mbar_wait_bounded(full + i % kDw2Stages, (i / kDw2Stages) & 1u, nullptr);
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(64, 96, true, true);
      uint32_t it = 0;
      for (int u = u0; u < u1; ++u, ++it) {
        const int s = it % kDw2Stages;
        if (!conv_wait(full + s, (it / kDw2Stages) & 1u, abort_flag, status)) break;
        tc::fence_after_sync();
        const uint64_t A = tc::sdesc_none(ring + s * kStage, 128, 256);
        const uint64_t B = tc::sdesc_none(ring + s * kStage + kDy2Box, 128, 288);
#pragma unroll
        for (int h = 0; h < 4; ++h)
          tc::mma_bf16(tmem, A + h * (kC2 / 8) * 256 / 16, B + h * (kC1 / 8) * 288 / 16 + kw, idesc,
                       it > 0 || h > 0);
        tc::mma_commit(empty + s);
      }
      tc::mma_commit(done);
      mbar_wait_bounded(done, 0, nullptr);
    }
  } else if (warp < kDw2Threads / 32) {
    const bool ok = mbar_wait_bounded(done, 0, nullptr);
    if (!__all_sync(0xffffffffu, ok) && lane == 0) raise_status(status, GBSGMC_ERR_TIMEOUT);
    tc::fence_after_sync();
    // Accumulator row r of an M = 64 tile is TMEM lane 32 (r / 16) + r % 16.
    const int q = warp & 3;
    float* dst = part + (static_cast<int64_t>(c) * S + split) * kK2 * kC2 + 16 * q + lane;
#pragma unroll 1
    for (int kh = 0; kh < 3; ++kh) {
      float v[32];
      tc::tmem_ld32(tmem + 32 * kh + (static_cast<uint32_t>(q * 32) << 16), v);
      const int tap = 3 * kh + kw;
      if (lane < 16) {
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[(tap * kC1 + j) * kC2] = v[j];
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 128);
  }
}

// ---------------------------------------------------------------------------
// conv3 (8 x 8 images) and its gradients: as conv2, on pairs of images.
//
// P2 and dY3 are stored as [pair][h][image of the pair][octet][w][8], so that
// a pair's box with its halo ([h][image][octet][10 columns] words) has 16 rows
// of 8 pixels a uniform stride apart: a tile of M = 128.  W3 ([tap][output
// octet][input][8], MN-major B of the forward GEMM and K-major B of the
// transposed one) streams through a ring, 16 KB a tap: resident it would leave
// no room for two boxes of dY3.  2,048 images: conv3 18 us against 27 with a
// swizzled box per tap, dP2 26 with its routing against 41 + 21.
//
// Forward (CK = 64, N = 128) or transposed (CK = 128, N = 64).  Roles: warp 0
// loads boxes, warp 1 issues the MMAs into two accumulators, warp 2 loads
// weights, warps 4-11 run the epilogue
//   epi.tile(pair, chain, lane quarter, half, accumulator)
// on 32 lanes and the columns [half N / 2, (half + 1) N / 2).  One CTA per SM,
// pairs blockIdx.x, + gridDim.x, ...
// ---------------------------------------------------------------------------
constexpr int kW3Tap = kC2 * kC3 * 2, kW3Stages = 5;
constexpr int kConv3Threads = 128 + 8 * 32;
constexpr int pair_box(int channels) { return 10 * 2 * (channels / 8) * 160; }
template <int CK>
constexpr int conv3_stages() { return CK == kC2 ? 3 : 2; }
template <int CK, class Epi>
constexpr int conv3_smem() {
  return kW3Stages * kW3Tap + conv3_stages<CK>() * pair_box(CK) + Epi::kStage + 128 + 256;
}

// Whether `ok` holds for all eight epilogue warps; a barrier among them.
__device__ __forceinline__ bool epilogue_vote(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(ok))
      : "memory");
  return r != 0;
}

template <int CK, int N, class Epi>
__global__ void __launch_bounds__(kConv3Threads, 1)
    cnn_conv3_kernel(const __grid_constant__ CUtensorMap map, const bf16* wts, int chains, int n,
                     int* status, const __grid_constant__ Epi epi) {
  constexpr bool kFwd = N == kC3;
  constexpr int kBox = pair_box(CK), kRow = (CK / 8) * 160, kStages = conv3_stages<CK>();
  constexpr uint32_t kCols = 2 * N;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* w_s = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* ring = w_s + kW3Stages * kW3Tap;
  uint8_t* stage = ring + kStages * kBox;
  uint64_t* full = reinterpret_cast<uint64_t*>(stage + Epi::kStage);
  uint64_t* empty = full + kStages;
  uint64_t* wfull = empty + kStages;
  uint64_t* wempty = wfull + kW3Stages;
  uint64_t* tfull = wempty + kW3Stages;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    for (int i = 0; i < kW3Stages; ++i) {
      mbar_init(wfull + i, 1);
      mbar_init(wempty + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tfull + i, 1);
      mbar_init(tempty + i, 8);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, kCols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int pairs = chains * (n / 2), per = n / 2;

  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t it = 0;
      for (int p = blockIdx.x; p < pairs; p += gridDim.x, ++it) {
        const int s = it % kStages;
        if (!conv_wait(empty + s, ((it / kStages) & 1u) ^ 1u, abort_flag, status)) break;
        mbar_arrive_expect_tx(full + s, kBox);
        tc::tma_load_4d(ring + s * kBox, &map, -8, 0, -1, p, full + s);
      }
      if (*abort_flag)   // copies in flight land before the CTA ends
        for (uint32_t i = it > kStages ? it - kStages : 0; i < it; ++i)
          mbar_wait_bounded(full + i % kStages, (i / kStages) & 1u, nullptr);
    }
  } else if (warp == 2) {
    if (tc::elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int p = blockIdx.x; ok && p < pairs; p += gridDim.x) {
        const bf16* src = wts + static_cast<int64_t>(p / per) * kK3 * kC3;
        for (int tap = 0; tap < 9; ++tap, ++it) {
          const int s = it % kW3Stages;
          ok = conv_wait(wempty + s, ((it / kW3Stages) & 1u) ^ 1u, abort_flag, status);
          if (!ok) break;
          mbar_arrive_expect_tx(wfull + s, kW3Tap);
          bulk_g2s(w_s + s * kW3Tap, src + tap * kC2 * kC3, kW3Tap, wfull + s);
        }
      }
      if (*abort_flag)
        for (uint32_t i = it > kW3Stages ? it - kW3Stages : 0; i < it; ++i)
          mbar_wait_bounded(wfull + i % kW3Stages, (i / kW3Stages) & 1u, nullptr);
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(128, N, false, kFwd);
      uint32_t it = 0, wt = 0;
      bool ok = true;
      for (int p = blockIdx.x; ok && p < pairs; p += gridDim.x, ++it) {
        const int s = it % kStages;
        const uint32_t buf = it & 1u;
        if (!conv_wait(tempty + buf, ((it >> 1) & 1u) ^ 1u, abort_flag, status) ||
            !conv_wait(full + s, (it / kStages) & 1u, abort_flag, status))
          break;
        const uint64_t A = tc::sdesc_none(ring + s * kBox, 160, kRow);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap, ++wt) {
          const int ws = wt % kW3Stages;
          ok = ok && conv_wait(wfull + ws, (wt / kW3Stages) & 1u, abort_flag, status);
          if (!ok) break;
          tc::fence_after_sync();
          const uint64_t B = kFwd ? tc::sdesc_none(w_s + ws * kW3Tap, 128, 1024)
                                  : tc::sdesc_none(w_s + ws * kW3Tap, 1024, 128);
          const int kh = kFwd ? tap / 3 : 2 - tap / 3, kw = kFwd ? tap % 3 : 2 - tap % 3;
#pragma unroll
          for (int k = 0; k < CK / 16; ++k)
            tc::mma_bf16(tmem + buf * N, A + (2 * kh * kRow + kw * 16 + k * 320) / 16,
                         B + k * (kFwd ? 16 : 128), idesc, (tap | k) != 0);
          tc::mma_commit(wempty + ws);
        }
        tc::mma_commit(empty + s);
        if (ok) tc::mma_commit(tfull + buf);
      }
      tc::mma_commit(drain);   // every MMA of this CTA has completed once it flips
      mbar_wait_bounded(drain, 0, nullptr);
    }
  } else if (warp >= 4) {
    const int q = warp & 3, half = (warp - 4) >> 2;
    uint32_t it = 0;
    for (int p = blockIdx.x; p < pairs; p += gridDim.x, ++it) {
      const uint32_t buf = it & 1u;
      // The eight warps leave together: the epilogue synchronises them.
      if (!epilogue_vote(conv_wait(tfull + buf, (it >> 1) & 1u, abort_flag, status))) break;
      tc::fence_after_sync();
      const tc::TmemRows load{tmem + buf * N + half * (N / 2) +
                              (static_cast<uint32_t>(q * 32) << 16)};
      epi.tile(p, p / per, q, half, load, stage);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty + buf);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kCols);
  }
}

// conv3's pooling: lane 16 i + 8 m + x of quarter q is the pixel (2 q + i, x)
// of the pair's image m.
struct EpiPairPool {
  static constexpr int kStage = 0;
  const float* w;
  bf16* P;      // [images, 4, 4, 128]
  uint8_t* M;
  template <class Load>
  __device__ __forceinline__ void tile(int pair, int c, int q, int half, const Load& load,
                                       uint8_t*) const {
    const int lane = epi::lane_id();
    const int64_t pix = (2 * static_cast<int64_t>(pair) + ((lane >> 3) & 1)) * 16 + 4 * q +
                        ((lane & 7) >> 1);
#pragma unroll 1
    for (int cb = 0; cb < 2; ++cb) {
      const int col0 = 64 * half + 32 * cb;
      const float bl = __ldg(w + static_cast<int64_t>(c) * kP + ob3 + col0 + lane);
      float v[32];
      load(cb, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j] + __shfl_sync(0xffffffffu, bl, j), 0.f);
      uint4 p;
      uint2 m;
      const int wp = pool_windows<16>(v, p, m);
      const int64_t at = pix * kC3 + col0 + 8 * wp;
      *reinterpret_cast<uint4*>(P + at) = p;
      *reinterpret_cast<uint2*>(M + at) = m;
    }
  }
};

// dP2 never leaves the chip: a lane routes its pooled pixel's 32 channels into
// dY2 [image][h][octet][w][8], and db2's partials add the routed values of 32
// pooled pixels (half an image) in order.
struct EpiPairRoute {
  static constexpr int kLd = kC2 + 1, kStage = 128 * kLd * 4;
  const uint8_t* M;
  bf16* dy;
  float* bpart;   // [chain, blocks, 64], block 2 (image of the chain) + half
  template <class Load>
  __device__ __forceinline__ void tile(int pair, int, int q, int half, const Load& load,
                                       uint8_t* stage) const {
    float* st = reinterpret_cast<float*>(stage);
    const int lane = epi::lane_id(), x = lane & 7, im = (lane >> 3) & 1, h = 2 * q + (lane >> 4);
    const int64_t img = 2 * static_cast<int64_t>(pair) + im;
    const uint2* mk = reinterpret_cast<const uint2*>(M + (img * 64 + h * 8 + x) * kC2) + 4 * half;
    uint2 mark[4];
#pragma unroll
    for (int o = 0; o < 4; ++o) mark[o] = __ldg(mk + o);
    float v[32];
    load(0, v);
    float* mine = st + (64 * im + 8 * h + x) * kLd + 32 * half;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      float g[8], val[8];
      uint32_t w[4][4];
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] = v[8 * o + e];
      route_octet(g, mark[o], w, val);
#pragma unroll
      for (int e = 0; e < 8; ++e) mine[8 * o + e] = val[e];
      bf16* at = dy + ((img * 16 + 2 * h) * 8 + 4 * half + o) * 128 + 16 * x;
      store_sector(at, w[0], w[1]);
      store_sector(at + 8 * 128, w[2], w[3]);
    }
    epilogue_vote(true);
    const int t = threadIdx.x - 128, col = t & 63, blk = t >> 6;
    float sum = 0.f;
#pragma unroll 8
    for (int u = 0; u < 32; ++u) sum += st[(32 * blk + u) * kLd + col];
    bpart[(4 * static_cast<int64_t>(pair) + blk) * kC2 + col] = sum;
  }   // the next tile's vote comes before anything is written here again
};

// dW3 = dY3^T Col3: per image the boxes of dY3 and of P2 with its halo, two
// image rows (16 pixels) as K; M = 128 outputs.  A CTA takes a split and one of
// Z = 3 column shifts, N = 192 (three kernel rows x 64 inputs, words 160 bytes
// apart), or of Z = 9 taps, N = 64; it writes a split-K partial [tap,
// input][output] of a run of a chain's images.
constexpr int kDy3Box = 8 * (kC3 / 8) * 128, kP2Box = 10 * (kC2 / 8) * 160;
constexpr int kDw3Stages = 3, kDw3Threads = 64 + 4 * 32;   // two CTAs an SM
constexpr int kDw3Smem = kDw3Stages * (kDy3Box + kP2Box) + 128 + 256;

__device__ __forceinline__ void conv3_dw(const CUtensorMap& mdy, const CUtensorMap& mp2,
                                         float* part, int n, int* status, uint8_t* smem_raw, int c,
                                         int split, int S, int z, int Z) {
  constexpr int kStage = kDy3Box + kP2Box, kRow = (kC2 / 8) * 160;
  uint8_t* ring = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + kDw3Stages * kStage);
  uint64_t* empty = full + kDw3Stages;
  uint64_t* done = empty + kDw3Stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool single = Z == 9;
  const uint32_t cols = single ? 64 : 256;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kDw3Stages; ++i) {
      mbar_init(full + i, 1);
      mbar_init(empty + i, 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, cols);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();
  const int each = n / S, u0 = c * n + each * split, u1 = u0 + each;   // images
  const int kw = z % 3, kh0 = single ? z / 3 : 0;
  if (warp == 0) {
    if (tc::elect_one()) {
      uint32_t it = 0;
      for (int u = u0; u < u1; ++u, ++it) {
        const int s = it % kDw3Stages;
        if (!conv_wait(empty + s, ((it / kDw3Stages) & 1u) ^ 1u, abort_flag, status)) break;
        uint8_t* dst = ring + s * kStage;
        mbar_arrive_expect_tx(full + s, kStage);
        tc::tma_load_4d(dst, &mdy, 0, (u & 1) * (kC3 / 8), 0, u >> 1, full + s);
        tc::tma_load_4d(dst + kDy3Box, &mp2, -8, (u & 1) * (kC2 / 8), -1, u >> 1, full + s);
      }
      if (*abort_flag)
        for (uint32_t i = it > kDw3Stages ? it - kDw3Stages : 0; i < it; ++i)
          mbar_wait_bounded(full + i % kDw3Stages, (i / kDw3Stages) & 1u, nullptr);
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      const uint32_t idesc = single ? tc::idesc_bf16_f32(128, 64, true, true)
                                    : tc::idesc_bf16_f32(128, 192, true, true);
      uint32_t it = 0;
      for (int u = u0; u < u1; ++u, ++it) {
        const int s = it % kDw3Stages;
        if (!conv_wait(full + s, (it / kDw3Stages) & 1u, abort_flag, status)) break;
        tc::fence_after_sync();
        const uint64_t A = tc::sdesc_none(ring + s * kStage, (kC3 / 8) * 128, 128);
        const uint64_t B = tc::sdesc_none(ring + s * kStage + kDy3Box, kRow, 160) +
                           (kh0 * kRow + kw * 16) / 16;
#pragma unroll
        for (int h = 0; h < 8; h += 2)
          tc::mma_bf16(tmem, A + h * (kC3 / 8) * 128 / 16, B + h * kRow / 16, idesc,
                       it > 0 || h > 0);
        tc::mma_commit(empty + s);
      }
      tc::mma_commit(done);
      mbar_wait_bounded(done, 0, nullptr);
    }
  } else if (warp < kDw3Threads / 32) {
    const bool ok = mbar_wait_bounded(done, 0, nullptr);
    if (!__all_sync(0xffffffffu, ok) && lane == 0) raise_status(status, GBSGMC_ERR_TIMEOUT);
    tc::fence_after_sync();
    const int q = warp & 3;
    float* dst = part + (static_cast<int64_t>(c) * S + split) * kK3 * kC3 + 32 * q + lane;
#pragma unroll 1
    for (int g = 0; g < (single ? 2 : 6); ++g) {   // kh, input half
      float v[32];
      tc::tmem_ld32(tmem + 32 * g + (static_cast<uint32_t>(q * 32) << 16), v);
      const int k0 = (3 * (kh0 + (g >> 1)) + kw) * kC2 + 32 * (g & 1);
#pragma unroll
      for (int j = 0; j < 32; ++j) dst[(k0 + j) * kC3] = v[j];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, cols);
  }
}

// The three weight gradients in one launch, two CTAs an SM: none depends on
// another, and their launches one after the other, each with a tail that
// leaves SMs idle and MMAs of small N that wait on the issue, took 279 us of a
// gradient of 8 x 256 images where the one launch leaves 266; with few images,
// where each is mostly latency, 4 chains of 50: 83 to 69, 2 of 256: 152 to 118,
// 2 of 2,048: 966 to 726.  Grid (parts, chains): a chain's splits of dW1 (the
// longest), then of dW2 by column shift, then of dW3 in z3 parts.
constexpr int kGradsSmem = std::max({kUnitSmem, kDw2Smem, kDw3Smem});

__global__ void __launch_bounds__(kUnitThreads, 2)
    cnn_weight_grads_kernel(const __grid_constant__ CnnArgs a, int pair,
                            const __grid_constant__ CUtensorMap mdy2,
                            const __grid_constant__ CUtensorMap mp1,
                            const __grid_constant__ CUtensorMap mdy3,
                            const __grid_constant__ CUtensorMap mp2, int z3) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int c = blockIdx.y, S1 = a.split[0], S2 = a.split[1], S3 = a.split[2];
  int b = blockIdx.x;
  if (b < S1) return conv1_grad(a, pair, smem_raw, c, b, S1);
  b -= S1;
  if (b < 3 * S2)
    return conv2_dw(mdy2, mp1, a.part[1], a.n, a.status, smem_raw, c, b % S2, S2, b / S2);
  b -= 3 * S2;
  conv3_dw(mdy3, mp2, a.part[2], a.n, a.status, smem_raw, c, b % S3, S3, b / S3, z3);
}

// Parts of a split of dW3: a tap each while all CTAs of the launch run at once
// (4 chains of 50 images 71 to 69 us), else a column shift each, which reads
// dY3 a third as often (8 of 256: 281 and 266 us).
int dw3_parts(const CnnArgs& a, int sms) {
  return a.chains * (a.split[0] + 3 * a.split[1] + 9 * a.split[2]) <= 2 * sms ? 9 : 3;
}

// ---------------------------------------------------------------------------
// Dense layer, softmax likelihood and its adjoint for kImgs images of a chain
// per block.  Writes lk, dlogits g = dU/dlogits (fp32), dP3 = g Wd^T and the
// per-image likelihood terms.  Grid (ceil(n / kImgs), chains), 80 threads per
// kPer images: thread (class pair p, images j, slice s) handles the features
// f = s, s + 16, ... of two classes; the 16 threads of a pair are one
// half-warp and reduce by shuffles.  The block first copies Wd (80 KB) and its
// images' P3 rows (4 KB each) into shared memory with all loads in flight: a
// half-warp then reads 8 bytes of 16 Wd rows 40 bytes apart, 32 distinct banks,
// and 16 consecutive P3 features of each image.  Shared memory's words are the
// limit: kPer images share what is read of Wd.
// Few images leave most SMs without a block of 16, so blocks take 4 then, one
// a thread: what a block takes is the latency of its loads and of 128 steps.
// ---------------------------------------------------------------------------
static_assert(oWd % 2 == 0 && kP % 2 == 0, "Wd is copied as float2");
constexpr size_t dense_smem(int imgs) {
  return sizeof(float) * kFlat * kClasses + sizeof(bf16) * imgs * kFlat;
}

template <int kDenseImgs, int kPer>
__global__ void __launch_bounds__(kDenseImgs / kPer * 80)
    cnn_dense_kernel(const CnnArgs a, float scale) {
  pdl_trigger();
  pdl_wait();
  constexpr int kSets = kDenseImgs / kPer, kDenseThreads = kSets * 80;
  extern __shared__ __align__(16) float wd_s[];  // Wd [2048][10], then P3 rows [kDenseImgs][2048]
  bf16* x_s = reinterpret_cast<bf16*>(wd_s + kFlat * kClasses);
  __shared__ __align__(8) float g_s[kDenseImgs][kClasses];   // logits, then their adjoints
  const unsigned full = 0xffffffffu;
  const int c = blockIdx.y, t = threadIdx.x;
  const int part = t / (kSets * 16), set = (t >> 4) % kSets, sl = t & 15;
  const float* w = a.w + static_cast<int64_t>(c) * kP;
  {
    // oWd and kP are even: the chain's Wd starts 8-byte aligned.
    const float2* src = reinterpret_cast<const float2*>(w + oWd);
    float2* dst = reinterpret_cast<float2*>(wd_s);
    // The block's images, 16 bytes per load (rows past n are not read).
    const int i0 = blockIdx.x * kDenseImgs;
    const int rows = min(kDenseImgs, a.n - i0);
    const uint4* xs =
        reinterpret_cast<const uint4*>(a.p3 + (static_cast<int64_t>(c) * a.n + i0) * kFlat);
    uint4* xd = reinterpret_cast<uint4*>(x_s);
#pragma unroll 16
    for (int e = t; e < kFlat * kClasses / 2; e += kDenseThreads) dst[e] = __ldg(src + e);
#pragma unroll 4
    for (int e = t; e < kDenseImgs * kFlat / 8; e += kDenseThreads)
      if (e < rows * (kFlat / 8)) xd[e] = __ldg(xs + e);
  }
  __syncthreads();
  {
    const bf16* x = x_s + set * kPer * kFlat;
    float acc[kPer][2] = {};
#pragma unroll 8
    for (int f = sl; f < kFlat; f += 16) {
      const float2 wr = *reinterpret_cast<const float2*>(wd_s + f * kClasses + 2 * part);
#pragma unroll
      for (int r = 0; r < kPer; ++r) {   // rows past n are not set: their sums go nowhere
        const float xv = bf(x[r * kFlat + f]);
        acc[r][0] = fmaf(xv, wr.x, acc[r][0]);
        acc[r][1] = fmaf(xv, wr.y, acc[r][1]);
      }
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
          acc[r][k] += __shfl_xor_sync(full, acc[r][k], off);
        if (sl == 0)
          g_s[set * kPer + r][2 * part + k] = acc[r][k] + __ldg(w + obd + 2 * part + k);
      }
  }
  __syncthreads();
  const int j = t, i = blockIdx.x * kDenseImgs + j;
  if (j < kDenseImgs && i < a.n) {
    float logit[kClasses], mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < kClasses; ++k) {
      logit[k] = g_s[j][k];
      mx = fmaxf(mx, logit[k]);
    }
    float se = 0.f;
#pragma unroll
    for (int k = 0; k < kClasses; ++k) se += expf(logit[k] - mx);
    const float lse = mx + logf(se);
    const int lab = a.lab[static_cast<int64_t>(c) * a.n + i];
    const float lk = g_s[j][lab] - lse;
    const float m = a.mask != nullptr ? __ldg(a.mask + static_cast<int64_t>(c) * a.n + i) : 1.f;
#pragma unroll
    for (int k = 0; k < kClasses; ++k) {
      const float pk = expf(logit[k] - lse);
      const float g = -scale * m * ((k == lab ? 1.f : 0.f) - pk);
      g_s[j][k] = g;
      a.gl[(static_cast<int64_t>(c) * a.n + i) * kClasses + k] = g;
    }
    if (a.lk != nullptr) a.lk[static_cast<int64_t>(c) * a.n + i] = lk;
    double* pl = a.plk + (static_cast<int64_t>(c) * a.n + i) * 4;
    pl[0] = static_cast<double>(m) * lk;
    pl[1] = lk;
    pl[2] = static_cast<double>(lk) * lk;
    pl[3] = 0.0;
  }
  if (!a.want_grad) return;
  __syncthreads();
  // dP3 rows of the block's images, two features of a thread at a time.
  const int rows = min(kDenseImgs, a.n - static_cast<int>(blockIdx.x) * kDenseImgs);
  float* dx = a.dp3 + (static_cast<int64_t>(c) * a.n + blockIdx.x * kDenseImgs) * kFlat;
  for (int f0 = t; f0 < kFlat; f0 += 2 * kDenseThreads) {
    const int f1 = f0 + kDenseThreads < kFlat ? f0 + kDenseThreads : f0;
    float2 wr[2][kClasses / 2];
#pragma unroll
    for (int k = 0; k < kClasses / 2; ++k) {
      wr[0][k] = reinterpret_cast<const float2*>(wd_s + f0 * kClasses)[k];
      wr[1][k] = reinterpret_cast<const float2*>(wd_s + f1 * kClasses)[k];
    }
#pragma unroll 2
    for (int r = 0; r < rows; ++r) {
      const float2* g = reinterpret_cast<const float2*>(g_s[r]);
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int k = 0; k < kClasses / 2; ++k) {
        const float2 gv = g[k];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          sum[u] = fmaf(gv.x, wr[u][k].x, sum[u]);
          sum[u] = fmaf(gv.y, wr[u][k].y, sum[u]);
        }
      }
      dx[static_cast<int64_t>(r) * kFlat + f0] = sum[0];
      dx[static_cast<int64_t>(r) * kFlat + f1] = sum[1];
    }
  }
}

// What depends on the dense layer's adjoint alone, in one launch.  Blocks
// 0 .. kFlat / 128: dWd [2048, 10] = sum_i P3_i (x) g_i and dbd = sum_i g_i
// (likelihood part); feature f = 128 x + t % 128, image group q = t / 128 adds
// the images i = q (mod 4) in order; the four partial sums are added in group
// order; dlogits are staged in shared memory 512 images at a time.  The other
// blocks: the routing of dP3 into dY3 [pair][h][image of the pair][octet][w]
// [8], a thread per pooled pixel and octet, 256 threads (16 pooled pixels, an
// image) of a block for each partial of db3: the routed (BF16-rounded) values
// of a channel, added in order.  Grid (kFlat / 128 + 1 + n / 2, chains).
constexpr int kDenseGradBlocks = kFlat / 128 + 1;

__global__ void __launch_bounds__(512) cnn_dense_grad_kernel(const CnnArgs a) {
  pdl_trigger();
  pdl_wait();
  __shared__ __align__(16) float smem[512 * kClasses + 3 * 128 * kClasses];
  const int c = blockIdx.y, t = threadIdx.x;
  if (blockIdx.x >= kDenseGradBlocks) {
    float* red = smem + (t >> 8) * 2048;
    const int i = 2 * (blockIdx.x - kDenseGradBlocks) + (t >> 8), tt = t & 255;
    const int px = tt & 3, oct = (tt >> 2) & 15, py = tt >> 6;
    const int in = (4 * py + px) * kC3 + 8 * oct;
    const int64_t img = static_cast<int64_t>(c) * a.n + i, at = img * kFlat + in;
    const float4* d = reinterpret_cast<const float4*>(a.dp3 + at);
    const float4 u = __ldg(d), v = __ldg(d + 1);
    const float g[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    uint32_t o[4][4];
    float val[8];
    route_octet(g, __ldg(reinterpret_cast<const uint2*>(a.m3 + at)), o, val);
    bf16* dst = a.dy3 + ((((img >> 1) * 8 + 2 * py) * 2 + (img & 1)) * 16 + oct) * 64 + 16 * px;
    store_sector(dst, o[0], o[1]);
    store_sector(dst + 2 * 16 * 64, o[2], o[3]);
#pragma unroll
    for (int e = 0; e < 8; ++e) red[in + e] = val[e];
    __syncthreads();
    if (tt < kC3) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 16; ++w) s += red[w * kC3 + tt];
      a.bpart[2][img * kC3 + tt] = s;
    }
    return;
  }
  float* gs = smem;
  float(*red)[128 * kClasses] = reinterpret_cast<float(*)[128 * kClasses]>(smem + 512 * kClasses);
  const int q = t >> 7;
  float* g = a.grad + static_cast<int64_t>(c) * kP;
  const float* gl = a.gl + static_cast<int64_t>(c) * a.n * kClasses;
  if (blockIdx.x == kFlat / 128) {
    float s = 0.f;
    for (int i0 = 0; i0 < a.n; i0 += 512) {
      const int cnt = min(512, a.n - i0);
      __syncthreads();
      for (int e = t; e < cnt * kClasses; e += 512) gs[e] = gl[i0 * kClasses + e];
      __syncthreads();
      if (t < kClasses) {
#pragma unroll 16
        for (int i = 0; i < cnt; ++i) s += gs[i * kClasses + t];
      }
    }
    if (t < kClasses) g[obd + t] = s;
    return;
  }
  const int f = blockIdx.x * 128 + (t & 127);
  const bf16* x = a.p3 + static_cast<int64_t>(c) * a.n * kFlat + f;
  float acc[kClasses];
#pragma unroll
  for (int k = 0; k < kClasses; ++k) acc[k] = 0.f;
  for (int i0 = 0; i0 < a.n; i0 += 512) {
    const int cnt = min(512, a.n - i0);
    __syncthreads();
    for (int e = t; e < cnt * kClasses; e += 512) gs[e] = gl[i0 * kClasses + e];
    __syncthreads();
    int i = q;
    for (; i + 28 < cnt; i += 32) {
      float xv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) xv[u] = bf(x[static_cast<int64_t>(i0 + i + 4 * u) * kFlat]);
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int k = 0; k < kClasses; k += 2) {   // rows of 40 bytes
          const float2 gv = *reinterpret_cast<const float2*>(gs + (i + 4 * u) * kClasses + k);
          acc[k] = fmaf(xv[u], gv.x, acc[k]);
          acc[k + 1] = fmaf(xv[u], gv.y, acc[k + 1]);
        }
    }
    for (; i < cnt; i += 4) {
      const float xv = bf(x[static_cast<int64_t>(i0 + i) * kFlat]);
#pragma unroll
      for (int k = 0; k < kClasses; ++k) acc[k] = fmaf(xv, gs[i * kClasses + k], acc[k]);
    }
  }
  if (q > 0) {
#pragma unroll
    for (int k = 0; k < kClasses; ++k) red[q - 1][(t & 127) * kClasses + k] = acc[k];
  }
  __syncthreads();
  if (q == 0) {
#pragma unroll
    for (int k = 0; k < kClasses; ++k) {
      float s = acc[k];
      for (int r = 0; r < 3; ++r) s += red[r][t * kClasses + k];
      g[oWd + static_cast<int64_t>(f) * kClasses + k] = s;
    }
  }
}

// What remains when the GEMMs are done, in one launch: the split-K partials of
// the three weight gradients and the unpool blocks' bias partials summed in a
// fixed order, the prior's w / (s^2 T) added to every parameter's gradient,
// U and var(lk).  (As seven launches, most of them a few microseconds of
// latency: 42 us of an 850 us gradient of 8 x 256 images, 26 us of 160 at 2 x
// 50.)  Grid (weight blocks + kBiasBlocks + 1, chains), 256 threads: the
// first ceil(P / 256) blocks take a parameter per thread, then four blocks a
// layer's bias (C / 4 channels each, 1024 / C groups of partials), the last
// block the values.
constexpr int kBiasBlocks = 12;

// Partials added in order, all loads in flight at once.
template <int S>
__device__ __forceinline__ float sum_splits(const float* p, int64_t count) {
  float x[S], v = 0.f;
#pragma unroll
  for (int q = 0; q < S; ++q) x[q] = __ldg(p + q * count);
#pragma unroll
  for (int q = 0; q < S; ++q) v += x[q];
  return v;
}

__global__ void __launch_bounds__(256) cnn_finalize_kernel(const CnnArgs a) {
  __shared__ float acc[256];
  __shared__ double red[4];
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.y, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const float* w = a.w + static_cast<int64_t>(c) * kP;
  const int weights = static_cast<int>(gridDim.x) - 1 - kBiasBlocks;
  const int bx = static_cast<int>(blockIdx.x) - weights;
  if (bx < 0) {
    const int64_t j = static_cast<int64_t>(blockIdx.x) * 256 + t;
    if (!a.want_grad || j >= kP) return;
    float* g = a.grad + static_cast<int64_t>(c) * kP + j;
    float v;
    if (j >= obd) {
      v = *g;   // the dense layer's, already in place
    } else {
      const int l = j >= ob3 ? 2 : (j >= ob2 ? 1 : 0);
      const int64_t off = l == 2 ? oW3 : (l == 1 ? oW2 : oW1);
      if (j < off) return;   // a bias
      const int64_t count = l == 2 ? kK3 * kC3 : (l == 1 ? kK2 * kC2 : kK1 * kC1);
      const float* p = a.part[l] + static_cast<int64_t>(c) * a.split[l] * count + (j - off);
      const int splits = a.split[l];
      v = splits == 32   ? sum_splits<32>(p, count)
          : splits == 16 ? sum_splits<16>(p, count)
          : splits == 8  ? sum_splits<8>(p, count)
          : splits == 4  ? sum_splits<4>(p, count)
                         : sum_splits<2>(p, count);
    }
    *g = a.pf != 0.f ? fmaf(a.pf, __ldg(w + j), v) : v;
    return;
  }
  if (bx < kBiasBlocks) {
    if (!a.want_grad) return;
    const int l = bx >> 2, C = l == 2 ? kC3 : (l == 1 ? kC2 : kC1);
    const int64_t off = l == 2 ? ob3 : (l == 1 ? ob2 : ob1);
    const int own = C / 4, groups = 256 / own, blocks = a.bblocks[l];
    const int ch = (bx & 3) * own + t % own;
    const float* p = a.bpart[l] + static_cast<int64_t>(c) * blocks * C + ch;
    float v = 0.f;
#pragma unroll 8
    for (int q = t / own; q < blocks; q += groups) v += p[static_cast<int64_t>(q) * C];
    acc[t] = v;
    __syncthreads();
    if (t < own) {
      float tot = 0.f;
      for (int u = 0; u < groups; ++u) tot += acc[u * own + t];
      const int64_t j = off + ch;
      a.grad[static_cast<int64_t>(c) * kP + j] =
          a.pf != 0.f ? fmaf(a.pf, __ldg(w + j), tot) : tot;
    }
    return;
  }
  // The chain's values: four FP64 sums, a warp each.
  if (warp < 4) {
    double v = 0.0;
    if (warp == 0) {
      for (int i = lane; i < kPrepBlocks; i += 32) v += a.psq[c * kPrepBlocks + i];
    } else {
      const double* p = a.plk + static_cast<int64_t>(c) * a.n * 4 + (warp - 1);
      for (int i = lane; i < a.n; i += 32) v += p[4 * static_cast<int64_t>(i)];
    }
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
  }
  __syncthreads();
  if (t != 0) return;
  const double sq = red[0], lm = red[1], l1 = red[2], l2 = red[3];
  double log_prior = 0.0;
  if (a.prior_scale > 0.f) {
    const double s2 = static_cast<double>(a.prior_scale) * a.prior_scale;
    log_prior = -0.5 * sq / s2 - a.prior_const;
  }
  const double U = (-static_cast<double>(a.n_obs) * (lm / a.n) - log_prior) / a.temperature;
  a.U[c] = U;
  if (a.lk_var != nullptr) {
    const double mean = l1 / a.n;
    a.lk_var[c] = fmax(l2 / a.n - mean * mean, 0.0);
  }
  if (!isfinite(U)) raise_status(a.status, GBSGMC_ERR_NONFINITE);
}

template <class T>
T* view(void* ws, size_t off) {
  return reinterpret_cast<T*>(static_cast<unsigned char*>(ws) + off);
}

int grid1(int64_t work) { return static_cast<int>((work + 255) / 256); }

int run_cnn(CnnArgs& a, const CnnLayout& L, void* ws, cudaStream_t st) {
  a.w2b = view<bf16>(ws, L.w2b);
  a.w3b = view<bf16>(ws, L.w3b);
  a.p1 = view<bf16>(ws, L.p1);
  a.dy2 = view<bf16>(ws, L.dy2);
  a.p2 = view<bf16>(ws, L.p2);
  a.dy3 = view<bf16>(ws, L.dy3);
  a.p3 = view<bf16>(ws, L.p3);
  a.m1 = view<uint8_t>(ws, L.m1);
  a.m2 = view<uint8_t>(ws, L.m2);
  a.m3 = view<uint8_t>(ws, L.m3);
  a.dp1 = view<float>(ws, L.dp1);
  a.lab = view<int32_t>(ws, L.labels);
  a.dp3 = view<float>(ws, L.dp3);
  a.gl = view<float>(ws, L.gl);
  a.psq = view<double>(ws, L.psq);
  a.plk = view<double>(ws, L.plk);
  const int C = a.chains, n = a.n;
  const int sizes[3] = {32, 16, 8}, couts[3] = {kC1, kC2, kC3};
  for (int l = 0; l < 3; ++l) {
    a.part[l] = view<float>(ws, L.part[l]);
    a.bpart[l] = view<float>(ws, L.bpart[l]);
    a.split[l] = wsplit(l + 1, n);
    a.bblocks[l] = grid1(int64_t(n) * (sizes[l] / 2) * (sizes[l] / 2) * couts[l] / 8);
  }
  a.pf = 0.f;
  a.prior_const = 0.0;
  if (a.prior_scale > 0.f) {
    const double ps = a.prior_scale;
    a.pf = static_cast<float>(1.0 / (ps * ps * a.temperature));
    a.prior_const = static_cast<double>(kP) * (std::log(ps) + 0.91893853320467274178);
  }
  int rc;
  auto launched = [&](const char* what) { return check_launch(what); };
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return set_error(GBSGMC_ERR_CUDA, "cnn: cannot query the device");
  const int pair = reinterpret_cast<uintptr_t>(a.X) % 8 == 0 && a.ld % 2 == 0;
  launch_pdl(cnn_conv1_kernel,
             static_cast<int>(std::min<int64_t>(
                 4 * sms, 2 * int64_t(C) * n + int64_t(C) * kPrepBlocks)),
             kStripThreads, 0, st, a, pair);
  if ((rc = launched("cnn_conv1_kernel"))) return rc;

  // 4-D maps of the octet layouts, with the boxes that the kernels take.
  const int64_t imgs = int64_t(C) * n, pairs = imgs / 2;
  CUtensorMap m_p1, m_p2;
  if ((rc = make_tmap_bf16_4d_plain(&m_p1, a.p1, {128, kC1 / 8, 16, imgs},
                                    {128, 16 * kC1, 256 * kC1}, {80, kC1 / 8, 18, 1})) ||
      (rc = make_tmap_bf16_4d_plain(&m_p2, a.p2, {64, kC2 / 4, 8, pairs},
                                    {64, 16 * kC2, 128 * kC2}, {80, kC2 / 4, 10, 1})))
    return rc;

  // conv1+pool1 -> conv2+pool2 -> conv3+pool3: each epilogue writes the pooled
  // BF16 map and the marks.
  const auto conv2 = [&](auto kern, int bytes, const CUtensorMap& map, const auto& epi) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "cnn_conv2_kernel: %s", cudaGetErrorString(e));
    launch_pdl(kern, static_cast<int>(std::min<int64_t>(2 * sms, 2 * imgs)), kConvThreads, bytes,
               st, map, static_cast<const bf16*>(a.w2b), C, n, a.status, epi);
    return launched("cnn_conv2_kernel");
  };
  if ((rc = conv2(cnn_conv2_kernel<kC1, kC2, EpiStripPool>, conv_smem<kC1>(), m_p1,
                  EpiStripPool{a.w, a.p2, a.m2})))
    return rc;
  const auto conv3 = [&](auto kern, int bytes, const CUtensorMap& map, const auto& epi) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "cnn_conv3_kernel: %s", cudaGetErrorString(e));
    launch_pdl(kern, static_cast<int>(std::min<int64_t>(sms, pairs)), kConv3Threads, bytes, st,
               map, static_cast<const bf16*>(a.w3b), C, n, a.status, epi);
    return launched("cnn_conv3_kernel");
  };
  if ((rc = conv3(cnn_conv3_kernel<kC2, kC3, EpiPairPool>, conv3_smem<kC2, EpiPairPool>(), m_p2,
                  EpiPairPool{a.w, a.p3, a.m3})))
    return rc;
  const auto dense = [&](auto kern, int imgs, int per) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(dense_smem(imgs)));
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "cnn_dense_kernel: %s", cudaGetErrorString(e));
    const float scale = static_cast<float>(static_cast<double>(a.n_obs) / n / a.temperature);
    launch_pdl(kern, dim3(ceil_div(n, imgs), C), imgs / per * 80, dense_smem(imgs), st, a, scale);
    return launched("cnn_dense_kernel");
  };
  // Sixteen images share a block's copy of Wd once that fills the SMs.
  rc = int64_t(C) * n >= 16 * (sms / 2) ? dense(cnn_dense_kernel<16, 2>, 16, 2)
                                        : dense(cnn_dense_kernel<4, 1>, 4, 1);
  if (rc) return rc;

  if (a.want_grad) {
    // dWd, dbd; layer 3: dY3 (routing of dP3) and db3.
    launch_pdl(cnn_dense_grad_kernel, dim3(kDenseGradBlocks + n / 2, C), 512, 0, st, a);
    if ((rc = launched("cnn_dense_grad_kernel"))) return rc;
    // Layer 3: dP2, the transposed convolution of dY3, routed into dY2, and db2.
    CUtensorMap m_dy3, m_dy3h, m_p2w;
    if ((rc = make_tmap_bf16_4d_plain(&m_dy3, a.dy3, {64, kC3 / 4, 8, pairs},
                                      {64, 16 * kC3, 128 * kC3}, {64, kC3 / 8, 8, 1})) ||
        (rc = make_tmap_bf16_4d_plain(&m_p2w, a.p2, {64, kC2 / 4, 8, pairs},
                                      {64, 16 * kC2, 128 * kC2}, {80, kC2 / 8, 10, 1})) ||
        (rc = make_tmap_bf16_4d_plain(&m_dy3h, a.dy3, {64, kC3 / 4, 8, pairs},
                                      {64, 16 * kC3, 128 * kC3}, {80, kC3 / 4, 10, 1})))
      return rc;
    if ((rc = conv3(cnn_conv3_kernel<kC3, kC2, EpiPairRoute>, conv3_smem<kC3, EpiPairRoute>(),
                    m_dy3h, EpiPairRoute{a.m2, a.dy2, a.bpart[1]})))
      return rc;
    // Layer 2: dP1, the transposed convolution of dY2.
    CUtensorMap m_dy2, m_dy2h, m_p1w;
    if ((rc = make_tmap_bf16_4d_plain(&m_dy2, a.dy2, {128, kC2 / 8, 16, imgs},
                                      {128, 16 * kC2, 256 * kC2}, {128, kC2 / 8, 4, 1})) ||
        (rc = make_tmap_bf16_4d_plain(&m_p1w, a.p1, {128, kC1 / 8, 16, imgs},
                                      {128, 16 * kC1, 256 * kC1}, {144, kC1 / 8, 6, 1})) ||
        (rc = make_tmap_bf16_4d_plain(&m_dy2h, a.dy2, {128, kC2 / 8, 16, imgs},
                                      {128, 16 * kC2, 256 * kC2}, {80, kC2 / 8, 18, 1})))
      return rc;
    if ((rc = conv2(cnn_conv2_kernel<kC2, kC1, EpiStripDX>, conv_smem<kC2>(), m_dy2h,
                    EpiStripDX{a.dp1})))
      return rc;
    // Routing of dP1 and db1; all dW.
    const cudaError_t e = cudaFuncSetAttribute(
        cnn_weight_grads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradsSmem);
    if (e != cudaSuccess)
      return set_error(GBSGMC_ERR_CUDA, "cnn_weight_grads_kernel: %s", cudaGetErrorString(e));
    const int z3 = dw3_parts(a, sms);
    launch_pdl(cnn_weight_grads_kernel, dim3(a.split[0] + 3 * a.split[1] + z3 * a.split[2], C),
               kUnitThreads, kGradsSmem, st, a, pair, m_dy2, m_p1w, m_dy3, m_p2w, z3);
    if ((rc = launched("cnn_weight_grads_kernel"))) return rc;
  }

  launch_pdl(cnn_finalize_kernel, dim3((a.want_grad ? grid1(kP) : 0) + kBiasBlocks + 1, C), 256, 0,
             st, a);
  return launched("cnn_finalize_kernel");
}

}  // namespace
}  // namespace gbsgmc

using namespace gbsgmc;

extern "C" int64_t gbsgmc_cnn_param_count(void) { return kP; }

extern "C" size_t gbsgmc_cnn_workspace_bytes(int chains, int n) {
  if (chains <= 0 || n <= 0 || n % 2 != 0) return 0;
  return cnn_layout(chains, n).total;
}

extern "C" int gbsgmc_cnn_value_and_grad(const gbsgmc_cnn* model, int chains, int n,
                                         const int32_t* idx_dev, int64_t idx_stride,
                                         const float* mask_dev, const float* w_dev,
                                         double* U_dev, float* grad_dev, float* lk_dev,
                                         double* lk_var_dev, void* workspace_dev,
                                         size_t workspace_bytes, int* status_dev,
                                         gbsgmc_stream_t stream) {
  if (model == nullptr || model->X == nullptr || model->labels == nullptr)
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: null model or data");
  if (chains < 0 || n < 0) return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: negative size");
  if (chains == 0) return GBSGMC_OK;
  if (n == 0 || n % 2 != 0 || chains > 65535 || n > 65536)
    return set_error(GBSGMC_ERR_SHAPE,
                     "cnn_value_and_grad: n must be a positive even number (got %d)", n);
  if (model->ld < kImg * kImg * kInC || model->label_ld < 1 || model->n_obs < 1 ||
      model->n_rows < 0 || model->n_rows >= (1ll << 31))
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: bad strides or sizes");
  if (!(model->temperature > 0.f) || !(model->prior_scale >= 0.f))
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: bad temperature or prior scale");
  if (idx_dev == nullptr || w_dev == nullptr || U_dev == nullptr || workspace_dev == nullptr ||
      status_dev == nullptr)
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: null pointer");
  if (idx_stride < n) return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: idx_stride < n");
  if (reinterpret_cast<uintptr_t>(workspace_dev) % 256 != 0)
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: workspace must be 256-byte aligned");
  const CnnLayout L = cnn_layout(chains, n);
  if (workspace_bytes < L.total)
    return set_error(GBSGMC_ERR_ARG, "cnn_value_and_grad: workspace of %zu bytes, need %zu",
                     workspace_bytes, L.total);
  CnnArgs a{};
  a.chains = chains;
  a.n = n;
  a.want_grad = grad_dev != nullptr;
  a.n_obs = model->n_obs;
  a.n_rows = model->n_rows > 0 ? model->n_rows : model->n_obs;
  a.ld = model->ld;
  a.X = model->X;
  a.labels = model->labels;
  a.label_ld = model->label_ld;
  a.mask = mask_dev;
  a.idx = idx_dev;
  a.idx_stride = idx_stride;
  a.w = w_dev;
  a.prior_scale = model->prior_scale;
  a.temperature = model->temperature;
  a.U = U_dev;
  a.grad = grad_dev;
  a.lk = lk_dev;
  a.lk_var = lk_var_dev;
  a.status = status_dev;
  return run_cnn(a, L, workspace_dev, static_cast<cudaStream_t>(stream));
}
