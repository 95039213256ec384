// Per-node MLP kernels (see eb_mlp.cuh) and the C-ABI training/evaluation
// entry points.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

#include "../../include/endobeams_gb300.h"
#include "eb_internal.cuh"
#include "eb_mlp.cuh"

int eb_internal_fail(int code, const char* msg);

namespace eb {
namespace {

constexpr int kThr = 256;      // threads per CTA
constexpr int kWarps = kThr / 32;
constexpr int kOutP = 8;       // padded output width
constexpr int kRows = 32;      // rows of a tile: a gradient partial's unit, whatever the launch
// Shared arrays of rows hold pairs of consecutive rows: entry k of pair p is the float2 at p ld + k.
constexpr int kLdX = 52, kLdH = 132;   // ld of the inputs and of the hidden activations (float2)
constexpr int kLdW2 = 132;             // row stride of W2 and of W3 transposed (BF16 values)

static_assert(kMlpIn == 48 && kMlpHidden == 128 && kMlpOut == 6, "kernel tiling assumes 48-128-128-6");

// A warp owns NP row pairs: 1 (16 rows a CTA), 2 (a tile) or 4 (two tiles).  FP32 arithmetic on CUDA
// cores bounds a tile (63,700 FMAs per row forward and backward), so the products are packed two to
// an instruction, both halves the same product of two rows, and every shared-memory operand feeds at
// least four of them.
template <int NP>
struct Smem {
  __nv_bfloat16 W1[kMlpIn * kMlpHidden];
  __nv_bfloat16 W2[kMlpHidden * kLdW2];
  __nv_bfloat16 W3T[kOutP * kLdW2];
  float b1[kMlpHidden], b2[kMlpHidden], b3[kOutP];
  float2 x[kWarps * NP * kLdX];
  // hidden activations and the derivatives of silu there, later the gradients by z (in place)
  float2 h1[kWarps * NP * kLdH], d1[kWarps * NP * kLdH], h2[kWarps * NP * kLdH], d2[kWarps * NP * kLdH];
  float2 dy[kWarps * NP * kOutP];  // targets, then the gradient by y
  double red[kWarps];
};

__device__ __forceinline__ float sigm(float z) { return 1.f / (1.f + expf(-z)); }

// d = a b + d on both halves, each rounded as fmaf does
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 both_lo(unsigned w) { return both(__uint_as_float(w << 16)); }
__device__ __forceinline__ float2 both_hi(unsigned w) { return both(__uint_as_float(w & 0xffff0000u)); }

// Row pair q of this warp (NP of them); pairs 16 .. are the second tile's.
template <int NP>
__device__ __forceinline__ int pair_of(int q) {
  const int warp = threadIdx.x >> 5;
  return NP == 1 ? warp : 2 * warp + (q & 1) + kRows / 2 * (q >> 1);
}

// acc[q][c] += Σ_k in[row][k] W[k][4 lane + c] for the warp's first CNT row pairs, k in increasing
// order in one chain per output.
template <int NP, int CNT, int K, int LDI, int LDW>
__device__ __forceinline__ void dot_rows(const float2* in, const __nv_bfloat16* W, float2 (&acc)[CNT][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 2
  for (int k = 0; k < K; k += 2) {
    const uint2 w0 = *reinterpret_cast<const uint2*>(W + k * LDW + 4 * lane);
    const uint2 w1 = *reinterpret_cast<const uint2*>(W + (k + 1) * LDW + 4 * lane);
    const float2 a[4] = {both_lo(w0.x), both_hi(w0.x), both_lo(w0.y), both_hi(w0.y)};
    const float2 b[4] = {both_lo(w1.x), both_hi(w1.x), both_lo(w1.y), both_hi(w1.y)};
#pragma unroll
    for (int q = 0; q < CNT; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(in + pair_of<NP>(q) * LDI + k);
#pragma unroll
      for (int c = 0; c < 4; ++c) fma2(acc[q][c], make_float2(v.x, v.y), a[c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) fma2(acc[q][c], make_float2(v.z, v.w), b[c]);
    }
  }
}

// acc[q][c] += Σ_j in[row][j] W2[lane + 32 c][j], j in increasing order.
template <int NP, int CNT>
__device__ __forceinline__ void dot_cols(const float2* in, const __nv_bfloat16* W, float2 (&acc)[CNT][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int j = 0; j < kMlpHidden; j += 4) {
    uint2 w[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) w[c] = *reinterpret_cast<const uint2*>(W + (lane + 32 * c) * kLdW2 + j);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 a[4], b[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const unsigned u = h ? w[c].y : w[c].x;
        a[c] = both_lo(u);
        b[c] = both_hi(u);
      }
#pragma unroll
      for (int q = 0; q < CNT; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(in + pair_of<NP>(q) * kLdH + j + 2 * h);
#pragma unroll
        for (int c = 0; c < 4; ++c) fma2(acc[q][c], make_float2(v.x, v.y), a[c]);
#pragma unroll
        for (int c = 0; c < 4; ++c) fma2(acc[q][c], make_float2(v.z, v.w), b[c]);
      }
    }
  }
}

// h = silu(in W + b) of the warp's first CNT row pairs, and silu' (TRAIN).
template <bool TRAIN, int NP, int CNT, int K, int LDI, int LDW>
__device__ __forceinline__ void dense_silu(const float2* in, const __nv_bfloat16* W, const float* b, float2* h, float2* d) {
  const int lane = threadIdx.x & 31;
  float2 acc[CNT][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int q = 0; q < CNT; ++q) acc[q][c] = both(b[4 * lane + c]);
  dot_rows<NP, CNT, K, LDI, LDW>(in, W, acc);
#pragma unroll
  for (int q = 0; q < CNT; ++q) {
    float hv[8], dv[8];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float z = r ? acc[q][c].y : acc[q][c].x, s = sigm(z);
        hv[2 * c + r] = z * s;
        if (TRAIN) dv[2 * c + r] = s + z * s * (1.f - s);
      }
    const int at = pair_of<NP>(q) * kLdH + 4 * lane;
    float4* hp = reinterpret_cast<float4*>(h + at);
    hp[0] = make_float4(hv[0], hv[1], hv[2], hv[3]);
    hp[1] = make_float4(hv[4], hv[5], hv[6], hv[7]);
    if (TRAIN) {
      float4* dp = reinterpret_cast<float4*>(d + at);
      dp[0] = make_float4(dv[0], dv[1], dv[2], dv[3]);
      dp[1] = make_float4(dv[4], dv[5], dv[6], dv[7]);
    }
  }
}

// g += Σ_rows inᵀ dz over `pairs` row pairs in row order: rows NR tk .. of the gradient, columns
// 2 tj, 2 tj + 1 of each quarter of 32.
template <int LDI, int NR>
__device__ __forceinline__ void weight_grad(const float2* in, const float2* dz, int pairs, float2 (&g)[NR][4]) {
  const int tk = threadIdx.x >> 4, tj = threadIdx.x & 15;
#pragma unroll 1
  for (int p = 0; p < pairs; ++p) {
    float2 v[NR];
    if (NR == 8) {
#pragma unroll
      for (int a = 0; a < NR; a += 2) {
        const float4 q = *reinterpret_cast<const float4*>(in + p * LDI + NR * tk + a);
        v[a] = make_float2(q.x, q.y);
        v[(a + 1) % NR] = make_float2(q.z, q.w);
      }
    } else {
#pragma unroll
      for (int a = 0; a < NR; ++a) v[a] = in[p * LDI + NR * tk + a];
    }
    float2 d0[4], d1[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 q = *reinterpret_cast<const float4*>(dz + p * kLdH + 2 * tj + 32 * c);
      d0[c] = make_float2(q.x, q.z);
      d1[c] = make_float2(q.y, q.w);
    }
#pragma unroll
    for (int a = 0; a < NR; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) fma2(g[a][c], both(v[a].x), d0[c]);
#pragma unroll
    for (int a = 0; a < NR; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) fma2(g[a][c], both(v[a].y), d1[c]);
  }
}

__device__ __forceinline__ void put_grad(float* G, int row, const float2 (&g)[4]) {
  const int tj = threadIdx.x & 15;
#pragma unroll
  for (int c = 0; c < 4; ++c) *reinterpret_cast<float2*>(G + row * kMlpHidden + 2 * tj + 32 * c) = g[c];
}

// One CTA processes tiles blockIdx.x, blockIdx.x + gridDim.x, ... (two at a time where NP = 4) of 32
// rows, 16 where NP = 1; X is 16-byte aligned.  TRAIN: targets T, gradient partials per CTA in gpart,
// loss partial in lpart.  Every sum has one order: over k in increasing order from the bias, over
// rows tile by tile, over CTAs in order (k_mlp_reduce), so outputs and gradients depend neither on
// NP nor on how the products are packed.  A batch of 8192 rows: 84 us with a 4 x 4 tile per thread and
// scalar operands, 40 us with sums split over even and odd k and 56-row tiles (another order: a loss
// after one epoch moved by 8e-8), 42 us now.
template <bool TRAIN, int NP>
__global__ void __launch_bounds__(kThr, 1)
    k_mlp(MlpDev m, const float* __restrict__ X, const int* __restrict__ rows, int64_t n,
          const float* __restrict__ T, float* __restrict__ Y, float* __restrict__ gpart, double* __restrict__ lpart,
          float gscale) {
  constexpr int kTile = NP == 1 ? 16 : kRows, kParts = NP == 4 ? 2 : 1, kPairs = kWarps * NP;
  extern __shared__ __align__(16) unsigned char smraw[];
  Smem<NP>& S = *reinterpret_cast<Smem<NP>*>(smraw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int64_t ntiles = (n + kTile - 1) / kTile;
  // ---- a round's input rows and targets, first into registers so that they arrive while other
  // work goes on; a row past the end is zero and carries no sample
  constexpr int kVecs = kPairs * (kMlpIn / 4), kNx = (kVecs + kThr - 1) / kThr;
  static_assert(kPairs * kOutP <= kThr, "one target pair per thread");
  float4 xin[kNx][2];
  float2 tin;
  auto row0 = [&](int64_t tile, int pair) { return (tile + pair / (kTile / 2) * (int64_t)gridDim.x) * kTile + 2 * (pair % (kTile / 2)); };
  auto load_tile = [&](int64_t tile) {
#pragma unroll
    for (int q = 0; q < kNx; ++q) {
      const int e = t + q * kThr, p = e / (kMlpIn / 4), k = e % (kMlpIn / 4);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t r = row0(tile, p) + u;
        xin[q][u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < kVecs && r < n) xin[q][u] = reinterpret_cast<const float4*>(X + (rows ? (int64_t)rows[r] : r) * kMlpIn)[k];
      }
    }
    if (TRAIN) {
      const int p = t / kOutP, o = t % kOutP;
      const bool on = t < kPairs * kOutP && o < kMlpOut;
      const int64_t r = row0(tile, p);
      tin = both(nanf(""));
      if (on && r < n) tin.x = T[(rows ? (int64_t)rows[r] : r) * kMlpOut + o];
      if (on && r + 1 < n) tin.y = T[(rows ? (int64_t)rows[r + 1] : r + 1) * kMlpOut + o];
    }
  };
  auto store_tile = [&]() {
#pragma unroll
    for (int q = 0; q < kNx; ++q) {
      const int e = t + q * kThr;
      if (e >= kVecs) continue;
      const float4 a = xin[q][0], b = xin[q][1];
      float4* dst = reinterpret_cast<float4*>(S.x + e / (kMlpIn / 4) * kLdX + 4 * (e % (kMlpIn / 4)));
      dst[0] = make_float4(a.x, b.x, a.y, b.y);
      dst[1] = make_float4(a.z, b.z, a.w, b.w);
    }
    if (TRAIN && t < kPairs * kOutP) S.dy[t] = tin;
  };
  // ---- weights: all loads are in flight before the first store waits
  constexpr int kIt1 = kMlpIn * kMlpHidden / 8 / kThr, kIt2 = kMlpHidden * kMlpHidden / 8 / kThr;
  static_assert(kIt1 * kThr * 8 == kMlpIn * kMlpHidden, "whole rounds");
  uint4 w1[kIt1], w2[kIt2];
  load_tile(blockIdx.x);
#pragma unroll
  for (int q = 0; q < kIt1; ++q) w1[q] = reinterpret_cast<const uint4*>(m.W + kOffW1)[t + q * kThr];
#pragma unroll
  for (int q = 0; q < kIt2; ++q) w2[q] = reinterpret_cast<const uint4*>(m.W + kOffW2)[t + q * kThr];
  for (int i = t; i < kMlpHidden * kOutP; i += kThr) {
    const int k = i / kOutP, o = i % kOutP;
    S.W3T[o * kLdW2 + k] = o < kMlpOut ? m.W[kOffW3 + k * kMlpOut + o] : __float2bfloat16_rn(0.f);
  }
  if (t < kMlpHidden) {
    S.b1[t] = m.P[kOffB1 + t];
    S.b2[t] = m.P[kOffB2 + t];
  }
  if (t < kOutP) S.b3[t] = t < kMlpOut ? m.P[kOffB3 + t] : 0.f;
#pragma unroll
  for (int q = 0; q < kIt1; ++q) reinterpret_cast<uint4*>(S.W1)[t + q * kThr] = w1[q];
#pragma unroll
  for (int q = 0; q < kIt2; ++q) {
    const int e = t + q * kThr;
    uint2* dst = reinterpret_cast<uint2*>(S.W2 + e / (kMlpHidden / 8) * kLdW2 + 8 * (e % (kMlpHidden / 8)));
    dst[0] = make_uint2(w2[q].x, w2[q].y);  // rows are 8-byte aligned
    dst[1] = make_uint2(w2[q].z, w2[q].w);
  }

  // gradient accumulators (TRAIN): weights as in weight_grad, biases: thread t < 128 of b2, t >= 128 of b1
  float2 g2[8][4], g1[3][4];
  float g3[4], gb = 0.f, gb3 = 0.f;
  double loss = 0.0;
  if (TRAIN) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int a = 0; a < 8; ++a) g2[a][c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < 3; ++a) g1[a][c] = make_float2(0.f, 0.f);
      g3[c] = 0.f;
    }
  }

  // a warp's row pairs through the network and back: a warp reads only its own rows
  auto through = [&](auto count, int64_t tile) {
    constexpr int CNT = decltype(count)::value;
    dense_silu<TRAIN, NP, CNT, kMlpIn, kLdX, kMlpHidden>(S.x, S.W1, S.b1, S.h1, S.d1);
    __syncwarp();
    dense_silu<TRAIN, NP, CNT, kMlpHidden, kLdH, kLdW2>(S.h1, S.W2, S.b2, S.h2, S.d2);
    __syncwarp();
    // ---- output layer: lane (pair, output)
    const int q = lane >> 3, o = lane & 7;
    if (q < CNT) {
      const int p = pair_of<NP>(q);
      float2 acc = both(S.b3[o]);
#pragma unroll 4
      for (int k = 0; k < kMlpHidden; k += 4) {
        const uint2 w = *reinterpret_cast<const uint2*>(S.W3T + o * kLdW2 + k);
        const float4 u = *reinterpret_cast<const float4*>(S.h2 + p * kLdH + k);
        const float4 v = *reinterpret_cast<const float4*>(S.h2 + p * kLdH + k + 2);
        fma2(acc, make_float2(u.x, u.y), both_lo(w.x));
        fma2(acc, make_float2(u.z, u.w), both_hi(w.x));
        fma2(acc, make_float2(v.x, v.y), both_lo(w.y));
        fma2(acc, make_float2(v.z, v.w), both_hi(w.y));
      }
      if (!TRAIN) {
        const int64_t r = row0(tile, p);
        if (o < kMlpOut && r < n) Y[r * kMlpOut + o] = acc.x;
        if (o < kMlpOut && r + 1 < n) Y[(r + 1) * kMlpOut + o] = acc.y;
      } else {
        const float2 tv = S.dy[p * kOutP + o];
        // NaN target: row carries no sample
        const float da = tv.x == tv.x ? acc.x - tv.x : 0.f, db = tv.y == tv.y ? acc.y - tv.y : 0.f;
        loss += (double)da * (double)da;
        loss += (double)db * (double)db;
        S.dy[p * kOutP + o] = make_float2(da * gscale, db * gscale);
      }
    }
    if (!TRAIN) return;
    __syncwarp();
    // ---- dz2 = (dy W3ᵀ) ⊙ silu'(z2), in place in d2
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float w[kMlpOut];
#pragma unroll
      for (int k = 0; k < kMlpOut; ++k) w[k] = __bfloat162float(S.W3T[k * kLdW2 + lane + 32 * c]);
#pragma unroll
      for (int a = 0; a < CNT; ++a) {
        const int p = pair_of<NP>(a);
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < kMlpOut; ++k) fma2(s, S.dy[p * kOutP + k], both(w[k]));
        const float2 d = S.d2[p * kLdH + lane + 32 * c];
        S.d2[p * kLdH + lane + 32 * c] = make_float2(s.x * d.x, s.y * d.y);
      }
    }
    __syncwarp();
    // ---- dz1 = (dz2 W2ᵀ) ⊙ silu'(z1), in place in d1
    float2 acc[CNT][4];
#pragma unroll
    for (int a = 0; a < CNT; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = make_float2(0.f, 0.f);
    dot_cols<NP, CNT>(S.d2, S.W2, acc);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int a = 0; a < CNT; ++a) {
        float2& d = S.d1[pair_of<NP>(a) * kLdH + lane + 32 * c];
        d = make_float2(acc[a][c].x * d.x, acc[a][c].y * d.y);
      }
  };

  for (int64_t tile = blockIdx.x; tile < ntiles; tile += kParts * (int64_t)gridDim.x) {
    store_tile();
    __syncthreads();
    if (tile + kParts * (int64_t)gridDim.x < ntiles) load_tile(tile + kParts * (int64_t)gridDim.x);
    const bool all = kParts == 1 || tile + gridDim.x < ntiles;  // else the second tile does not exist
    if (all) through(std::integral_constant<int, NP>{}, tile);
    else through(std::integral_constant<int, NP == 4 ? 2 : NP>{}, tile);
    if (TRAIN) {
      __syncthreads();
      // ---- weight gradients over all rows of the round
      const int pairs = all ? kPairs : kRows / 2;
      weight_grad<kLdH, 8>(S.h1, S.d2, pairs, g2);
      weight_grad<kLdX, 3>(S.x, S.d1, pairs, g1);
      const int k = t >> 1, o0 = (t & 1) * 4;
      const float2* db = (t < kMlpHidden ? S.d2 : S.d1) + (t & (kMlpHidden - 1));
#pragma unroll 4
      for (int p = 0; p < pairs; ++p) {
        const float2 hv = S.h2[p * kLdH + k], bv = db[p * kLdH];
        const float4 u = *reinterpret_cast<const float4*>(S.dy + p * kOutP + o0);
        const float4 v = *reinterpret_cast<const float4*>(S.dy + p * kOutP + o0 + 2);
        g3[0] = fmaf(hv.x, u.x, g3[0]); g3[1] = fmaf(hv.x, u.z, g3[1]);
        g3[2] = fmaf(hv.x, v.x, g3[2]); g3[3] = fmaf(hv.x, v.z, g3[3]);
        g3[0] = fmaf(hv.y, u.y, g3[0]); g3[1] = fmaf(hv.y, u.w, g3[1]);
        g3[2] = fmaf(hv.y, v.y, g3[2]); g3[3] = fmaf(hv.y, v.w, g3[3]);
        gb += bv.x;
        gb += bv.y;
      }
      if (t < kOutP)
        for (int p = 0; p < pairs; ++p) {
          const float2 v = S.dy[p * kOutP + t];
          gb3 += v.x;
          gb3 += v.y;
        }
    }
    __syncthreads();
  }

  if (TRAIN) {
    float* G = gpart + (int64_t)blockIdx.x * kMlpParams;  // kMlpParams and every offset are even
    const int tk = t >> 4;
#pragma unroll
    for (int a = 0; a < 8; ++a) put_grad(G + kOffW2, 8 * tk + a, g2[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) put_grad(G + kOffW1, 3 * tk + a, g1[a]);
    const int k = t >> 1, o0 = (t & 1) * 4;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (o0 + c < kMlpOut) G[kOffW3 + k * kMlpOut + o0 + c] = g3[c];
    G[t < kMlpHidden ? kOffB2 + t : kOffB1 + t - kMlpHidden] = gb;
    if (t < kMlpOut) G[kOffB3 + t] = gb3;
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
    if (lane == 0) S.red[warp] = loss;
    __syncthreads();
    if (t == 0) {
      double sum = 0.0;
      for (int w = 0; w < kWarps; ++w) sum += S.red[w];
      lpart[blockIdx.x] = sum;
    }
  }
}

// g[p] = Σ_c gpart[c][p] in CTA order; loss = Σ_c lpart[c] · lscale.  A CTA owns 32 parameters: its
// warps bring the partials into shared memory, one warp adds them.  With ADAM the parameter is
// updated at once, and its BF16 copy.  152 partials are 14.3 MB, read from L2: 17 us with a thread
// per parameter plus 3.6 us for Adam's own launch, 12 us now.
constexpr int kRedParams = 32, kRedWarps = 8, kRedChunk = 160;
constexpr int kRedCtas = (kMlpParams + kRedParams - 1) / kRedParams;

template <bool ADAM>
__global__ void __launch_bounds__(kRedParams * kRedWarps)
    k_mlp_reduce(const float* __restrict__ gpart, int grid, MlpTrainer t, const double* __restrict__ lpart,
                 double* __restrict__ loss, double lscale, float lr, float c1, float c2) {
  __shared__ float part[kRedChunk][kRedParams];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x == kRedCtas) {
    if (warp == 0 && loss) {
      double s = 0.0;
      for (int c = lane; c < grid; c += 32) s += lpart[c];
      for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
      if (lane == 0) *loss = s * lscale;
    }
    return;
  }
  const int p = blockIdx.x * kRedParams + lane;
  float gp = 0.f;
  for (int c0 = 0; c0 < grid; c0 += kRedChunk) {
    const int cnt = min(kRedChunk, grid - c0);
    if (p < kMlpParams)
#pragma unroll 20
      for (int c = warp; c < cnt; c += kRedWarps) part[c][lane] = gpart[(int64_t)(c0 + c) * kMlpParams + p];
    __syncthreads();
    if (warp == 0)
#pragma unroll 8
      for (int c = 0; c < cnt; ++c) gp += part[c][lane];
    __syncthreads();
  }
  if (warp != 0 || p >= kMlpParams) return;
  if (!ADAM) {
    t.G[p] = gp;
    return;
  }
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float a = b1 * t.M1[p] + (1.f - b1) * gp;
  const float v = b2 * t.M2[p] + (1.f - b2) * gp * gp;
  t.M1[p] = a;
  t.M2[p] = v;
  const float w = t.P[p] - lr * (a * c1) / (sqrtf(v * c2) + eps);
  t.P[p] = w;
  t.W[p] = __float2bfloat16_rn(w);
}

__global__ void k_mlp_bf16(const float* __restrict__ P, __nv_bfloat16* __restrict__ W) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < kMlpParams) W[p] = __float2bfloat16_rn(P[p]);
}

template <bool TRAIN, int NP>
cudaError_t launch_mlp(int sms, const MlpDev& m, const float* X, const int* rows, int64_t n, const float* T, float* Y,
                       float* gpart, double* lpart, float gscale, int* grid_out, cudaStream_t s) {
  constexpr int kTile = NP == 1 ? 16 : kRows;
  const void* k = (const void*)k_mlp<TRAIN, NP>;
  cudaError_t e = raise_smem_limit(k, sizeof(Smem<NP>));
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<int64_t>((n + kTile - 1) / kTile, sms);
  k_mlp<TRAIN, NP><<<grid, kThr, sizeof(Smem<NP>), s>>>(m, X, rows, n, T, Y, gpart, lpart, gscale);
  *grid_out = grid;
  return cudaGetLastError();
}

// Rows per round of a CTA: one tile where every tile has an SM to itself, else two tiles, whose weights
// are read half as often; without gradients also half a tile, where as many have an SM each
// (2000 rows forward: 10.4 us in sixteens, 13.2 in tiles).  A gradient partial is whole tiles, so that its sums keep one order.
template <bool TRAIN>
cudaError_t run_mlp(const MlpDev& m, const float* X, const int* rows, int64_t n, const float* T, float* Y, float* gpart,
                    double* lpart, float gscale, int* grid, cudaStream_t s) {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  auto go = n > (int64_t)sms * kRows            ? launch_mlp<TRAIN, 4>
            : TRAIN || n > (int64_t)sms * 16    ? launch_mlp<TRAIN, 2>
                                                : launch_mlp<TRAIN, TRAIN ? 2 : 1>;
  return go(sms, m, X, rows, n, T, Y, gpart, lpart, gscale, grid, s);
}

}  // namespace

cudaError_t mlp_forward(const MlpDev& m, const float* X, int64_t n, float* Y, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int grid = 0;
  return run_mlp<false>(m, X, nullptr, n, nullptr, Y, nullptr, nullptr, 0.f, &grid, s);
}

cudaError_t mlp_to_bf16(const float* P, __nv_bfloat16* W, cudaStream_t s) {
  k_mlp_bf16<<<(kMlpParams + 255) / 256, 256, 0, s>>>(P, W);
  return cudaGetLastError();
}

cudaError_t MlpSlab::make() {
  cudaError_t e = cudaMalloc(&base, bytes ? bytes : 1);
  if (e != cudaSuccess) return e;
  for (int i = 0; i < n_parts; ++i) *parts[i].to = (char*)base + parts[i].off;
  return cudaSuccess;
}

cudaError_t mlp_trainer_init(MlpTrainer& t, MlpSlab& slab, const float* params_host, cudaStream_t s) {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  t.grid = sms;
  for (float** p : {&t.P, &t.G, &t.M1, &t.M2}) slab.want(p, kMlpParams);
  slab.want(&t.W, kMlpParams);
  slab.want(&t.gpart, (size_t)kMlpParams * t.grid);
  slab.want(&t.loss, (size_t)t.grid + 1);
  cudaError_t e = slab.make();
  if (e != cudaSuccess) return e;
  const size_t pb = sizeof(float) * kMlpParams;
  if ((e = cudaMemcpyAsync(t.P, params_host, pb, cudaMemcpyHostToDevice, s)) ||
      (e = cudaMemsetAsync(t.M1, 0, pb, s)) || (e = cudaMemsetAsync(t.M2, 0, pb, s)))
    return e;
  t.step = 0;
  return mlp_to_bf16(t.P, t.W, s);
}

template <bool ADAM>
static cudaError_t grad_step(MlpTrainer& t, const float* X, const float* T, const int* rows, int64_t n, float lr,
                             double* loss_dev, cudaStream_t s) {
  const float gscale = 2.f / (float)((double)n * kMlpOut);
  int grid = 0;
  cudaError_t e = run_mlp<true>(MlpDev{t.P, t.W}, X, rows, n, T, nullptr, t.gpart, t.loss, gscale, &grid, s);
  if (e != cudaSuccess) return e;
  if (ADAM) t.step += 1;
  const float c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)t.step)));
  const float c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)t.step)));
  k_mlp_reduce<ADAM><<<kRedCtas + 1, kRedParams * kRedWarps, 0, s>>>(t.gpart, grid, t, t.loss, loss_dev,
                                                                     1.0 / ((double)n * kMlpOut), lr, c1, c2);
  return cudaGetLastError();
}

cudaError_t mlp_loss_grad(MlpTrainer& t, const float* X, const float* T, const int* rows, int64_t n, double* loss_dev,
                          cudaStream_t s) {
  return grad_step<false>(t, X, T, rows, n, 0.f, loss_dev, s);
}

cudaError_t mlp_train_step(MlpTrainer& t, const float* X, const float* T, const int* rows, int64_t n, float lr,
                           double* loss_dev, cudaStream_t s) {
  return grad_step<true>(t, X, T, rows, n, lr, loss_dev, s);
}

}  // namespace eb

// ---------------------------------------------------------------- C ABI
using namespace eb;

namespace {
int cuda_fail(cudaError_t e, const char* what) {
  char buf[256];
  std::snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  return eb_internal_fail(EB_ERR_CUDA, buf);
}
#define MCK(x, what)                          \
  do {                                        \
    cudaError_t _e = (x);                     \
    if (_e != cudaSuccess) return cuda_fail(_e, what); \
  } while (0)
}  // namespace

extern "C" {

int eb_mlp_forward(const float* params, const float* X, int64_t n, float* Y) {
  if (!params || n < 0 || (n > 0 && (!X || !Y))) return eb_internal_fail(EB_ERR_ARG, "eb_mlp_forward: bad arguments");
  MlpSlab slab;
  float *P = nullptr, *Xd = nullptr, *Yd = nullptr;
  __nv_bfloat16* W = nullptr;
  slab.want(&P, kMlpParams);
  slab.want(&W, kMlpParams);
  slab.want(&Xd, (size_t)n * kMlpIn);
  slab.want(&Yd, (size_t)n * kMlpOut);
  MCK(slab.make(), "eb_mlp_forward");
  MCK(cudaMemcpy(P, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice), "eb_mlp_forward");
  if (n) MCK(cudaMemcpy(Xd, X, sizeof(float) * (size_t)n * kMlpIn, cudaMemcpyHostToDevice), "eb_mlp_forward");
  MCK(mlp_to_bf16(P, W, 0), "eb_mlp_forward");
  MCK(mlp_forward(MlpDev{P, W}, Xd, n, Yd, 0), "eb_mlp_forward");
  MCK(cudaMemcpy(Y, Yd, sizeof(float) * (size_t)n * kMlpOut, cudaMemcpyDeviceToHost), "eb_mlp_forward");
  return EB_OK;
}

int eb_mlp_loss_grad(const float* params, const float* X, const float* T, int64_t n, double* loss, float* grad) {
  if (!params || !X || !T || n <= 0 || !loss || !grad)
    return eb_internal_fail(EB_ERR_ARG, "eb_mlp_loss_grad: bad arguments");
  MlpTrainer tr;
  MlpSlab slab;
  float *Xd = nullptr, *Td = nullptr;
  slab.want(&Xd, (size_t)n * kMlpIn);
  slab.want(&Td, (size_t)n * kMlpOut);
  MCK(mlp_trainer_init(tr, slab, params, 0), "eb_mlp_loss_grad");
  MCK(cudaMemcpy(Xd, X, sizeof(float) * (size_t)n * kMlpIn, cudaMemcpyHostToDevice), "eb_mlp_loss_grad");
  MCK(cudaMemcpy(Td, T, sizeof(float) * (size_t)n * kMlpOut, cudaMemcpyHostToDevice), "eb_mlp_loss_grad");
  MCK(mlp_loss_grad(tr, Xd, Td, nullptr, n, tr.loss + tr.grid, 0), "eb_mlp_loss_grad");
  MCK(cudaMemcpy(grad, tr.G, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost), "eb_mlp_loss_grad");
  MCK(cudaMemcpy(loss, tr.loss + tr.grid, sizeof(double), cudaMemcpyDeviceToHost), "eb_mlp_loss_grad");
  return EB_OK;
}

int eb_mlp_train(float* params, const float* X, const float* T, int64_t n, int32_t epochs, int32_t batch, float lr,
                 uint64_t seed, double* loss_per_epoch) {
  if (!params || !X || !T || n <= 0 || epochs < 0 || batch <= 0 || !(lr > 0))
    return eb_internal_fail(EB_ERR_ARG, "eb_mlp_train: bad arguments");
  if (n > INT32_MAX) return eb_internal_fail(EB_ERR_ARG, "eb_mlp_train: too many samples");
  const int64_t nb = (n + batch - 1) / batch;
  MlpTrainer tr;
  MlpSlab slab;
  float *Xd = nullptr, *Td = nullptr;
  int* Rd = nullptr;
  double* Ld = nullptr;
  slab.want(&Xd, (size_t)n * kMlpIn);
  slab.want(&Td, (size_t)n * kMlpOut);
  slab.want(&Rd, (size_t)n);
  slab.want(&Ld, (size_t)nb);
  MCK(mlp_trainer_init(tr, slab, params, 0), "eb_mlp_train");
  MCK(cudaMemcpy(Xd, X, sizeof(float) * (size_t)n * kMlpIn, cudaMemcpyHostToDevice), "eb_mlp_train");
  MCK(cudaMemcpy(Td, T, sizeof(float) * (size_t)n * kMlpOut, cudaMemcpyHostToDevice), "eb_mlp_train");
  std::vector<int> perm((size_t)n);
  std::mt19937_64 rng(seed);
  std::vector<double> bl((size_t)nb);
  for (int ep = 0; ep < epochs; ++ep) {
    for (int64_t i = 0; i < n; ++i) perm[(size_t)i] = (int)i;
    for (int64_t i = n - 1; i > 0; --i) {  // Fisher-Yates with the seeded engine
      const int64_t j = (int64_t)(rng() % (uint64_t)(i + 1));
      std::swap(perm[(size_t)i], perm[(size_t)j]);
    }
    MCK(cudaMemcpy(Rd, perm.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice), "eb_mlp_train");
    for (int64_t b = 0; b < nb; ++b) {
      const int64_t r0 = b * batch, m = std::min<int64_t>(batch, n - r0);
      MCK(mlp_train_step(tr, Xd, Td, Rd + r0, m, lr, Ld + b, 0), "eb_mlp_train");
    }
    MCK(cudaMemcpy(bl.data(), Ld, sizeof(double) * (size_t)nb, cudaMemcpyDeviceToHost), "eb_mlp_train");
    if (loss_per_epoch) {
      double s = 0.0;
      for (int64_t b = 0; b < nb; ++b) s += bl[(size_t)b];
      loss_per_epoch[ep] = s / (double)nb;
    }
  }
  MCK(cudaMemcpy(params, tr.P, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost), "eb_mlp_train");
  return EB_OK;
}

}  // extern "C"
