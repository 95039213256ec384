// Per-node MLP kernels (see eb_mlp.cuh) and the C-ABI training/evaluation
// entry points.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/endobeams_gb300.h"
#include "eb_internal.cuh"
#include "eb_mlp.cuh"

int eb_internal_fail(int code, const char* msg);

namespace eb {
namespace {

constexpr int kThr = 256;      // threads per CTA
constexpr int kLdX = 52;       // shared row stride of the input tile (floats)
constexpr int kLdH = 132;      // shared row stride of hidden activations (floats)
constexpr int kLdW1 = 52;      // shared row stride of W1 transposed (BF16 values)
constexpr int kLdW2 = 132;     // shared row stride of W2, W2 and W3 transposed
constexpr int kOutP = 8;       // padded output width
constexpr int kWarps = kThr / 32;

static_assert(kMlpIn == 48 && kMlpHidden == 128 && kMlpOut == 6, "kernel tiling assumes 48-128-128-6");

// A CTA's tile has RW rows per warp.  FP32 arithmetic on CUDA cores bounds a tile (63,700 FMAs per
// row forward and backward: 14.6 us for 56 rows on one SM), so the products are packed two to an
// instruction and every shared-memory operand feeds at least four of them.
template <int RW>
struct Smem {
  __nv_bfloat16 W1T[kMlpHidden * kLdW1];
  __nv_bfloat16 W2T[kMlpHidden * kLdW2];
  __nv_bfloat16 W2[kMlpHidden * kLdW2];  // as stored (backward only)
  __nv_bfloat16 W3T[kOutP * kLdW2];
  float b1[kMlpHidden], b2[kMlpHidden], b3[kOutP];
  float x[kWarps * RW * kLdX];
  // hidden activations and the derivatives of silu there, later the gradients by z (in place)
  float h1[kWarps * RW * kLdH], d1[kWarps * RW * kLdH], h2[kWarps * RW * kLdH], d2[kWarps * RW * kLdH];
  float dy[kWarps * RW * kOutP];  // targets, then the gradient by y
  float gb[kWarps * (2 * kMlpHidden + kOutP)];
  double red[kWarps];
};

__device__ __forceinline__ float sigm(float z) { return 1.f / (1.f + expf(-z)); }

// d = a b + d on both halves, each rounded as fmaf does
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

__device__ __forceinline__ float2 unpack(unsigned w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// acc[a][c] = Σ_k in[row][k] W[col][k] for this warp's RW rows and columns lane + 32 c, even and
// odd k in the two halves: both operands then are read along k, the inputs as one address per
// warp, the weights without bank conflicts (row strides of 26 and 66 words).
template <int K, int LDI, int LDW, int RW>
__device__ __forceinline__ void tile_dot(const float* in, const __nv_bfloat16* W, float2 (&acc)[RW][4]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < RW; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[a][c] = make_float2(0.f, 0.f);
  const float* ip = in + warp * RW * LDI;
  const __nv_bfloat16* wp = W + lane * LDW;
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float4 v[RW];
#pragma unroll
    for (int a = 0; a < RW; ++a) v[a] = *reinterpret_cast<const float4*>(ip + a * LDI + k);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint2 w = *reinterpret_cast<const uint2*>(wp + 32 * c * LDW + k);
      const float2 w0 = unpack(w.x), w1 = unpack(w.y);
#pragma unroll
      for (int a = 0; a < RW; ++a) {
        fma2(acc[a][c], make_float2(v[a].x, v[a].y), w0);
        fma2(acc[a][c], make_float2(v[a].z, v[a].w), w1);
      }
    }
  }
}

// h = silu(in W + b) of this warp's rows, and silu' (TRAIN).
template <int K, int LDI, int LDW, int RW, bool TRAIN>
__device__ __forceinline__ void dense_silu(const float* in, const __nv_bfloat16* W, const float* b, float* h, float* d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2 acc[RW][4];
  tile_dot<K, LDI, LDW, RW>(in, W, acc);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float bc = b[lane + 32 * c];
#pragma unroll
    for (int a = 0; a < RW; ++a) {
      const float z = (acc[a][c].x + acc[a][c].y) + bc, s = sigm(z);
      const int at = (warp * RW + a) * kLdH + lane + 32 * c;
      h[at] = z * s;
      if (TRAIN) d[at] = s + z * s * (1.f - s);
    }
  }
}

// g += Σ_rows inᵀ dz over the tile: rows 4 tk .. +3 and K/2 + 4 tk .. +3 of the gradient (K = 48:
// 3 tk .. +2), columns 4 tj .. +3 and 64 + 4 tj .. +3; 16-byte reads without bank conflicts.
template <int K, int LDI, int ROWS, int NR>
__device__ __forceinline__ void weight_grad(const float* in, const float* dz, float2 (&g)[NR][4]) {
  const int tk = threadIdx.x >> 4, tj = threadIdx.x & 15;
#pragma unroll 2
  for (int i = 0; i < ROWS; ++i) {
    float v[NR];
    if (NR == 8) {
      const float4 p = *reinterpret_cast<const float4*>(in + i * LDI + 4 * tk);
      const float4 q = *reinterpret_cast<const float4*>(in + i * LDI + K / 2 + 4 * tk);
      v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3 % NR] = p.w;
      v[4 % NR] = q.x; v[5 % NR] = q.y; v[6 % NR] = q.z; v[7 % NR] = q.w;
    } else {
#pragma unroll
      for (int a = 0; a < NR; ++a) v[a] = in[i * LDI + NR * tk + a];
    }
    const float4 da = *reinterpret_cast<const float4*>(dz + i * kLdH + 4 * tj);
    const float4 db = *reinterpret_cast<const float4*>(dz + i * kLdH + kMlpHidden / 2 + 4 * tj);
#pragma unroll
    for (int a = 0; a < NR; ++a) {
      const float2 vv = make_float2(v[a], v[a]);
      fma2(g[a][0], vv, make_float2(da.x, da.y));
      fma2(g[a][1], vv, make_float2(da.z, da.w));
      fma2(g[a][2], vv, make_float2(db.x, db.y));
      fma2(g[a][3], vv, make_float2(db.z, db.w));
    }
  }
}

__device__ __forceinline__ void put_grad(float* G, int row, const float2 (&g)[4]) {
  const int tj = threadIdx.x & 15;
  float2* p = reinterpret_cast<float2*>(G + row * kMlpHidden + 4 * tj);
  p[0] = g[0];
  p[1] = g[1];
  float2* q = reinterpret_cast<float2*>(G + row * kMlpHidden + kMlpHidden / 2 + 4 * tj);
  q[0] = g[2];
  q[1] = g[3];
}

// One CTA processes tiles blockIdx.x, blockIdx.x + gridDim.x, ... of 8 RW rows; X is 16-byte
// aligned.  TRAIN: targets T, gradient partials per CTA in gpart, loss partial in lpart.  A batch
// of 8192 rows on 147 SMs: 84 us with a 4 x 4 tile per thread, scalar operands and two rounds of
// 32 rows, 40 us now (10 of them weights in and gradients out).
template <bool TRAIN, int RW>
__global__ void __launch_bounds__(kThr, 1)
    k_mlp(MlpDev m, const float* __restrict__ X, const int* __restrict__ rows, int64_t n,
          const float* __restrict__ T, float* __restrict__ Y, float* __restrict__ gpart, double* __restrict__ lpart,
          float gscale) {
  constexpr int kTile = kWarps * RW;
  extern __shared__ __align__(16) unsigned char smraw[];
  Smem<RW>& S = *reinterpret_cast<Smem<RW>*>(smraw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int64_t ntiles = (n + kTile - 1) / kTile;
  // ---- a tile's input rows and targets, first into registers so that they arrive while other
  // work goes on; a row past the end is zero and carries no sample
  constexpr int kVecs = kTile * (kMlpIn / 4), kNx = (kVecs + kThr - 1) / kThr;
  constexpr int kOuts = kTile * kOutP, kNt = (kOuts + kThr - 1) / kThr;
  float4 xin[kNx];
  float tin[kNt];
  auto load_tile = [&](int64_t tile) {
    const int64_t r0 = tile * kTile;
#pragma unroll
    for (int q = 0; q < kNx; ++q) {
      const int e = t + q * kThr, i = e / (kMlpIn / 4), k = e % (kMlpIn / 4);
      const int64_t r = r0 + i;
      xin[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < kVecs && r < n) xin[q] = reinterpret_cast<const float4*>(X + (rows ? (int64_t)rows[r] : r) * kMlpIn)[k];
    }
    if (TRAIN)
#pragma unroll
      for (int q = 0; q < kNt; ++q) {
        const int e = t + q * kThr, o = e % kOutP;
        const int64_t r = r0 + e / kOutP;
        tin[q] = e < kOuts && r < n && o < kMlpOut ? T[(rows ? (int64_t)rows[r] : r) * kMlpOut + o] : nanf("");
      }
  };
  auto store_tile = [&]() {
#pragma unroll
    for (int q = 0; q < kNx; ++q) {
      const int e = t + q * kThr;
      if (e < kVecs) *reinterpret_cast<float4*>(S.x + e / (kMlpIn / 4) * kLdX + 4 * (e % (kMlpIn / 4))) = xin[q];
    }
    if (TRAIN)
#pragma unroll
      for (int q = 0; q < kNt; ++q)
        if (t + q * kThr < kOuts) S.dy[t + q * kThr] = tin[q];
  };
  // ---- weights: a thread takes eight columns of two rows k, k + 1 and stores the pairs along k
  // (lanes along k: no bank conflicts); all loads are in flight before the first store waits
  constexpr int kIt1 = (kMlpIn / 2 * 16 + kThr - 1) / kThr, kIt2 = kMlpHidden / 2 * 16 / kThr;
  uint4 w1[kIt1][2], w2[kIt2][2];
  load_tile(blockIdx.x);
  auto load2 = [&](const __nv_bfloat16* W, int pairs, int e, uint4 (&v)[2]) {
    const uint4* src = reinterpret_cast<const uint4*>(W + (2 * (e % pairs)) * kMlpHidden + 8 * (e / pairs));
    v[0] = src[0];
    v[1] = src[kMlpHidden / 8];
  };
  auto store2 = [&](const uint4 (&v)[2], int pairs, int e, __nv_bfloat16* WT, int ld) {
    const unsigned a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {v[1].x, v[1].y, v[1].z, v[1].w};
    unsigned* dst = reinterpret_cast<unsigned*>(WT + 8 * (e / pairs) * ld) + e % pairs;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      dst[c * ld / 2] = __byte_perm(a[c / 2], b[c / 2], c % 2 ? 0x7632 : 0x5410);
  };
#pragma unroll
  for (int q = 0; q < kIt1; ++q)
    if (t + q * kThr < kMlpIn / 2 * 16) load2(m.W + kOffW1, kMlpIn / 2, t + q * kThr, w1[q]);
#pragma unroll
  for (int q = 0; q < kIt2; ++q) load2(m.W + kOffW2, kMlpHidden / 2, t + q * kThr, w2[q]);
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
  for (int q = 0; q < kIt1; ++q)
    if (t + q * kThr < kMlpIn / 2 * 16) store2(w1[q], kMlpIn / 2, t + q * kThr, S.W1T, kLdW1);
#pragma unroll
  for (int q = 0; q < kIt2; ++q) {
    const int e = t + q * kThr, k = 2 * (e % (kMlpHidden / 2)), j = 8 * (e / (kMlpHidden / 2));
    store2(w2[q], kMlpHidden / 2, e, S.W2T, kLdW2);
    if (TRAIN)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint2* dst = reinterpret_cast<uint2*>(S.W2 + (k + h) * kLdW2 + j);  // rows are 8-byte aligned
        dst[0] = make_uint2(w2[q][h].x, w2[q][h].y);
        dst[1] = make_uint2(w2[q][h].z, w2[q][h].w);
      }
  }

  // gradient accumulators (TRAIN): weights as in weight_grad, biases of this warp's rows
  float2 g2[8][4], g1[3][4];
  float g3[4], gb1[4], gb2[4], gb3 = 0.f;
  double loss = 0.0;
  if (TRAIN) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int a = 0; a < 8; ++a) g2[a][c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int a = 0; a < 3; ++a) g1[a][c] = make_float2(0.f, 0.f);
      g3[c] = gb1[c] = gb2[c] = 0.f;
    }
  }

  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t r0 = tile * kTile;
    store_tile();
    __syncthreads();
    if (tile + gridDim.x < ntiles) load_tile(tile + gridDim.x);
    // a warp reads only its own rows up to y
    dense_silu<kMlpIn, kLdX, kLdW1, RW, TRAIN>(S.x, S.W1T, S.b1, S.h1, S.d1);
    __syncwarp();
    dense_silu<kMlpHidden, kLdH, kLdW2, RW, TRAIN>(S.h1, S.W2T, S.b2, S.h2, S.d2);
    __syncwarp();
    // ---- output layer: lane (o, q) sums the k of quarter q, interleaved by four
    {
      const int o = lane & 7, q = lane >> 3;
      float2 acc[RW];
#pragma unroll
      for (int a = 0; a < RW; ++a) acc[a] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int k = 4 * q; k < kMlpHidden; k += 16) {
        const uint2 w = *reinterpret_cast<const uint2*>(S.W3T + o * kLdW2 + k);
        const float2 w0 = unpack(w.x), w1 = unpack(w.y);
#pragma unroll
        for (int a = 0; a < RW; ++a) {
          const float4 v = *reinterpret_cast<const float4*>(S.h2 + (warp * RW + a) * kLdH + k);
          fma2(acc[a], make_float2(v.x, v.y), w0);
          fma2(acc[a], make_float2(v.z, v.w), w1);
        }
      }
#pragma unroll
      for (int a = 0; a < RW; ++a) {
        float y = acc[a].x + acc[a].y;
        y += __shfl_xor_sync(0xffffffffu, y, 8);
        y += __shfl_xor_sync(0xffffffffu, y, 16);
        y += S.b3[o];
        const int i = warp * RW + a;
        const int64_t r = r0 + i;
        if (q != 0) continue;
        if (!TRAIN) {
          if (r < n && o < kMlpOut) Y[r * kMlpOut + o] = y;
        } else {
          const float tv = S.dy[i * kOutP + o];
          const float d = tv == tv ? y - tv : 0.f;  // NaN target: row carries no sample
          loss += (double)d * (double)d;
          gb3 += d * gscale;
          S.dy[i * kOutP + o] = d * gscale;
        }
      }
    }
    if (TRAIN) {
      __syncwarp();
      // ---- dz2 = (dy W3ᵀ) ⊙ silu'(z2) of this warp's rows, in place in d2
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float w[kMlpOut];
#pragma unroll
        for (int o = 0; o < kMlpOut; ++o) w[o] = __bfloat162float(S.W3T[o * kLdW2 + lane + 32 * c]);
#pragma unroll
        for (int a = 0; a < RW; ++a) {
          const int i = warp * RW + a;
          float s = 0.f;
#pragma unroll
          for (int o = 0; o < kMlpOut; ++o) s = fmaf(S.dy[i * kOutP + o], w[o], s);
          s *= S.d2[i * kLdH + lane + 32 * c];
          S.d2[i * kLdH + lane + 32 * c] = s;
          gb2[c] += s;
        }
      }
      __syncwarp();
      // ---- dz1 = (dz2 W2ᵀ) ⊙ silu'(z1) of this warp's rows, in place in d1
      {
        float2 acc[RW][4];
        tile_dot<kMlpHidden, kLdH, kLdW2, RW>(S.d2, S.W2, acc);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int a = 0; a < RW; ++a) {
            const int at = (warp * RW + a) * kLdH + lane + 32 * c;
            const float s = (acc[a][c].x + acc[a][c].y) * S.d1[at];
            S.d1[at] = s;
            gb1[c] += s;
          }
      }
      __syncthreads();
      // ---- weight gradients over all rows of the tile
      weight_grad<kMlpHidden, kLdH, kTile, 8>(S.h1, S.d2, g2);
      weight_grad<kMlpIn, kLdX, kTile, 3>(S.x, S.d1, g1);
      {
        const int k = t >> 1, o0 = (t & 1) * 4;
#pragma unroll 4
        for (int i = 0; i < kTile; ++i) {
          const float hv = S.h2[i * kLdH + k];
          const float4 dv = *reinterpret_cast<const float4*>(S.dy + i * kOutP + o0);
          g3[0] = fmaf(hv, dv.x, g3[0]);
          g3[1] = fmaf(hv, dv.y, g3[1]);
          g3[2] = fmaf(hv, dv.z, g3[2]);
          g3[3] = fmaf(hv, dv.w, g3[3]);
        }
      }
    }
    __syncthreads();
  }

  if (TRAIN) {
    float* G = gpart + (int64_t)blockIdx.x * kMlpParams;  // kMlpParams and every offset are even
    {
      const int tk = t >> 4;
#pragma unroll
      for (int a = 0; a < 8; ++a) put_grad(G + kOffW2, (a < 4 ? 0 : kMlpHidden / 2) + 4 * tk + (a & 3), g2[a]);
#pragma unroll
      for (int a = 0; a < 3; ++a) put_grad(G + kOffW1, 3 * tk + a, g1[a]);
    }
    {
      const int k = t >> 1, o0 = (t & 1) * 4;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (o0 + c < kMlpOut) G[kOffW3 + k * kMlpOut + o0 + c] = g3[c];
    }
    // biases and loss: the warps' sums in warp order
    float* gb = S.gb + warp * (2 * kMlpHidden + kOutP);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      gb[lane + 32 * c] = gb1[c];
      gb[kMlpHidden + lane + 32 * c] = gb2[c];
    }
    if (lane < kOutP) gb[2 * kMlpHidden + lane] = gb3;
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
    if (lane == 0) S.red[warp] = loss;
    __syncthreads();
    for (int e = t; e < 2 * kMlpHidden + kMlpOut; e += kThr) {
      float sum = 0.f;
      for (int w = 0; w < kWarps; ++w) sum += S.gb[w * (2 * kMlpHidden + kOutP) + e];
      G[e < kMlpHidden ? kOffB1 + e : e < 2 * kMlpHidden ? kOffB2 + e - kMlpHidden : kOffB3 + e - 2 * kMlpHidden] = sum;
    }
    if (t == 0) {
      double sum = 0.0;
      for (int w = 0; w < kWarps; ++w) sum += S.red[w];
      lpart[blockIdx.x] = sum;
    }
  }
}

// g[p] = Σ_c gpart[c][p]; loss = Σ_c lpart[c] · lscale.  A CTA owns 32 parameters: warp w sums the
// partials w, w + 8, ... and the eight sums are added in warp order.  With ADAM the parameter is
// updated at once, and its BF16 copy.  147 partials are 13.9 MB, read from L2: 17 us with a thread
// per parameter plus 3.6 us for Adam's own launch, 7.4 us now.
constexpr int kRedParams = 32, kRedWarps = 8;
constexpr int kRedCtas = (kMlpParams + kRedParams - 1) / kRedParams;

template <bool ADAM>
__global__ void __launch_bounds__(kRedParams * kRedWarps)
    k_mlp_reduce(const float* __restrict__ gpart, int grid, MlpTrainer t, const double* __restrict__ lpart,
                 double* __restrict__ loss, double lscale, float lr, float c1, float c2) {
  __shared__ float part[kRedWarps][kRedParams];
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
  float s = 0.f;
  if (p < kMlpParams) {
#pragma unroll 8
    for (int c = warp; c < grid; c += kRedWarps) s += gpart[(int64_t)c * kMlpParams + p];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || p >= kMlpParams) return;
  float gp = part[0][lane];
#pragma unroll
  for (int w = 1; w < kRedWarps; ++w) gp += part[w][lane];
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

template <bool TRAIN, int RW>
cudaError_t launch_mlp(int sms, const MlpDev& m, const float* X, const int* rows, int64_t n, const float* T, float* Y,
                       float* gpart, double* lpart, float gscale, int* grid_out, cudaStream_t s) {
  const void* k = (const void*)k_mlp<TRAIN, RW>;
  cudaError_t e = raise_smem_limit(k, sizeof(Smem<RW>));
  if (e != cudaSuccess) return e;
  const int grid = (int)std::min<int64_t>((n + kWarps * RW - 1) / (kWarps * RW), sms);
  k_mlp<TRAIN, RW><<<grid, kThr, sizeof(Smem<RW>), s>>>(m, X, rows, n, T, Y, gpart, lpart, gscale);
  *grid_out = grid;
  return cudaGetLastError();
}

// Rows per tile: the smallest of 16, 32 and 56 for which every tile has an SM to itself (forward
// and gradient: 11 and 20 us at 16 rows, 14 and 27 at 32; 27 and 54 with the 32-row tile of four by
// four per thread), else 56, whose weights and gradients are loaded and stored least often.  A
// row's outputs do not depend on the choice.
template <bool TRAIN>
cudaError_t run_mlp(const MlpDev& m, const float* X, const int* rows, int64_t n, const float* T, float* Y, float* gpart,
                    double* lpart, float gscale, int* grid, cudaStream_t s) {
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  auto go = n <= (int64_t)sms * kWarps * 2   ? launch_mlp<TRAIN, 2>
            : n <= (int64_t)sms * kWarps * 4 ? launch_mlp<TRAIN, 4>
                                             : launch_mlp<TRAIN, 7>;
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
