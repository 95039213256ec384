// Explicit inverse of the condensed tangent: where the condensation keeps few
// enough nodes, the kept system K_r (N x N) is inverted once per
// factorisation and the preconditioner applies it as one dense product,
// instead of two chains of N / 32 dependent block steps on one SM.
//
// The line is drawn at N = kDenseMax = 2048 by both sides' times: at N = 1782 (48-wire
// stent, b = 443) the band sweeps took 0.27 ms an application on one SM, the product reads
// 12.7 MB from L2 over the simulation's whole team (about 12 us on 16 SMs); the 2 N^3
// operations of the inversion grow past the band LU's latency beyond it, and its memory
// (4 N^2 bytes) past the band's.
#pragma once
#include <vector>

#include "eb_cond.cuh"

namespace eb {

constexpr int kDenseMax = 2048;
constexpr int kDenseTile = 64;

struct DenseDev {
  float* G;             // row-major ld x ld matrices, ld = N rounded up to 64 (identity beyond N)
  const int64_t* off;   // per sim: offset of its matrix in G
  const int* n;         // per sim: N, 0 = not dense
  const int* b;         // per sim: half bandwidth of the kept system before its inversion
};

__host__ __device__ __forceinline__ int dense_ld(int n) { return (n + kDenseTile - 1) / kDenseTile * kDenseTile; }

struct DenseWork {
  float *Ct, *O, *D;    // per sim: scaled pivot block column (transposed, 64 x ld), old pivot block row
                        // (64 x ld), inverses of two consecutive diagonal blocks (2 x 64 x 64)
  const int64_t* poff;  // per sim: offset in Ct and O (64 x the ld of the simulations before)
  int max_ld;           // largest ld of the handle, 0 = no dense simulation
};

// grids: dense_grids of the handle's simulations; sms: the device's multiprocessors.
// Returns the number of launches.
int launch_dense_inverse(const Dev& d, const DenseDev& g, const DenseWork& w, const CondFactor& f,
                         const std::vector<int>& grids, int sms, const int* refactor, cudaStream_t s);

// Rows of z = G x by whole warps, four rows at a time (x in shared memory, ld entries, zero
// beyond N); a row's sum has one order, whatever the number of warps.
template <typename T>
__device__ __forceinline__ void dense_rows(const float* __restrict__ G, int n, int ld, const float* xsm, float* xk, T* zk,
                                           int warp, int nwarps) {
  const int lane = threadIdx.x & 31;
  for (int r0 = 4 * warp; r0 < n; r0 += 4 * nwarps) {  // rows up to ld exist
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const float* row = G + (int64_t)r0 * ld;
#pragma unroll 4
    for (int c = 4 * lane; c < ld; c += 128) {
      const float4 v = *reinterpret_cast<const float4*>(xsm + c);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 m = __ldg(reinterpret_cast<const float4*>(row + (int64_t)u * ld + c));
        acc[u] = fmaf(m.x, v.x, acc[u]);
        acc[u] = fmaf(m.y, v.y, acc[u]);
        acc[u] = fmaf(m.z, v.z, acc[u]);
        acc[u] = fmaf(m.w, v.w, acc[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
      if (lane == u && r0 + u < n) {
        xk[r0 + u] = acc[u];
        zk[r0 + u] = (T)acc[u];
      }
    }
  }
}

}  // namespace eb
