// Blocked in-place Gauss-Jordan inversion of the condensed tangents (see eb_dense.cuh), without
// pivoting (the dynamic tangent carries the positive mass term on its diagonal, as for the band
// LU), FP32.  All marked simulations advance together, one 64-wide pivot block per step:
//   k_dense_panel   C_i = A_ik D⁻¹ for every block row i and a copy O_j of the pivot block row;
//   k_dense_update  A_ij -= C_i O_j; the pivot block row becomes D⁻¹ O_j, the pivot block column
//                   -C_i, the pivot block D⁻¹; the CTA of the next diagonal block inverts it at once.
// The kept system is a band in its order (half bandwidth b); a step leaves out the blocks past what the
// pivots so far have filled (dense_reach), whose C_i and O_j are zero: 2 (N^3 - b^3) / 3 + 2 b N^2
// operations instead of 2 N^3, the same values (304 nets of 33 x 33, N = 1,578 and b = 479: 90.9 -> 65.4 ms a
// factorisation; 512 of 20 x 20: 33.3 -> 23.6; 1,024 of 12 x 12, N = 864 and b = 77: 50.6 -> 30.4).  The
// chain is N / 64 steps of two launches.  Tiles of 128 x 128 and 128 x 64 outputs (eight by eight and eight by four a
// thread) were no faster than 64 x 64: shared memory's 16-byte reads bound both (ncu: L1 72%, FP32 41% busy).  In
// launches of many waves a tile has 64 threads with 8 x 8 outputs each (k_dense_update_many).
#include <algorithm>

#include "eb_dense.cuh"
#include "eb_launch_rules.hpp"

namespace eb {

namespace {

constexpr int kT = kDenseTile;
constexpr int kMm = 256;   // threads per CTA: 16 x 16, 4 x 4 outputs each
constexpr int kMany = 64;  // threads per CTA of k_dense_update_many: 8 x 8, 8 x 8 outputs each
constexpr int kStages = 4;
constexpr int kLd = kT + 4;

// acc (+)= Aᵀ-stored (k, m) times B (k, n), both kT x kT in shared memory with stride kLd
__device__ __forceinline__ void mm64(const float* At, const float* B, float (&acc)[4][4]) {
  const int tm = threadIdx.x >> 4, tn = threadIdx.x & 15;
#pragma unroll 8
  for (int k = 0; k < kT; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(At + k * kLd + 4 * tm);
    const float4 b = *reinterpret_cast<const float4*>(B + k * kLd + 4 * tn);
    const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
}

// 64 x 64 tile (row stride ld) into shared memory, as it is or transposed, by THR threads
template <int THR = kMm>
__device__ __forceinline__ void load_tile(float* sm, const float* g, int64_t ld) {
#pragma unroll 8
  for (int e = threadIdx.x; e < kT * kT / 4; e += THR) {
    const int r = e >> 4, c = 4 * (e & 15);
    *reinterpret_cast<float4*>(sm + r * kLd + c) = *reinterpret_cast<const float4*>(g + r * ld + c);
  }
}
template <int THR = kMm>
__device__ __forceinline__ void load_tile_t(float* sm, const float* g, int64_t ld) {
#pragma unroll 8
  for (int e = threadIdx.x; e < kT * kT / 4; e += THR) {
    const int r = e & 63, c = 4 * (e >> 6);  // lanes along the rows: the transposed stores are conflict free
    const float4 v = *reinterpret_cast<const float4*>(g + r * ld + c);
    sm[c * kLd + r] = v.x; sm[(c + 1) * kLd + r] = v.y; sm[(c + 2) * kLd + r] = v.z; sm[(c + 3) * kLd + r] = v.w;
  }
}

// Rows of group h of a 64 x 64 tile (row stride ld) into shared memory, asynchronously, by kMany threads.
__device__ __forceinline__ void copy_rows(float* sm, const float* g, int64_t ld, int h) {
  constexpr int rows = kT / kStages;
#pragma unroll
  for (int e = threadIdx.x; e < rows * kT / 4; e += kMany) {
    const int r = rows * h + (e >> 4), c = 4 * (e & 15);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sm + r * kLd + c);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(g + r * ld + c) : "memory");
  }
}

// In-place Gauss-Jordan of a 64 x 64 matrix held by the CTA: thread t has row t / 4, columns
// 16 (t % 4) .. of it in v; row buffers in shared memory, one barrier per pivot.
__device__ __forceinline__ void invert64(float (&v)[16], float* rows /* 2 x 64 */) {
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3, lane = threadIdx.x & 31;
  for (int pb = 0; pb < 4; ++pb) {
#pragma unroll
    for (int pi = 0; pi < 16; ++pi) {
      const int p = 16 * pb + pi;
      float* row = rows + (pi & 1) * kT;
      const float f = __shfl_sync(0xffffffffu, v[pi], (lane & ~3) | pb);  // a(r, p)
      if (r == p) {
        const float d = 1.f / f;
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] *= d;
        if (q == pb) v[pi] = d;
#pragma unroll
        for (int c = 0; c < 16; c += 4)
          *reinterpret_cast<float4*>(row + 16 * q + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
      }
      __syncthreads();
      if (r != p) {
        if (q == pb) v[pi] = 0.f;  // becomes -f d
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          const float4 w = *reinterpret_cast<const float4*>(row + 16 * q + c);
          v[c] = fmaf(-f, w.x, v[c]);
          v[c + 1] = fmaf(-f, w.y, v[c + 1]);
          v[c + 2] = fmaf(-f, w.z, v[c + 2]);
          v[c + 3] = fmaf(-f, w.w, v[c + 3]);
        }
      }
    }
  }
}

__device__ __forceinline__ void store_inverse(const float (&v)[16], float* dst) {
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int c = 0; c < 16; c += 4)
    *reinterpret_cast<float4*>(dst + r * kT + 16 * q + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
}

// Simulation of this CTA and its index among the simulation's `per` CTAs: everything on the grid's x
// axis, whose limit no handle reaches (y ends at 65,535).
__device__ __forceinline__ int sim_of(int per, int* i) {
  const int s = (int)(blockIdx.x / (unsigned)per);
  *i = (int)(blockIdx.x - (unsigned)s * (unsigned)per);
  return s;
}

__device__ __forceinline__ bool marked(const Dev& d, const DenseDev& g, const int* refactor, int s) {
  return g.n[s] > 0 && d.active[s] && refactor[s];
}

}  // namespace

// Zeros, with ones on the diagonal beyond N; `per` CTAs per simulation.
__global__ void k_dense_zero(Dev d, DenseDev g, const int* refactor, int per) {
  int part;
  const int s = sim_of(per, &part);
  if (!marked(d, g, refactor, s)) return;
  const int n = g.n[s], ld = dense_ld(n);
  float* G = g.G + g.off[s];
  const int64_t len = (int64_t)ld * ld;
  for (int64_t i = 4 * ((int64_t)part * blockDim.x + threadIdx.x); i < len; i += 4 * (int64_t)per * blockDim.x) {
    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    const int r = (int)(i / ld), c = (int)(i - (int64_t)r * ld);
    if (r >= n && r >= c && r < c + 4) (&z.x)[r - c] = 1.f;
    *reinterpret_cast<float4*>(G + i) = z;
  }
}

// Thread per (block among the kept nodes, entry).
__global__ void k_dense_fill(Dev d, DenseDev g, CondFactor f, const int* refactor) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.red_n * 36) return;
  const int blk = f.red[t / 36], k = (int)(t % 36);
  const int s = d.node_sim[f.rnode[blk]];
  if (!marked(d, g, refactor, s)) return;
  const int ne = f.c.ne[s], ld = dense_ld(g.n[s]);
  const int i = 6 * (f.rpos[t / 36] - ne) + k / 6, j = 6 * (f.c.scol[blk] - ne) + k % 6;
  g.G[g.off[s] + (int64_t)i * ld + j] = f.c.S[(int64_t)blk * 36 + k];
}

// The first diagonal block's inverse.
__global__ void __launch_bounds__(kMm) k_dense_first(Dev d, DenseDev g, DenseWork w, const int* refactor) {
  const int s = blockIdx.x;
  if (!marked(d, g, refactor, s)) return;
  __shared__ __align__(16) float rows[2 * kT];
  const int ld = dense_ld(g.n[s]);
  const float* A = g.G + g.off[s];
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
  float v[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) v[c] = A[(int64_t)r * ld + 16 * q + c];
  invert64(v, rows);
  store_inverse(v, w.D + (int64_t)s * 2 * kT * kT);
}

// CTA (i, s): C_i = A_ik D⁻¹ (stored transposed) and O_i = A_ki, for i != k.
__global__ void __launch_bounds__(kMm) k_dense_panel(Dev d, DenseDev g, DenseWork w, const int* refactor, int k, int per) {
  int i;
  const int s = sim_of(per, &i);
  if (!marked(d, g, refactor, s)) return;
  const int ld = dense_ld(g.n[s]);
  if (kT * k >= ld || kT * i >= ld || i == k || i >= dense_reach(k, g.b[s])) return;
  __shared__ __align__(16) float At[kT * kLd], B[kT * kLd];
  const float* A = g.G + g.off[s];
  load_tile_t(At, A + (int64_t)kT * i * ld + kT * k, ld);
  load_tile(B, w.D + ((int64_t)s * 2 + (k & 1)) * kT * kT, kT);
  float* O = w.O + w.poff[s] + kT * i;
  for (int e = threadIdx.x; e < kT * kT / 4; e += kMm) {
    const int r = e >> 4, c = 4 * (e & 15);
    *reinterpret_cast<float4*>(O + (int64_t)r * ld + c) =
        *reinterpret_cast<const float4*>(A + (int64_t)(kT * k + r) * ld + kT * i + c);
  }
  __syncthreads();
  float acc[4][4] = {};
  mm64(At, B, acc);
  const int tm = threadIdx.x >> 4, tn = threadIdx.x & 15;
  float* Ct = w.Ct + w.poff[s] + kT * i;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<float4*>(Ct + (int64_t)(4 * tn + c) * ld + 4 * tm) =
        make_float4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
}

// CTA (tile, s) of step k; the next diagonal block's tile comes first, so that its inversion
// runs beside the other tiles.
__global__ void __launch_bounds__(kMm) k_dense_update(Dev d, DenseDev g, DenseWork w, const int* refactor, int k, int side) {
  int at;
  const int s = sim_of(side * side, &at);
  if (!marked(d, g, refactor, s)) return;
  const int ld = dense_ld(g.n[s]), nb = ld / kT, reach = min(nb, dense_reach(k, g.b[s]));
  if (k >= nb || at >= reach * reach) return;  // beyond the reach C_i or O_j is zero
  const int first = k + 1 < nb ? (k + 1) * reach + k + 1 : 0;
  const int tile = at == 0 ? first : (at <= first ? at - 1 : at);
  const int i = tile / reach, j = tile - i * reach;
  __shared__ __align__(16) float At[kT * kLd], B[kT * kLd];
  __shared__ __align__(16) float rows[2 * kT];
  float* A = g.G + g.off[s] + (int64_t)kT * i * ld + kT * j;
  const float* Dk = w.D + ((int64_t)s * 2 + (k & 1)) * kT * kT;
  const float* Ct = w.Ct + w.poff[s] + kT * i;
  const float* O = w.O + w.poff[s] + kT * j;
  const int tm = threadIdx.x >> 4, tn = threadIdx.x & 15;
  if (j == k) {  // pivot block column: -C_i, or D⁻¹ itself
    for (int e = threadIdx.x; e < kT * kT; e += kMm) {
      const int r = e & 63, c = e >> 6;
      A[(int64_t)r * ld + c] = i == k ? Dk[r * kT + c] : -Ct[(int64_t)c * ld + r];
    }
    return;
  }
  if (i == k) load_tile_t(At, Dk, kT);  // D⁻¹ O_j
  else load_tile(At, Ct, ld);
  load_tile(B, O, ld);
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[a][c] = 0.f;
  float4 old[4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
    old[a] = i == k ? make_float4(0.f, 0.f, 0.f, 0.f)
                    : *reinterpret_cast<const float4*>(A + (int64_t)(4 * tm + a) * ld + 4 * tn);
  __syncthreads();
  mm64(At, B, acc);
  const float sg = i == k ? 1.f : -1.f;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float4 v = make_float4(fmaf(sg, acc[a][0], old[a].x), fmaf(sg, acc[a][1], old[a].y),
                                 fmaf(sg, acc[a][2], old[a].z), fmaf(sg, acc[a][3], old[a].w));
    *reinterpret_cast<float4*>(A + (int64_t)(4 * tm + a) * ld + 4 * tn) = v;
    old[a] = v;
  }
  if (at != 0 || k + 1 >= nb) return;
  // the next diagonal block: invert it from the updated values
  __syncthreads();  // every thread is done with At
#pragma unroll
  for (int a = 0; a < 4; ++a) *reinterpret_cast<float4*>(At + (4 * tm + a) * kLd + 4 * tn) = old[a];
  __syncthreads();
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
  float v[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) v[c] = At[r * kLd + 16 * q + c];
  invert64(v, rows);
  store_inverse(v, w.D + ((int64_t)s * 2 + ((k + 1) & 1)) * kT * kT);
}

// The same for launches of many waves, without the next diagonal block's tile (k_dense_update's): 64 threads of
// 8 x 8 outputs each, so that a k takes four 16-byte reads of shared memory for 64 multiply-adds instead of two for
// 16.  Each output's sum has the same order.  Bound by the FP32 pipe and the wait for the tiles (36 TFLOP/s at
// 48,400 tiles before their rows came in groups; 304 nets of 33 x 33: a factorisation 62 -> 55 ms, with groups 53).
__global__ void __launch_bounds__(kMany) k_dense_update_many(Dev d, DenseDev g, DenseWork w, const int* refactor, int k,
                                                             int side) {
  int tile;
  const int s = sim_of(side * side, &tile);
  if (!marked(d, g, refactor, s)) return;
  const int ld = dense_ld(g.n[s]), nb = ld / kT, reach = min(nb, dense_reach(k, g.b[s]));
  const int first = k + 1 < nb ? (k + 1) * reach + k + 1 : 0;
  if (k >= nb || tile >= reach * reach || tile == first) return;
  const int i = tile / reach, j = tile - i * reach;
  __shared__ __align__(16) float At[kT * kLd], B[kT * kLd];
  float* A = g.G + g.off[s] + (int64_t)kT * i * ld + kT * j;
  const float* Dk = w.D + ((int64_t)s * 2 + (k & 1)) * kT * kT;
  const float* Ct = w.Ct + w.poff[s] + kT * i;
  if (j == k) {  // pivot block column: -C_i, or D⁻¹ itself
    for (int e = threadIdx.x; e < kT * kT; e += kMany) {
      const int r = e & 63, c = e >> 6;
      A[(int64_t)r * ld + c] = i == k ? Dk[r * kT + c] : -Ct[(int64_t)c * ld + r];
    }
    return;
  }
  // rows of both operands in four asynchronous groups: the products of one run while the next arrive
  const float* O = w.O + w.poff[s] + kT * j;
  if (i == k) load_tile_t<kMany>(At, Dk, kT);  // D⁻¹ O_j
#pragma unroll
  for (int h = 0; h < kStages; ++h) {
    if (i != k) copy_rows(At, Ct, ld, h);
    copy_rows(B, O, ld, h);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int tm = threadIdx.x >> 3, tn = threadIdx.x & 7;  // rows and columns 4 t .. + 3 and 32 + 4 t .. + 3
  float acc[8][8];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[a][c] = 0.f;
#pragma unroll
  for (int h = 0; h < kStages; ++h) {
    if (h == 0) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (h == 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (h == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll 4
    for (int q = h * (kT / kStages); q < (h + 1) * (kT / kStages); ++q) {
      float av[8], bv[8];
      *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(At + q * kLd + 4 * tm);
      *reinterpret_cast<float4*>(av + 4) = *reinterpret_cast<const float4*>(At + q * kLd + 32 + 4 * tm);
      *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(B + q * kLd + 4 * tn);
      *reinterpret_cast<float4*>(bv + 4) = *reinterpret_cast<const float4*>(B + q * kLd + 32 + 4 * tn);
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[a][c] = fmaf(av[a], bv[c], acc[a][c]);
    }
  }
  const float sg = i == k ? 1.f : -1.f;
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4* p = reinterpret_cast<float4*>(A + (int64_t)(32 * (a >> 2) + 4 * tm + (a & 3)) * ld + 32 * h + 4 * tn);
      const float4 o = i == k ? make_float4(0.f, 0.f, 0.f, 0.f) : *p;
      const float* v = &acc[a][4 * h];
      *p = make_float4(fmaf(sg, v[0], o.x), fmaf(sg, v[1], o.y), fmaf(sg, v[2], o.z), fmaf(sg, v[3], o.w));
    }
}

int launch_dense_inverse(const Dev& d, const DenseDev& g, const DenseWork& w, const CondFactor& f,
                         const std::vector<int>& grids, int sms, const int* refactor, cudaStream_t s) {
  if (w.max_ld == 0) return 0;
  const unsigned S = (unsigned)d.n_sims;
  const int nb = w.max_ld / kT, zero = std::max(1, nb * nb / 2);
  int launches = 2;
  // float4 stores of the largest matrix over 256-thread CTAs, eight per thread
  k_dense_zero<<<zero * S, 256, 0, s>>>(d, g, refactor, zero);
  if (f.red_n) {
    k_dense_fill<<<nblocks(f.red_n * 36, 256), 256, 0, s>>>(d, g, f, refactor);
    ++launches;
  }
  k_dense_first<<<S, kMm, 0, s>>>(d, g, w, refactor);
  for (int k = 0; k < nb; ++k) {
    const int side = grids[k];
    const bool many = dense_many((int64_t)side * side * S, sms);
    if (nb > 1) k_dense_panel<<<side * S, kMm, 0, s>>>(d, g, w, refactor, k, side);
    k_dense_update<<<(many ? 1 : side * side) * S, kMm, 0, s>>>(d, g, w, refactor, k, many ? 1 : side);
    if (many) k_dense_update_many<<<side * side * S, kMany, 0, s>>>(d, g, w, refactor, k, side);
    launches += (nb > 1) + 1 + many;
  }
  return launches;
}

}  // namespace eb
