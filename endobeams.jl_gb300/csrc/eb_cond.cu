// Numeric condensation kernels (see eb_cond.cuh).
#include "eb_cond.cuh"

namespace eb {

// Thread per (block, entry): the tangent's block (column-major FP64) as FP32 row-major; fixed
// DOFs become identity rows/columns (the free-DOF system of extract_free_dofs!,
// src/utils_solver.jl:94-102, embedded in the full size); fill blocks start at zero.
__global__ void k_cond_fill(Dev d, CondFactor f, const int* __restrict__ refactor) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.n_blocks * 36) return;
  const int64_t blk = t / 36;
  const int k = (int)(t - 36 * blk);
  const int rn = f.rnode[blk];
  const int s = d.node_sim[rn];
  if (!d.active[s] || !refactor[s]) return;
  const int src = f.src[blk], r = k / 6, c = k - 6 * r;
  const int64_t gr = 6 * (int64_t)rn + r, gc = 6 * (int64_t)f.cnode[blk] + c;
  float v = src >= 0 ? (float)d.Kt[(int64_t)src * 36 + 6 * c + r] : 0.f;
  if (d.fixed[gr] || d.fixed[gc]) v = gr == gc ? 1.f : 0.f;
  f.c.S[t] = v;
}

// Warp per eliminated node: Gauss-Jordan with partial pivoting on [D | I | A(p, c) ...], one
// column per lane (lanes 0-5 carry D, the others up to 26 right-hand columns at a time); D is
// overwritten by D⁻¹ and A(p, c) by -D⁻¹ A(p, c).
__global__ void __launch_bounds__(128) k_cond_elim(Dev d, CondFactor f, const int* __restrict__ refactor, int64_t q0,
                                                   int64_t q1) {
  const int64_t q = q0 + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  if (q >= q1) return;
  const int s = d.node_sim[f.elim_node[q]];
  if (!d.active[s] || !refactor[s]) return;
  const int lane = threadIdx.x & 31;
  const CondRange g = f.c.range[f.elim[q]];
  float* D = f.c.S + (int64_t)g.w0 * 36;
  float dc[6];  // lanes 0-5: a column of D
#pragma unroll
  for (int r = 0; r < 6; ++r) dc[r] = lane < 6 ? D[6 * r + lane] : 0.f;
  __syncwarp();
  const int ncol = 6 * (g.w1 - g.w0);  // identity (in D's place) and the W blocks' columns
  for (int c0 = 0; c0 < ncol; c0 += 26) {
    const int c = c0 + lane - 6;
    const bool rhs = lane >= 6 && c < ncol;
    float* col = f.c.S + ((int64_t)g.w0 + (rhs ? c / 6 : 0)) * 36 + (rhs ? c % 6 : 0);
    float a[6];
#pragma unroll
    for (int r = 0; r < 6; ++r) a[r] = lane < 6 ? dc[r] : (!rhs ? 0.f : (c < 6 ? (c == r ? 1.f : 0.f) : col[6 * r]));
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      float m[6];  // column k of D as it stands
#pragma unroll
      for (int r = 0; r < 6; ++r) m[r] = __shfl_sync(0xffffffffu, a[r], k);
      int p = k;
      float best = fabsf(m[k]);
#pragma unroll
      for (int r = k + 1; r < 6; ++r)
        if (fabsf(m[r]) > best) { best = fabsf(m[r]); p = r; }
#pragma unroll
      for (int r = k + 1; r < 6; ++r)
        if (p == r) {
          float t = a[k]; a[k] = a[r]; a[r] = t;
          t = m[k]; m[k] = m[r]; m[r] = t;
        }
      const float pk = a[k] / m[k];
#pragma unroll
      for (int r = 0; r < 6; ++r) a[r] = r == k ? pk : fmaf(-m[r], pk, a[r]);
    }
    if (rhs) {
      const float sg = c < 6 ? 1.f : -1.f;
#pragma unroll
      for (int r = 0; r < 6; ++r) col[6 * r] = sg * a[r];
    }
    __syncwarp();
  }
}

// Thread per (target block, entry): S_t += Σ L W over the level's nodes in elimination order
// (L = A(r, e) not yet scaled, W = -D⁻¹ A(e, c)).
__global__ void k_cond_update(Dev d, CondFactor f, const int* __restrict__ refactor, int64_t t0, int64_t t1) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t q = t0 + i / 36;
  if (q >= t1) return;
  const int k = (int)(i % 36), r = k / 6, c = k - 6 * r;
  const int t = f.tgt[q];
  const int s = d.node_sim[f.rnode[t]];
  if (!d.active[s] || !refactor[s]) return;
  float acc = f.c.S[(int64_t)t * 36 + k];
  for (int u = f.tptr[q]; u < f.tptr[q + 1]; ++u) {
    const float* L = f.c.S + (int64_t)f.cl[u] * 36 + 6 * r;
    const float* W = f.c.S + (int64_t)f.cw[u] * 36 + c;
#pragma unroll
    for (int j = 0; j < 6; ++j) acc = fmaf(L[j], W[6 * j], acc);
  }
  f.c.S[(int64_t)t * 36 + k] = acc;
}

// Thread per (L block, row): L <- -A(r, e) D_e⁻¹, in place.
__global__ void k_cond_scale(Dev d, CondFactor f, const int* __restrict__ refactor) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= f.n_blocks * 6) return;
  const int64_t blk = t / 6;
  const int dg = f.ldiag[blk];
  if (dg < 0) return;
  const int s = d.node_sim[f.rnode[blk]];
  if (!d.active[s] || !refactor[s]) return;
  float* row = f.c.S + blk * 36 + 6 * (t - 6 * blk);
  const float* D = f.c.S + (int64_t)dg * 36;
  float a[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) a[j] = row[j];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < 6; ++j) v = fmaf(a[j], D[6 * j + c], v);
    row[c] = -v;
  }
}

void launch_cond_factor(const Dev& d, const CondFactor& f, const CondLevels& lv, const int* refactor, cudaStream_t s) {
  if (f.n_blocks == 0) return;
  k_cond_fill<<<nblocks(f.n_blocks * 36, 256), 256, 0, s>>>(d, f, refactor);
  for (int l = 0; l < lv.n; ++l) {
    const int64_t q0 = lv.elim_off[l], q1 = lv.elim_off[l + 1], t0 = lv.tgt_off[l], t1 = lv.tgt_off[l + 1];
    if (q1 > q0) k_cond_elim<<<nblocks((q1 - q0) * 32), kThreads, 0, s>>>(d, f, refactor, q0, q1);
    if (t1 > t0) k_cond_update<<<nblocks((t1 - t0) * 36, 288), 288, 0, s>>>(d, f, refactor, t0, t1);
  }
  k_cond_scale<<<nblocks(f.n_blocks * 6, 256), 256, 0, s>>>(d, f, refactor);
}

}  // namespace eb
