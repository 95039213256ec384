// Condensation in front of the band LU: level-by-level block elimination of
// low-degree nodes (plan in eb_cond_plan.hpp) and its part of the
// preconditioner application.
//
// Blocks are 6x6 FP32, row-major (entry (r, c) at 6 r + c), so the thread that
// owns a row reads its 24 bytes as three 8-byte words and six neighbouring
// threads read one contiguous block.  After the factorisation the blocks of an
// eliminated position p hold D⁻¹ (first) and -D⁻¹ A(p, c) (W), and the blocks of
// a row towards earlier positions hold -A(p, e) D_e⁻¹ (L), so that both sweeps
// are plain block-row products:
//   forward   x_p += Σ_e L(p, e) x_e       (levels in increasing order, then the kept nodes)
//   backward  z_p  = D_p⁻¹ x_p + Σ_c W(p, c) z_c   (levels in decreasing order)
#pragma once
#include "eb_internal.cuh"

namespace eb {

struct CondRange {
  int w0, w1;  // blocks: diagonal, W (eliminated positions only)
  int l0, l1;  // blocks: L
};

struct CondDev {
  float* S;                 // blocks, 36 floats each
  const int* scol;          // per block: position of its column in its simulation
  const CondRange* range;   // per global position (node_off[s] + p)
  const int* ne;            // per sim: eliminated nodes
  const int* lev_off;       // per sim (n_sims + 1): its range in lev_ptr
  const int* lev_ptr;       // per sim: first position of each level, then ne
  const int64_t* roff;      // per sim (n_sims + 1): kept nodes before it (offsets of the diagonal-block inverses)
};

// Lists of the numeric factorisation (kernel arguments of the launches below).
struct CondFactor {
  CondDev c;
  int64_t n_blocks;
  const int* src;           // per block: BSR block of the tangent, -1 = fill
  const int* rnode;         // per block: global node of its row
  const int* cnode;         // per block: global node of its column
  const int* ldiag;         // per block: diagonal block of its column for L blocks, else -1
  const int* elim;          // global positions of the eliminated nodes, level by level over all simulations
  const int* elim_node;     // their global nodes
  const int* tgt;           // target blocks, level by level
  const int* tptr;          // per target: its range of cl / cw
  const int* cl;
  const int* cw;
  int64_t red_n;            // blocks among the kept nodes
  const int* red;           // their block ids
  const int* rpos;          // positions of their rows
};

// Rows of positions [p0, p1) of one sweep phase, five positions per warp (`warp` of `nwarps`
// working together), a position's six rows read before any of them is written (x is updated
// in place unless `out` is another vector).  x: the simulation's permuted vector; z (backward
// sweep): the result in T besides.
template <bool FWD, typename T>
__device__ __forceinline__ void cond_rows(const CondDev& c, int64_t base, int p0, int p1, float* x, float* out, T* z,
                                          int warp, int nwarps) {
  const int lane = threadIdx.x & 31;
  const int sub = lane / 6, r = lane - 6 * sub;
  for (int q = p0 + 5 * warp; q < p1; q += 5 * nwarps) {
    const int p = q + sub;
    const bool on = sub < 5 && p < p1;
    float a0 = 0.f, a1 = 0.f;
    if (on) {
      const CondRange g = c.range[base + p];
      if (FWD) a0 = x[6 * p + r];
      const int b0 = FWD ? g.l0 : g.w0, b1 = FWD ? g.l1 : g.w1;
      for (int b = b0; b < b1; ++b) {
        const float2* s = reinterpret_cast<const float2*>(c.S + (int64_t)b * 36 + 6 * r);
        const float2* v = reinterpret_cast<const float2*>(x + 6 * c.scol[b]);
        const float2 s0 = s[0], s1 = s[1], s2 = s[2], v0 = v[0], v1 = v[1], v2 = v[2];
        a0 = fmaf(s0.x, v0.x, a0); a1 = fmaf(s0.y, v0.y, a1);
        a0 = fmaf(s1.x, v1.x, a0); a1 = fmaf(s1.y, v1.y, a1);
        a0 = fmaf(s2.x, v2.x, a0); a1 = fmaf(s2.y, v2.y, a1);
      }
    }
    __syncwarp();
    if (on) {
      const float y = a0 + a1;
      out[6 * p + r] = y;
      if (!FWD) z[6 * p + r] = (T)y;
    }
  }
}

// The tangent's blocks into S, the level-by-level elimination and the final scaling of the L
// blocks, for the active simulations marked in `refactor`.  lev_elim / lev_tgt: host offsets of
// every level in elim / tgt.  The kept nodes' Schur complement is left in S for k_band_fill.
struct CondLevels {
  const int64_t *elim_off, *tgt_off;  // n + 1 each
  int n;
};
void launch_cond_factor(const Dev& d, const CondFactor& f, const CondLevels& lv, const int* refactor, cudaStream_t s);

}  // namespace eb
