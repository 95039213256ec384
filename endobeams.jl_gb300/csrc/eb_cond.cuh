// Condensation in front of the kept nodes' explicit inverse or band LU:
// level-by-level block elimination of low-degree nodes (plan in
// eb_cond_plan.hpp) and its part of the preconditioner application.
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
  const int* lev_wide;      // beside lev_ptr: rows of many blocks, kWideFwd | kWideBwd (last: the kept rows)
  const int* solo;          // per sim: first of the last levels that one CTA walks alone
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

constexpr int kWideFwd = 1, kWideBwd = 2;
// Rows of at least this many blocks (on average over a level) are summed by a warp each, five lanes
// per row: the last levels of a net have a few dozen rows of 20 to 40 blocks, a serial chain of
// loads for one lane per row (33 x 33 net, ten levels: a backward sweep 46 us with lanes per row
// throughout, 29 us with this rule).
constexpr int kWideBlocks = 6;

// A level that one CTA of sixteen warps finishes in two rounds (positions of warps, of lanes).
constexpr int kSoloWide = 32, kSoloNarrow = 160;

// What a lane's first row of a sweep phase needs besides the vector: its blocks' range, and the
// first kAhead blocks' columns and values.  Loaded between the halves of the barrier that ends the
// previous phase (none of it changes during a solve), so that after it only the vector's loads are
// left of a chain of three; a team's barrier drops the L1 contents, so each was an L2 round trip.
// The columns of eight blocks ahead instead were no faster (48 x 200 stent: 28 and 29 us a sweep).
constexpr int kAhead = 3;
struct CondAhead {
  int b, b1;             // first and past the last block of this lane
  int col[kAhead];
  float2 s[kAhead][3];
};
template <bool FWD>
__device__ __forceinline__ void cond_ahead(const CondDev& c, int64_t base, int p0, int p1, bool wide, int warp, CondAhead& a) {
  const int lane = threadIdx.x & 31, sub = lane / 6, r = lane - 6 * sub;
  const int p = wide ? p0 + warp : p0 + 5 * warp + sub, step = wide ? 5 : 1;
  a.b = a.b1 = 0;
  if (sub >= 5 || p >= p1) return;
  const CondRange g = c.range[base + p];
  a.b = (FWD ? g.l0 : g.w0) + (wide ? sub : 0);
  a.b1 = FWD ? g.l1 : g.w1;
#pragma unroll
  for (int k = 0; k < kAhead; ++k)
    if (a.b + k * step < a.b1) {
      const int64_t b = a.b + k * step;
      const float2* s = reinterpret_cast<const float2*>(c.S + b * 36 + 6 * r);
      a.col[k] = c.scol[b];
      a.s[k][0] = s[0]; a.s[k][1] = s[1]; a.s[k][2] = s[2];
    }
}

// Rows of positions [p0, p1) of one sweep phase (`warp` of `nwarps` working together): five
// positions per warp, one lane per row, or with `wide` one position per warp, five lanes per row.  A
// position's six rows are read before any of them is written (in place unless `out` is another
// vector).  x: the simulation's permuted vector; z (backward sweep): the result in T besides;
// ahead: this phase's cond_ahead.
template <bool FWD, typename T>
__device__ __forceinline__ void cond_rows(const CondDev& c, int64_t base, int p0, int p1, bool wide, float* x, float* out,
                                          T* z, int warp, int nwarps, const CondAhead& ahead) {
  const int lane = threadIdx.x & 31;
  const int sub = lane / 6, r = lane - 6 * sub;
  const int per = wide ? 1 : 5, step = wide ? 5 : 1, first = wide ? sub : 0;
  for (int q = p0 + per * warp; q < p1; q += per * nwarps) {
    const int p = wide ? q : q + sub;
    const bool on = sub < 5 && p < p1;
    float a0 = 0.f, a1 = 0.f;
    auto add = [&](const float2 (&s)[3], int col) {
      const float2* v = reinterpret_cast<const float2*>(x + 6 * col);
      const float2 v0 = v[0], v1 = v[1], v2 = v[2];
      a0 = fmaf(s[0].x, v0.x, a0); a1 = fmaf(s[0].y, v0.y, a1);
      a0 = fmaf(s[1].x, v1.x, a0); a1 = fmaf(s[1].y, v1.y, a1);
      a0 = fmaf(s[2].x, v2.x, a0); a1 = fmaf(s[2].y, v2.y, a1);
    };
    if (on) {
      if (FWD && first == 0) a0 = x[6 * p + r];
      int b, b1;
      if (q == p0 + per * warp) {
        b = ahead.b;
        b1 = ahead.b1;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          if (b < b1) add(ahead.s[k], ahead.col[k]);
          b += step;
        }
      } else {
        const CondRange g = c.range[base + p];
        b = (FWD ? g.l0 : g.w0) + first;
        b1 = FWD ? g.l1 : g.w1;
      }
#pragma unroll 2
      for (; b < b1; b += step) {
        const float2* s = reinterpret_cast<const float2*>(c.S + (int64_t)b * 36 + 6 * r);
        const float2 sv[3] = {s[0], s[1], s[2]};
        add(sv, c.scol[b]);
      }
    }
    float y = a0 + a1;
    if (wide) {  // lanes r, r + 6 .. r + 24
      const float y1 = __shfl_sync(0xffffffffu, y, r + 6), y2 = __shfl_sync(0xffffffffu, y, r + 12),
                  y3 = __shfl_sync(0xffffffffu, y, r + 18), y4 = __shfl_sync(0xffffffffu, y, r + 24);
      y += (y1 + y2) + (y3 + y4);
    }
    __syncwarp();
    if (on && (!wide || sub == 0)) {
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
