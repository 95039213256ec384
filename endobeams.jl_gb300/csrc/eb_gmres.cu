// Linear solve of the Newton step, replacing MKL PARDISO (src/linearsolvers.jl,
// called from solve_free_dofs!, src/utils_solver.jl:107-120).
//
// Ktan_free ΔD_free = r_free is solved per simulation by right-preconditioned
// GMRES; the preconditioner is the condensation with the explicit inverse or the
// band LU of the kept nodes (eb_cond.cuh, eb_dense.cuh, eb_band.cuh) or 6x6
// block-Jacobi (the LU of each node's diagonal block, fixed DOFs replaced by
// identity rows/columns).  Each
// simulation is owned by one team of CTAs (a cluster of 1 to 16, so that few
// simulations use many SMs) for the whole solve: its Krylov basis lives in
// global memory in the preconditioner's node order, its Hessenberg matrix and
// Givens rotations in every CTA's shared memory, and every sum has an order
// fixed by the simulation's size, so results do not depend on how many CTAs
// work on a simulation or how many simulations share the launch.
//
// Precision: the outer loop always measures the true residual b - A x in
// FP64.  Each pass runs one GMRES(m) cycle on that residual, in FP64
// (EB_PREC_FP64) or with an FP32 basis and preconditioner, the products with the
// tangent in FP32 pairs (EB_PREC_MIXED: iterative refinement).  A pass is therefore
// both the GMRES restart and the refinement sweep.
#include <cfloat>
#include <type_traits>

#include "eb_band.cuh"
#include "eb_gmres.cuh"
#include "eb_launch_rules.hpp"

namespace eb {

// The CTAs of one simulation: a cluster of `size` (1: a single CTA).
struct Team {
  int rank, size;
  // Barrier in two halves: what needs no other CTA's results is loaded between them.  Release /
  // acquire at cluster scope: global and shared writes of the other CTAs are seen after wait().
  __device__ __forceinline__ void arrive() const {
    if (size > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  }
  __device__ __forceinline__ void wait() const {
    if (size > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    else __syncthreads();
  }
  __device__ __forceinline__ void sync() const {
    arrive();
    wait();
  }
};

// Vectors are cut into chunks whose length depends on the simulation alone (at most
// kMaxChunks of them); a warp owns whole chunks, and sums are formed chunk by chunk and then
// over the chunks in one fixed order, so no result depends on the number of CTAs or threads.
constexpr int kMaxChunks = 256;
__device__ __forceinline__ int chunk_len(int n) { return ((n + kMaxChunks - 1) / kMaxChunks + 31) / 32 * 32; }

struct Work {
  Team t;
  int n, ch, nchunk;     // DOFs, chunk length, chunks
  int warp0, nwarps;     // this warp's first chunk, stride between its chunks
  double* part[2];       // chunk sums of a reduction (kMaxChunks x SolverArgs::dots), used in turn
  double* sums;          // 8
  int flip;
  template <typename F>
  __device__ __forceinline__ void each(F f) const {  // f(i) over this warp's chunks
    const int lane = threadIdx.x & 31;
    for (int c = warp0; c < nchunk; c += nwarps) {
      const int i1 = min(n, (c + 1) * ch);
      for (int i = c * ch + lane; i < i1; i += 32) f(i);
    }
  }
};

// Sums NQ values over the warp, NQ a power of two: while a lane holds several values it keeps half of
// them and sends the others' partial sums to the lane that keeps those, so that eight values take 9
// FP64 additions instead of 40 (each holds the SM's FP64 pipe for 16 cycles).  Afterwards the
// lanes q (32 / NQ) .. hold the sum of value q.
template <int NQ>
__device__ __forceinline__ double warp_sums(const double (&in)[NQ]) {
  const int lane = threadIdx.x & 31;
  double v[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) v[q] = in[q];
#pragma unroll
  for (int off = 16, cnt = NQ; off > 0; off >>= 1) {
    if (cnt > 1) {
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int q = 0; q < cnt / 2; ++q) {
        const double keep = up ? v[q + cnt / 2] : v[q], send = up ? v[q] : v[q + cnt / 2];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
      cnt /= 2;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  return v[0];
}

// out[q] = Σ_i of what f(i, acc) adds to acc[q]: per lane in TA, over lanes and chunks in FP64.  Each
// chunk's sums go to every CTA of the team; one team barrier; two buffers in turn, so that a CTA
// that is ahead does not overwrite sums that another still reads.  root: out is the sum's square
// root, with its reciprocal left in w.sums[NQ + q] (one thread's work: a square root and a division
// by every warp of a CTA hold the FP64 pipe for 2 us).
template <int NQ, typename TA, typename F>
__device__ __forceinline__ void team_sum(Work& w, double (&out)[NQ], F f, bool root = false) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  constexpr int G = 32 / NQ;  // lanes that hold the same sum
  double* part = w.flip ? w.part[1] : w.part[0];
  w.flip ^= 1;
  for (int c = w.warp0; c < w.nchunk; c += w.nwarps) {
    TA acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0;
    const int i1 = min(w.n, (c + 1) * w.ch);
#pragma unroll 4
    for (int i = c * w.ch + lane; i < i1; i += 32) f(i, acc);
    double v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = (double)acc[q];
    const double sum = warp_sums<NQ>(v);
    double* mine = part + lane / G * kMaxChunks + c;
    if (w.t.size == 1) {
      if (lane % G == 0) *mine = sum;
    } else {  // the lanes of a sum write the CTAs' copies
      for (int r = lane % G; r < w.t.size; r += G) {
        uint32_t a;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(mine)), "r"(r));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(sum) : "memory");
      }
    }
  }
  w.t.sync();
  for (int q = warp; q < NQ; q += nw) {
    double s = 0.0;
    for (int c = lane; c < w.nchunk; c += 32) s += part[q * kMaxChunks + c];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) {
      if (root) s = sqrt(s);
      w.sums[q] = s;
      if (root) w.sums[q + NQ] = 1.0 / s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) out[q] = w.sums[q];
}

// Row i of P A x in FP64 (P zeroes fixed rows); vectors are in the solver's order.
template <typename TX>
__device__ __forceinline__ double row64(const SolverArgs& a, int64_t n0, int i, const TX* x) {
  const int p = i / 6, k = i - 6 * p;
  if ((a.pfix[n0 + p] >> k) & 1) return 0.0;
  const int2 blocks = a.prow[n0 + p];
  double acc0 = 0.0, acc1 = 0.0;
  for (int bb = blocks.x; bb < blocks.y; ++bb) {
    const double* Ab = a.Kt + (int64_t)bb * 36 + k;
    const TX* xc = x + 6 * a.pcol[bb];
#pragma unroll
    for (int j = 0; j < 6; j += 2) {
      acc0 += Ab[6 * j] * (double)xc[j];
      acc1 += Ab[6 * j + 6] * (double)xc[j + 1];
    }
  }
  return acc0 + acc1;
}

// The same row from the tangent as FP32 pairs (hi + lo carry 48 bits of it), summed as FP32
// pairs (exact products by FMA, Knuth's two-sum): an FP64 sum's error in FP32 operations, of
// which an SM does 64 times as many.  With plain FP32 products the Arnoldi relation was off by
// 1e-4 of the residual and most solves to 1e-4 ended just above their target, one cycle more
// each (24-wire stent: 12 cycles and 36 iterations a step, now 6 and 32).
__device__ __forceinline__ float row_pairs(const SolverArgs& a, int64_t n0, int i, const float* x) {
  const int p = i / 6, k = i - 6 * p;
  if ((a.pfix[n0 + p] >> k) & 1) return 0.f;
  const int2 blocks = a.prow[n0 + p];
  float hi = 0.f, lo = 0.f;
  for (int bb = blocks.x; bb < blocks.y; ++bb) {
    const float2* Ab = a.Ktp + (int64_t)bb * 36 + k;
    const float* xc = x + 6 * a.pcol[bb];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const float2 e = Ab[6 * j];
      const float xv = xc[j];
      const float q = __fmul_rn(e.x, xv), qe = __fmaf_rn(e.x, xv, -q);
      const float s = __fadd_rn(hi, q), t = __fsub_rn(s, hi);
      const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(q, t));
      hi = s;
      lo = __fadd_rn(lo, __fadd_rn(err, __fmaf_rn(e.y, xv, qe)));
    }
  }
  return hi + lo;
}

template <typename T>
__global__ void __launch_bounds__(kGmresMaxThreads) k_gmres(SolverArgs a) {
  Work wk;
  {
    uint32_t r, c;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(c));
    wk.t = Team{(int)r, (int)c};
  }
  const Team& team = wk.t;
  const int warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int s = a.cta_sim[blockIdx.x / team.size];
  if (!a.active[s]) return;
  const int m = a.m;
  const int64_t n0 = a.sim_node_off[s];
  const int64_t o = 6 * n0;
  const int n = (int)(6 * (a.sim_node_off[s + 1] - n0));
  extern __shared__ double sm[];
  double* H = sm;                  // (m+1) x m, column j at H + (m+1) j; every CTA keeps its own copy
  double* cs = H + (m + 1) * m;
  double* sn = cs + m;
  double* g = sn + m;              // m+1
  double* y = g + m + 1;           // m + 1
  T* yt = reinterpret_cast<T*>(y + m + 1);  // y in the cycle's precision
  wk.part[0] = y + 2 * m + 2;
  wk.part[1] = wk.part[0] + a.dots * kMaxChunks;
  wk.sums = wk.part[1] + a.dots * kMaxChunks;  // 16
  wk.flip = 0;
  wk.n = n;
  wk.ch = chunk_len(n);
  wk.nchunk = (n + wk.ch - 1) / wk.ch;
  wk.warp0 = team.rank + team.size * (threadIdx.x >> 5);  // neighbouring work on different CTAs
  wk.nwarps = team.size * (blockDim.x >> 5);
  T* V = reinterpret_cast<T*>(a.V) + (int64_t)(m + 1) * o;
  T* Zb = reinterpret_cast<T*>(a.Z) + (int64_t)m * o;  // z_j = M⁻¹ v_j at Zb + j n
  double* X = a.X + o;
  double* R = a.R64 + o;
  // the vector the preconditioner works on, z_j and w: in shared memory where one CTA owns a small
  // simulation (every phase reads what another thread has just written, an L2 round trip each)
  const bool vs = a.vec_smem > 0 && team.size == 1;
  float* xa = a.band.work + o;
  const int* node_at = a.band.node_at + n0;
  auto dof = [&](int i) { return 6 * (int64_t)node_at[i / 6] + i % 6; };  // caller's DOF of entry i
  const T* Dm = std::is_same<T, double>::value ? reinterpret_cast<const T*>(a.Dinv64)
                                              : reinterpret_cast<const T*>(a.Dinv32);
  const bool use_band = a.band.bw != nullptr && a.band.bw[s] > 0;
  const int dn = a.dense.n[s];     // kept DOFs of the explicit inverse, 0 = none
  const CondDev& cd = a.band.cond;
  const int ne = cd.ne[s];
  const int* lev = cd.lev_ptr + cd.lev_off[s];
  const int* wide = cd.lev_wide + cd.lev_off[s];
  const int nlev = max(0, cd.lev_off[s + 1] - cd.lev_off[s] - 1);
  // the dense product's input, dense_ld entries, read as float4
  float* xd = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(wk.sums + 16) + 15) & ~uintptr_t(15));
  float* xs = a.x_in_smem ? xd + a.dense_ld + a.vec_smem : nullptr;  // the kept entries during the band sweeps
  T* zs = reinterpret_cast<T*>(xd + a.dense_ld);  // vec_smem floats: z_j, w, xa
  T* ws = zs + n;
  if (vs) xa = reinterpret_cast<float*>(ws + n);
  // shared-memory staging of band blocks for the triangular solves (bulk async copies)
  __shared__ __align__(8) uint64_t bars[4];
  __shared__ int stage_fail;
  __shared__ int stage_pend[4];
  Stage stage;
  const Stage* stp = nullptr;
  uint32_t ph = 0u;  // bit k: next phase of staging barrier k
  if (use_band && a.stage_floats > 0 && team.rank == 0) {
    char* base = reinterpret_cast<char*>(xd + a.dense_ld + a.vec_smem + (xs ? a.max_n : 0));
    base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(base) + 127) & ~uintptr_t(127));
    // two band-column buffers of stage_floats = 32 (b_max + 1) floats, then the inverses
    float* f = reinterpret_cast<float*>(base);
    stage.buf[0] = f;
    stage.buf[1] = f + a.stage_floats;
    stage.inv[0] = f + 2 * (int64_t)a.stage_floats;
    stage.inv[1] = stage.inv[0] + kPanel * kPanel;
    stage.bar = bars;
    stage.fail = &stage_fail;
    stage.pend = stage_pend;
    stage.extra = (uint32_t)a.stage_test_extra;
    if (threadIdx.x == 0) {
      for (int k = 0; k < 4; ++k) {
        mbar_init(&bars[k], 1);
        stage_pend[k] = -1;
      }
      stage_fail = 0;
      fence_async_smem();
    }
    __syncthreads();
    stp = &stage;
  }
  team.sync();  // every CTA of the team runs before any writes another's shared memory

  const bool use_x0 = a.x0_on != nullptr && a.x0_on[s] != 0;
  double v1[1];
  team_sum<1, double>(wk, v1, [&](int i, double (&q)[1]) {
    const int64_t d = dof(i);
    const bool fx = a.fixed[d];
    const double bi = fx ? 0.0 : a.b[d];
    X[i] = (use_x0 && !fx) ? a.dD[d] : 0.0;
    R[i] = bi;
    q[0] += bi * bi;
  }, true);
  const double bnorm = v1[0];
  double rnorm = bnorm;
  if (use_x0 && isfinite(bnorm)) {
    // initial guess: X = α x0 with α = <A x0, b> / <A x0, A x0> clipped to [0, 1], so that
    // ‖b − A X‖ <= ‖b‖ (a guess that does not help costs one FP64 product)
    double yb[2];
    team_sum<2, double>(wk, yb, [&](int i, double (&q)[2]) {
      const double bi = R[i], ax = row64(a, n0, i, X);
      q[0] += ax * bi;
      q[1] += ax * ax;
    });
    double alpha = yb[1] > 0.0 ? yb[0] / yb[1] : 0.0;
    if (!(alpha > 0.0)) alpha = 0.0;
    if (alpha > 1.0) alpha = 1.0;
    team_sum<1, double>(wk, v1, [&](int i, double (&q)[1]) {
      const double ri = R[i] - alpha * row64(a, n0, i, X);
      R[i] = ri;
      q[0] += ri * ri;
    }, true);
    wk.each([&](int i) { X[i] *= alpha; });
    rnorm = v1[0];
  }
  int its = 0, refs = 0, status = 0;
  if (!isfinite(bnorm)) status = 2;  // EB_SIM_NAN
  // the tensor-core factorisation of these factors stopped at a bounded wait: not trusted
  if (use_band && a.band.lu_fail && a.band.lu_fail[s]) status = 4;

  // relative tolerance of this solve (inexact Newton, Eisenstat-Walker choice 2)
  double rtol = a.tol;
  if (a.forcing) {
    const double prev = a.prev_bnorm[s], pe = a.prev_eta[s];
    double eta = a.forcing_max;
    if (prev > 0.0) {
      const double q = bnorm / prev;
      eta = 0.9 * q * q;
      if (0.9 * pe * pe > 0.1) eta = fmax(eta, 0.9 * pe * pe);
      eta = fmin(fmax(eta, a.tol), a.forcing_max);
    }
    rtol = eta;
    team.sync();  // every thread has read the previous values
    if (threadIdx.x == 0 && team.rank == 0) {
      a.prev_bnorm[s] = bnorm;
      a.prev_eta[s] = eta;
    }
  }
  if (status == 0 && bnorm > 0.0) {
    const double target = rtol * bnorm;
    for (int ref = 0; ref < a.max_ref && rnorm > target && its < a.max_iter; ++ref) {
      // ---- one GMRES(m) cycle on the FP64 residual R
      const double beta = rnorm;
      const double ib = wk.sums[1];  // 1 / beta: beta is the last sum's root
      wk.each([&](int i) {
        const T v = (T)(R[i] * ib);
        V[i] = v;
        xa[i] = (float)v;
      });
      if (threadIdx.x == 0) g[0] = beta;
      CondAhead ahead;
      auto first_ahead = [&] {
        const int l = min(1, nlev);
        if (use_band || dn)
          cond_ahead<true>(cd, n0, l < nlev ? lev[l] : ne, l < nlev ? lev[l + 1] : n / 6, wide[l] & kWideFwd, wk.warp0, ahead);
      };
      team.arrive();
      first_ahead();
      team.wait();
      // a cycle that can reach the target aims at half of it, from zero as from an initial guess: its
      // estimate differs from the true residual by rounding, and a residual left just above the
      // target costs another cycle
      double inner_target = a.inner_tol * beta;
      if (inner_target <= target) inner_target = 0.5 * target;
      int k = 0;  // dimension of the Krylov space built in this cycle
      const int jmax = min(m, a.max_iter - its);
      for (int j = 0; j < jmax; ++j) {
        T* vn = V + (int64_t)(j + 1) * n;
        T* w = vs ? ws : vn;
        T* zg = Zb + (int64_t)j * n;
        T* zj = vs ? zs : zg;
        // ---- z_j = M⁻¹ v_j; v_j lies in xa (FP32) when the preconditioner starts
        if (use_band || dn) {
          // phases: forward levels 1 .. (level 0 receives nothing), the kept rows (phase nlev), the kept
          // system, backward levels; `ahead` always holds the next phase's first blocks
          auto fwd_ahead = [&](int l) {
            cond_ahead<true>(cd, n0, l < nlev ? lev[l] : ne, l < nlev ? lev[l + 1] : n / 6, wide[l] & kWideFwd, wk.warp0, ahead);
          };
          auto bwd_ahead = [&](int l) {
            if (l >= 0) cond_ahead<false>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideBwd, wk.warp0, ahead);
          };
          float* kin = dn ? a.kin + 6 * cd.roff[s] - 6 * ne : xa;
          // levels from `solo` on are so small that one CTA walks them faster by its own barriers (1.1
          // us a phase on a ring, whose levels are all that small) than the team by its own (2.4 us)
          const int solo = team.size > 1 ? max(1, cd.solo[s]) : nlev;
          for (int l = 1; l < min(solo, nlev); ++l) {
            cond_rows<true>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideFwd, xa, xa, (T*)nullptr, wk.warp0, wk.nwarps, ahead);
            team.arrive();
            if (l + 1 < solo || solo >= nlev) fwd_ahead(l + 1);
            team.wait();
          }
          if (solo < nlev) {
            if (team.rank == 0)
              for (int l = solo; l < nlev; ++l) {
                cond_ahead<true>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideFwd, warp, ahead);
                if (l > solo) __syncthreads();
                cond_rows<true>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideFwd, xa, xa, (T*)nullptr, warp, nwarp, ahead);
              }
            team.arrive();
            fwd_ahead(nlev);
            team.wait();
          }
          cond_rows<true>(cd, n0, ne, n / 6, wide[nlev] & kWideFwd, xa, kin, (T*)nullptr, wk.warp0, wk.nwarps, ahead);
          team.sync();
          if (dn) {
            const int ld = dense_ld(dn);
            for (int i = threadIdx.x; i < ld; i += blockDim.x) xd[i] = i < dn ? kin[6 * ne + i] : 0.f;
            __syncthreads();
            dense_rows(a.dense.G + a.dense.off[s], dn, ld, xd, xa + 6 * ne, zj + 6 * ne, wk.warp0, wk.nwarps);
          } else {
            if (team.rank == 0) band_sweeps(a.band, s, xa + 6 * ne, xs, stp, ph);
            team.sync();
            for (int i = 6 * ne + wk.warp0 * 32 + (threadIdx.x & 31); i < n; i += 32 * wk.nwarps) zj[i] = (T)xa[i];
          }
          team.arrive();
          if (solo >= nlev) bwd_ahead(nlev - 1);
          team.wait();
          if (solo < nlev) {
            if (team.rank == 0)
              for (int l = nlev - 1; l >= solo; --l) {
                cond_ahead<false>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideBwd, warp, ahead);
                if (l < nlev - 1) __syncthreads();
                cond_rows<false>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideBwd, xa, xa, zj, warp, nwarp, ahead);
              }
            team.arrive();
            bwd_ahead(solo - 1);
            team.wait();
          }
          for (int l = min(solo, nlev) - 1; l >= 0; --l) {
            cond_rows<false>(cd, n0, lev[l], lev[l + 1], wide[l] & kWideBwd, xa, xa, zj, wk.warp0, wk.nwarps, ahead);
            team.arrive();
            bwd_ahead(l - 1);
            team.wait();
          }
        } else {
          const T* vj = V + (int64_t)j * n;
          wk.each([&](int i) {
            const int p = i / 6, r = i - 6 * p;
            const T* Db = Dm + (int64_t)node_at[p] * 36 + r;
            T acc = 0;
#pragma unroll
            for (int q = 0; q < 6; ++q) acc += Db[6 * q] * vj[6 * p + q];
            zj[i] = acc;
          });
          team.sync();
        }
        // ---- w = A z_j, orthogonalised by classical Gram-Schmidt, twice
        wk.each([&](int i) {
          if constexpr (std::is_same<T, double>::value) w[i] = row64(a, n0, i, zj);
          else w[i] = row_pairs(a, n0, i, zj);
          if (vs) zg[i] = zj[i];
        });
        __syncwarp();
        // The second pass also forms w·w: ‖w - Σ y v‖² = w·w - Σ y², of which the first pass has left next
        // to nothing to subtract, so that its update can normalise w at once.
        for (int pass = 0; pass < 2; ++pass) {
          const int last = j + pass;  // in the second pass, "v_(j+1)" is w itself
          for (int i0 = 0; i0 <= last;) {
            // inner products with v_i0 .., as many at a time as are left (at most a.dots; a sum's order
            // does not depend on how many there are)
            auto dots = [&](auto width) {
              constexpr int NQ = decltype(width)::value;
              const int nq = min(NQ, last + 1 - i0);
              const T* Vq = V + (int64_t)i0 * n;
              double hp[NQ];
              team_sum<NQ, T>(wk, hp, [&](int i, T (&q)[NQ]) {
                const T wi = w[i];
#pragma unroll
                for (int u = 0; u < NQ; ++u)
                  if (u < nq) q[u] += (i0 + u > j ? wi : Vq[(int64_t)u * n + i]) * wi;
              });
              if (threadIdx.x == 0)
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                  if (q < nq) {
                    y[i0 + q] = hp[q];
                    if (i0 + q <= j) {
                      double* h = H + (m + 1) * j + i0 + q;
                      *h = (pass == 0 ? 0.0 : *h) + hp[q];
                      yt[i0 + q] = (T)hp[q];  // this pass's coefficients
                    }
                  }
              i0 += NQ;
            };
            const int left = last + 1 - i0;
            if (left > 4 && a.dots > 4) dots(std::integral_constant<int, 8>{});
            else if (left > 2) dots(std::integral_constant<int, 4>{});
            else if (left > 1) dots(std::integral_constant<int, 2>{});
            else dots(std::integral_constant<int, 1>{});
          }
          if (pass == 0) {
            __syncthreads();
            wk.each([&](int i) {
              T acc = w[i];
#pragma unroll 4
              for (int q = 0; q <= j; ++q) acc -= yt[q] * V[(int64_t)q * n + i];
              w[i] = acc;
            });
            __syncthreads();  // yt is read before the next pass rewrites it
          }
        }
        if (threadIdx.x == 0) {
          double ww = y[j + 1], yy = 0.0;
          for (int q = 0; q <= j; ++q) yy += y[q] * y[q];
          const double h2 = ww - yy;
          const double hn = h2 > 0.25 * ww ? sqrt(h2) : -1.0;  // else too much was subtracted (or NaN)
          wk.sums[8] = hn;
          wk.sums[9] = hn > 0.0 ? 1.0 / hn : 0.0;
        }
        __syncthreads();
        double hn = wk.sums[8];
        const bool direct = !(hn >= 0.0);  // the same in every CTA: the sums are
        T ihn = (T)wk.sums[9];
        if (direct) ihn = (T)1;
        wk.each([&](int i) {
          T acc = w[i];
#pragma unroll 4
          for (int q = 0; q <= j; ++q) acc -= yt[q] * V[(int64_t)q * n + i];
          const T v = acc * ihn;
          if (direct) w[i] = v;
          vn[i] = v;
          xa[i] = (float)v;
        });
        if (direct) {
          double nn[1];
          team_sum<1, T>(wk, nn, [&](int i, T (&q)[1]) { q[0] += w[i] * w[i]; }, true);
          hn = nn[0];
          if (hn > 0.0) {
            ihn = (T)wk.sums[1];
            wk.each([&](int i) {
              const T v = w[i] * ihn;
              vn[i] = v;
              xa[i] = (float)v;
            });
          }
        }
        if (threadIdx.x == 0) {
          double* Hj = H + (m + 1) * j;
          Hj[j + 1] = hn;
          for (int i = 0; i < j; ++i) {
            const double t = cs[i] * Hj[i] + sn[i] * Hj[i + 1];
            Hj[i + 1] = -sn[i] * Hj[i] + cs[i] * Hj[i + 1];
            Hj[i] = t;
          }
          const double den = sqrt(Hj[j] * Hj[j] + hn * hn);
          const double rden = den > 0.0 ? 1.0 / den : 0.0;
          const double c = den > 0.0 ? Hj[j] * rden : 1.0;
          const double sv = hn * rden;
          cs[j] = c;
          sn[j] = sv;
          Hj[j] = den;
          Hj[j + 1] = 0.0;
          g[j + 1] = -sv * g[j];
          g[j] = c * g[j];
        }
        team.arrive();
        first_ahead();
        team.wait();
        ++its;
        k = j + 1;
        const double gres = fabs(g[j + 1]);
        if (!(gres > inner_target) || hn <= DBL_MIN || !isfinite(gres)) break;
      }
      // back-substitution H y = g (k x k upper triangular)
      if (threadIdx.x < 32) {  // a lane per row (four beyond 32), column by column
        const int lane = threadIdx.x;
        double t[4], inv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int q = lane + 32 * u;
          t[u] = q < k ? g[q] : 0.0;
          inv[u] = q < k ? 1.0 / H[(m + 1) * q + q] : 0.0;
        }
        for (int i = k - 1; i >= 0; --i) {
          double yi = 0.0;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if ((i >> 5) == u) yi = __shfl_sync(0xffffffffu, t[u] * inv[u], i & 31);
          if (lane == 0) y[i] = yi;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int q = lane + 32 * u;
            if (q < i) t[u] -= H[(m + 1) * i + q] * yi;
          }
        }
      }
      __syncthreads();
      // X += M⁻¹ V y = Z y: the preconditioned basis was kept, so the update needs no further
      // preconditioner application (one band solve per cycle saved)
      wk.each([&](int i) {
        double acc = 0.0;
        for (int q = 0; q < k; ++q) acc += y[q] * (double)Zb[(int64_t)q * n + i];
        X[i] += acc;
      });
      team.sync();
      // true FP64 residual R = b - Ktan X
      team_sum<1, double>(wk, v1, [&](int i, double (&q)[1]) {
        const int64_t d = dof(i);
        const double ri = (a.fixed[d] ? 0.0 : a.b[d]) - row64(a, n0, i, X);
        R[i] = ri;
        q[0] += ri * ri;
      }, true);
      rnorm = v1[0];
      ++refs;
      if (!isfinite(rnorm)) { status = 2; break; }
    }
    if (status == 0 && rnorm > target) status = 3;  // EB_SIM_KRYLOV_STAGNATED
  }
  __syncthreads();
  if (stp && stage_fail) {
    status = 4;  // EB_SIM_WAIT_TIMEOUT: a bulk copy did not complete in time
    stage_drain(stp);
  }

  // ΔD[free] = x; Newton norms of compute_norms_corrector (utils_solver.jl:126-151).  The
  // increment is written whenever the solve was finite, also where a staging wait ran out (rank 0
  // knows it and reports the step as not converged).
  double q[4];
  team_sum<4, double>(wk, q, [&](int i, double (&v)[4]) {
    const int64_t d = dof(i);
    const double f = (a.fext1[d] + a.Tc1[d]) + a.Tk1[d];
    if (a.fixed[d]) {
      v[3] += f * f;
    } else {
      const double x = (bnorm > 0.0 && status != 2) ? X[i] : 0.0;
      a.dD[d] = x;
      v[0] += x * x;
      v[1] += a.b[d] * a.b[d];
      v[2] += f * f;
    }
  });
  if (threadIdx.x == 0 && team.rank == 0) {
    a.norms[5 * s + 0] = q[0];
    a.norms[5 * s + 1] = q[1];
    a.norms[5 * s + 2] = q[2];
    a.norms[5 * s + 3] = q[3];
    a.norms[5 * s + 4] = status == 4 ? -1.0 : (double)its;  // iterations of this solve (-1: a wait ran out)
    a.its[s] += its;
    a.refs[s] += refs;
    const double rel = bnorm > 0.0 ? rnorm / bnorm : 0.0;
    a.relres[s] = fmax(a.relres[s], rel);
    if (status > a.status[s]) a.status[s] = status;
  }
}

// 6x6 block-Jacobi factors: inverse of each node's diagonal block of Ktan with
// fixed DOFs replaced by identity rows/columns (Gauss-Jordan, partial pivoting).
__global__ void k_block_jacobi(const Dev d, double* Dinv64, float* Dinv32) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (!d.active[d.node_sim[i]]) return;
  double A[36], B[36];
  const double* blk = d.Kt + (int64_t)d.diag_blk[i] * 36;
#pragma unroll
  for (int c = 0; c < 6; ++c)
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const bool fr = d.fixed[6 * i + r], fc = d.fixed[6 * i + c];
      A[6 * c + r] = (fr || fc) ? (r == c ? 1.0 : 0.0) : blk[6 * c + r];
      B[6 * c + r] = (r == c) ? 1.0 : 0.0;
    }
  for (int c = 0; c < 6; ++c) {
    int p = c;
    double best = fabs(A[6 * c + c]);
    for (int r = c + 1; r < 6; ++r)
      if (fabs(A[6 * c + r]) > best) { best = fabs(A[6 * c + r]); p = r; }
    if (p != c)
      for (int q = 0; q < 6; ++q) {
        double t = A[6 * q + c]; A[6 * q + c] = A[6 * q + p]; A[6 * q + p] = t;
        t = B[6 * q + c]; B[6 * q + c] = B[6 * q + p]; B[6 * q + p] = t;
      }
    const double piv = A[6 * c + c];
    const double ip = piv != 0.0 ? 1.0 / piv : 0.0;
    for (int q = 0; q < 6; ++q) { A[6 * q + c] *= ip; B[6 * q + c] *= ip; }
    for (int r = 0; r < 6; ++r) {
      if (r == c) continue;
      const double f = A[6 * c + r];
      if (f == 0.0) continue;
      for (int q = 0; q < 6; ++q) { A[6 * q + r] -= f * A[6 * q + c]; B[6 * q + r] -= f * B[6 * q + c]; }
    }
  }
  double* o64 = Dinv64 + i * 36;
  float* o32 = Dinv32 + i * 36;
#pragma unroll
  for (int k = 0; k < 36; ++k) { o64[k] = B[k]; o32[k] = (float)B[k]; }
}

void launch_block_jacobi(const Dev& d, double* Dinv64, float* Dinv32, cudaStream_t s) {
  if (d.n_nodes) k_block_jacobi<<<nblocks(d.n_nodes), kThreads, 0, s>>>(d, Dinv64, Dinv32);
}

size_t gmres_smem(int m, int dots) {
  return sizeof(double) * ((size_t)(m + 1) * m + 5 * (size_t)m + 3 + 2 * (size_t)dots * kMaxChunks + 16 + 1);
}

size_t gmres_smem_total(const SolverArgs& a) {
  return gmres_smem(a.m, a.dots) + sizeof(float) * ((size_t)a.dense_ld + (size_t)a.vec_smem) + (a.x_in_smem ? sizeof(float) * (size_t)a.max_n : 0) +
         (a.stage_floats > 0 ? 128 + sizeof(float) * 2 * (size_t)a.stage_floats +
                                   sizeof(float) * 2 * kPanel * kPanel
                             : 0);
}

int gmres_stage_b(int m) {
  const size_t rest = gmres_smem(m, 4) + sizeof(float) * (kDenseMax + 2 * kPanel * kPanel) + 128;
  return rest >= kGmresSmemLimit ? 0 : (int)((kGmresSmemLimit - rest) / (2 * sizeof(float) * kPanel)) - 1;
}

namespace {
const void* gmres_kernel(bool fp32) { return fp32 ? (const void*)k_gmres<float> : (const void*)k_gmres<double>; }

cudaLaunchConfig_t gmres_config(const SolverArgs& a, int threads, cudaStream_t s, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)(a.n_sims * a.team));
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = gmres_smem_total(a);
  c.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)a.team;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  c.attrs = at;
  c.numAttrs = 1;
  return c;
}
}  // namespace

// CTAs per simulation of a launch: the largest power of two up to 16 for which all teams are
// resident at once and every CTA still has kTeamDofs entries of the largest simulation.
int gmres_team(const SolverArgs& a, bool fp32, int threads, int max_dofs) {
  const void* k = gmres_kernel(fp32);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 1;
  if (raise_smem_limit(k, gmres_smem_total(a)) != cudaSuccess) return 1;
  cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  for (int t = 16; t > 1; t /= 2) {
    if (a.n_sims * t > sms || (t / 2) * kTeamDofs >= max_dofs) continue;
    SolverArgs b = a;
    b.team = t;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t c = gmres_config(b, threads, 0, at);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k, &c) == cudaSuccess && clusters >= a.n_sims) return t;
    cudaGetLastError();
  }
  return 1;
}

cudaError_t launch_gmres(const SolverArgs& a, bool fp32, int threads, cudaStream_t s) {
  // shared memory is the occupancy limit: prefer the largest carveout so two CTAs fit when they can
  const void* k = gmres_kernel(fp32);
  cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  cudaError_t e = raise_smem_limit(k, gmres_smem_total(a));
  if (e != cudaSuccess) return e;
  if (a.team > 8) cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t c = gmres_config(a, threads, s, at);
  void* args[1] = {const_cast<SolverArgs*>(&a)};
  e = cudaLaunchKernelExC(&c, k, args);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace eb
