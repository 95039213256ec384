// Element, contact, assembly and HHT step-algebra kernels.
#include "eb_internal.cuh"

namespace eb {
using namespace ebd;

// ------------------------------------------------------------------ loads
__device__ __forceinline__ V3 node3(const double* f, int64_t n, int i) {
  return v3(f[i], f[n + i], f[2 * n + i]);
}
__device__ __forceinline__ M3 node9(const double* f, int64_t n, int i) {
  M3 m;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.a[k] = f[k * n + i];
  return m;
}
__device__ __forceinline__ void store3(double* f, int64_t n, int i, V3 v) {
  f[i] = v.x; f[n + i] = v.y; f[2 * n + i] = v.z;
}
__device__ __forceinline__ void store9(double* f, int64_t n, int i, const M3& m) {
#pragma unroll
  for (int k = 0; k < 9; ++k) f[k * n + i] = m.a[k];
}
__device__ __forceinline__ V3 elem3(const double* f, int64_t ne, int64_t e) {
  return v3(f[e], f[ne + e], f[2 * ne + e]);
}

// ------------------------------------------------------------------ assemble! element pass
// compute_beams via assemble_beams.jl:21-48, ten or thirty elements per CTA (eb_beam.cuh).
struct BeamElem {
  const Dev& d;
  int64_t e;
  int nd[2];
  __device__ __forceinline__ V3 x(int n) const { return node3(d.X0, d.n_nodes, nd[n]) + node3(d.u, d.n_nodes, nd[n]); }
  __device__ __forceinline__ M3 R(int n) const { return node9(d.R, d.n_nodes, nd[n]); }
  __device__ __forceinline__ M3 dR(int n) const { return node9(d.dR, d.n_nodes, nd[n]); }
  __device__ __forceinline__ M3 Re0() const {
    M3 m;
#pragma unroll
    for (int k = 0; k < 9; ++k) m.a[k] = d.Re0[k * d.n_elem + e];
    return m;
  }
  __device__ __forceinline__ V3 ud(int n) const { return node3(d.ud, d.n_nodes, nd[n]); }
  __device__ __forceinline__ V3 wd(int n) const { return node3(d.wd, d.n_nodes, nd[n]); }
  __device__ __forceinline__ V3 udd(int n) const { return node3(d.udd, d.n_nodes, nd[n]); }
  __device__ __forceinline__ V3 wdd(int n) const { return node3(d.wdd, d.n_nodes, nd[n]); }
  __device__ __forceinline__ double l0() const { return d.l0[e]; }
  __device__ __forceinline__ double Ku() const { return d.Kbar[e]; }
  __device__ __forceinline__ V3 KT() const { return elem3(d.Kbar + d.n_elem, d.n_elem, e); }
  __device__ __forceinline__ V3 KTT() const { return elem3(d.Kbar + 4 * d.n_elem, d.n_elem, e); }
  __device__ __forceinline__ V3 Jr() const { return elem3(d.Jr, d.n_elem, e); }
  __device__ __forceinline__ double Ar() const { return d.Ar[e]; }
  __device__ __forceinline__ double damping() const { return d.damp[e]; }
  __device__ __forceinline__ BeamOut out() const {
    return BeamOut{d.stK + e * 144, d.stM + e * 144, d.stC + e * 144, d.stTi + e * 12, d.stTk + e * 12, d.stE + e * 2};
  }
};

__global__ void __launch_bounds__(kBeamCta, 3) k_beam(const __grid_constant__ Dev d, Gauss3 g, int nb) {
  extern __shared__ double beam_tab[];
  beam_cta(d.n_elem, nb, g, beam_tab, [&](int64_t e) { return BeamElem{d, e, {d.ea[e], d.eb[e]}}; },
           [&](int64_t e) { return d.active[d.elem_sim[e]] != 0; });
}

// The same with a thread per element, for launches of many waves (many_elements).
__global__ void __launch_bounds__(kBeamCta, 3) k_beam_thread(const __grid_constant__ Dev d, Gauss3 g) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= d.n_elem || !d.active[d.elem_sim[e]]) return;
  beam_thread(BeamElem{d, e, {d.ea[e], d.eb[e]}}, g);
}

// compute_contact_beams via compute&assemble…:460-482, ten or thirty elements per CTA (eb_contact.cuh).
struct ContactElem : BeamElem {
  __device__ __forceinline__ double radius() const { return d.radius[e]; }
  __device__ __forceinline__ const SurfaceDev& surf() const { return d.surf[d.elem_sim[e]]; }
  __device__ __forceinline__ const ContactProps& props() const { return d.props[d.elem_sim[e]]; }
  __device__ __forceinline__ ContactOut out() const {
    return ContactOut{d.scK + e * 144, d.scC + e * 144, d.scT + e * 12, d.scE + e};
  }
  __device__ __forceinline__ void touched(bool any) const { d.sc_on[e] = any ? 1 : 0; }
};

__global__ void __launch_bounds__(kContactCta) k_contact(const __grid_constant__ Dev d, Gauss3 g, int nb) {
  extern __shared__ double beam_tab[];
  contact_cta(d.n_elem, nb, g, beam_tab, [&](int64_t e) { return ContactElem{{d, e, {d.ea[e], d.eb[e]}}}; },
              [&](int64_t e) { return d.is_contact[e] && d.active[d.elem_sim[e]]; });
}

void launch_beam(const Dev& d, const Gauss3& g, cudaStream_t s) {
  if (!d.n_elem) return;
  const int nb = beam_groups(d.beam_threads);
  if (nb == 3 && d.many_elements) {
    k_beam_thread<<<nblocks(d.n_elem, kBeamCta), kBeamCta, 0, s>>>(d, g);
    return;
  }
  const size_t smem = beam_smem(nb);
  if (smem > 48 * 1024) raise_smem_limit((const void*)k_beam, smem);
  k_beam<<<nblocks(d.n_elem, kBeamGroup * nb), kBeamCta, smem, s>>>(d, g, nb);
}
void launch_contact(const Dev& d, const Gauss3& g, cudaStream_t s) {
  if (!d.n_elem) return;
  const int nb = beam_groups(d.contact_threads);
  const size_t smem = contact_smem(nb);
  if (smem > 48 * 1024) raise_smem_limit((const void*)k_contact, smem);
  k_contact<<<nblocks(d.n_elem, kBeamGroup * nb), kContactCta, smem, s>>>(d, g, nb);
}

// v as an unevaluated sum of two FP32 numbers (48 bits of it)
__device__ __forceinline__ float2 fp32_pair(double v) {
  const float hi = (float)v;
  return make_float2(hi, (float)(v - (double)hi));
}

// ------------------------------------------------------------------ ordered block assembly
// Thread per (block, entry): the reference's `nzval[global_sparsity_map] += vec(K)`
// (assemble_beams.jl:64-66, compute&assemble…:496-497) as a fixed-order sum over
// the contributions of each block, fused with the tangent
// Ktan = (1+α)K + γ/(βΔt) C + 1/(βΔt²) M (utils_solver.jl:83).
__global__ void k_gather_mat(Dev d, double alpha, int with_contact) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.nnzb * 36) return;
  const int b = (int)(t / 36), k = (int)(t % 36);
  const int s = d.blk_sim[b];
  if (!d.active[s]) return;
  const int i = k % 6, j = k / 6;
  double Ks = 0.0, Cs = 0.0, Ms = 0.0;
  const int c0 = d.blk_cptr[b], c1 = d.blk_cptr[b + 1];
  for (int c = c0; c < c1; ++c) {
    const int v = d.blk_contrib[c];
    const int64_t e = v >> 2;
    const int I = v & 1, J = (v >> 1) & 1;
    const int64_t idx = e * 144 + (6 * J + j) * 12 + (6 * I + i);
    Ks += d.stK[idx];
    Cs += d.stC[idx];
    Ms += d.stM[idx];
  }
  if (with_contact) {
    const double ca = 1 + alpha;
    for (int c = c0; c < c1; ++c) {
      const int v = d.blk_contrib[c];
      const int64_t e = v >> 2;
      if (!d.sc_on[e]) continue;
      const int I = v & 1, J = (v >> 1) & 1;
      const int64_t idx = e * 144 + (6 * J + j) * 12 + (6 * I + i);
      Ks += -d.scK[idx];
      Cs += -(ca * d.scC[idx]);
    }
  }
  d.K1[t] = Ks;
  d.C1[t] = Cs;
  d.M1[t] = Ms;
  const double kt = (d.cK[s] * Ks + d.cC[s] * Cs) + d.cM[s] * Ms;
  d.Kt[t] = kt;
  if (d.Ktp) d.Ktp[t] = fp32_pair(kt);
}

// ΔD[fixed] = imposed - D[fixed] (apply_boundary_conditions!, utils_bcs_and_loads.jl:5-29); the
// other part, r -= Ktan[:, fixed] ΔD[fixed], is k_bc_lift.
__device__ __forceinline__ void bc_delta(const Dev& d, int64_t t) {
  if (d.fixed[t]) d.dD[t] = d.imposed[t] - d.D[t];
}

// Thread per (node, dof): Tⁱⁿᵗ, Tᵏ, Tᶜ as ordered sums over incident elements
// (assemble_beams.jl:60-61, compute&assemble…:493); with `rhs` also the residual
// (compute_tangent_and_residuals_corrector!, utils_solver.jl:87) and the imposed increments: as
// launches of their own these two cost 4.3 and 2.7 us of a 64-element ring's iteration.
__global__ void k_gather_vec(Dev d, double alpha, int with_contact, int rhs) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.n_dof) return;
  const int i = (int)(t / 6), k = (int)(t % 6);
  if (!d.active[d.node_sim[i]]) return;
  double Ti = 0.0, Tk = 0.0, Tc = 0.0;
  const int c0 = d.node_cptr[i], c1 = d.node_cptr[i + 1];
  for (int c = c0; c < c1; ++c) {
    const int v = d.node_contrib[c];
    const int64_t e = v >> 1;
    const int I = v & 1;
    Ti += d.stTi[e * 12 + 6 * I + k];
    Tk += d.stTk[e * 12 + 6 * I + k];
  }
  if (with_contact) {
    for (int c = c0; c < c1; ++c) {
      const int v = d.node_contrib[c];
      const int64_t e = v >> 1;
      if (!d.sc_on[e]) continue;
      Tc += d.scT[e * 12 + 6 * (v & 1) + k];
    }
  }
  if (rhs) {
    d.r[t] = ((1 + alpha) * ((d.fext1[t] + Tc) - Ti) - alpha * ((d.fextn[t] + d.Tcn[t]) - d.Tin[t])) - Tk;
    bc_delta(d, t);
  }
  d.Ti1[t] = Ti;
  d.Tk1[t] = Tk;
  d.Tc1[t] = Tc;
}

void launch_gather(const Dev& d, double alpha, bool with_contact, bool rhs, cudaStream_t s) {
  if (d.nnzb) k_gather_mat<<<nblocks(d.nnzb * 36, d.gmat_threads), d.gmat_threads, 0, s>>>(d, alpha, with_contact ? 1 : 0);
  if (d.n_dof) k_gather_vec<<<nblocks(d.n_dof, d.gvec_threads), d.gvec_threads, 0, s>>>(d, alpha, with_contact ? 1 : 0, rhs ? 1 : 0);
}

// ------------------------------------------------------------------ predictor
// initialize_global_predictor! (utils_solver.jl:30-48)
__global__ void k_init_predictor(Dev d) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  if (!d.active[d.node_sim[i]]) return;
  const int64_t n = d.n_nodes;
  V3 u = node3(d.u, n, i), ud = node3(d.ud, n, i), udd = node3(d.udd, n, i);
  V3 wd = node3(d.wd, n, i), wdd = node3(d.wdd, n, i);
  double* D = d.D + 6 * i;
  double* Dd = d.Dd + 6 * i;
  double* Ddd = d.Ddd + 6 * i;
  double* dD = d.dD + 6 * i;
  D[0] = u.x; D[1] = u.y; D[2] = u.z; D[3] = 0.0; D[4] = 0.0; D[5] = 0.0;
  Dd[0] = ud.x; Dd[1] = ud.y; Dd[2] = ud.z; Dd[3] = wd.x; Dd[4] = wd.y; Dd[5] = wd.z;
  Ddd[0] = udd.x; Ddd[1] = udd.y; Ddd[2] = udd.z; Ddd[3] = wdd.x; Ddd[4] = wdd.y; Ddd[5] = wdd.z;
#pragma unroll
  for (int k = 0; k < 6; ++k) dD[k] = 0.0;
}

// compute_tangent_and_residuals_predictor! (utils_solver.jl:54-74), thread per (node, dof):
// Ktan from the matrices at n, r = (1+α)fⁿ⁺¹ - Tⁱⁿᵗⁿ - Tᵏⁿ - αfⁿ + Cⁿ t₁ + Mⁿ t₂ /(βΔt²); the
// imposed increments.  A block's 30 values are loaded before any is stored: with loads and stores
// in turn a thread waited for L2 six times per block (64-element ring: 19.7 us).
__global__ void k_predictor_rhs(Dev d, double alpha, double beta, double gamma) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.n_dof) return;
  const int i = (int)(t / 6), k = (int)(t % 6);
  const int s = d.node_sim[i];
  if (!d.active[s]) return;
  const double dt = d.dt[s];
  const double cK = d.cK[s], cC = d.cC[s], cM = d.cM[s];
  const double a1 = gamma / beta, a2 = (dt / 2 * (2 * beta - gamma)) / beta;
  const double b2 = (dt * dt) / 2;
  double r = (((1 + alpha) * d.fext1[t] - d.Tin[t]) - d.Tkn[t]) - alpha * d.fextn[t];
  double cv = 0.0, mv = 0.0;
  for (int bb = d.row_ptr[i]; bb < d.row_ptr[i + 1]; ++bb) {
    const int c = d.col[bb];
    const double* Cb = d.Cn + (int64_t)bb * 36;
    const double* Mb = d.Mn + (int64_t)bb * 36;
    const double* Kb = d.Kn + (int64_t)bb * 36;
    double vd[6], va[6], kv[6], cw[6], mw[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      kv[j] = Kb[6 * j + k];
      cw[j] = Cb[6 * j + k];
      mw[j] = Mb[6 * j + k];
      vd[j] = d.Dd[6 * c + j];
      va[j] = d.Ddd[6 * c + j];
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const double t1 = a1 * vd[j] - a2 * va[j];
      const double t2 = dt * vd[j] + b2 * va[j];
      cv += cw[j] * t1;
      mv += mw[j] * t2;
      const double kt = (cK * kv[j] + cC * cw[j]) + cM * mw[j];
      d.Kt[(int64_t)bb * 36 + 6 * j + k] = kt;
      if (d.Ktp) d.Ktp[(int64_t)bb * 36 + 6 * j + k] = fp32_pair(kt);
    }
  }
  r = cv + r;
  r = cM * mv + r;
  d.r[t] = r;
  bc_delta(d, t);
}

void launch_init_predictor(const Dev& d, cudaStream_t s) {
  if (d.n_nodes) k_init_predictor<<<nblocks(d.n_nodes), kThreads, 0, s>>>(d);
}
void launch_predictor_rhs(const Dev& d, double alpha, double beta, double gamma, cudaStream_t s) {
  if (d.n_dof) k_predictor_rhs<<<nblocks(d.n_dof, 256), 256, 0, s>>>(d, alpha, beta, gamma);
}

__global__ void k_bc_lift(Dev d) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.n_dof) return;
  const int i = (int)(t / 6), k = (int)(t % 6);
  const int s = d.node_sim[i];
  if (!d.active[s] || !d.has_fixed[s]) return;
  double acc = 0.0;
  for (int bb = d.row_ptr[i]; bb < d.row_ptr[i + 1]; ++bb) {
    const int c = d.col[bb];
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (d.fixed[6 * c + j]) acc += d.dD[6 * c + j] * d.Kt[(int64_t)bb * 36 + 6 * j + k];
  }
  d.r[t] -= acc;
}
void launch_bc_lift(const Dev& d, cudaStream_t s) {
  if (!d.n_dof) return;
  k_bc_lift<<<nblocks(d.n_dof, 256), 256, 0, s>>>(d);
}

// A node's six values of a vector in DOF order (48 bytes, 16-byte aligned).
__device__ __forceinline__ void load6(const double* p, int64_t i, double* v) {
  const double2* q = reinterpret_cast<const double2*>(p + 6 * i);
  const double2 a = q[0], b = q[1], c = q[2];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y;
}
__device__ __forceinline__ void store6(double* p, int64_t i, V3 a, V3 b) {
  double2* q = reinterpret_cast<double2*>(p + 6 * i);
  q[0] = make_double2(a.x, a.y);
  q[1] = make_double2(a.z, b.x);
  q[2] = make_double2(b.y, b.z);
}

// angular rates of utils_solver.jl:214-215 / :239-240
__device__ __forceinline__ void rates(const M3& dR, V3 w, V3 wdn, V3 wddn, double beta, double gamma, double dt,
                                      V3* wd, V3* wdd) {
  V3 a = (gamma / (beta * dt)) * w + ((beta - gamma) / beta) * wdn + ((dt * (beta - gamma / 2)) / beta) * wddn;
  V3 b = (1 / (beta * (dt * dt))) * w - (1 / (beta * dt)) * wdn - (1 / (2 * beta) - 1) * wddn;
  *wd = dR * a;
  *wdd = dR * b;
}

// End of the predictor, thread per node: compute_global_predictor! (utils_solver.jl:157-172),
// compute_local_predictor! (:197-217) and initialize_global_corrector! (:6-24).  Everything a node
// needs is loaded before the first store, one round trip to L2 instead of one per field (64-element
// ring: 7.4 + 13.5 + 5 us as three launches with loads and stores in turn).
__global__ void k_predictor_update(Dev d, double beta, double gamma) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  const int s = d.node_sim[i];
  if (!d.active[s]) return;
  const int64_t n = d.n_nodes;
  const double dt = d.dt[s];
  double D[6], Dd[6], Ddd[6], dD[6];
  load6(d.D, i, D);
  load6(d.Dd, i, Dd);
  load6(d.Ddd, i, Ddd);
  load6(d.dD, i, dD);
  const V3 wdn = node3(d.wdn, n, i), wddn = node3(d.wddn, n, i);
  const M3 Rn = node9(d.Rn, n, i);
  const double g_bdt = gamma / (beta * dt), g_b = gamma / beta, inv = 1 / (beta * (dt * dt));
  const double dt2b = (dt * (2 * beta - gamma)) / (2 * beta);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double v = Dd[k], a = Ddd[k];
    D[k] += dD[k];
    Dd[k] += (g_bdt * dD[k] - g_b * v) + dt2b * a;
    Ddd[k] += inv * ((dD[k] - dt * v) - ((dt * dt) / 2) * a);
  }
  const V3 u = v3(D[0], D[1], D[2]), ud = v3(Dd[0], Dd[1], Dd[2]), udd = v3(Ddd[0], Ddd[1], Ddd[2]);
  const V3 th = v3(D[3], D[4], D[5]);
  const M3 dR = rotation_matrix(th);
  V3 wd, wdd;
  rates(dR, th, wdn, wddn, beta, gamma, dt, &wd, &wdd);
  store3(d.u, n, i, u);
  store3(d.ud, n, i, ud);
  store3(d.udd, n, i, udd);
  store3(d.w, n, i, th);
  store9(d.dR, n, i, dR);
  store9(d.R, n, i, dR * Rn);
  store3(d.wd, n, i, wd);
  store3(d.wdd, n, i, wdd);
  store6(d.D, i, u, th);
  store6(d.Dd, i, ud, wd);
  store6(d.Ddd, i, udd, wdd);
  store6(d.dD, i, v3(0.0, 0.0, 0.0), v3(0.0, 0.0, 0.0));
}
void launch_predictor_update(const Dev& d, double beta, double gamma, cudaStream_t s) {
  if (d.n_nodes) k_predictor_update<<<nblocks(d.n_nodes), kThreads, 0, s>>>(d, beta, gamma);
}

// End of a corrector iteration, thread per node: compute_global_corrector! (utils_solver.jl:178-190)
// and compute_local_corrector! (:224-245); node w is not written, as in the reference.  Loads first,
// as above (64-element ring: 4.5 + 16.3 us as two launches with loads and stores in turn).
__global__ void k_corrector_update(Dev d, double beta, double gamma) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n_nodes) return;
  const int s = d.node_sim[i];
  if (!d.active[s]) return;
  const int64_t n = d.n_nodes;
  const double dt = d.dt[s], cC = d.cC[s], cM = d.cM[s];
  double D[6], Dd[6], Ddd[6], dD[6];
  load6(d.D, i, D);
  load6(d.Dd, i, Dd);
  load6(d.Ddd, i, Ddd);
  load6(d.dD, i, dD);
  const V3 wdn = node3(d.wdn, n, i), wddn = node3(d.wddn, n, i);
  const M3 dR0 = node9(d.dR, n, i), Rn = node9(d.Rn, n, i);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    D[k] += dD[k];
    Dd[k] += cC * dD[k];
    Ddd[k] += cM * dD[k];
  }
  const V3 u = v3(D[0], D[1], D[2]), ud = v3(Dd[0], Dd[1], Dd[2]), udd = v3(Ddd[0], Ddd[1], Ddd[2]);
  const M3 dR = rotation_matrix(v3(dD[3], dD[4], dD[5])) * dR0;
  const V3 w1 = toangle(dR);
  V3 wd, wdd;
  rates(dR, w1, wdn, wddn, beta, gamma, dt, &wd, &wdd);
  store6(d.D, i, u, v3(D[3], D[4], D[5]));
  store6(d.Dd, i, ud, v3(Dd[3], Dd[4], Dd[5]));
  store6(d.Ddd, i, udd, v3(Ddd[3], Ddd[4], Ddd[5]));
  store3(d.u, n, i, u);
  store3(d.ud, n, i, ud);
  store3(d.udd, n, i, udd);
  store9(d.dR, n, i, dR);
  store3(d.wd, n, i, wd);
  store3(d.wdd, n, i, wdd);
  store9(d.R, n, i, dR * Rn);
}
void launch_corrector_update(const Dev& d, double beta, double gamma, cudaStream_t s) {
  if (d.n_nodes) k_corrector_update<<<nblocks(d.n_nodes), kThreads, 0, s>>>(d, beta, gamma);
}

// ------------------------------------------------------------------ commit / rollback
// update_converged! (utils_solver.jl:252-275) when commit, else update_not_converged! (:282-305).
// One launch: a thread per value of the node fields (component-major, 36 per node), then one per
// DOF, then one per block entry.  A thread's loads precede its stores; a thread per node went through
// 36 of them in turn (19 us for 64 nodes, and two more launches).
struct NodeFields {
  double* p[8];
};
constexpr int kNodeValues = 36;
__global__ void k_commit(const __grid_constant__ Dev d, const __grid_constant__ NodeFields work,
                         const __grid_constant__ NodeFields kept, const int* mask, int commit, int64_t total) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int64_t n = d.n_nodes;
  if (t < kNodeValues * n) {
    const int c = (int)(t / n);
    const int64_t i = t - c * n;
    if (!mask[d.node_sim[i]]) return;
    const int f = c < 18 ? c / 3 : 6 + (c - 18) / 9;
    const int64_t at = (c < 18 ? c % 3 : (c - 18) % 9) * n + i;
    if (commit) kept.p[f][at] = work.p[f][at];
    else work.p[f][at] = kept.p[f][at];
    return;
  }
  t -= kNodeValues * n;
  if (t < d.n_dof) {
    if (!mask[d.node_sim[t / 6]]) return;
    if (commit) {
      const double a = d.Ti1[t], b = d.Tk1[t], c = d.Tc1[t], e = d.fext1[t];
      d.Tin[t] = a; d.Tkn[t] = b; d.Tcn[t] = c; d.fextn[t] = e;
    } else {
      const double a = d.Tin[t], b = d.Tkn[t], c = d.Tcn[t], e = d.fextn[t];
      d.Ti1[t] = a; d.Tk1[t] = b; d.Tc1[t] = c; d.fext1[t] = e;
    }
    return;
  }
  t -= d.n_dof;
  if (!mask[d.blk_sim[t / 36]]) return;
  if (commit) {
    const double a = d.K1[t], b = d.C1[t], c = d.M1[t];
    d.Kn[t] = a; d.Cn[t] = b; d.Mn[t] = c;
  } else {
    const double a = d.Kn[t], b = d.Cn[t], c = d.Mn[t];
    d.K1[t] = a; d.C1[t] = b; d.M1[t] = c;
  }
}

static NodeFields node_fields(const Dev& d, bool at_n) {
  return at_n ? NodeFields{{d.un, d.udn, d.uddn, d.wn, d.wdn, d.wddn, d.Rn, d.dRn}}
              : NodeFields{{d.u, d.ud, d.udd, d.w, d.wd, d.wdd, d.R, d.dR}};
}
static void commit_values(const Dev& d, const int* mask, bool commit, int64_t total, cudaStream_t s) {
  if (total) k_commit<<<nblocks(total, 256), 256, 0, s>>>(d, node_fields(d, false), node_fields(d, true), mask, commit ? 1 : 0, total);
}
void launch_commit(const Dev& d, const int* mask, bool commit, cudaStream_t s) {
  commit_values(d, mask, commit, kNodeValues * d.n_nodes + d.n_dof + 36 * d.nnzb, s);
}

void launch_restore_nodes(const Dev& d, const int* mask, cudaStream_t s) {
  commit_values(d, mask, false, kNodeValues * d.n_nodes, s);
}

// Node fields of m nodes from `first` as arrays of structures, field by field, into `out` (pinned
// host memory: the values go straight there, one launch instead of a copy per component).
__global__ void k_state(const __grid_constant__ NodeFields f, int64_t n, int64_t first, int m, double* out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)kNodeValues * m) return;
  const bool vec = t < 18 * (int64_t)m;
  const int nc = vec ? 3 : 9;
  const int64_t u = vec ? t : t - 18 * (int64_t)m;
  const int k = (int)(u / ((int64_t)nc * m));
  const int64_t e = u - (int64_t)k * nc * m;
  const double* src = f.p[vec ? k : 6 + k];
  if (src) out[t] = src[(e % nc) * n + first + e / nc];
}
void launch_state(const Dev& d, bool at_n, unsigned fields, int64_t first, int m, double* out, cudaStream_t s) {
  NodeFields f = node_fields(d, at_n);
  for (int k = 0; k < 8; ++k)
    if (!(fields >> k & 1)) f.p[k] = nullptr;
  if (m) k_state<<<nblocks((int64_t)kNodeValues * m, 256), 256, 0, s>>>(f, d.n_nodes, first, m, out);
}

}  // namespace eb
