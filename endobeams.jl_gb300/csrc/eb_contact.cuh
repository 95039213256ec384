// Beam-to-rigid-surface contact element on the GPU (FP64): compute_contact_beams of
// src/interactions/compute&assemble_interactions_beams.jl:1-445 with the
// surfaces of src/interactions/utils_compute_interactions_beams.jl and the
// regularisations of interactions_beams_regularization.jl.
//
// As in the reference, the normal damping ηₙ is a function-level variable
// that the Gauss loop overwrites with its smoothstep value (:100), so an
// in-contact Gauss point sees the value left by the previous one.
//
// An element with three Gauss points in contact is about 18,000 FP64 operations;
// one thread per element ran them as one chain with spills (0.44 ms a launch
// even for 64 elements, 0.62 ms for 9,600 in contact against a floor of 0.14 ms).
// Like the beam element it is cut into pieces that share a table: frame, end
// nodes, one lane per element and Gauss point for the gap test and the point's
// quantities (contact_point), and the block columns of Kᶜ and Cᶜ (contact_column).
#pragma once
#include "eb_beam.cuh"

namespace ebd {

struct ContactProps {
  double kn, mu, eps_t, eta_n;
};

// Rigid surface: analytic sphere, quadratic B-spline SDF on a voxel grid, or
// analytic plane.
struct SurfaceDev {
  int kind;                // 0 sphere, 1 SDF, 2 plane
  double cx, cy, cz, R;    // sphere
  int axis;                // plane: x[axis] = pos, body on the positive side
  double pos;
  const double* coef;      // (nx+2)(ny+2)(nz+2) prefiltered coefficients (interp 1: the samples), x fastest
  int interp;              // 0 quadratic B-spline (the reference's), 1 trilinear
  int nx, ny, nz;          // grid points
  double x0, y0, z0;       // first grid point
  double ihx, ihy, ihz;    // 1 / spacing
  double xl, yl, zl;       // domain extents (n-1)*h
};

struct ContactIn {
  V3 X1, X2, u1, u2, ud1, ud2, wd1, wd2;
  M3 R1, R2, dR1, dR2, Re0;
  double l0, radius;
};

struct ContactOut {
  double* K;   // 144
  double* C;   // 144
  double* T;   // 12
  double* E;   // 1
};

// interactions_beams_regularization.jl:2-26
EB_DEV void regularize_gap_penalty(double gap, double rb, double* p, double* dp, double* Pi) {
  double gt = rb / 4, hg = gt / 2;
  if (gap <= 0) {
    *p = hg - gap;
    *dp = -1.0;
    *Pi = (gap * gap) / 2 - hg * gap + (gt * gt) / 6;
  } else {
    double aux = (gt - hg) / (gt * gt);
    *p = aux * (gap * gap) - gap + hg;
    *dp = 2 * aux * gap - 1;
    *Pi = (gt - hg) / (3 * (gt * gt)) * (gap * gap * gap) - (gap * gap) / 2 + hg * gap - (gt * gt) / 6;
  }
}

// interactions_beams_regularization.jl:29-46
EB_DEV void smoothstep_transition(double value, double pos, double rb, double* s, double* ds) {
  double ul = rb / 4;
  if (pos <= 0) {
    *s = value;
    *ds = 0.0;
  } else {
    double np = (pos - ul) / ul;
    *s = np * np * (3 + 2 * np) * value;
    *ds = 6 / ul * np * (1 + np) * value;
  }
}

// Per-axis quadratic B-spline weights around the nearest grid point.
EB_DEV int bspline_axis(double t, int n, double w[3], double d[3]) {
  int i = (int)floor(t + 0.5);
  i = i < 0 ? 0 : (i > n - 1 ? n - 1 : i);
  double del = t - (double)i;
  double lo = 0.5 - del, hi = 0.5 + del;
  w[0] = 0.5 * (lo * lo);
  w[1] = 0.75 - del * del;
  w[2] = 0.5 * (hi * hi);
  d[0] = del - 0.5;
  d[1] = -2 * del;
  d[2] = del + 0.5;
  return i;
}

// Cell index (clamped to the grid's n-1 cells) and fraction along one axis.
EB_DEV int linear_axis(double t, int n, double* f) {
  int i = (int)floor(t);
  i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
  *f = t - (double)i;
  return i;
}

// Trilinear interpolant of the samples (8 taps of the padded grid, sample (i,j,k) at
// padded (i+1,j+1,k+1)): value, gradient and Hessian of the interpolating polynomial of
// the cell (its diagonal second derivatives vanish; the mixed ones do not).
EB_DEV double sdf_eval_linear(const SurfaceDev& s, V3 x, V3* grad, M3* hess) {
  double fx, fy, fz;
  const int ix = linear_axis((x.x - s.x0) * s.ihx, s.nx, &fx);
  const int iy = linear_axis((x.y - s.y0) * s.ihy, s.ny, &fy);
  const int iz = linear_axis((x.z - s.z0) * s.ihz, s.nz, &fz);
  const long px = s.nx + 2, py = s.ny + 2;
  const double* base = s.coef + ((ix + 1) + px * ((iy + 1) + py * (long)(iz + 1)));
  const double wx[2] = {1 - fx, fx}, wy[2] = {1 - fy, fy}, wz[2] = {1 - fz, fz};
  const double dd[2] = {-1.0, 1.0};
  double v = 0, gx = 0, gy = 0, gz = 0, hxy = 0, hxz = 0, hyz = 0;
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const double* row = base + px * (b + py * c);
      const double q0 = __ldg(row), q1 = __ldg(row + 1);
      const double sw = wx[0] * q0 + wx[1] * q1, sd = q1 - q0;
      v += wy[b] * wz[c] * sw;
      gx += wy[b] * wz[c] * sd;
      gy += dd[b] * wz[c] * sw;
      gz += wy[b] * dd[c] * sw;
      hxy += dd[b] * wz[c] * sd;
      hxz += wy[b] * dd[c] * sd;
      hyz += dd[b] * dd[c] * sw;
    }
  if (grad) {
    *grad = v3(gx * s.ihx, gy * s.ihy, gz * s.ihz);
    const double exy = hxy * (s.ihx * s.ihy), exz = hxz * (s.ihx * s.ihz), eyz = hyz * (s.ihy * s.ihz);
    *hess = rows(0.0, exy, exz, exy, 0.0, eyz, exz, eyz, 0.0);
  }
  return v;
}

// Value (and optionally gradient and Hessian) of the scaled quadratic
// B-spline interpolant at world point x (27 taps of the padded grid).
EB_DEV double sdf_eval(const SurfaceDev& s, V3 x, V3* grad, M3* hess) {
  if (s.interp == 1) return sdf_eval_linear(s, x, grad, hess);
  double wx[3], wy[3], wz[3], dx[3], dy[3], dz[3];
  int ix = bspline_axis((x.x - s.x0) * s.ihx, s.nx, wx, dx);
  int iy = bspline_axis((x.y - s.y0) * s.ihy, s.ny, wy, dy);
  int iz = bspline_axis((x.z - s.z0) * s.ihz, s.nz, wz, dz);
  const long px = s.nx + 2, py = s.ny + 2;
  const double* base = s.coef + (ix + px * (iy + py * (long)iz));
  double v = 0, gx = 0, gy = 0, gz = 0, hxx = 0, hyy = 0, hzz = 0, hxy = 0, hxz = 0, hyz = 0;
  const double dd[3] = {1.0, -2.0, 1.0};
  const bool full = grad != nullptr;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double* row = base + px * (b + py * c);
      double q0 = __ldg(row), q1 = __ldg(row + 1), q2 = __ldg(row + 2);
      double sw = wx[0] * q0 + wx[1] * q1 + wx[2] * q2;   // Σ wx q
      double wyz = wy[b] * wz[c];
      v += wyz * sw;
      if (full) {
        double sd = dx[0] * q0 + dx[1] * q1 + dx[2] * q2;  // Σ dx q
        double s2 = q0 - 2 * q1 + q2;                      // Σ ddx q
        gx += wyz * sd;
        gy += dy[b] * wz[c] * sw;
        gz += wy[b] * dz[c] * sw;
        hxx += wyz * s2;
        hyy += dd[b] * wz[c] * sw;
        hzz += wy[b] * dd[c] * sw;
        hxy += dy[b] * wz[c] * sd;
        hxz += wy[b] * dz[c] * sd;
        hyz += dy[b] * dz[c] * sw;
      }
    }
  }
  if (full) {
    *grad = v3(gx * s.ihx, gy * s.ihy, gz * s.ihz);
    double exy = hxy * (s.ihx * s.ihy), exz = hxz * (s.ihx * s.ihz), eyz = hyz * (s.ihy * s.ihz);
    *hess = rows(hxx * (s.ihx * s.ihx), exy, exz, exy, hyy * (s.ihy * s.ihy), eyz, exz, eyz, hzz * (s.ihz * s.ihz));
  }
  return v;
}

EB_DEV double axis_coord(V3 x, int a) { return a == 0 ? x.x : (a == 1 ? x.y : x.z); }

// PlaneSurface (def_interactions.jl:24-27) has no gap method in the reference; the one
// here follows the sphere's convention (utils_compute…:2-36): gap = x[axis] - pos - r,
// gradient e_axis, Hessian zero, contact when gap <= r/4.
EB_DEV bool incontact(const SurfaceDev& s, V3 x, double rb) {
  double gbar = rb / 4;
  if (s.kind == 2) return axis_coord(x, s.axis) - s.pos - rb <= gbar;
  if (s.kind == 0) {  // utils_compute_interactions_beams.jl:23-36
    V3 aux = x - v3(s.cx, s.cy, s.cz);
    return norm(aux) - s.R - rb <= gbar;
  }
  // isinside (utils_compute…:39-47) && φ - r ≤ r/4 (:67-75)
  double lx = x.x - s.x0, ly = x.y - s.y0, lz = x.z - s.z0;
  bool in = lx >= 0 && lx <= s.xl && ly >= 0 && ly <= s.yl && lz >= 0 && lz <= s.zl;
  if (!in) return false;
  return sdf_eval(s, x, nullptr, nullptr) - rb <= gbar;
}

EB_DEV void contact_gap(const SurfaceDev& s, V3 x, double rb, double* g, V3* dg, M3* d2g) {
  if (s.kind == 2) {
    *g = axis_coord(x, s.axis) - s.pos - rb;
    *dg = v3(s.axis == 0 ? 1.0 : 0.0, s.axis == 1 ? 1.0 : 0.0, s.axis == 2 ? 1.0 : 0.0);
    *d2g = zm3();
    return;
  }
  if (s.kind == 0) {  // utils_compute…:2-20
    V3 aux = x - v3(s.cx, s.cy, s.cz);
    double na = norm(aux);
    *g = na - s.R - rb;
    double inv = 1 / na;
    *dg = inv * aux;
    M3 h = (-(inv * inv * inv)) * outer(aux, aux);
    h.a[0] += inv; h.a[4] += inv; h.a[8] += inv;
    *d2g = h;
    return;
  }
  // utils_compute…:50-64 (Hessian projected with the already-normalised gradient)
  V3 gr;
  M3 H;
  double v = sdf_eval(s, x, &gr, &H);
  double nn = dot(gr, gr);
  double nmaginv = 1 / sqrt(nn);
  gr = nmaginv * gr;
  M3 P = (-1.0 / nn) * outer(gr, gr);
  P.a[0] += 1; P.a[4] += 1; P.a[8] += 1;
  *g = v - rb;
  *dg = gr;
  *d2g = (nmaginv * H) * P;
}

// Table of a contact element: the beam element's frame entries (eb_beam.cuh), then
enum {
  kCtVel = 25,    // 2 x 6: u̇, ẇ of the end nodes in the element frame
  kCtTa = 37,     // 2 x 9: Ts⁻¹(Δθ)ᵀ of the end rotations
  kCtSize = 55
};
// Table of a Gauss point in contact.
enum {
  kPtRHR = 0,     // 3 x 9: Rₑ H₁ⁱ Rₑᵀ, i = 1, 2, 4 (the third is the first's complement)
  kPtA1 = 27,     // 9
  kPtA2 = 36,     // 9
  kPtD = 45,      // 9: Rₑ (H₁F₁ - S(h₁))
  kPtRS = 54,     // 9: Rₑ S(Ẇᵉ)
  kPtW = 63,      // 3 x 9: H₁ⁱᵀ S(𝓕ᶜ) - S(H₁ⁱᵀ𝓕ᶜ), i = 1, 2, 4
  kPtF = 90,      // 3: 𝓕ᶜ
  kPtN = 93,      // N₇/l, N₇/l², N₃, N₄
  kPtSize = 97
};

// The pieces read an element through IO: x(n), R(n), dR(n), Re0(), ud(n), wd(n), l0(), radius().
// Node n's local rotation and velocities.
template <typename IO>
EB_PIECE void contact_node(const IO& io, int n, Tab t) {
  const M3 Re = t.m(kTabRe);
  t.put(kTabTh + 3 * n, toangle(mulTN(Re, io.R(n)) * io.Re0()));
  t.put(kCtVel + 6 * n, mulTv(Re, io.ud(n)));
  t.put(kCtVel + 6 * n + 3, mulTv(Re, io.wd(n)));
}
template <typename IO>
EB_PIECE void contact_exact(const IO& io, int n, Tab t) {
  t.put(kCtTa + 9 * n, tr(Ts_inv(toangle(io.dR(n)))));
}

struct ContactShape {
  double N1, N2, N3, N4;
  V3 ut, xG;
};
template <typename IO>
EB_DEV ContactShape contact_shape(const IO& io, const Tab& t, double zg) {
  ContactShape q;
  const double l0 = io.l0();
  const V3 Th1 = t.v(kTabTh), Th2 = t.v(kTabTh + 3);
  double xi = l0 * (zg + 1) / 2;
  double s = xi / l0;
  q.N1 = 1 - s;
  q.N2 = 1 - q.N1;
  q.N3 = xi * ((1 - s) * (1 - s));
  q.N4 = -(1 - s) * ((xi * xi) / l0);
  q.ut = v3(0.0, q.N3 * Th1.z + q.N4 * Th2.z, -q.N3 * Th1.y - q.N4 * Th2.y);
  q.xG = q.N1 * io.x(0) + q.N2 * io.x(1) + t.m(kTabRe) * q.ut;
  return q;
}
// Whether a Gauss point is in contact (:72, :95).
template <typename IO>
EB_PIECE bool contact_test(const IO& io, const SurfaceDev& srf, Tab t, double zg) {
  return incontact(srf, contact_shape(io, t, zg).xG, io.radius());
}
template <typename IO>
EB_PIECE void contact_distance(const IO& io, const SurfaceDev& srf, Tab t, double zg, double* gn, V3* dg, M3* d2g) {
  contact_gap(srf, contact_shape(io, t, zg).xG, io.radius(), gn, dg, d2g);
}

// A Gauss point's quantities into its table p, A1, A2, W and 𝓕ᶜ scaled by the weight wl = w lₒ/2, so
// that every block is too; `eta_n` and `deta_n` as the reference's scoping leaves them at this
// point.  emit.T(i, x) and emit.E(x) add over the Gauss points.
template <typename IO, typename EMIT>
EB_PIECE void contact_point(const IO& io, const ContactProps& cp, Tab t, Tab p, double zg, double wl, double gn, V3 dg,
                            const M3& d2g, double eta_n, double deta_n, EMIT emit) {
  const M3 I3 = eye3();
  const M3 Re = t.m(kTabRe);
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const double il = t.at(kTabLn + 1), rb = io.radius();
  const double kn = cp.kn, mu = cp.mu, eps_t = cp.eps_t;
  const ContactShape q = contact_shape(io, t, zg);
  const V3 Ud1 = t.v(kCtVel), Wd1 = t.v(kCtVel + 3), Ud2 = t.v(kCtVel + 6), Wd2 = t.v(kCtVel + 9);
  const double N1 = q.N1, N2 = q.N2, N3 = q.N3, N4 = q.N4, N7 = N3 + N4;
  const double N7l = N7 * il, N7l2 = N7l * il;
  M3 Sut = skew(q.ut);
  M3 SutG1 = mulG(Sut, G1);
  M3 H1[4];
  H1[0] = diag3(N1, N1 + N7l, N1 + N7l) - SutG1;
  H1[1] = rows(0, 0, 0, 0, 0, N3, 0, -N3, 0) - mulG(Sut, G2);
  H1[2] = diag3(N2, N2 - N7l, N2 - N7l) + SutG1;
  H1[3] = rows(0, 0, 0, 0, 0, N4, 0, -N4, 0) - mulG(Sut, G4);
  V3 h1 = H1[0] * Ud1 + H1[1] * Wd1 + H1[2] * Ud2 + H1[3] * Wd2;
  M3 H1F1 = mulskew(H1[0], Ud1) + mulskew(H1[1], Wd1) + mulskew(H1[2], Ud2) + mulskew(H1[3], Wd2);
  V3 ud0 = Re * h1;

  double pn, dpn, Pie;
  regularize_gap_penalty(gn, rb, &pn, &dpn, &Pie);
  double udn_mag = dot(ud0, dg);
  V3 udn = udn_mag * dg;
  V3 udt = ud0 - udn;
  double udt2 = dot(udt, udt);
  emit.E(wl * kn * Pie);
  V3 fn = (kn * pn) * dg - eta_n * udn;
  double mureg = mu / sqrt(udt2 + eps_t);
  V3 ft = (-(kn * pn) * mureg) * udt;
  V3 fc = wl * (fn + ft);
  V3 Fc = mulTv(Re, fc);
  p.put(kPtF, Fc);
  p.at(kPtN) = N7l; p.at(kPtN + 1) = N7l2; p.at(kPtN + 2) = N3; p.at(kPtN + 3) = N4;
  {  // H₁¹ + H₁³ = I (N₁ + N₂ = 1)
    const M3 R0 = mulNT(Re * H1[0], Re);
    const V3 T0 = mulTv(R0, fc);
    emit.T(0, T0);
    emit.T(2, fc - T0);
    p.put(kPtRHR, R0);
  }
#pragma unroll
  for (int i = 1; i < 4; i += 2) {
    const M3 Ri = mulNT(Re * H1[i], Re);
    emit.T(i, mulTv(Ri, fc));
    p.put(kPtRHR + 9 * (i == 3 ? 2 : 1), Ri);
  }
  const M3 SFc = skew(Fc);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i != 2) p.put(kPtW + 9 * (i == 3 ? 2 : i), mulTN(H1[i], SFc) - skew(mulTv(H1[i], Fc)));

  // ∂u̇₀/∂d (:211-238)
  const V3 We = Gv(G1, Ud1 - Ud2) + Gv(G2, Wd1) + Gv(G4, Wd2);
  p.put(kPtD, Re * (H1F1 - skew(h1)));
  p.put(kPtRS, mulskew(Re, We));
  M3 aux = dot(dg, ud0) * d2g + outer(dg, d2g * ud0);
  M3 nn = outer(dg, dg);
  M3 auxK = (kn * dpn) * nn + (kn * pn) * d2g - outer(deta_n * udn, dg);
  M3 aux1 = outer(((-mureg) * kn * dpn) * udt, dg);
  M3 aux2 = ((-mureg) * kn * pn) * (I3 - (1 / (udt2 + eps_t)) * outer(udt, udt));
  // The reference's ∂u̇ₙ/∂d = aux Rⱼ + nn D⁰ⱼ, ∂u̇ₜ/∂d = D⁰ⱼ - ∂u̇ₙ/∂d and ∂u̇ₜ/∂u̇ = Rⱼ - nn Rⱼ,
  // substituted and collected (14 products instead of 32):
  //   Kfcⱼ = A1 Rⱼ + A2 D⁰ⱼ,  Cfcⱼ = A2 Rⱼ,
  //   A1 = auxK + aux1 - (ηₙ I + aux2) aux,  A2 = aux2 - aux2 nn - ηₙ nn.
  M3 eta_aux2 = aux2;
  eta_aux2.a[0] += eta_n; eta_aux2.a[4] += eta_n; eta_aux2.a[8] += eta_n;
  p.put(kPtA1, wl * ((auxK + aux1) - eta_aux2 * aux));
  p.put(kPtA2, wl * (aux2 - (aux2 * nn + eta_n * nn)));
}

// Block columns of Kᶜ and Cᶜ at a Gauss point (:332-370): c = 0: columns 1 and 3, 1: column 2, 2:
// column 4.  Per row block i:
//   t₁ + t₃ (:128-155, :186-209): Rₑ[-S(H₁ⁱᵀ𝓕ᶜ) + H₁ⁱᵀS(𝓕ᶜ)] Gʲ Rₑᵀ (column 3 is minus column 1),
//   t₂ (:157-184) = -Rₑ Gⁱᵀ (S(𝓕ᶜ) P₁ʲ Rₑᵀ), for i = j = 1 with A₁.
// H₁¹ + H₁³ = I, so row block 3 is row block 1's complement: its t₁+t₃ and t₂ are minus row 1's, and
// its Rₑ H₁³ Rₑᵀ = I - Rₑ H₁¹ Rₑᵀ gives Kᶜ/Cᶜ terms Kfcⱼ - t₄¹ʲ; likewise Kfc₃ = A1 - Kfc₁, Cfc₃ = A2 - Cfc₁.
// emit.K(i, j, x), emit.C(i, j, x) add over the Gauss points.
template <int COL, typename EMIT>
EB_PIECE void contact_column(Tab t, Tab p, EMIT emit) {
  const M3 Re = t.m(kTabRe);
  const M3 ReT = tr(Re);
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const V3 Fc = p.v(kPtF), v1 = col(Re, 0);
  const M3 SFc = skew(Fc), RS = p.m(kPtRS);
  M3 SFP, du0, A1F;  // S(𝓕ᶜ) P₁ʲ Rₑᵀ, D⁰ⱼ
  if (COL == 0) {
    const V3 dU = t.v(kCtVel) - t.v(kCtVel + 6);
    const double N7l = p.at(kPtN), N7l2 = p.at(kPtN + 1);
    const V3 d = v3(0.0, N7l, N7l);
    SFP = muld(SFc, d) * ReT;
    du0 = p.m(kPtD) * Gmul(G1, ReT) + muld(RS, d) * ReT;
    du0 += N7l2 * (Re * rows(0, 0, 0, v1.x * dU.y, v1.y * dU.y, v1.z * dU.y, v1.x * dU.z, v1.y * dU.z, v1.z * dU.z));
    A1F = N7l2 * rows(0, 0, 0, Fc.y * v1.x, Fc.y * v1.y, Fc.y * v1.z, Fc.z * v1.x, Fc.z * v1.y, Fc.z * v1.z);
  } else {
    const double N = p.at(COL == 1 ? kPtN + 2 : kPtN + 3);
    const M3 P = rows(0, 0, 0, 0, 0, N, 0, -N, 0);
    SFP = (SFc * P) * ReT;
    du0 = p.m(kPtD) * Gmul(COL == 1 ? G2 : G4, ReT) + (RS * P) * ReT;
    A1F = zm3();
  }
  constexpr int j = COL == 2 ? 3 : COL;
  const M3 A1 = p.m(kPtA1), A2 = p.m(kPtA2), Rj = p.m(kPtRHR + 9 * COL);
  const M3 Kf = A1 * Rj + A2 * du0, Cf = A2 * Rj;
  // W Gʲ Rₑᵀ: Gᵀ¹ has three entries, Gᵀ² and Gᵀ⁴ one row
  const V3 r0 = col(Re, 0), r1 = col(Re, 1), r2 = col(Re, 2);
  const Gt G = COL == 1 ? G2 : G4;
  const V3 rg = G.a * r0 + G.b * r1;
#pragma unroll
  for (int row = 0; row < 3; ++row) {
    const int i = row == 2 ? 3 : row;
    const M3 W = p.m(kPtW + 9 * row);
    const M3 GS = i == 0 ? GTmul(G1, SFP) : (i == 1 ? GTmul(G2, SFP) : GTmul(G4, SFP));
    M3 in = COL == 0 ? outer(G1.g13 * col(W, 0) + G1.g23 * col(W, 1), r2) + outer(G1.g32 * col(W, 2), r1)
                     : outer(col(W, 0), rg);
    in = in - GS;
    if (COL == 0 && i == 0) in += A1F;
    const M3 t12 = Re * in, Ri = p.m(kPtRHR + 9 * row);
    const M3 t4 = mulTN(Ri, Kf), tc = mulTN(Ri, Cf);
    emit.K(i, j, t12 + t4);
    emit.C(i, j, tc);
    if (i == 0) {
      emit.K(2, j, (Kf - t4) - t12);
      emit.C(2, j, Cf - tc);
    }
    if (COL == 0) {
      const M3 t43 = mulTN(Ri, A1) - t4, tc3 = mulTN(Ri, A2) - tc;
      emit.K(i, 2, t43 - t12);
      emit.C(i, 2, tc3);
      if (i == 0) {
        emit.K(2, 2, ((A1 - Kf) - t43) + t12);
        emit.C(2, 2, (A2 - Cf) - tc3);
      }
    }
  }
}

#if !defined(__CUDACC__)
// One element in sequence (host checks of the pieces).
struct ContactRecord {
  const ContactIn& in;
  V3 x(int n) const { return n ? in.X2 + in.u2 : in.X1 + in.u1; }
  M3 R(int n) const { return n ? in.R2 : in.R1; }
  M3 dR(int n) const { return n ? in.dR2 : in.dR1; }
  M3 Re0() const { return in.Re0; }
  V3 ud(int n) const { return n ? in.ud2 : in.ud1; }
  V3 wd(int n) const { return n ? in.wd2 : in.wd1; }
  double l0() const { return in.l0; }
  double radius() const { return in.radius; }
};

inline void contact_element(const ContactIn& in, const Gauss3& gs, const ContactProps& cp, const SurfaceDev& srf,
                            ContactOut out, bool* any_contact) {
  const ContactRecord io{in};
  double tab[kCtSize], pt[kPtSize];
  const Tab t{tab, 1}, p{pt, 1};
  beam_frame(io, t);
  for (int n = 0; n < 2; ++n) contact_node(io, n, t);
  bool inc[3];
  *any_contact = false;
  for (int g = 0; g < 3; ++g) *any_contact |= inc[g] = contact_test(io, srf, t, gs.z[g]);
  if (!*any_contact) return;
  for (int n = 0; n < 2; ++n) contact_exact(io, n, t);
  struct Add {
    ContactOut o;
    void T(int i, V3 x) const { o.T[3 * i] += x.x; o.T[3 * i + 1] += x.y; o.T[3 * i + 2] += x.z; }
    void E(double x) const { o.E[0] += x; }
    void K(int i, int j, const M3& x) const { acc_block(o.K, i, j, 1.0, x); }
    void C(int i, int j, const M3& x) const { acc_block(o.C, i, j, 1.0, x); }
  } emit{out};
  for (int k = 0; k < 144; ++k) out.K[k] = out.C[k] = 0.0;
  for (int k = 0; k < 12; ++k) out.T[k] = 0.0;
  out.E[0] = 0.0;
  double eta_n = cp.eta_n;  // overwritten by each in-contact Gauss point (reference scoping)
  for (int g = 0; g < 3; ++g) {
    if (!inc[g]) continue;
    double gn, deta_n;
    V3 dg;
    M3 d2g;
    contact_distance(io, srf, t, gs.z[g], &gn, &dg, &d2g);
    smoothstep_transition(eta_n, gn, in.radius, &eta_n, &deta_n);
    contact_point(io, cp, t, p, gs.z[g], gs.w[g] * (in.l0 / 2), gn, dg, d2g, eta_n, deta_n, emit);
    contact_column<0>(t, p, emit);
    contact_column<1>(t, p, emit);
    contact_column<2>(t, p, emit);
  }
  for (int i = 1; i < 4; i += 2)
    for (int j = 0; j < 4; ++j) put_block(out.C, i, j, get_block(out.C, i, j) * t.m(kCtTa + (i == 3 ? 9 : 0)));
}
#else
// ------------------------------------------------------------------ cooperative evaluation
// A CTA of three warps evaluates ten elements (the Gauss points on one warp, the block columns on
// three: the shortest chain, for launches that leave SMs idle) or thirty (each warp its own ten,
// nothing formed twice).  Elements without contact stop after the gap test.
constexpr int kContactCta = 96;
__host__ __device__ inline size_t contact_smem(int nb) {
  return sizeof(double) * ((size_t)kCtSize * kBeamGroup + (size_t)kPtSize * 32) * nb;
}

// Sums over the three lanes of an element in Gauss order (points not in contact add nothing) into
// its outputs.  Lane g sums the g-th of three values, so of a 3x3 block it holds row g, and
// the rows of Cᶜ that take Tₐᵀ / T_bᵀ are transformed by the lane that holds them.
struct EmitContact {
  ContactOut o;
  Tab t;
  int base, g;
  bool inc, store;
  __device__ __forceinline__ double sum(V3 x) const {
    if (!inc) x = zv3();
    const double up = g == 0 ? x.z : (g == 1 ? x.x : x.y);    // to lane g - 1 (mod 3)
    const double down = g == 0 ? x.y : (g == 1 ? x.z : x.x);  // to lane g + 1 (mod 3)
    const double own = g == 0 ? x.x : (g == 1 ? x.y : x.z);
    const double next = __shfl_sync(0xffffffffu, up, base + (g == 2 ? 0 : g + 1));
    const double prev = __shfl_sync(0xffffffffu, down, base + (g == 0 ? 2 : g - 1));
    const double v0 = g == 0 ? own : (g == 1 ? prev : next);
    const double v1 = g == 1 ? own : (g == 2 ? prev : next);
    const double v2 = g == 2 ? own : (g == 0 ? prev : next);
    return (v0 + v1) + v2;
  }
  __device__ __forceinline__ void T(int i, V3 x) const {
    const double v = sum(x);
    if (store) o.T[3 * i + g] = v;
  }
  __device__ __forceinline__ void E(double x) const {
    const double v = sum(v3(x, 0.0, 0.0));
    if (store && g == 0) o.E[0] = v;
  }
  __device__ __forceinline__ V3 row(const M3& x) const {
    return v3(sum(col(x, 0)), sum(col(x, 1)), sum(col(x, 2)));
  }
  __device__ __forceinline__ void put(double* m, int i, int j, V3 r) const {
    if (!store) return;
    double* q = m + 3 * i + g + 36 * j;
    q[0] = r.x; q[12] = r.y; q[24] = r.z;
  }
  __device__ __forceinline__ void K(int i, int j, const M3& x) const { put(o.K, i, j, row(x)); }
  __device__ __forceinline__ void C(int i, int j, const M3& x) const {
    V3 r = row(x);
    if (i & 1) r = mulTv(t.m(kCtTa + (i == 3 ? 9 : 0)), r);
    put(o.C, i, j, r);
  }
};

// nb = 1 or 3 groups of ten elements.  make(e): element e's IO with surf(), props(), out() and
// touched(bool); on(e): whether it is evaluated (both for e < n only).
template <typename MAKE, typename ON>
__device__ __forceinline__ void contact_cta(int64_t n, int nb, const Gauss3& gs, double* tab, MAKE make, ON on) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = kBeamGroup * nb;
  const int64_t e0 = (int64_t)blockIdx.x * E;
  __shared__ unsigned char act[32];
  __shared__ unsigned inc_mask[3];
  bool mine = false;
  if (threadIdx.x < E) {
    mine = e0 + threadIdx.x < n && on(e0 + threadIdx.x);
    act[threadIdx.x] = mine;
  }
  if (!__syncthreads_or(mine)) return;
  auto table = [&](int e) { return Tab{tab + e, E}; };
  if (warp == 0 && lane < E && act[lane]) beam_frame(make(e0 + lane), table(lane));
  __syncthreads();
  if (threadIdx.x < 2 * E && act[threadIdx.x >> 1])
    contact_node(make(e0 + (threadIdx.x >> 1)), threadIdx.x & 1, table(threadIdx.x >> 1));
  __syncthreads();
  // lanes without an element of their own repeat another's, but are never in contact (30, 31: the
  // last element's first two points)
  const int group = nb == 1 ? 0 : warp;
  const bool own = lane < 3 * kBeamGroup;
  const int sub = own ? lane / 3 : kBeamGroup - 1, g = own ? lane - 3 * sub : lane - 30;
  const int el = kBeamGroup * group + sub;
  const bool mineg = own && act[el];
  int e = el;
  if (!act[e])
    for (e = 0; !act[e]; ++e) {
    }
  const auto io = make(e0 + e);
  const Tab t = table(e);
  const double zg = g == 0 ? gs.z[0] : (g == 1 ? gs.z[1] : gs.z[2]);
  const double wg = g == 0 ? gs.w[0] : (g == 1 ? gs.w[1] : gs.w[2]);
  if (nb > 1 || warp == 0) {
    const bool in = mineg && contact_test(io, io.surf(), t, zg);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) inc_mask[group] = m;
    if (mineg && g == 0) io.touched(((m >> (3 * sub)) & 7u) != 0);
  }
  __syncthreads();
  const unsigned mask = inc_mask[group];
  if (!__syncthreads_or(mask != 0)) return;
  const bool inc = own && ((mask >> lane) & 1u);
  const bool touched = mineg && ((mask >> (3 * sub)) & 7u) != 0;
  Tab p{tab + (int64_t)kCtSize * E + 32 * kPtSize * group + lane, 32};
  const EmitContact emit{io.out(), t, 3 * sub, g, inc, touched};
  // exact-mode transforms of the touched elements: beside the Gauss points, or by the group's own warp
  if (mask && (nb > 1 || warp == 1)) {
    const int pe = lane >> 1;
    if (pe < kBeamGroup && act[kBeamGroup * group + pe] && ((mask >> (3 * pe)) & 7u))
      contact_exact(make(e0 + kBeamGroup * group + pe), lane & 1, table(kBeamGroup * group + pe));
  }
  if (mask && (nb > 1 || warp == 0)) {
    double gn = 0.0;
    V3 dg = v3(1.0, 0.0, 0.0);
    M3 d2g = zm3();
    if (inc) contact_distance(io, io.surf(), t, zg, &gn, &dg, &d2g);
    // ηₙ as the in-contact points before this one, and this one, leave it
    double eta = io.props().eta_n, deta = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double gk = __shfl_sync(0xffffffffu, gn, 3 * sub + k);
      if (k <= g && ((mask >> (3 * sub + k)) & 1u)) smoothstep_transition(eta, gk, io.radius(), &eta, &deta);
    }
    contact_point(io, io.props(), t, p, zg, wg * (io.l0() / 2), gn, dg, d2g, eta, deta, emit);
  }
  __syncthreads();
  if (!mask) return;
  if (nb > 1 || warp == 0) contact_column<0>(t, p, emit);
  if (nb > 1 || warp == 1) contact_column<1>(t, p, emit);
  if (nb > 1 || warp == 2) contact_column<2>(t, p, emit);
}
#endif

}  // namespace ebd
