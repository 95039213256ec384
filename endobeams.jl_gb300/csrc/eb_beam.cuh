// Corotational beam element on the GPU, FP64.
//
// Same quantities as compute_beams (src/beams/compute_beams.jl:1-538, the
// `exact=true, isdynamic=true` path used by assemble!): strain and kinetic
// energy, Tⁱⁿᵗ, Tᵏ (12) and Kⁱⁿᵗ, M, Cᵏ (12x12, column-major).  The
// formulas are the reference's; the evaluation exploits their structure
// (sparse Gᵀ/P/H₂ matrices, skew commutators, reuse of Bᵀ·K̄ₕ products) to
// cut FP64 instructions, which bound this kernel on GB300.
//
// An element is about 16,400 FP64 operations.  One thread per element runs them
// as one dependent chain (0.40 ms a launch even for 20 elements), which is best for
// tens of thousands of elements only; here the element is cut into pieces that
// share a table (shared memory on the device): its frame, angles and velocities
// (beam_frame, beam_exact, beam_velocity, one lane per end node), the static
// stiffness in two halves (beam_static), the mass and the gyroscopic blocks per
// Gauss point (beam_mass, beam_gyro, one lane per element and Gauss point) and the
// rotation of every 3x3 block back to global axes (beam_block, one lane per
// element and block).  The pieces are functions of their own, not inlined: how they
// are spread over warps does not change a bit of their results.
#pragma once
#include "eb_device_math.cuh"

#if defined(__CUDACC__)
#define EB_PIECE static __device__ __noinline__
#else
#define EB_PIECE inline
#endif

namespace ebd {

struct BeamIn {
  V3 X1, X2, u1, u2, ud1, ud2, wd1, wd2, udd1, udd2, wdd1, wdd2;
  M3 R1, R2, dR1, dR2, Re0;
  double l0, Ku, Ar, damping;
  V3 KT, KTT, Jr;
};

struct BeamOut {  // destinations (any stride-1 buffers)
  double* K;    // 144
  double* M;    // 144
  double* C;    // 144
  double* Tint; // 12
  double* Tk;   // 12
  double* E;    // 2: strain, kinetic
};

struct Gauss3 {
  double w[3], z[3];
};

EB_DEV void put_block(double* m, int bi, int bj, const M3& b) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) m[(3 * bi + i) + 12 * (3 * bj + j)] = b(i, j);
}
EB_DEV void put_blockT(double* m, int bi, int bj, const M3& b) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) m[(3 * bi + i) + 12 * (3 * bj + j)] = b(j, i);
}
EB_DEV void put_vec(double* v, int bi, V3 x) { v[3 * bi] = x.x; v[3 * bi + 1] = x.y; v[3 * bi + 2] = x.z; }
EB_DEV M3 get_block(const double* m, int bi, int bj) {
  M3 b;
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) b(i, j) = m[(3 * bi + i) + 12 * (3 * bj + j)];
  return b;
}
// block (bi, bj) of a 12x12 column-major matrix += s q (fused multiply-add per entry)
EB_DEV void acc_block(double* m, int bi, int bj, double s, const M3& q) {
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double& x = m[(3 * bi + i) + 12 * (3 * bj + j)];
      x = fma(s, q(i, j), x);
    }
}

// Element frame and auxiliaries of local_Rₑ_and_aux (utils_beams.jl:35-87).
struct Frame {
  M3 Re;
  V3 v1;
  double eta, ln;
  Gu G1;      // Gᵀ¹ ; Gᵀ³ = -Gᵀ¹
  Gt G2, G4;  // Gᵀ², Gᵀ⁴
};

EB_DEV Frame local_frame(V3 x1, V3 x2, const M3& R1, const M3& R2, V3 e2, double ln) {
  Frame f;
  f.ln = ln;
  V3 v1 = (1.0 / ln) * (x2 - x1);
  V3 p1 = R1 * e2, p2 = R2 * e2;
  V3 p = 0.5 * (p1 + p2);
  V3 v3_ = cross(v1, p);
  v3_ = (1.0 / norm(v3_)) * v3_;
  V3 v2 = cross(v3_, v1);
  f.Re = hcat3(v1, v2, v3_);
  f.v1 = v1;
  double q2 = dot(v2, p);
  double iq2 = 1.0 / q2;
  double eta = dot(v1, p) * iq2;
  double eta11 = dot(v1, p1) * iq2, eta12 = dot(v2, p1) * iq2;
  double eta21 = dot(v1, p2) * iq2, eta22 = dot(v2, p2) * iq2;
  f.eta = eta;
  double il = 1.0 / ln;
  f.G1 = Gu{eta * il, il, -il};
  f.G2 = Gt{eta12 / 2, -eta11 / 2};
  f.G4 = Gt{eta22 / 2, -eta21 / 2};
  return f;
}

// compute_K̄ₕ (utils_beams.jl:201-215)
EB_DEV M3 compute_Kh(V3 th, V3 Mb, const M3& Ts, double eta, double mu) {
  M3 MtT = outer(Mb, th);  // M̄Θ̅ᵀ
  M3 inner = eta * (outer(th, Mb) - 2.0 * MtT);
  double d = eta * dot(th, Mb);
  inner.a[0] += d; inner.a[4] += d; inner.a[8] += d;
  axpy(inner, mu, skewmul(th, skewmul(th, MtT)));
  axpy(inner, -0.5, skew(Mb));
  return inner * Ts;
}

// Gᵀ v for the GᵀΘ shape [a b 0; 0 0 0; 0 0 0]
EB_DEV V3 GTv(Gt g, V3 v) { return v3(g.a * v.x, g.b * v.x, 0.0); }

// Table of an element: entry i at p[i * ld].
enum {
  kTabRe = 0,     // 9: element frame
  kTabG = 9,      // 7: Gᵀ¹ (3), Gᵀ² (2), Gᵀ⁴ (2)
  kTabLn = 16,    // length, 1 / length, η
  kTabTh = 19,    // 2 x 3: Θ̄₁, Θ̄₂
  kTabT = 25,     // 2 x 9: Ts⁻¹(Θ̄)
  kTabEm = 43,    // 2 x 2: η, μ of K̄ₕ
  kTabVel = 47,   // 2 x 12: u̇, ẇ, ü, ẅ in the element frame
  kTabTa = 71,    // 2 x 9: Ts⁻¹(Δθ)ᵀ of the end rotations (exact mode)
  kTabM = 89,     // 10 x 9: M11 M12 M13 M14 M22 M23 M24 M33 M34 M44, Gauss sums in the element frame
  kTabTk = 179,   // 4 x 3, then the kinetic energy
  kTabC = 192,    // 12 x 9: C11 C12 C14 C21 C22 C24 C31 C32 C34 C41 C42 C44
  kTabSize = 300
};
struct Tab {
  double* p;
  int ld;
  EB_DEV double& at(int i) const { return p[(int64_t)i * ld]; }
  EB_DEV V3 v(int i) const { return v3(at(i), at(i + 1), at(i + 2)); }
  EB_DEV M3 m(int i) const {
    M3 r;
#pragma unroll
    for (int k = 0; k < 9; ++k) r.a[k] = at(i + k);
    return r;
  }
  EB_DEV void put(int i, V3 x) const { at(i) = x.x; at(i + 1) = x.y; at(i + 2) = x.z; }
  EB_DEV void put(int i, const M3& x) const {
#pragma unroll
    for (int k = 0; k < 9; ++k) at(i + k) = x.a[k];
  }
  EB_DEV Gu G1() const { return Gu{at(kTabG), at(kTabG + 1), at(kTabG + 2)}; }
  EB_DEV Gt G2() const { return Gt{at(kTabG + 3), at(kTabG + 4)}; }
  EB_DEV Gt G4() const { return Gt{at(kTabG + 5), at(kTabG + 6)}; }
};

// The pieces read an element through IO (node n of 0, 1):
//   V3 x(n) = X + u; M3 R(n), dR(n), Re0(); V3 ud(n), wd(n), udd(n), wdd(n);
//   double l0(), Ku(), Ar(), damping(); V3 KT(), KTT(), Jr(); BeamOut out().
// Element frame and auxiliaries.
template <typename IO>
EB_PIECE void beam_frame(const IO& io, Tab t) {
  const V3 x1 = io.x(0), x2 = io.x(1);
  const Frame f = local_frame(x1, x2, io.R(0), io.R(1), col(io.Re0(), 1), norm(x2 - x1));
  t.put(kTabRe, f.Re);
  t.at(kTabG) = f.G1.g13; t.at(kTabG + 1) = f.G1.g23; t.at(kTabG + 2) = f.G1.g32;
  t.at(kTabG + 3) = f.G2.a; t.at(kTabG + 4) = f.G2.b; t.at(kTabG + 5) = f.G4.a; t.at(kTabG + 6) = f.G4.b;
  t.at(kTabLn) = f.ln; t.at(kTabLn + 1) = 1.0 / f.ln; t.at(kTabLn + 2) = f.eta;
}
// Node n's local rotation with its Ts⁻¹, η, μ.
template <typename IO>
EB_PIECE void beam_angle(const IO& io, int n, Tab t) {
  const V3 Th = toangle(mulTN(t.m(kTabRe), io.R(n)) * io.Re0());
  t.put(kTabTh + 3 * n, Th);
  t.put(kTabT + 9 * n, Ts_inv(Th));
  double eta, mu;
  compute_eta_mu(Th, &eta, &mu);
  t.at(kTabEm + 2 * n) = eta;
  t.at(kTabEm + 2 * n + 1) = mu;
}
// Ts⁻¹(Δθ_n)ᵀ of the exact-mode transforms (:480-506)
template <typename IO>
EB_PIECE void beam_exact(const IO& io, int n, Tab t) {
  t.put(kTabTa + 9 * n, tr(Ts_inv(toangle(io.dR(n)))));
}
// Node n's velocities and accelerations in the element frame.
template <typename IO>
EB_PIECE void beam_velocity(const IO& io, int n, Tab t) {
  const M3 Re = t.m(kTabRe);
  const int o = kTabVel + 12 * n;
  t.put(o, mulTv(Re, io.ud(n)));
  t.put(o + 3, mulTv(Re, io.wd(n)));
  t.put(o + 6, mulTv(Re, io.udd(n)));
  t.put(o + 9, mulTv(Re, io.wdd(n)));
}

// Static part (:13-159): what both halves use, then half 0, the first block row of Kⁱⁿᵗ, and half
// 1, the other rows and Tⁱⁿᵗ.
struct BeamStatic {
  M3 Bp11, Bp12, Bp22, Bp14, Bp24, B11, B12, B14, B21, B22, B24, Kh1, Kh2, Z12, Z22, Z14, Z24;
  V3 TT1, TT2, Mps, Qs1, Qs2, Qs4;
  double Tu, ubar;
};
template <typename IO>
EB_PIECE void beam_static_common(const IO& io, Tab t, BeamStatic& q) {
  const M3 ReT = tr(t.m(kTabRe));
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const V3 Th1 = t.v(kTabTh), Th2 = t.v(kTabTh + 3);
  const M3 T1 = t.m(kTabT), T2 = t.m(kTabT + 9);
  const V3 KT = io.KT(), KTT = io.KTT();
  M3 G1ReT = Gmul(G1, ReT), G2ReT = Gmul(G2, ReT), G4ReT = Gmul(G4, ReT);
  q.Bp11 = -G1ReT;          // P¹¹Rₑᵀ = B̄⁺¹¹ = B̄⁺²¹
  q.Bp12 = ReT - G2ReT;     // (I-Gᵀ²)Rₑᵀ
  q.Bp22 = -G2ReT;
  q.Bp14 = -G4ReT;
  q.Bp24 = ReT - G4ReT;
  q.B11 = T1 * q.Bp11; q.B12 = T1 * q.Bp12; q.B14 = T1 * q.Bp14;
  q.B21 = T2 * q.Bp11; q.B22 = T2 * q.Bp22; q.B24 = T2 * q.Bp24;
  q.ubar = t.at(kTabLn) - io.l0();
  q.Tu = io.Ku() * q.ubar;
  q.TT1 = dmulv(KT, Th1) + dmulv(KTT, Th2);
  q.TT2 = dmulv(KTT, Th1) + dmulv(KT, Th2);
  V3 Mp1 = mulTv(T1, q.TT1), Mp2 = mulTv(T2, q.TT2);
  q.Mps = Mp1 + Mp2;
  q.Qs1 = -GTv(G1, q.Mps);                       // P¹¹ᵀM̄⁺₁ + P²¹ᵀM̄⁺₂
  q.Qs2 = Mp1 - GTv(G2, q.Mps);                  // (I-Gᵀ²)ᵀM̄⁺₁ - Gᵀ²ᵀM̄⁺₂
  q.Qs4 = Mp2 - GTv(G4, q.Mps);                  // -Gᵀ⁴ᵀM̄⁺₁ + (I-Gᵀ⁴)ᵀM̄⁺₂
  q.Kh1 = compute_Kh(Th1, q.TT1, T1, t.at(kTabEm), t.at(kTabEm + 1));
  q.Kh2 = compute_Kh(Th2, q.TT2, T2, t.at(kTabEm + 2), t.at(kTabEm + 3));
  q.Z12 = dmul(KT, q.B12) + dmul(KTT, q.B22); q.Z22 = dmul(KTT, q.B12) + dmul(KT, q.B22);
  q.Z14 = dmul(KT, q.B14) + dmul(KTT, q.B24); q.Z24 = dmul(KTT, q.B14) + dmul(KT, q.B24);
}
template <typename IO>
EB_PIECE void beam_static(const IO& io, Tab t, const BeamStatic& q, int half) {
  const M3 Re = t.m(kTabRe);
  const M3 ReT = tr(Re);
  const V3 v1 = col(Re, 0);
  const V3 r1 = -v1;  // B̄⁺¹ = ru₁
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const double il = t.at(kTabLn + 1), eta = t.at(kTabLn + 2), Tu = q.Tu;
  const V3 KT = io.KT(), KTT = io.KTT();
  const BeamOut out = io.out();
  double* K = out.K;
  if (half == 0) {
    M3 Q1 = skew(q.Qs1);
    V3 a = v3(0.0, eta * q.Mps.x * il + q.Mps.y * il, q.Mps.z * il);
    // D₃ N̄ = (I - v₁v₁ᵀ) N̄ / lₙ
    M3 Km11 = (Tu * il) * (eye3() - outer(v1, v1));
    Km11 = Km11 - (Re * mulG(Q1, G1)) * ReT;
    Km11 += outer(Re * GTv(G1, a), r1);
    M3 Km12 = -((Re * mulG(Q1, G2)) * ReT);
    M3 Km14 = -((Re * mulG(Q1, G4)) * ReT);
    // K̃ (:131-136) with the B̄⁺ᵀK̄ₕ left factors shared between blocks
    M3 Y11 = mulTN(q.Bp11, q.Kh1), Y21 = mulTN(q.Bp11, q.Kh2);
    M3 Kt11 = Y11 * q.Bp11 + Y21 * q.Bp11 + Km11;
    M3 Kt12 = Y11 * q.Bp12 + Y21 * q.Bp22 + Km12;
    M3 Kt14 = Y11 * q.Bp14 + Y21 * q.Bp24 + Km14;
    // BᵀK̄ⁱⁿᵗB (:139-146)
    M3 Z11 = dmul(KT, q.B11) + dmul(KTT, q.B21), Z21 = dmul(KTT, q.B11) + dmul(KT, q.B21);
    M3 K11 = outer(io.Ku() * r1, r1) + mulTN(q.B11, Z11) + mulTN(q.B21, Z21) + Kt11;
    M3 K12 = mulTN(q.B11, q.Z12) + mulTN(q.B21, q.Z22) + Kt12;
    M3 K14 = mulTN(q.B11, q.Z14) + mulTN(q.B21, q.Z24) + Kt14;
    // Kⁱⁿᵗ layout of :159 (blocks below the diagonal are transposes):
    // K¹³ = -K¹¹, K²³ = -K¹²ᵀ, K³³ = K¹¹, K³⁴ = -K¹⁴ (:150-156)
    M3 K13 = -K11, K34 = -K14, mK12 = -K12;
    put_block(K, 0, 0, K11);  put_blockT(K, 1, 0, K12);  put_blockT(K, 2, 0, K13); put_blockT(K, 3, 0, K14);
    put_block(K, 0, 1, K12);  put_block(K, 2, 1, mK12);
    put_block(K, 0, 2, K13);  put_blockT(K, 1, 2, mK12); put_block(K, 2, 2, K11);  put_blockT(K, 3, 2, K34);
    put_block(K, 0, 3, K14);  put_block(K, 2, 3, K34);
  } else {
    V3 Ti1 = Tu * r1 + mulTv(q.B11, q.TT1) + mulTv(q.B21, q.TT2);
    V3 Ti2 = mulTv(q.B12, q.TT1) + mulTv(q.B22, q.TT2);
    V3 Ti4 = mulTv(q.B14, q.TT1) + mulTv(q.B24, q.TT2);
    put_vec(out.Tint, 0, Ti1); put_vec(out.Tint, 1, Ti2); put_vec(out.Tint, 2, -Ti1); put_vec(out.Tint, 3, Ti4);
    out.E[0] = (q.ubar * Tu + dot(t.v(kTabTh), q.TT1) + dot(t.v(kTabTh + 3), q.TT2)) / 2;
    M3 Q2 = skew(q.Qs2), Q4 = skew(q.Qs4);
    M3 Km22 = -((Re * mulG(Q2, G2)) * ReT);
    M3 Km24 = -((Re * mulG(Q2, G4)) * ReT);
    M3 Km44 = -((Re * mulG(Q4, G4)) * ReT);
    M3 Y12 = mulTN(q.Bp12, q.Kh1), Y22 = mulTN(q.Bp22, q.Kh2);
    M3 Kt22 = Y12 * q.Bp12 + Y22 * q.Bp22 + Km22;
    M3 Kt24 = Y12 * q.Bp14 + Y22 * q.Bp24 + Km24;
    M3 Kt44 = mulTN(q.Bp14, q.Kh1) * q.Bp14 + mulTN(q.Bp24, q.Kh2) * q.Bp24 + Km44;
    M3 K22 = mulTN(q.B12, q.Z12) + mulTN(q.B22, q.Z22) + Kt22;
    M3 K24 = mulTN(q.B12, q.Z14) + mulTN(q.B22, q.Z24) + Kt24;
    M3 K44 = mulTN(q.B14, q.Z14) + mulTN(q.B24, q.Z24) + Kt44;
    put_block(K, 1, 1, K22); put_blockT(K, 3, 1, K24); put_block(K, 1, 3, K24); put_block(K, 3, 3, K44);
  }
}

// What the mass and gyroscopic pieces share at one Gauss point (:202-300).
struct GaussPoint {
  double N1, N2, N3, N4, N5, N6, N7l, N7l2, N8l, N8l2, wg;
  M3 H11, H12, H13, H14, Ir, P1P2, P1P4;
  V3 s21, d22, d24;   // H₂¹ = skew(s21), H₂³ = -H₂¹, H₂² = diag(d22), H₂⁴ = diag(d24)
  V3 dU, Wd1, Wd2, We, h1, h2;
  M3 C11, C12, C14, C21, C22, C24;
};

EB_PIECE void gauss_point(Tab t, double l0, V3 Jr, double zg, double wg, GaussPoint& q) {
  q.wg = wg;
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const V3 Th1 = t.v(kTabTh), Th2 = t.v(kTabTh + 3);
  const V3 Ud1 = t.v(kTabVel), Wd1 = t.v(kTabVel + 3), Ud2 = t.v(kTabVel + 12), Wd2 = t.v(kTabVel + 15);
  const double il = t.at(kTabLn + 1);
  const V3 dU = Ud1 - Ud2;
  const double rd = -dU.x;  // r¹·u̇₁ + r³·u̇₂, r³ = -r¹ = v₁
  q.dU = dU; q.Wd1 = Wd1; q.Wd2 = Wd2;
  q.We = Gv(G1, dU) + Gv(G2, Wd1) + Gv(G4, Wd2);  // Gᵀ³ = -Gᵀ¹
  double xi = l0 * (zg + 1) / 2;
  double s = xi / l0;
  q.N1 = 1 - s;
  q.N2 = 1 - q.N1;
  q.N3 = xi * ((1 - s) * (1 - s));
  q.N4 = -(1 - s) * ((xi * xi) / l0);
  q.N5 = (1 - 3 * s) * (1 - s);
  q.N6 = (3 * s - 2) * s;
  const double N7 = q.N3 + q.N4, N8 = q.N5 + q.N6 - 1;
  const double N1 = q.N1, N2 = q.N2, N3 = q.N3, N4 = q.N4, N5 = q.N5, N6 = q.N6;

  V3 ut = v3(0.0, N3 * Th1.z + N4 * Th2.z, -N3 * Th1.y - N4 * Th2.y);
  V3 Thb = v3(N1 * Th1.x + N2 * Th2.x, N5 * Th1.y + N6 * Th2.y, N5 * Th1.z + N6 * Th2.z);
  M3 Rb = eye3() + skew(Thb);
  q.Ir = mulNT(muld(Rb, Jr), Rb);  // R̄ Jᵨ R̄ᵀ

  q.N7l = N7 * il; q.N7l2 = q.N7l * il; q.N8l = N8 * il; q.N8l2 = q.N8l * il;
  const double N7l = q.N7l;
  M3 Sut = skew(ut);
  M3 SutG1 = mulG(Sut, G1);
  q.P1P2 = rows(0, 0, 0, 0, 0, N3, 0, -N3, 0);
  q.P1P4 = rows(0, 0, 0, 0, 0, N4, 0, -N4, 0);
  q.H11 = diag3(N1, N1 + N7l, N1 + N7l) - SutG1;
  q.H12 = q.P1P2 - mulG(Sut, G2);
  q.H13 = diag3(N2, N2 - N7l, N2 - N7l) + SutG1;
  q.H14 = q.P1P4 - mulG(Sut, G4);
  q.s21 = v3(q.N8l, 0.0, 0.0);
  q.d22 = v3(N1, N5, N5);
  q.d24 = v3(N2, N6, N6);

  V3 udt = v3(0.0, N7l * dU.y + N3 * Wd1.z + N4 * Wd2.z, N7l * dU.z - N3 * Wd1.y - N4 * Wd2.y);
  M3 Sudt = skew(udt);
  double N7rd = q.N7l2 * rd, N8rd = q.N8l2 * rd;
  M3 Hd11 = diag3(0.0, -N7rd, -N7rd) - mulG(Sudt, G1);
  M3 Hd12 = -mulG(Sudt, G2);
  M3 Hd14 = -mulG(Sudt, G4);

  q.h1 = q.H11 * Ud1 + q.H12 * Wd1 + q.H13 * Ud2 + q.H14 * Wd2;
  q.h2 = cross(q.s21, dU) + dmulv(q.d22, Wd1) + dmulv(q.d24, Wd2);

  const V3 We = q.We;
  q.C11 = skewmul(We, q.H11) + Hd11 - mulskew(q.H11, We);   // C₁¹
  q.C12 = skewmul(We, q.H12) + Hd12 - mulskew(q.H12, We);   // C₁²
  q.C14 = skewmul(We, q.H14) + Hd14 - mulskew(q.H14, We);   // C₁⁴
  // C₂¹ = [S(Ẇᵉ), S(s21)] + Ḣ₂¹ = S(Ẇᵉ × s21) + S((-N₈ṙ,0,0))
  q.C21 = skew(cross(We, q.s21) + v3(-N8rd, 0.0, 0.0));
  // C₂² = S(Ẇᵉ)D - D S(Ẇᵉ) for D = diag(d): entry (i,j) scales by d_j - d_i
  double e2 = N5 - N1, e4 = N6 - N2;
  q.C22 = rows(0, -We.z * e2, We.y * e2, -We.z * e2, 0, 0, We.y * e2, 0, 0);
  q.C24 = rows(0, -We.z * e4, We.y * e4, -We.z * e4, 0, 0, We.y * e4, 0, 0);
}

// Mass blocks, Tᵏ and the kinetic energy at one Gauss point (:302-378); emit(i, x) adds x to the
// table's entries i .. over the Gauss points.
template <typename EMIT>
EB_PIECE void beam_mass(Tab t, const GaussPoint& q, double Ar, double damping, EMIT emit) {
  const double wg = q.wg;
  {
    const V3 Udd1 = t.v(kTabVel + 6), Wdd1 = t.v(kTabVel + 9), Udd2 = t.v(kTabVel + 18), Wdd2 = t.v(kTabVel + 21);
    V3 ReTudd0 = (q.H11 * Udd1 + q.H12 * Wdd1 + q.H13 * Udd2 + q.H14 * Wdd2) +
                 (q.C11 * q.dU + q.C12 * q.Wd1 + q.C14 * q.Wd2);
    V3 W0 = q.h2;
    V3 ReTwdd0 = (cross(q.s21, Udd1 - Udd2) + dmulv(q.d22, Wdd1) + dmulv(q.d24, Wdd2)) +
                 (q.C21 * q.dU + q.C22 * q.Wd1 + q.C24 * q.Wd2);
    V3 IrW0 = q.Ir * W0;
    V3 Fw = q.Ir * ReTwdd0 + cross(W0, IrW0);
    V3 Tk1 = wg * (Ar * mulTv(q.H11, ReTudd0) - cross(q.s21, Fw));  // H₂¹ᵀ = -S(s21)
    V3 Tk2 = wg * (Ar * mulTv(q.H12, ReTudd0) + dmulv(q.d22, Fw));
    V3 Tk3 = (wg * Ar) * ReTudd0 - Tk1;
    V3 Tk4 = wg * (Ar * mulTv(q.H14, ReTudd0) + dmulv(q.d24, Fw));
    if (damping > 0) {
      V3 Td1G = (wg * damping) * (Ar * mulTv(q.H11, q.h1) - cross(q.s21, IrW0));
      Tk1 += Td1G;
      Tk2 += (wg * damping) * (Ar * mulTv(q.H12, q.h1) + dmulv(q.d22, IrW0));
      Tk3 += ((wg * Ar) * damping) * q.h1 - Td1G;
      Tk4 += (wg * damping) * (Ar * mulTv(q.H14, q.h1) + dmulv(q.d24, IrW0));
    }
    emit(kTabTk, Tk1); emit(kTabTk + 3, Tk2); emit(kTabTk + 6, Tk3); emit(kTabTk + 9, Tk4);
    // |u̇₀| does not depend on the frame
    emit(kTabTk + 12, wg / 2 * (Ar * dot(q.h1, q.h1) + dot(W0, IrW0)));
  }
  M3 H21TIr = -skewmul(q.s21, q.Ir);
  const double wA = wg * Ar;
  const M3 I3 = eye3();
  M3 M11G = wA * mulTN(q.H11, q.H11) + wg * mulskew(H21TIr, q.s21);
  emit(kTabM, M11G);
  emit(kTabM + 18, wA * tr(q.H11) - M11G);
  emit(kTabM + 63, M11G + wA * ((I3 - q.H11) - tr(q.H11)));
  M3 M12G = wA * mulTN(q.H11, q.H12) + wg * muld(H21TIr, q.d22);
  emit(kTabM + 9, M12G);
  emit(kTabM + 45, wA * tr(q.H12) - tr(M12G));
  M3 M14G = wA * mulTN(q.H11, q.H14) + wg * muld(H21TIr, q.d24);
  emit(kTabM + 27, M14G);
  emit(kTabM + 72, wA * q.H14 - M14G);
  emit(kTabM + 36, wA * mulTN(q.H12, q.H12) + wg * dmul(q.d22, muld(q.Ir, q.d22)));
  emit(kTabM + 54, wA * mulTN(q.H12, q.H14) + wg * dmul(q.d22, muld(q.Ir, q.d24)));
  emit(kTabM + 81, wA * mulTN(q.H14, q.H14) + wg * dmul(q.d24, muld(q.Ir, q.d24)));
}

// Gyroscopic / damping blocks at one Gauss point (:380-416).
template <typename EMIT>
EB_PIECE void beam_gyro(Tab t, const GaussPoint& q, double Ar, EMIT emit) {
  const double wg = q.wg;
  const Gu G1 = t.G1();
  const Gt G2 = t.G2(), G4 = t.G4();
  const V3 Ud1 = t.v(kTabVel), Ud2 = t.v(kTabVel + 12);
  M3 H1F1 = mulskew(q.H11, Ud1) + mulskew(q.H12, q.Wd1) + mulskew(q.H13, Ud2) + mulskew(q.H14, q.Wd2);
  M3 H2F1 = skewmul(q.s21, skew(q.dU)) + dmul(q.d22, skew(q.Wd1)) + dmul(q.d24, skew(q.Wd2));
  M3 F1 = H1F1 - skew(q.h1), F2 = H2F1 - skew(q.h2);
  M3 A1 = rows(0, 0, 0, q.N7l2 * q.dU.y, 0, 0, q.N7l2 * q.dU.z, 0, 0);
  M3 C31 = mulG(F1, G1) + A1 + muld(skew(q.We), v3(0.0, q.N7l, q.N7l));
  M3 C32 = mulG(F1, G2) + skewmul(q.We, q.P1P2);
  M3 C34 = mulG(F1, G4) + skewmul(q.We, q.P1P4);
  M3 A2 = rows(0, 0, 0, -q.N8l2 * q.dU.z, 0, 0, q.N8l2 * q.dU.y, 0, 0);
  M3 C41 = mulG(F2, G1) + A2;
  M3 C42 = mulG(F2, G2);
  M3 C44 = mulG(F2, G4);
  M3 SWm = skewmul(q.h2, q.Ir) - skew(q.Ir * q.h2);
  // column 1, 2 and 4 in turn: first and third block row from H₁¹, second from H₁², fourth from H₁⁴
  auto column = [&](int k, const M3& Ac, const M3& X) {
    M3 c1 = wg * (mulTN(q.H11, Ac) - skewmul(q.s21, X));
    emit(kTabC + 9 * k, c1);
    emit(kTabC + 9 * (6 + k), wg * Ac - c1);
    emit(kTabC + 9 * (3 + k), wg * (mulTN(q.H12, Ac) + dmul(q.d22, X)));
    emit(kTabC + 9 * (9 + k), wg * (mulTN(q.H14, Ac) + dmul(q.d24, X)));
  };
  column(0, Ar * (q.C11 + C31), q.Ir * (q.C21 + C41) + mulskew(SWm, q.s21));
  column(1, Ar * (q.C12 + C32), q.Ir * (q.C22 + C42) + muld(SWm, q.d22));
  column(2, Ar * (q.C14 + C34), q.Ir * (q.C24 + C44) + muld(SWm, q.d24));
}

// Output block b of an element from the table's Gauss sums: lₒ/2 Rₑ X Rₑᵀ (:431-457), the damping
// terms (:461-478) and the exact-mode transforms (:480-506).  0..9: the mass blocks
// (b = index in kTabM), 10..21: the gyroscopic blocks, 22: Tᵏ and the kinetic energy.
constexpr int kBeamBlocks = 23;
template <typename IO>
EB_PIECE void beam_block(const IO& io, Tab t, int b) {
  const M3 Re = t.m(kTabRe);
  const double l02 = io.l0() / 2;
  const M3 lRe = l02 * Re;
  const BeamOut out = io.out();
  if (b < 10) {
    // (row, column) of the block; M²ʲ and M⁴⁴ take Tₐᵀ / T_bᵀ; M²¹ = M¹²ᵀTₐᵀ, M³¹ = M¹³ᵀ, M⁴¹ = M¹⁴ᵀT_bᵀ,
    // M³² = (M²³Tₐᵀ)ᵀ, M⁴² = (M²⁴Tₐᵀ)ᵀT_bᵀ (the reassigned M²³, M²⁴ are read, :493), M⁴³ = M³⁴ᵀT_bᵀ
    const int i = b < 4 ? 0 : (b < 7 ? 1 : (b < 9 ? 2 : 3));
    const int j = b < 4 ? b : (b < 7 ? b - 3 : (b < 9 ? b - 5 : 3));
    M3 X = mulNT(lRe * t.m(kTabM + 9 * b), Re);
    if (i == 1) X = X * t.m(kTabTa);
    if (i == 3) X = X * t.m(kTabTa + 9);
    put_block(out.M, i, j, X);
    if (i == j) return;
    if (j == 2) put_blockT(out.M, 2, i, X);
    else put_block(out.M, j, i, mulTN(X, t.m(j == 1 ? kTabTa : kTabTa + 9)));
  } else if (b < 22) {
    const int c = b - 10, i = c / 3, k = c - 3 * i, j = k == 2 ? 3 : k;
    const double damping = io.damping();
    M3 X = t.m(kTabC + 9 * c), Y = -X;  // Cᵏⁱ³ = -Cᵏⁱ¹
    if (damping > 0) {
      // M of block (i, j): stored for i <= j, else its transpose
      auto Mij = [&](int r, int s2) {
        const int lo = r < s2 ? r : s2, hi = r < s2 ? s2 : r;
        const M3 m = t.m(kTabM + 9 * (lo == 0 ? hi : (lo == 1 ? hi + 3 : (lo == 2 ? hi + 5 : 9))));
        return r <= s2 ? m : tr(m);
      };
      axpy(X, damping, Mij(i, j));
      if (j == 0) axpy(Y, damping, Mij(i, 2));
    }
    const M3 Ta = t.m(i == 3 ? kTabTa + 9 : kTabTa);
    X = mulNT(lRe * X, Re);
    if (i & 1) X = X * Ta;
    put_block(out.C, i, j, X);
    if (j == 0) {
      if (damping > 0) {
        Y = mulNT(lRe * Y, Re);
        if (i & 1) Y = Y * Ta;
      } else {
        Y = -X;
      }
      put_block(out.C, i, 2, Y);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) put_vec(out.Tk, k, lRe * t.v(kTabTk + 3 * k));
    out.E[1] = l02 * t.at(kTabTk + 12);
  }
}

#if !defined(__CUDACC__)
// One element in sequence (host checks of the pieces).
template <typename IO>
EB_DEV void beam_element(const IO& io, const Gauss3& gs) {
  double tab[kTabSize];
  const Tab t{tab, 1};
  for (int k = 0; k < kTabSize; ++k) tab[k] = 0.0;
  beam_frame(io, t);
  for (int n = 0; n < 2; ++n) {
    beam_angle(io, n, t);
    beam_exact(io, n, t);
    beam_velocity(io, n, t);
  }
  BeamStatic st;
  beam_static_common(io, t, st);
  beam_static(io, t, st, 0);
  beam_static(io, t, st, 1);
  struct Add {
    const Tab& t;
    void operator()(int i, double x) const { t.at(i) += x; }
    void operator()(int i, V3 x) const { t.put(i, t.v(i) + x); }
    void operator()(int i, const M3& x) const { t.put(i, t.m(i) + x); }
  };
  for (int g = 0; g < 3; ++g) {
    GaussPoint q;
    gauss_point(t, io.l0(), io.Jr(), gs.z[g], gs.w[g], q);
    beam_mass(t, q, io.Ar(), io.damping(), Add{t});
    beam_gyro(t, q, io.Ar(), Add{t});
  }
  for (int b = 0; b < kBeamBlocks; ++b) beam_block(io, t, b);
}

// An element whose inputs lie in a BeamIn record.
struct BeamRecord {
  const BeamIn& in;
  BeamOut o;
  EB_DEV V3 x(int n) const { return n ? in.X2 + in.u2 : in.X1 + in.u1; }
  EB_DEV M3 R(int n) const { return n ? in.R2 : in.R1; }
  EB_DEV M3 dR(int n) const { return n ? in.dR2 : in.dR1; }
  EB_DEV M3 Re0() const { return in.Re0; }
  EB_DEV V3 ud(int n) const { return n ? in.ud2 : in.ud1; }
  EB_DEV V3 wd(int n) const { return n ? in.wd2 : in.wd1; }
  EB_DEV V3 udd(int n) const { return n ? in.udd2 : in.udd1; }
  EB_DEV V3 wdd(int n) const { return n ? in.wdd2 : in.wdd1; }
  EB_DEV double l0() const { return in.l0; }
  EB_DEV double Ku() const { return in.Ku; }
  EB_DEV double Ar() const { return in.Ar; }
  EB_DEV double damping() const { return in.damping; }
  EB_DEV V3 KT() const { return in.KT; }
  EB_DEV V3 KTT() const { return in.KTT; }
  EB_DEV V3 Jr() const { return in.Jr; }
  EB_DEV BeamOut out() const { return o; }
};
#else
// ------------------------------------------------------------------ cooperative evaluation
// A CTA of four warps evaluates 10 or 30 elements, a Gauss-point lane per element and point, ten
// elements a warp.  FP64 instructions occupy the SM's pipe for 16 cycles a warp, however many
// lanes work.  Ten: two warps for the static halves, one each for the mass and the gyroscopic
// blocks, the shortest chain, for launches that leave SMs idle.  Thirty: one warp for the static part
// and three for the Gauss points, every lane busy and nothing formed twice, for the others.
constexpr int kBeamGroup = 10;
constexpr int kBeamCta = 128;
__host__ __device__ inline int beam_groups(int threads) { return threads >= 256 ? 3 : 1; }
__host__ __device__ inline size_t beam_smem(int nb) { return sizeof(double) * kTabSize * kBeamGroup * nb; }

// Adds Gauss-point values over the three lanes of an element, in Gauss order, into its table.
// Three values at a time: lane g sums the g-th and stores it (two additions for three values; the
// exchanges run on other pipes).
struct EmitSum {
  Tab t;
  int base, g;   // lane of the element's first Gauss point, this lane's point
  bool store;
  __device__ __forceinline__ void operator()(int i, V3 x) const {
    // the other two lanes' value g: each lane sends what the receiver sums
    const double up = g == 0 ? x.z : (g == 1 ? x.x : x.y);    // to lane g - 1 (mod 3)
    const double down = g == 0 ? x.y : (g == 1 ? x.z : x.x);  // to lane g + 1 (mod 3)
    const double own = g == 0 ? x.x : (g == 1 ? x.y : x.z);
    const double next = __shfl_sync(0xffffffffu, up, base + (g == 2 ? 0 : g + 1));
    const double prev = __shfl_sync(0xffffffffu, down, base + (g == 0 ? 2 : g - 1));
    const double v0 = g == 0 ? own : (g == 1 ? prev : next);
    const double v1 = g == 1 ? own : (g == 2 ? prev : next);
    const double v2 = g == 2 ? own : (g == 0 ? prev : next);
    if (store) t.at(i + g) = (v0 + v1) + v2;
  }
  __device__ __forceinline__ void operator()(int i, double x) const {
    const double a = __shfl_sync(0xffffffffu, x, base), b = __shfl_sync(0xffffffffu, x, base + 1),
                 c = __shfl_sync(0xffffffffu, x, base + 2);
    if (store && g == 0) t.at(i) = (a + b) + c;
  }
  __device__ __forceinline__ void operator()(int i, const M3& x) const {
#pragma unroll
    for (int k = 0; k < 9; k += 3) (*this)(i + k, v3(x.a[k], x.a[k + 1], x.a[k + 2]));
  }
};

// nb = 1 or 3 groups of ten elements; make(e) gives element e's IO, on(e) whether it is evaluated
// (both for e < n only).  All threads of the CTA call it.
template <typename MAKE, typename ON>
__device__ __forceinline__ void beam_cta(int64_t n, int nb, const Gauss3& gs, double* tab, MAKE make, ON on) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int nw = kBeamCta / 32;
  const int E = kBeamGroup * nb;
  const int64_t e0 = (int64_t)blockIdx.x * E;
  __shared__ unsigned char act[32];
  bool mine = false;
  if (threadIdx.x < E) {
    mine = e0 + threadIdx.x < n && on(e0 + threadIdx.x);
    act[threadIdx.x] = mine;
  }
  if (!__syncthreads_or(mine)) return;
  auto table = [&](int e) { return Tab{tab + e, E}; };
  // frames on warp 0; then one lane per (element, node): angles on warps 0 and 1, velocities and
  // exact-mode transforms on the others
  if (warp == 0 && lane < E && act[lane]) beam_frame(make(e0 + lane), table(lane));
  const int pair = 32 * (warp & 1) + lane, pe = pair >> 1, pn = pair & 1;
  if (warp >= 2 && pe < E && act[pe]) beam_exact(make(e0 + pe), pn, table(pe));
  __syncthreads();
  if (pe < E && act[pe]) {
    if (warp < 2) beam_angle(make(e0 + pe), pn, table(pe));
    else beam_velocity(make(e0 + pe), pn, table(pe));
  }
  __syncthreads();
  const int gauss0 = nb == 1 ? 2 : 1;  // first warp of the Gauss-point pieces
  if (warp < gauss0) {
    if (lane < E && act[lane]) {
      const auto io = make(e0 + lane);
      const Tab t = table(lane);
      BeamStatic q;
      beam_static_common(io, t, q);
      for (int half = 0; half < 2; ++half)
        if (nb > 1 || half == warp) beam_static(io, t, q, half);
    }
  } else {
    // lanes without an element of their own repeat another's (no divergence at the shuffles); lanes
    // 30 and 31 repeat the last element's first two points
    const int group = nb == 1 ? 0 : warp - 1, own = lane < 3 * kBeamGroup;
    const int sub = own ? lane / 3 : kBeamGroup - 1, g = own ? lane - 3 * sub : lane - 30;
    int e = kBeamGroup * group + sub;
    const bool store = own && act[e];
    if (!act[e])
      for (e = 0; !act[e]; ++e) {
      }
    const auto io = make(e0 + e);
    const Tab t = table(e);
    const EmitSum emit{t, 3 * sub, g, store};
    GaussPoint q;
    gauss_point(t, io.l0(), io.Jr(), g == 0 ? gs.z[0] : (g == 1 ? gs.z[1] : gs.z[2]),
                g == 0 ? gs.w[0] : (g == 1 ? gs.w[1] : gs.w[2]), q);
    if (nb > 1 || warp == 2) beam_mass(t, q, io.Ar(), io.damping(), emit);
    if (nb > 1 || warp == 3) beam_gyro(t, q, io.Ar(), emit);
  }
  __syncthreads();
  const int per = 32 / E, sub = lane / E, e = lane - sub * E;  // blocks per warp pass
  if (sub < per && act[e]) {
    const auto io = make(e0 + e);
    const Tab t = table(e);
    for (int b = warp * per + sub; b < kBeamBlocks; b += nw * per) beam_block(io, t, b);
  }
}

// Adds Gauss-point values into the table, point after point: EmitSum's order (an addition of its own, never
// part of a multiply-add).
struct EmitAdd {
  Tab t;
  bool first;
  __device__ __forceinline__ void operator()(int i, double x) const { t.at(i) = first ? x : __dadd_rn(t.at(i), x); }
  __device__ __forceinline__ void operator()(int i, V3 x) const {
    (*this)(i, x.x);
    (*this)(i + 1, x.y);
    (*this)(i + 2, x.z);
  }
  __device__ __forceinline__ void operator()(int i, const M3& x) const {
#pragma unroll
    for (int k = 0; k < 9; ++k) (*this)(i + k, x.a[k]);
  }
};

// The same pieces by one thread, its table in local memory.
template <typename IO>
__device__ __forceinline__ void beam_thread(const IO& io, const Gauss3& gs) {
  double tab[kTabSize];
  const Tab t{tab, 1};
  beam_frame(io, t);
  for (int n = 0; n < 2; ++n) {
    beam_exact(io, n, t);
    beam_angle(io, n, t);
    beam_velocity(io, n, t);
  }
  {
    BeamStatic q;
    beam_static_common(io, t, q);
    for (int half = 0; half < 2; ++half) beam_static(io, t, q, half);
  }
  for (int g = 0; g < 3; ++g) {
    GaussPoint q;
    gauss_point(t, io.l0(), io.Jr(), gs.z[g], gs.w[g], q);
    const EmitAdd emit{t, g == 0};
    beam_mass(t, q, io.Ar(), io.damping(), emit);
    beam_gyro(t, q, io.Ar(), emit);
  }
  for (int b = 0; b < kBeamBlocks; ++b) beam_block(io, t, b);
}
#endif

}  // namespace ebd
