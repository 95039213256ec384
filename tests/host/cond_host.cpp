// Test infrastructure: the condensation plan (endobeams.jl_gb300/csrc/eb_cond_plan.hpp) walked
// in FP64 on the host with the operations of the device kernels, the kept system by dense LU.
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

#include "../../endobeams.jl_gb300/csrc/eb_cond_plan.hpp"

using namespace eb;
using Blk = std::vector<double>;  // 36, row-major

namespace {
Blk inv6(const Blk& A) {
  std::vector<double> m(72, 0.0);
  for (int r = 0; r < 6; ++r) {
    for (int c = 0; c < 6; ++c) m[12 * r + c] = A[6 * r + c];
    m[12 * r + 6 + r] = 1.0;
  }
  for (int k = 0; k < 6; ++k) {
    int p = k;
    for (int r = k + 1; r < 6; ++r)
      if (std::fabs(m[12 * r + k]) > std::fabs(m[12 * p + k])) p = r;
    for (int c = 0; c < 12; ++c) std::swap(m[12 * k + c], m[12 * p + c]);
    const double d = m[12 * k + k];
    for (int c = 0; c < 12; ++c) m[12 * k + c] /= d;
    for (int r = 0; r < 6; ++r)
      if (r != k) {
        const double f = m[12 * r + k];
        for (int c = 0; c < 12; ++c) m[12 * r + c] -= f * m[12 * k + c];
      }
  }
  Blk I(36);
  for (int r = 0; r < 6; ++r)
    for (int c = 0; c < 6; ++c) I[6 * r + c] = m[12 * r + 6 + c];
  return I;
}
void madd(Blk& t, double s, const Blk& a, const Blk& b) {
  for (int r = 0; r < 6; ++r)
    for (int c = 0; c < 6; ++c)
      for (int j = 0; j < 6; ++j) t[6 * r + c] += s * a[6 * r + j] * b[6 * j + c];
}
Blk mul(double s, const Blk& a, const Blk& b) {
  Blk t(36, 0.0);
  madd(t, s, a, b);
  return t;
}
}  // namespace

// Relative residual |A z - v| / |v| of z = M^-1 v for a random block matrix on the graph with the
// m edges (pairs of nodes); out: eliminated nodes, levels, half bandwidth of the kept graph.
extern "C" double host_cond_residual(int n, int m, const int32_t* edges, int max_w, int max_dense, int seed,
                                     int32_t* out) {
  std::vector<std::vector<int>> adj(n);
  for (int e = 0; e < m; ++e) {
    adj[edges[2 * e]].push_back(edges[2 * e + 1]);
    adj[edges[2 * e + 1]].push_back(edges[2 * e]);
  }
  for (auto& a : adj) {
    std::sort(a.begin(), a.end());
    a.erase(std::unique(a.begin(), a.end()), a.end());
  }
  CondPlan P;
  cond_plan(adj, max_w, max_dense, P);
  out[0] = P.ne; out[1] = (int)P.lev_ptr.size() - 1; out[2] = P.w;
  std::mt19937 rng(seed);
  std::uniform_real_distribution<double> U(-1, 1);
  std::vector<Blk> S(P.n_blocks, Blk(36, 0.0));
  std::vector<std::vector<std::pair<int, Blk>>> A(n);  // by position
  std::vector<int> node_at(n);
  for (int v = 0; v < n; ++v) node_at[P.pos[v]] = v;
  for (int p = 0; p < n; ++p) {
    std::vector<int> cols{p};
    for (int u : adj[node_at[p]]) cols.push_back(P.pos[u]);
    for (int c : cols) {
      Blk b(36);
      for (double& x : b) x = U(rng);
      if (c == p)
        for (int k = 0; k < 6; ++k) b[7 * k] += 6.0 * (adj[node_at[p]].size() + 1.0);
      const int id = P.find(p, c);
      if (id < 0 || P.srow[id] != p || P.scol[id] != c) return 1e30;  // an edge outside the pattern
      S[id] = b;
      A[p].push_back({c, b});
    }
  }
  const int nlev = (int)P.lev_ptr.size() - 1;
  for (int l = 0; l < nlev; ++l) {
    for (int p = P.lev_ptr[l]; p < P.lev_ptr[l + 1]; ++p) {
      const Blk D = inv6(S[P.wptr[p]]);
      S[P.wptr[p]] = D;
      for (int b = P.wptr[p] + 1; b < P.wptr[p + 1]; ++b) S[b] = mul(-1.0, D, S[b]);
    }
    for (size_t k = 0; k < P.tgt[l].size(); ++k)
      for (int u = P.tptr[l][k]; u < P.tptr[l][k + 1]; ++u) {
        if (P.tgt[l][k] < 0 || P.cl[l][u] < 0) return 1e30;
        madd(S[P.tgt[l][k]], 1.0, S[P.cl[l][u]], S[P.cw[l][u]]);
      }
  }
  for (int b = P.lptr[0]; b < P.red0; ++b) S[b] = mul(-1.0, S[b], S[P.wptr[P.scol[b]]]);
  const int N = 6 * (n - P.ne);
  std::vector<double> K((size_t)N * N, 0.0);
  int w = 0;
  for (int b = P.red0; b < P.n_blocks; ++b) {
    const int r = P.srow[b] - P.ne, c = P.scol[b] - P.ne;
    w = std::max(w, std::abs(r - c));
    for (int i = 0; i < 6; ++i)
      for (int j = 0; j < 6; ++j) K[(size_t)(6 * r + i) * N + 6 * c + j] = S[b][6 * i + j];
  }
  if (w > P.w) return 1e30;
  std::vector<double> v(6 * n), x;
  for (double& t : v) t = U(rng);
  x = v;
  auto rows = [&](int p0, int p1, bool fwd) {
    for (int p = p0; p < p1; ++p) {
      double y[6];
      const int b0 = fwd ? P.lptr[p] : P.wptr[p], b1 = fwd ? P.lptr[p + 1] : P.wptr[p + 1];
      for (int r = 0; r < 6; ++r) {
        y[r] = fwd ? x[6 * p + r] : 0.0;
        for (int b = b0; b < b1; ++b)
          for (int c = 0; c < 6; ++c) y[r] += S[b][6 * r + c] * x[6 * P.scol[b] + c];
      }
      for (int r = 0; r < 6; ++r) x[6 * p + r] = y[r];
    }
  };
  for (int l = 1; l < nlev; ++l) rows(P.lev_ptr[l], P.lev_ptr[l + 1], true);
  rows(P.ne, n, true);
  double* xr = &x[6 * P.ne];
  for (int k = 0; k < N; ++k) {  // dense LU solve of the kept system
    for (int i = k + 1; i < N; ++i) {
      const double f = K[(size_t)i * N + k] / K[(size_t)k * N + k];
      if (f == 0.0) continue;
      for (int j = k; j < N; ++j) K[(size_t)i * N + j] -= f * K[(size_t)k * N + j];
      xr[i] -= f * xr[k];
    }
  }
  for (int i = N - 1; i >= 0; --i) {
    for (int j = i + 1; j < N; ++j) xr[i] -= K[(size_t)i * N + j] * xr[j];
    xr[i] /= K[(size_t)i * N + i];
  }
  for (int l = nlev - 1; l >= 0; --l) rows(P.lev_ptr[l], P.lev_ptr[l + 1], false);
  double e2 = 0, v2 = 0;
  for (int p = 0; p < n; ++p)
    for (int r = 0; r < 6; ++r) {
      double t = -v[6 * p + r];
      for (auto& [c, b] : A[p])
        for (int j = 0; j < 6; ++j) t += b[6 * r + j] * x[6 * c + j];
      e2 += t * t;
      v2 += v[6 * p + r] * v[6 * p + r];
    }
  return std::sqrt(e2 / v2);
}
