// Signed distance field of a closed triangle mesh on a regular grid.
//
// No counterpart in the reference: its DiscreteSignedDistanceField reads a
// precomputed grid (read_vtk_sdf, src/IO/read_input_files.jl:154-195), while
// its vessel geometries exist as triangle meshes (read_vtk_triangle_mesh,
// :81-152).  This turns such a mesh into the grid the contact kernels use.
//
// One thread per grid point, one CTA per brick of 8 x 4 x 4 points.  Per (point, triangle):
//   * squared distance to the closest point of the triangle, by the Voronoi-
//     region tests of Ericson, "Real-Time Collision Detection" (2005), §5.1.5;
//   * the triangle's signed solid angle seen from the point, by the formula of
//     Van Oosterom & Strackee, IEEE Trans. Biomed. Eng. 30 (1983) 125-126:
//     tan(Ω/2) = a·(b×c) / (|a||b||c| + (a·b)|c| + (a·c)|b| + (b·c)|a|).
// FP64 runs at 1/64 of FP32's rate here and only few pairs decide the result:
//   * distance: FP32 distances from the brick's centre leave the triangles within the brick's
//     diameter of its nearest one, FP32 distances from the point those within the FP32 error
//     bound of its nearest one; these are evaluated in FP64;
//   * sign: Ω is summed in FP32 over the triangles that are well conditioned from the point (the
//     denominator above a quarter of |a||b||c|, no vertex close by) and in FP64 over the others;
//     where the sum lies within its error bound of the threshold 2π, the point's whole sum is
//     repeated in FP64.
// 5,120 triangles x 64³ points, all pairs in FP64: 392 ms a call.
// The solid angles sum to 4π times the generalized winding number; the point is
// inside when |Σ Ω| > 2π (either orientation of the mesh).  The value is the
// distance, positive inside and negative outside — the sign convention of the
// reference's SDF files for bodies inside the surface (DiscreteSignedDistanceField
// with inside = true, def_interactions.jl:67-71).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/endobeams_gb300.h"

int eb_internal_fail(int code, const char* msg);  // sets eb_last_error (eb_abi.cu)

namespace {

constexpr int kSdfThreads = 128;
constexpr int kTile = 128;  // triangles per shared-memory tile of the solid angles

template <typename T>
struct P3T {
  T x, y, z;
};
using P3 = P3T<double>;
using P3f = P3T<float>;
template <typename T>
__device__ __forceinline__ P3T<T> sub(P3T<T> a, P3T<T> b) { return P3T<T>{a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename T>
__device__ __forceinline__ T dot(P3T<T> a, P3T<T> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <typename T>
__device__ __forceinline__ P3T<T> cross(P3T<T> a, P3T<T> b) {
  return P3T<T>{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <typename T>
__device__ __forceinline__ P3T<T> axpy(T s, P3T<T> a, P3T<T> b) {
  return P3T<T>{b.x + s * a.x, b.y + s * a.y, b.z + s * a.z};
}

// Squared distance from p to triangle abc (closest-point region tests).
template <typename T>
__device__ T dist2_point_triangle(P3T<T> p, P3T<T> a, P3T<T> b, P3T<T> c) {
  const P3T<T> ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
  const T d1 = dot(ab, ap), d2 = dot(ac, ap);
  P3T<T> q;
  if (d1 <= T(0) && d2 <= T(0)) {
    q = a;  // vertex region a
  } else {
    const P3T<T> bp = sub(p, b);
    const T d3 = dot(ab, bp), d4 = dot(ac, bp);
    if (d3 >= T(0) && d4 <= d3) {
      q = b;  // vertex region b
    } else {
      const T vc = d1 * d4 - d3 * d2;
      if (vc <= T(0) && d1 >= T(0) && d3 <= T(0)) {
        q = axpy(d1 / (d1 - d3), ab, a);  // edge ab
      } else {
        const P3T<T> cp = sub(p, c);
        const T d5 = dot(ab, cp), d6 = dot(ac, cp);
        if (d6 >= T(0) && d5 <= d6) {
          q = c;  // vertex region c
        } else {
          const T vb = d5 * d2 - d1 * d6;
          if (vb <= T(0) && d2 >= T(0) && d6 <= T(0)) {
            q = axpy(d2 / (d2 - d6), ac, a);  // edge ac
          } else {
            const T va = d3 * d6 - d5 * d4;
            if (va <= T(0) && (d4 - d3) >= T(0) && (d5 - d6) >= T(0)) {
              q = axpy((d4 - d3) / ((d4 - d3) + (d5 - d6)), sub(c, b), b);  // edge bc
            } else {
              const T den = T(1) / (va + vb + vc);  // face region
              const T v = vb * den, w = vc * den;
              q = axpy(w, ac, axpy(v, ab, a));
            }
          }
        }
      }
    }
  }
  const P3T<T> d = sub(p, q);
  return dot(d, d);
}

// Signed solid angle of triangle abc seen from p.
__device__ double solid_angle(P3 p, P3 A, P3 B, P3 C) {
  const P3 a = sub(A, p), b = sub(B, p), c = sub(C, p);
  const double la = sqrt(dot(a, a)), lb = sqrt(dot(b, b)), lc = sqrt(dot(c, c));
  const double num = dot(a, cross(b, c));
  const double den = la * lb * lc + dot(a, b) * lc + dot(a, c) * lb + dot(b, c) * la;
  return 2.0 * atan2(num, den);
}

struct Grid {
  int64_t nx, ny, nz;
  double ox, oy, oz, hx, hy, hz;
  double cx, cy, cz;  // origin of the FP32 coordinates ...
  double scale;       // ... and their unit's inverse: they are at most 1, whatever the mesh's units
  float margin;       // bound of the FP32 distances' error, twice
  float lmin2;        // squared length below which a vertex is close by
  double slack;       // bound of the FP32 solid-angle sum's error
};

__device__ __forceinline__ P3 tri_vertex(const double* tri, int64_t t, int k) {
  const double* v = tri + 9 * t + 3 * k;
  return P3{v[0], v[1], v[2]};
}

// FP32 copy of the triangles relative to the grid's centre, scaled.  The FP32 distance divides by the
// squared area: its error grows as the square of longest edge over height.  Host comparison with
// FP64, 1e8 triangles of 1e-9 to 1 of the extent: 13 times the margin below a height of 1.1e-3 of the longest
// edge, 0.6 of it at 5e-3, 0.04 at 2e-2.  A thinner triangle (a needle), also one that rounding to FP32 makes so,
// gets a NaN: no FP32 test ever discards it.  The same below 1e-8 of the extent, where products of four
// lengths come near FP32's smallest.
__global__ void k_mesh_prep(const double* __restrict__ tri, int64_t nt, Grid g, float* __restrict__ tf) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const P3 c{g.cx, g.cy, g.cz};
  float f[9];
  for (int k = 0; k < 3; ++k) {
    const P3 v = sub(tri_vertex(tri, t, k), c);
    f[3 * k] = (float)(v.x * g.scale);
    f[3 * k + 1] = (float)(v.y * g.scale);
    f[3 * k + 2] = (float)(v.z * g.scale);
  }
  const P3 a{f[0], f[1], f[2]}, b{f[3], f[4], f[5]}, q{f[6], f[7], f[8]};
  const P3 e0 = sub(b, a), e1 = sub(q, a), e2 = sub(q, b), n = cross(e0, e1);
  const double L2 = fmax(dot(e0, e0), fmax(dot(e1, e1), dot(e2, e2)));
  const bool needle = !(dot(n, n) > 4e-4 * L2 * L2) || L2 < 1e-16;
  for (int k = 0; k < 9; ++k) tf[9 * t + k] = needle && k % 3 == 0 ? nanf("") : f[k];
}

constexpr int kBx = 8, kBy = 4, kBz = 4;  // points of a brick
constexpr int kMaxCand = 2048;            // candidates kept; beyond it every triangle is one
static_assert(kBx * kBy * kBz == kSdfThreads, "one thread per point of the brick");

__device__ __forceinline__ float dist_f(const float* v, P3f p) {
  return sqrtf(dist2_point_triangle(p, P3f{v[0], v[1], v[2]}, P3f{v[3], v[4], v[5]}, P3f{v[6], v[7], v[8]}));
}

__global__ void __launch_bounds__(kSdfThreads) k_mesh_sdf(const double* __restrict__ tri, const float* __restrict__ tf,
                                                          int64_t nt, Grid g, double* __restrict__ out) {
  __shared__ float st[kTile * 9];
  __shared__ int cand[kMaxCand];
  __shared__ int ncand;
  __shared__ float red[kSdfThreads / 32];
  const int64_t bx = (g.nx + kBx - 1) / kBx, by = (g.ny + kBy - 1) / kBy;
  const int64_t bi = blockIdx.x % bx, bj = (blockIdx.x / bx) % by, bk = blockIdx.x / (bx * by);
  const int64_t i = bi * kBx + threadIdx.x % kBx, j = bj * kBy + (threadIdx.x / kBx) % kBy,
                k = bk * kBz + threadIdx.x / (kBx * kBy);
  const bool valid = i < g.nx && j < g.ny && k < g.nz;
  const P3 p{g.ox + (double)i * g.hx, g.oy + (double)j * g.hy, g.oz + (double)k * g.hz};
  const P3f pf{(float)((p.x - g.cx) * g.scale), (float)((p.y - g.cy) * g.scale), (float)((p.z - g.cz) * g.scale)};
  const int lane = threadIdx.x & 31;

  // ---- triangles that can be nearest to a point of the brick: d(centre) <= min d(centre) + 2 r
  const double sx = 0.5 * (kBx - 1) * g.hx, sy = 0.5 * (kBy - 1) * g.hy, sz = 0.5 * (kBz - 1) * g.hz;
  const P3f cf{(float)((g.ox + (double)(bi * kBx) * g.hx + sx - g.cx) * g.scale),
               (float)((g.oy + (double)(bj * kBy) * g.hy + sy - g.cy) * g.scale),
               (float)((g.oz + (double)(bk * kBz) * g.hz + sz - g.cz) * g.scale)};
  const float rx = (float)(sx * g.scale), ry = (float)(sy * g.scale), rz = (float)(sz * g.scale);
  const float rb = sqrtf(rx * rx + ry * ry + rz * rz);
  float dmin = INFINITY;
  for (int64_t t = threadIdx.x; t < nt; t += kSdfThreads) dmin = fminf(dmin, dist_f(tf + 9 * t, cf));
  for (int o = 16; o > 0; o >>= 1) dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
  if (lane == 0) red[threadIdx.x >> 5] = dmin;
  if (threadIdx.x == 0) ncand = 0;
  __syncthreads();
  for (int q = 0; q < kSdfThreads / 32; ++q) dmin = fminf(dmin, red[q]);
  const float bound = dmin + 2.0002f * rb + g.margin;
  for (int64_t t = threadIdx.x; t < nt; t += kSdfThreads)
    if (!(dist_f(tf + 9 * t, cf) > bound)) {
      const int q = atomicAdd(&ncand, 1);
      if (q < kMaxCand) cand[q] = (int)t;
    }
  __syncthreads();
  const bool all = ncand > kMaxCand;
  const int64_t nc = all ? nt : ncand;
  double d2 = INFINITY;
  if (valid) {
    float dp = INFINITY;
    for (int64_t q = 0; q < nc; ++q) dp = fminf(dp, dist_f(tf + 9 * (all ? q : (int64_t)cand[q]), pf));
    dp += g.margin;
    for (int64_t q = 0; q < nc; ++q) {
      const int64_t t = all ? q : (int64_t)cand[q];
      if (!(dist_f(tf + 9 * t, pf) > dp))
        d2 = fmin(d2, dist2_point_triangle(p, tri_vertex(tri, t, 0), tri_vertex(tri, t, 1), tri_vertex(tri, t, 2)));
    }
  }

  // ---- solid angles
  double omega = 0.0;
  for (int64_t t0 = 0; t0 < nt; t0 += kTile) {
    const int cnt = (int)(nt - t0 < kTile ? nt - t0 : kTile);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt * 9; q += blockDim.x) st[q] = tf[t0 * 9 + q];
    __syncthreads();
    if (valid) {
      float sum = 0.f;
      for (int t = 0; t < cnt; ++t) {
        const float* v = st + 9 * t;
        const P3f a = sub(P3f{v[0], v[1], v[2]}, pf), b = sub(P3f{v[3], v[4], v[5]}, pf), c = sub(P3f{v[6], v[7], v[8]}, pf);
        const float aa = dot(a, a), bb = dot(b, b), cc = dot(c, c);
        const float la = sqrtf(aa), lb = sqrtf(bb), lc = sqrtf(cc);
        const float num = dot(a, cross(b, c)), lll = la * lb * lc;
        const float den = lll + dot(a, b) * lc + dot(a, c) * lb + dot(b, c) * la;
        if (den > 0.25f * lll && fminf(aa, fminf(bb, cc)) > g.lmin2) {
          sum += atanf(num / den);
        } else {  // close by or seen from within its wedge (NaN: a needle)
          omega += solid_angle(p, tri_vertex(tri, t0 + t, 0), tri_vertex(tri, t0 + t, 1), tri_vertex(tri, t0 + t, 2));
        }
      }
      omega += 2.0 * (double)sum;
    }
  }
  if (valid) {
    if (fabs(fabs(omega) - 6.283185307179586) < g.slack) {
      omega = 0.0;
      for (int64_t t = 0; t < nt; ++t)
        omega += solid_angle(p, tri_vertex(tri, t, 0), tri_vertex(tri, t, 1), tri_vertex(tri, t, 2));
    }
    const double d = sqrt(d2);
    out[i + g.nx * (j + g.ny * k)] = fabs(omega) > 6.283185307179586 ? d : -d;  // |winding number| > 1/2: inside
  }
}

struct Buf {
  void* p = nullptr;
  ~Buf() {
    if (p) cudaFree(p);
  }
};

}  // namespace

extern "C" int eb_sdf_from_mesh(int64_t n_vert, const double* verts, int64_t n_tri, const int64_t* tris,
                                const int64_t* dims, const double* origin, const double* spacing, double* out) {
  if (n_vert < 3 || n_tri < 1 || !verts || !tris || !dims || !origin || !spacing || !out)
    return eb_internal_fail(EB_ERR_ARG, "eb_sdf_from_mesh: bad arguments");
  if (dims[0] < 1 || dims[1] < 1 || dims[2] < 1 || !(spacing[0] > 0) || !(spacing[1] > 0) || !(spacing[2] > 0))
    return eb_internal_fail(EB_ERR_ARG, "eb_sdf_from_mesh: bad grid");
  std::vector<double> tv(9 * (size_t)n_tri);
  for (int64_t t = 0; t < n_tri; ++t)
    for (int k = 0; k < 3; ++k) {
      const int64_t v = tris[3 * t + k];
      if (v < 0 || v >= n_vert) return eb_internal_fail(EB_ERR_ARG, "eb_sdf_from_mesh: triangle vertex out of range");
      std::memcpy(&tv[9 * t + 3 * k], verts + 3 * v, 3 * sizeof(double));
    }
  const int64_t N = dims[0] * dims[1] * dims[2];
  Grid g{dims[0], dims[1], dims[2], origin[0], origin[1], origin[2], spacing[0], spacing[1], spacing[2]};
  g.cx = origin[0] + 0.5 * (double)(dims[0] - 1) * spacing[0];
  g.cy = origin[1] + 0.5 * (double)(dims[1] - 1) * spacing[1];
  g.cz = origin[2] + 0.5 * (double)(dims[2] - 1) * spacing[2];
  // largest coordinate and longest edge; an FP32 coordinate is off by 2^-24 of the former, a
  // distance by that and, through the face region's quotient (needles are kept out), by 8e-5 of
  // the latter: the margin is 25 times the sum
  double ext = std::max(std::max(0.5 * (double)dims[0] * spacing[0], 0.5 * (double)dims[1] * spacing[1]),
                        0.5 * (double)dims[2] * spacing[2]);
  double L2 = 0.0;
  const double c[3] = {g.cx, g.cy, g.cz};
  for (int64_t t = 0; t < n_tri; ++t)
    for (int k = 0; k < 3; ++k) {
      double e2 = 0.0;
      for (int a = 0; a < 3; ++a) {
        ext = std::max(ext, std::fabs(tv[9 * t + 3 * k + a] - c[a]));
        const double e = tv[9 * t + 3 * ((k + 1) % 3) + a] - tv[9 * t + 3 * k + a];
        e2 += e * e;
      }
      L2 = std::max(L2, e2);
    }
  g.scale = 1.0 / ext;
  g.margin = (float)(2e-3 * std::sqrt(L2) * g.scale + 2e-5);
  // a vertex at 2e-3 of the extent is off by 3e-5 of its distance, a solid angle with den > |a||b||c| / 4
  // then by 3e-4 (the same for all triangles at a vertex: over a closed mesh it cancels), and by 1.8e-6
  // through rounding (1e8 triangles compared on the host): 4e-6 for each
  g.lmin2 = 4e-6f;
  g.slack = 0.2 + 4e-6 * (double)n_tri;
  Buf dt, df, dout;
  if (cudaMalloc(&dt.p, sizeof(double) * tv.size()) != cudaSuccess ||
      cudaMalloc(&df.p, sizeof(float) * tv.size()) != cudaSuccess ||
      cudaMalloc(&dout.p, sizeof(double) * (size_t)N) != cudaSuccess ||
      cudaMemcpy(dt.p, tv.data(), sizeof(double) * tv.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return eb_internal_fail(EB_ERR_CUDA, "eb_sdf_from_mesh: device allocation or copy failed");
  const int64_t bricks = ((dims[0] + kBx - 1) / kBx) * ((dims[1] + kBy - 1) / kBy) * ((dims[2] + kBz - 1) / kBz);
  k_mesh_prep<<<(unsigned)((n_tri + 127) / 128), 128>>>((const double*)dt.p, n_tri, g, (float*)df.p);
  k_mesh_sdf<<<(unsigned)bricks, kSdfThreads>>>((const double*)dt.p, (const float*)df.p, n_tri, g, (double*)dout.p);
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpy(out, dout.p, sizeof(double) * (size_t)N, cudaMemcpyDeviceToHost) != cudaSuccess)
    return eb_internal_fail(EB_ERR_CUDA, "eb_sdf_from_mesh: kernel or copy failed");
  return EB_OK;
}
