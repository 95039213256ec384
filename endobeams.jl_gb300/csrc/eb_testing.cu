// Element-level testing entry points: evaluate the device beam and contact
// elements on caller-supplied packed states, so the kernels can be compared
// with a CPU evaluation of compute_beams / compute_contact_beams for the
// same inputs.
//
// Packed input record (96 doubles): X1[3] X2[3] u1[3] u2[3] R1[9] R2[9] ΔR1[9]
// ΔR2[9] u̇1[3] u̇2[3] ẇ1[3] ẇ2[3] ü1[3] ü2[3] ẅ1[3] ẅ2[3] l0 Rₑ⁰[9] K̄ū K̄Θ[3]
// K̄ΘΘ[3] Jᵨ[3] Aᵨ damping radius (pad).  3x3 matrices column-major.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/endobeams_gb300.h"
#include "eb_internal.cuh"
#include "eb_launch_rules.hpp"

using namespace ebd;

namespace {
thread_local char g_err2[512];

__device__ __forceinline__ V3 P3(const double* p) { return v3(p[0], p[1], p[2]); }
__device__ __forceinline__ M3 P9(const double* p) {
  M3 m;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.a[k] = p[k];
  return m;
}

// Packed record p with outputs at o.
struct PackedElem {
  const double* p;
  double* o;
  __device__ __forceinline__ V3 x(int n) const { return P3(p + 3 * n) + P3(p + 6 + 3 * n); }
  __device__ __forceinline__ M3 R(int n) const { return P9(p + 12 + 9 * n); }
  __device__ __forceinline__ M3 dR(int n) const { return P9(p + 30 + 9 * n); }
  __device__ __forceinline__ M3 Re0() const { return P9(p + 73); }
  __device__ __forceinline__ V3 ud(int n) const { return P3(p + 48 + 3 * n); }
  __device__ __forceinline__ V3 wd(int n) const { return P3(p + 54 + 3 * n); }
  __device__ __forceinline__ V3 udd(int n) const { return P3(p + 60 + 3 * n); }
  __device__ __forceinline__ V3 wdd(int n) const { return P3(p + 66 + 3 * n); }
  __device__ __forceinline__ double l0() const { return p[72]; }
  __device__ __forceinline__ double Ku() const { return p[82]; }
  __device__ __forceinline__ V3 KT() const { return P3(p + 83); }
  __device__ __forceinline__ V3 KTT() const { return P3(p + 86); }
  __device__ __forceinline__ V3 Jr() const { return P3(p + 89); }
  __device__ __forceinline__ double Ar() const { return p[92]; }
  __device__ __forceinline__ double damping() const { return p[93]; }
  __device__ __forceinline__ BeamOut out() const { return BeamOut{o + 26, o + 170, o + 314, o + 2, o + 14, o}; }
};

__global__ void __launch_bounds__(kBeamCta) k_element_eval(int64_t n, int nb, const double* in, Gauss3 g, double* out) {
  extern __shared__ double beam_tab[];
  beam_cta(n, nb, g, beam_tab, [&](int64_t e) { return PackedElem{in + 96 * e, out + 458 * e}; }, [](int64_t) { return true; });
}

struct PackedContact : PackedElem {
  const SurfaceDev& s;
  const ContactProps& cp;
  int32_t* flag;
  __device__ __forceinline__ PackedContact(const double* p_, double* o_, const SurfaceDev& s_, const ContactProps& c_, int32_t* f_)
      : PackedElem{p_, o_}, s(s_), cp(c_), flag(f_) {}
  __device__ __forceinline__ double radius() const { return p[94]; }
  __device__ __forceinline__ const SurfaceDev& surf() const { return s; }
  __device__ __forceinline__ const ContactProps& props() const { return cp; }
  __device__ __forceinline__ ContactOut out() const { return ContactOut{o + 13, o + 157, o + 1, o}; }
  __device__ __forceinline__ void touched(bool any) const { *flag = any ? 1 : 0; }
};

__global__ void __launch_bounds__(kContactCta) k_contact_eval(int64_t n, int nb, const double* in, Gauss3 g,
                                                              const __grid_constant__ ContactProps cp,
                                                              const __grid_constant__ SurfaceDev s, double* out,
                                                              int32_t* flags) {
  extern __shared__ double beam_tab[];
  contact_cta(n, nb, g, beam_tab, [&](int64_t e) { return PackedContact(in + 96 * e, out + 301 * e, s, cp, flags + e); },
              [](int64_t) { return true; });
}

// Launch shape of n elements on the current device (as eb_create's).
int eval_groups(int64_t n) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return beam_groups(eb::wide_elements(n, sms) ? 256 : 128);
}

cudaError_t launch_contact_eval(int64_t n, const double* in, const Gauss3& g, const ContactProps& cp, const SurfaceDev& s,
                                double* out, int32_t* flags, cudaStream_t st) {
  const int nb = eval_groups(n);
  const cudaError_t e = eb::raise_smem_limit((const void*)k_contact_eval, contact_smem(nb));
  if (e != cudaSuccess) return e;
  k_contact_eval<<<eb::nblocks(n, kBeamGroup * nb), kContactCta, contact_smem(nb), st>>>(n, nb, in, g, cp, s, out, flags);
  return cudaGetLastError();
}

struct DBuf {
  void* p = nullptr;
  ~DBuf() { if (p) cudaFree(p); }
};

}  // namespace

// defined in eb_abi.cu
std::vector<double> eb_sdf_coefficients_host(const double* values, const int64_t dims[3], bool negate);
std::vector<double> eb_sdf_samples_padded_host(const double* values, const int64_t dims[3], bool negate);
int eb_internal_fail(int code, const char* msg);

namespace {
int err(const char* what, cudaError_t e) {
  std::snprintf(g_err2, sizeof(g_err2), "%s: %s", what, cudaGetErrorString(e));
  return eb_internal_fail(EB_ERR_CUDA, g_err2);
}
}  // namespace

extern "C" int eb_element_eval(int64_t n, const double* in, const double* gauss6, double* out) {
  if (n <= 0 || !in || !gauss6 || !out) return EB_ERR_ARG;
  Gauss3 g;
  for (int i = 0; i < 3; ++i) { g.w[i] = gauss6[i]; g.z[i] = gauss6[3 + i]; }
  DBuf di, dout;
  cudaError_t e;
  if ((e = cudaMalloc(&di.p, sizeof(double) * 96 * n)) != cudaSuccess) return err("cudaMalloc", e);
  if ((e = cudaMalloc(&dout.p, sizeof(double) * 458 * n)) != cudaSuccess) return err("cudaMalloc", e);
  cudaMemcpy(di.p, in, sizeof(double) * 96 * n, cudaMemcpyHostToDevice);
  cudaMemset(dout.p, 0, sizeof(double) * 458 * n);
  const int nb = eval_groups(n);
  if ((e = eb::raise_smem_limit((const void*)k_element_eval, beam_smem(nb))) != cudaSuccess) return err("k_element_eval", e);
  k_element_eval<<<eb::nblocks(n, kBeamGroup * nb), kBeamCta, beam_smem(nb)>>>(n, nb, (const double*)di.p, g,
                                                                                (double*)dout.p);
  if ((e = cudaGetLastError()) != cudaSuccess) return err("k_element_eval launch", e);
  if ((e = cudaMemcpy(out, dout.p, sizeof(double) * 458 * n, cudaMemcpyDeviceToHost)) != cudaSuccess)
    return err("k_element_eval", e);
  return EB_OK;
}

extern "C" int eb_contact_eval(int64_t n, const double* in, const double* gauss6, const double* props,
                               const double* surf, const double* values, double* out, int32_t* flags) {
  if (n <= 0 || !in || !gauss6 || !props || !surf || !out || !flags) return EB_ERR_ARG;
  Gauss3 g;
  for (int i = 0; i < 3; ++i) { g.w[i] = gauss6[i]; g.z[i] = gauss6[3 + i]; }
  ContactProps cp{props[0], props[1], props[2], props[3]};
  SurfaceDev s;
  std::memset(&s, 0, sizeof(s));
  s.kind = (int)surf[0];
  s.cx = surf[1]; s.cy = surf[2]; s.cz = surf[3]; s.R = surf[4];
  if (s.kind == 2) {
    s.axis = (int)surf[1];
    s.pos = surf[2];
  }
  if (s.kind < 0 || s.kind > 3 || s.axis < 0 || s.axis > 2) return EB_ERR_ARG;
  if (s.kind == 3) {  // voxel SDF, trilinear
    s.kind = 1;
    s.interp = 1;
    if (surf[5] < 2 || surf[6] < 2 || surf[7] < 2) return EB_ERR_ARG;
  }
  DBuf dcoef, di, dout, dfl;
  cudaError_t e;
  if (s.kind == 1) {
    if (!values) return EB_ERR_ARG;
    int64_t dims[3] = {(int64_t)surf[5], (int64_t)surf[6], (int64_t)surf[7]};
    std::vector<double> c = s.interp ? eb_sdf_samples_padded_host(values, dims, false)
                                     : eb_sdf_coefficients_host(values, dims, false);
    if ((e = cudaMalloc(&dcoef.p, sizeof(double) * c.size())) != cudaSuccess) return err("cudaMalloc", e);
    cudaMemcpy(dcoef.p, c.data(), sizeof(double) * c.size(), cudaMemcpyHostToDevice);
    s.coef = (const double*)dcoef.p;
    s.nx = (int)dims[0]; s.ny = (int)dims[1]; s.nz = (int)dims[2];
    s.x0 = surf[8]; s.y0 = surf[9]; s.z0 = surf[10];
    s.ihx = 1.0 / surf[11]; s.ihy = 1.0 / surf[12]; s.ihz = 1.0 / surf[13];
    s.xl = (s.nx - 1) * surf[11]; s.yl = (s.ny - 1) * surf[12]; s.zl = (s.nz - 1) * surf[13];
  }
  if ((e = cudaMalloc(&di.p, sizeof(double) * 96 * n)) != cudaSuccess) return err("cudaMalloc", e);
  if ((e = cudaMalloc(&dout.p, sizeof(double) * 301 * n)) != cudaSuccess) return err("cudaMalloc", e);
  if ((e = cudaMalloc(&dfl.p, sizeof(int32_t) * n)) != cudaSuccess) return err("cudaMalloc", e);
  cudaMemcpy(di.p, in, sizeof(double) * 96 * n, cudaMemcpyHostToDevice);
  cudaMemset(dout.p, 0, sizeof(double) * 301 * n);
  if ((e = launch_contact_eval(n, (const double*)di.p, g, cp, s, (double*)dout.p, (int32_t*)dfl.p, 0)) != cudaSuccess)
    return err("k_contact_eval launch", e);
  if ((e = cudaMemcpy(out, dout.p, sizeof(double) * 301 * n, cudaMemcpyDeviceToHost)) != cudaSuccess)
    return err("k_contact_eval", e);
  cudaMemcpy(flags, dfl.p, sizeof(int32_t) * n, cudaMemcpyDeviceToHost);
  return EB_OK;
}

// ---------------------------------------------------------------- contact evaluation without allocation
// Variant of eb_contact_eval for callers that cannot allocate device memory
// during the call (a host whose device memory belongs to its own pool
// allocator, a loop that forbids allocation after start-up): the caller's
// device buffers are used directly, and the prefiltered SDF coefficients go
// to the fixed array below instead of a cudaMalloc.
namespace {

__device__ __align__(256) double g_noalloc_coef[EB_NOALLOC_SDF_MAX_COEFS];

std::mutex g_noalloc_mu;
constexpr int kMaxDevices = 64;
// Device address of g_noalloc_coef per device ordinal, and the context it was looked up in:
// after cudaDeviceReset (or any other re-creation of the device's context) the address is
// looked up again.
double* g_noalloc_ptr[kMaxDevices] = {nullptr};
void* g_noalloc_ctx[kMaxDevices] = {nullptr};

// The calling thread's current driver context (an opaque handle), through the runtime's
// driver entry-point query so the library does not link the driver API; nullptr if unknown.
void* current_context() {
  using GetCurrent = int (*)(void**);
  static GetCurrent fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (GetCurrent)f;
  }();
  void* ctx = nullptr;
  if (!fn || fn(&ctx) != 0) return nullptr;
  return ctx;
}

__global__ void k_sdf_interior(const double* __restrict__ vals, int nx, int ny, int nz, double* __restrict__ c) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)nx * ny * nz) return;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / ((int64_t)nx * ny));
  c[(i + 1) + (int64_t)(nx + 2) * ((j + 1) + (int64_t)(ny + 2) * (k + 1))] = vals[t];
}

// In-place solve of the quadratic B-spline interpolation system
// ⅛c[i-1] + ¾c[i] + ⅛c[i+1] = y[i] along every grid line of `axis` with the
// reflected ends (first/last diagonal 7/8), then the two pads c[0] = c[1],
// c[n+1] = c[n].  Lines run over the padded range of axes already filtered.
//
// The elimination's factors do not depend on the samples and reach their fixed
// point within 32 rows: they come as a table.  A CTA takes 32 lines into shared
// memory (rows of consecutive lines, or whole lines along x, both coalesced) and
// one warp runs the recurrences there, a chain of two FP64 operations per row;
// with a thread per line in global memory every row waited for a load and a
// division (61³ points: 76 us a pass, 147 us at 128³).
struct LineFactors {
  double cp[32], im[32];  // super-diagonal factor, inverse pivot of rows 0 .. 31 (row 31: all later ones)
};
LineFactors line_factors() {
  LineFactors f;
  double cp = 0.0;
  for (int i = 0; i < 32; ++i) {
    const double m = i == 0 ? 0.875 : 0.75 - 0.125 * cp;
    cp = 0.125 / m;
    f.cp[i] = cp;
    f.im[i] = 1.0 / m;
  }
  return f;
}

constexpr int kLines = 32;       // lines per CTA, one per lane of the solving warp
constexpr int kLineStride = 33;  // doubles between rows in shared memory
constexpr int kLineThreads = 256;
constexpr int kMaxLine = 800;    // longest line whose tile fits in shared memory (211 KB)

__device__ __forceinline__ int64_t line_base(int64_t t, int nx, int ny, int nz, int axis, int64_t* stride) {
  const int64_t px = nx + 2, py = ny + 2;
  if (axis == 0) {  // lines (j, k), interior j and k
    *stride = 1;
    return px * ((1 + t % ny) + py * (1 + t / ny));
  }
  if (axis == 1) {  // lines (i, k), all i, interior k
    *stride = px;
    return t % px + px * py * (1 + t / px);
  }
  *stride = px * py;  // lines (i, j), all i and j
  return t;
}

__global__ void __launch_bounds__(kLineThreads) k_sdf_prefilter_axis(double* c, int nx, int ny, int nz, int axis,
                                                                     int64_t lines, LineFactors f) {
  extern __shared__ double row[];
  const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
  const int64_t l0 = (int64_t)blockIdx.x * kLines;
  const int nl = (int)(lines - l0 < kLines ? lines - l0 : kLines);
  int64_t stride;
  // element (row i, line l) of the tile: threads run along the contiguous direction
  auto each = [&](auto op) {
    for (int e = threadIdx.x; e < n * kLines; e += kLineThreads) {
      const int i = axis == 0 ? e % n : e / kLines, l = axis == 0 ? e / n : e % kLines;
      if (l < nl) op(i, l, c + line_base(l0 + l, nx, ny, nz, axis, &stride) + (int64_t)(i + 1) * stride);
    }
  };
  each([&](int i, int l, double* p) { row[i * kLineStride + l] = *p; });
  __syncthreads();
  if (threadIdx.x < nl && n > 1) {
    double* y = row + threadIdx.x;
    double v = y[0] * f.im[0];
    y[0] = v;
    for (int i = 1; i < n - 1; ++i) {
      v = (y[i * kLineStride] - 0.125 * v) * f.im[i < 32 ? i : 31];
      y[i * kLineStride] = v;
    }
    v = (y[(n - 1) * kLineStride] - 0.125 * v) / (0.875 - 0.125 * f.cp[n - 2 < 32 ? n - 2 : 31]);
    y[(n - 1) * kLineStride] = v;
    for (int i = n - 2; i >= 0; --i) {
      v = y[i * kLineStride] - f.cp[i < 32 ? i : 31] * v;
      y[i * kLineStride] = v;
    }
  }
  __syncthreads();
  each([&](int i, int l, double* p) {
    const double v = row[i * kLineStride + l];
    *p = v;
    if (i == 0) p[-stride] = v;
    if (i == n - 1) p[stride] = v;
  });
}

// The same for lines longer than kMaxLine: one thread per line, in place in global memory.
__global__ void k_sdf_prefilter_long(double* c, int nx, int ny, int nz, int axis, int64_t lines, LineFactors f) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= lines) return;
  const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
  int64_t stride;
  double* y = c + line_base(t, nx, ny, nz, axis, &stride);
  y += stride;
  double v = y[0] * f.im[0];
  y[0] = v;
  for (int i = 1; i < n - 1; ++i) y[i * stride] = v = (y[i * stride] - 0.125 * v) * f.im[i < 32 ? i : 31];
  v = (y[(n - 1) * stride] - 0.125 * v) / (0.875 - 0.125 * f.cp[31]);
  y[(n - 1) * stride] = y[n * stride] = v;
  for (int i = n - 2; i >= 0; --i) y[i * stride] = v = y[i * stride] - f.cp[i < 32 ? i : 31] * v;
  y[-stride] = v;
}

}  // namespace

// Prefilters a padded coefficient grid whose interior holds the SDF samples
// (three passes over the grid lines of an axis).
namespace eb {
void launch_sdf_prefilter(double* coef, int nx, int ny, int nz, cudaStream_t st) {
  static const LineFactors f = line_factors();
  const int64_t px = nx + 2, py = ny + 2, lines[3] = {(int64_t)ny * nz, px * nz, px * py};
  const int n[3] = {nx, ny, nz};
  for (int a = 0; a < 3; ++a) {
    const size_t smem = sizeof(double) * kLineStride * (size_t)n[a];
    if (n[a] <= kMaxLine && (smem <= 48 * 1024 || raise_smem_limit((const void*)k_sdf_prefilter_axis, smem) == cudaSuccess))
      k_sdf_prefilter_axis<<<(unsigned)((lines[a] + kLines - 1) / kLines), kLineThreads, smem, st>>>(coef, nx, ny, nz, a,
                                                                                                    lines[a], f);
    else
      k_sdf_prefilter_long<<<(unsigned)((lines[a] + 127) / 128), 128, 0, st>>>(coef, nx, ny, nz, a, lines[a], f);
  }
}
}  // namespace eb

extern "C" int eb_contact_eval_noalloc(int64_t n, const double* d_in, const double* gauss6, const double* props,
                                       const double* surf, const double* d_sdf_values, double* d_out,
                                       int32_t* d_flags, void* stream) {
  if (n < 0 || !gauss6 || !props || !surf) return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: bad arguments");
  if (n == 0) return EB_OK;
  if (!d_in || !d_out || !d_flags) return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: null device buffer");
  cudaStream_t st = (cudaStream_t)stream;
  Gauss3 g;
  for (int i = 0; i < 3; ++i) { g.w[i] = gauss6[i]; g.z[i] = gauss6[3 + i]; }
  ContactProps cp{props[0], props[1], props[2], props[3]};
  // surface kind (0 sphere, 1 SDF, 2 plane) and the plane's axis are whole numbers in range
  // before they are converted
  if (!(surf[0] == 0 || surf[0] == 1 || surf[0] == 2) ||
      (surf[0] == 2 && !(surf[1] == 0 || surf[1] == 1 || surf[1] == 2)))
    return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: bad surface kind or plane axis");
  SurfaceDev s;
  std::memset(&s, 0, sizeof(s));
  s.kind = (int)surf[0];
  s.cx = surf[1]; s.cy = surf[2]; s.cz = surf[3]; s.R = surf[4];
  if (s.kind == 2) {
    s.axis = (int)surf[1];
    s.pos = surf[2];
  }
  if (s.kind == 1) {
    if (!d_sdf_values) return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: SDF values missing");
    // every grid dimension is checked on its own (finite, at least 1, within the array) before
    // the padded product is formed, so the product cannot overflow
    const double lim = (double)EB_NOALLOC_SDF_MAX_COEFS;
    for (int a = 5; a < 8; ++a)
      if (!std::isfinite(surf[a]) || !(surf[a] >= 1) || !(surf[a] <= lim) || surf[a] != std::floor(surf[a]))
        return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: bad SDF grid dimension (surf[5..7] must be "
                                            "integers in [1, EB_NOALLOC_SDF_MAX_COEFS])");
    for (int a = 8; a < 14; ++a)
      if (!std::isfinite(surf[a]) || (a >= 11 && !(surf[a] > 0)))
        return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: bad SDF origin or spacing (surf[8..13])");
    const int64_t nx = (int64_t)surf[5], ny = (int64_t)surf[6], nz = (int64_t)surf[7];
    if ((nx + 2) > (int64_t)EB_NOALLOC_SDF_MAX_COEFS / ((ny + 2) * (nz + 2)) ||
        (nx + 2) * (ny + 2) * (nz + 2) > (int64_t)EB_NOALLOC_SDF_MAX_COEFS)
      return eb_internal_fail(EB_ERR_ARG,
                              "eb_contact_eval_noalloc: SDF grid too large for the fixed coefficient array "
                              "((nx+2)(ny+2)(nz+2) > EB_NOALLOC_SDF_MAX_COEFS = 287496)");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return err("cudaGetDevice", e);
    if (dev < 0 || dev >= kMaxDevices) return eb_internal_fail(EB_ERR_ARG, "eb_contact_eval_noalloc: device ordinal");
    double* coef = nullptr;
    {
      std::lock_guard<std::mutex> lk(g_noalloc_mu);
      void* ctx = current_context();
      if (!g_noalloc_ptr[dev] || !ctx || ctx != g_noalloc_ctx[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_coef);
        if (e != cudaSuccess) return err("cudaGetSymbolAddress", e);
        g_noalloc_ptr[dev] = (double*)p;
        g_noalloc_ctx[dev] = current_context();
      }
      coef = g_noalloc_ptr[dev];
    }
    const int NX = (int)nx, NY = (int)ny, NZ = (int)nz;
    const int64_t pts = nx * ny * nz;
    k_sdf_interior<<<(unsigned)((pts + 255) / 256), 256, 0, st>>>(d_sdf_values, NX, NY, NZ, coef);
    eb::launch_sdf_prefilter(coef, NX, NY, NZ, st);
    s.coef = coef;
    s.nx = NX; s.ny = NY; s.nz = NZ;
    s.x0 = surf[8]; s.y0 = surf[9]; s.z0 = surf[10];
    s.ihx = 1.0 / surf[11]; s.ihy = 1.0 / surf[12]; s.ihz = 1.0 / surf[13];
    s.xl = (NX - 1) * surf[11]; s.yl = (NY - 1) * surf[12]; s.zl = (NZ - 1) * surf[13];
  }
  // untouched elements leave zero records, as in eb_contact_eval
  cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(double) * 301 * n, st);
  if (e != cudaSuccess) return err("cudaMemsetAsync", e);
  e = launch_contact_eval(n, d_in, g, cp, s, d_out, d_flags, st);
  if (e != cudaSuccess) return err("k_contact_eval (no-alloc) launch", e);
  return EB_OK;
}

// ---------------------------------------------------------------- FP64 throughput probe
namespace {
__global__ void k_fp64_fma(double* out, int iters, double b, double c) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6,
         a7 = a0 + 7;
  for (int i = 0; i < iters; ++i) {
    a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
    a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
  }
  out[(int64_t)blockIdx.x * blockDim.x + threadIdx.x] = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
}
}  // namespace

extern "C" int eb_fp64_peak(double* tflops) {
  if (!tflops) return EB_ERR_ARG;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int threads = 256, blocks = sms * 8, iters = 4096;
  DBuf out;
  cudaError_t e;
  if ((e = cudaMalloc(&out.p, sizeof(double) * threads * blocks)) != cudaSuccess) return err("cudaMalloc", e);
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  k_fp64_fma<<<blocks, threads>>>((double*)out.p, iters, 0.999999, 1e-7);  // warm-up
  float best = 1e30f;
  for (int rep = 0; rep < 5; ++rep) {
    cudaEventRecord(a);
    k_fp64_fma<<<blocks, threads>>>((double*)out.p, iters, 0.999999, 1e-7);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    if (ms < best) best = ms;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if ((e = cudaGetLastError()) != cudaSuccess) return err("k_fp64_fma", e);
  const double flops = 2.0 * 8.0 * iters * (double)threads * blocks;
  *tflops = flops / (best * 1e-3) / 1e12;
  return EB_OK;
}
