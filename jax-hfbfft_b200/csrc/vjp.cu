// Nyquist-line terms for the vector-Jacobian products of hpsi and of the
// densities.
//
// The second derivative of cderv02 (levels.py:284-395) replaces the Nyquist
// bin of each line along the derivative axis by -(pi/d)^2 mean(B) x_N / n,
// x_N = sum_j (-1)^j x_j.  As an operator on x this is c mean(B) e e^T with
// e_j = (-1)^j and c = -(pi/d)^2 / n: Hermitian in x and linear in B.  The
// rest of hpsi's bilinear form <a|h[P]|b> is the integral of each field
// times the pair density of (a, b) that the density kernel computes, so
// these two kernels are all the VJPs add to the library's hpsi and density
// kernels:
//   hfb_nyquist_pair   the bmass cotangent from this term,
//   hfb_nyquist_apply  the term itself, with B a density cotangent (the
//                      density tau has no Nyquist term, so the density VJP,
//                      formed with hpsi, takes it back out).
// Lines along axis ax are numbered by the two other coordinates (u, v) in
// increasing order; every sum runs in a fixed order.
#include <math.h>
#include "hfb_ctx.cuh"

namespace hfb {
namespace {

constexpr int kVjThreads = 128;

struct LineGeo {
  size_t off, stride;
};

__device__ __forceinline__ LineGeo line_geo(int n, int ax, int line) {
  const int u = line / n, v = line % n;
  const size_t n2 = (size_t)n * n;
  if (ax == 0) return {(size_t)u * n + v, n2};
  if (ax == 1) return {(size_t)u * n2 + v, (size_t)n};
  return {(size_t)u * n2 + (size_t)v * n, 1};
}

// The sums over a line, sum_j (-1)^j x_j, are formed for every state and line
// at once (one thread each): per isospin with the states in a loop, 24 blocks
// did it all (532 us for 70 states at 32^3; 68 us with the two launches below).

// t[s][ax][line] = sum_c Re(conj(a_N) b_N)
template <class Z>
__global__ void __launch_bounds__(kVjThreads) nyq_pair_lines_kernel(int n, const Z* __restrict__ a,
                                                                    const Z* __restrict__ b, double* __restrict__ t) {
  const int line = blockIdx.x * kVjThreads + threadIdx.x, ax = blockIdx.y, s = blockIdx.z;
  if (line >= n * n) return;
  const LineGeo g = line_geo(n, ax, line);
  const size_t n3 = (size_t)n * n * n;
  double sum = 0.0;
  for (int c = 0; c < 2; ++c) {
    const Z* pa = a + ((size_t)s * 2 + c) * n3 + g.off;
    const Z* pb = b + ((size_t)s * 2 + c) * n3 + g.off;
    double ar = 0.0, ai = 0.0, br = 0.0, bi = 0.0;
#pragma unroll 4
    for (int j = 0; j < n; j += 2) {   // n is even
      const Z x = pa[(size_t)j * g.stride], y = pb[(size_t)j * g.stride];
      const Z u = pa[(size_t)(j + 1) * g.stride], v = pb[(size_t)(j + 1) * g.stride];
      ar += (double)x.x; ai += (double)x.y; br += (double)y.x; bi += (double)y.y;
      ar -= (double)u.x; ai -= (double)u.y; br -= (double)v.x; bi -= (double)v.y;
    }
    sum += ar * br + ai * bi;
  }
  t[((size_t)s * 3 + ax) * n * n + line] = sum;
}

// m[iq][ax][line] = sum_{s in iq} w_s t[s][ax][line]
__global__ void __launch_bounds__(kVjThreads) nyq_pair_sum_kernel(int n2, int nst, int nneut, const double* __restrict__ w,
                                                                  const double* __restrict__ t, double* __restrict__ m) {
  const int e = blockIdx.x * kVjThreads + threadIdx.x, iq = blockIdx.y;
  if (e >= 3 * n2) return;
  const int s0 = iq == 0 ? 0 : nneut, s1 = iq == 0 ? nneut : nst;
  double acc = 0.0;
#pragma unroll 8
  for (int s = s0; s < s1; ++s) acc += w[s] * t[(size_t)s * 3 * n2 + e];
  m[(size_t)iq * 3 * n2 + e] = acc;
}

// field[iq][x][y][z] += sum_ax (pi/d_ax)^2 / n^2 m[iq][ax][line_ax(x, y, z)]
__global__ void nyq_pair_field_kernel(int n, double k0, double k1, double k2, const double* __restrict__ m,
                                      double* __restrict__ field) {
  const size_t n3 = (size_t)n * n * n, n2 = (size_t)n * n;
  const size_t i = blockIdx.x * (size_t)kVjThreads + threadIdx.x;
  if (i >= 2 * n3) return;
  const int iq = (int)(i / n3);
  const size_t r = i % n3;
  const int x = (int)(r / n2), y = (int)((r / n) % n), z = (int)(r % n);
  const double* mq = m + (size_t)iq * 3 * n2;
  field[i] += k0 * mq[(size_t)y * n + z] + k1 * mq[n2 + (size_t)x * n + z] + k2 * mq[2 * n2 + (size_t)x * n + y];
}

// xn[sc][ax][line] = c_ax scale_s mean_line(field[iq(s)]) x_N, with sc the
// state and component
struct Nyq3 {
  double v[3];
};
template <class Z>
__global__ void __launch_bounds__(kVjThreads)
nyq_apply_lines_kernel(int n, int nneut, Nyq3 c, const double* __restrict__ field, const double* __restrict__ scale,
                       const Z* __restrict__ x, double2* __restrict__ xn) {
  const int line = blockIdx.x * kVjThreads + threadIdx.x, ax = blockIdx.y, sc = blockIdx.z, s = sc / 2;
  if (line >= n * n) return;
  const LineGeo g = line_geo(n, ax, line);
  const size_t n3 = (size_t)n * n * n;
  const double* f = field + (size_t)(s < nneut ? 0 : 1) * n3 + g.off;
  const Z* px = x + (size_t)sc * n3 + g.off;
  double fm = 0.0, xr = 0.0, xi = 0.0;
#pragma unroll 4
  for (int j = 0; j < n; j += 2) {   // n is even
    const Z u = px[(size_t)j * g.stride], v = px[(size_t)(j + 1) * g.stride];
    fm += f[(size_t)j * g.stride] + f[(size_t)(j + 1) * g.stride];
    xr += (double)u.x; xi += (double)u.y;
    xr -= (double)v.x; xi -= (double)v.y;
  }
  const double k = scale[s] * c.v[ax] * (fm / n);
  xn[((size_t)sc * 3 + ax) * n * n + line] = make_double2(k * xr, k * xi);
}

// y_s += sum_ax (-1)^j xn[sc][ax][line_ax]
template <class Z>
__global__ void __launch_bounds__(kVjThreads)
nyq_apply_points_kernel(int n, const double2* __restrict__ xn, Z* __restrict__ y) {
  const size_t n3 = (size_t)n * n * n, n2 = (size_t)n * n;
  const size_t i = blockIdx.x * (size_t)kVjThreads + threadIdx.x;
  if (i >= n3) return;
  const int px = (int)(i / n2), py = (int)((i / n) % n), pz = (int)(i % n);
  const double2* t = xn + (size_t)blockIdx.y * 3 * n2;
  const double2 a = t[(size_t)py * n + pz], b = t[n2 + (size_t)px * n + pz], c = t[2 * n2 + (size_t)px * n + py];
  const double sa = (px & 1) ? -1.0 : 1.0, sb = (py & 1) ? -1.0 : 1.0, sc = (pz & 1) ? -1.0 : 1.0;
  Z* o = y + (size_t)blockIdx.y * n3 + i;
  Z v = *o;
  v.x += sa * a.x + sb * b.x + sc * c.x;
  v.y += sa * a.y + sb * b.y + sc * c.y;
  *o = v;
}

}  // namespace
}  // namespace hfb

using namespace hfb;

extern "C" int hfb_nyquist_pair(hfb_ctx_t ctx, int prec, int nst, int nneut, const void* a, const void* b,
                                const double* w, double* field, void* stream) {
  if (!ctx || !a || !b || !w || !field || nst <= 0 || nneut < 0 || nneut > nst) return HFB_ERR_ARG;
  const int n = ctx->n;
  const size_t n2 = (size_t)n * n;
  double* t = (double*)scratch(ctx, hfb_ctx_s::S_VJP, sizeof(double) * 3 * n2 * ((size_t)nst + 2));
  if (!t) return HFB_ERR_ALLOC;
  double* m = t + 3 * n2 * nst;
  cudaStream_t st = as_stream(stream);
  // at most 65535 states a launch (the grid's third dimension)
  for (int s = 0; s < nst; s += 65535) {
    const dim3 grid((n * n + kVjThreads - 1) / kVjThreads, 3, nst - s < 65535 ? nst - s : 65535);
    const size_t o = (size_t)s * 2 * n2 * n;
    if (prec == HFB_F64)
      nyq_pair_lines_kernel<double2><<<grid, kVjThreads, 0, st>>>(n, (const double2*)a + o, (const double2*)b + o,
                                                                  t + 3 * n2 * s);
    else
      nyq_pair_lines_kernel<float2><<<grid, kVjThreads, 0, st>>>(n, (const float2*)a + o, (const float2*)b + o,
                                                                 t + 3 * n2 * s);
    HFB_CHECK_LAUNCH();
  }
  nyq_pair_sum_kernel<<<dim3((3 * n * n + kVjThreads - 1) / kVjThreads, 2), kVjThreads, 0, st>>>(n * n, nst, nneut, w, t,
                                                                                                 m);
  HFB_CHECK_LAUNCH();
  double k[3];
  for (int ax = 0; ax < 3; ++ax) k[ax] = (M_PI / ctx->d[ax]) * (M_PI / ctx->d[ax]) / ((double)n * n);
  const size_t tot = 2 * (size_t)n * n * n;
  nyq_pair_field_kernel<<<(unsigned)((tot + kVjThreads - 1) / kVjThreads), kVjThreads, 0, st>>>(n, k[0], k[1], k[2],
                                                                                               m, field);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

extern "C" int hfb_nyquist_apply(hfb_ctx_t ctx, int prec, int nst, int nneut, const double* field,
                                 const double* scale, const void* x, void* y, void* stream) {
  if (!ctx || !field || !scale || !x || !y || nst <= 0 || nneut < 0 || nneut > nst || x == y) return HFB_ERR_ARG;
  const int n = ctx->n;
  cudaStream_t st = as_stream(stream);
  const size_t n2 = (size_t)n * n, n3 = n2 * n;
  double2* xn = (double2*)scratch(ctx, hfb_ctx_s::S_VJP, sizeof(double2) * 6 * n2 * nst);
  if (!xn) return HFB_ERR_ALLOC;
  Nyq3 c;
  for (int ax = 0; ax < 3; ++ax) c.v[ax] = -(M_PI / ctx->d[ax]) * (M_PI / ctx->d[ax]) / n;
  for (int s = 0; s < nst; s += 32767) {   // two grid layers a state
    const int ns = nst - s < 32767 ? nst - s : 32767;
    const dim3 g1((n * n + kVjThreads - 1) / kVjThreads, 3, 2 * ns), g2((unsigned)((n3 + kVjThreads - 1) / kVjThreads), 2 * ns);
    const size_t o = (size_t)s * 2 * n3;
    if (prec == HFB_F64) {
      nyq_apply_lines_kernel<double2><<<g1, kVjThreads, 0, st>>>(n, nneut - s, c, field, scale + s, (const double2*)x + o,
                                                                 xn);
      HFB_CHECK_LAUNCH();
      nyq_apply_points_kernel<double2><<<g2, kVjThreads, 0, st>>>(n, xn, (double2*)y + o);
    } else {
      nyq_apply_lines_kernel<float2><<<g1, kVjThreads, 0, st>>>(n, nneut - s, c, field, scale + s, (const float2*)x + o,
                                                                xn);
      HFB_CHECK_LAUNCH();
      nyq_apply_points_kernel<float2><<<g2, kVjThreads, 0, st>>>(n, xn, (float2*)y + o);
    }
    HFB_CHECK_LAUNCH();
  }
  return HFB_OK;
}
