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

constexpr int kVjThreads = 128, kVjWarps = kVjThreads / 32;

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

// The sums over a line, sum_j (-1)^j x_j, are formed for every line and for
// runs of an isospin's states at once (one thread each): with all the states of
// an isospin in one loop, 24 blocks did it all (532 us for 70 states at 32^3;
// 64 us here, lines and their sum).  At most kVjGroups runs an isospin, so that
// their sums have one size whatever the state count.
constexpr int kVjGroups = 64;
struct VjRuns {
  int first[2], end[2], run[2], groups[2];   // states of each isospin, states a run, runs
};

// t[group][ax][line] = sum_{s in the group} w_s sum_c Re(conj(a_N) b_N); the
// neutrons' groups first
template <class Z>
__global__ void __launch_bounds__(kVjThreads)
nyq_pair_lines_kernel(int n, VjRuns r, const Z* __restrict__ a, const Z* __restrict__ b, const double* __restrict__ w,
                      double* __restrict__ t) {
  const int line = blockIdx.x * kVjThreads + threadIdx.x, ax = blockIdx.y;
  if (line >= n * n) return;
  const int iq = (int)blockIdx.z >= r.groups[0], group = blockIdx.z - (iq ? r.groups[0] : 0);
  const int s0 = r.first[iq] + group * r.run[iq], s1 = min(s0 + r.run[iq], r.end[iq]);
  const LineGeo g = line_geo(n, ax, line);
  const size_t n3 = (size_t)n * n * n;
  double acc = 0.0;
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    double sum = 0.0;
#pragma unroll
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
    acc += w[s] * sum;
  }
  t[((size_t)blockIdx.z * 3 + ax) * n * n + line] = acc;
}

// m[iq][ax][line] = sum of the isospin's groups
__global__ void __launch_bounds__(kVjThreads) nyq_pair_sum_kernel(int n2, VjRuns r, const double* __restrict__ t,
                                                                  double* __restrict__ m) {
  const int e = blockIdx.x * kVjThreads + threadIdx.x, iq = blockIdx.y;
  if (e >= 3 * n2) return;
  const double* p = t + (iq ? (size_t)r.groups[0] * 3 * n2 : 0) + e;
  double acc = 0.0;
#pragma unroll 8
  for (int g = 0; g < r.groups[iq]; ++g) acc += p[(size_t)g * 3 * n2];
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

// y_s += c scale_s sum over the lines through each point of mean_line(field)
// (-1)^j x_N: the x lines, then the y and z lines plane by plane.  Two passes,
// no scratch (held in a buffer between two launches, the lines' sums made the
// first call of a context allocate).

// x lines: a warp takes a quarter of the points (n / 4, even) of 32 lines
template <class Z>
__global__ void __launch_bounds__(kVjThreads)
nyq_apply_x_kernel(int n, int nneut, double c, const double* __restrict__ field, const double* __restrict__ scale,
                   const Z* __restrict__ x, Z* __restrict__ y) {
  __shared__ double part[kVjWarps][3][32];
  const int n2 = n * n, nb = n2 / 32, seg = n / kVjWarps;   // n is a multiple of 8
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int sc = blockIdx.x / nb, s = sc / 2, j0 = warp * seg;
  const size_t n3 = (size_t)n * n2, off = (size_t)j0 * n2 + blockIdx.x % nb * 32 + lane;
  const double* f = field + (s < nneut ? 0 : n3) + off;
  const Z* px = x + (size_t)sc * n3 + off;
  Z* py = y + (size_t)sc * n3 + off;
  double t[3] = {0.0, 0.0, 0.0};
#pragma unroll 6
  for (int j = 0; j < seg; j += 2) {
    const Z u = px[(size_t)j * n2], v = px[(size_t)(j + 1) * n2];
    t[0] += (double)u.x; t[1] += (double)u.y;
    t[0] -= (double)v.x; t[1] -= (double)v.y;
    t[2] += f[(size_t)j * n2] + f[(size_t)(j + 1) * n2];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) part[warp][i][lane] = t[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = part[0][i][lane];
    for (int w = 1; w < kVjWarps; ++w) t[i] += part[w][i][lane];
  }
  const double k = scale[s] * c * (t[2] / n), xr = k * t[0], xi = k * t[1];
#pragma unroll 6
  for (int j = 0; j < seg; j += 2) {
    Z u = py[(size_t)j * n2], v = py[(size_t)(j + 1) * n2];
    u.x += xr; u.y += xi;
    v.x -= xr; v.y -= xi;
    py[(size_t)j * n2] = u;
    py[(size_t)(j + 1) * n2] = v;
  }
}

// y and z lines of an x-plane: a warp per row, its lanes two columns each; the
// rows' sums by shuffles, the columns' over the warps in order.
constexpr int kVjMaxN = 48;

template <class Z>
__global__ void __launch_bounds__(kVjThreads)
nyq_apply_yz_kernel(int n, int nneut, double cy, double cz, const double* __restrict__ field,
                    const double* __restrict__ scale, const Z* __restrict__ x, Z* __restrict__ y) {
  __shared__ double2 rows[kVjMaxN], cols[kVjMaxN];
  __shared__ double part[kVjWarps][3][kVjMaxN];
  const int sc = blockIdx.x / n, plane = blockIdx.x % n, s = sc / 2;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const size_t n2 = (size_t)n * n, n3 = n2 * n, off = (size_t)sc * n3 + plane * n2;
  const double* f = field + (s < nneut ? 0 : n3) + plane * n2;
  const double k = scale[s];
  const double sz = (lane & 1) ? -1.0 : 1.0;   // of both columns
  double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0}, cf[2] = {0.0, 0.0};
  for (int r = warp; r < n; r += kVjWarps) {
    const double sy = (r & 1) ? -1.0 : 1.0;
    double xr = 0.0, xi = 0.0, fm = 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int z = lane + 32 * h;
      if (z >= n) continue;
      const Z v = x[off + (size_t)r * n + z];
      const double b = f[(size_t)r * n + z], vr = (double)v.x, vi = (double)v.y;
      xr += vr; xi += vi; fm += b;
      cr[h] += sy * vr; ci[h] += sy * vi; cf[h] += b;
    }
    xr *= sz;
    xi *= sz;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      xr += __shfl_xor_sync(0xffffffffu, xr, o);
      xi += __shfl_xor_sync(0xffffffffu, xi, o);
      fm += __shfl_xor_sync(0xffffffffu, fm, o);
    }
    const double kr = k * cz * (fm / n);
    if (lane == 0) rows[r] = make_double2(kr * xr, kr * xi);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (lane + 32 * h < n) {
      part[warp][0][lane + 32 * h] = cr[h];
      part[warp][1][lane + 32 * h] = ci[h];
      part[warp][2][lane + 32 * h] = cf[h];
    }
  __syncthreads();
  if ((int)threadIdx.x < n) {
    double t[3] = {0.0, 0.0, 0.0};
    for (int w = 0; w < kVjWarps; ++w)
      for (int i = 0; i < 3; ++i) t[i] += part[w][i][threadIdx.x];
    const double kc = k * cy * (t[2] / n);
    cols[threadIdx.x] = make_double2(kc * t[0], kc * t[1]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n * n; e += kVjThreads) {
    const int r = e / n, z = e % n;
    const double2 a = cols[z], b = rows[r];
    const double ry = (r & 1) ? -1.0 : 1.0, rz = (z & 1) ? -1.0 : 1.0;
    Z v = y[off + e];
    v.x += ry * a.x + rz * b.x;
    v.y += ry * a.y + rz * b.y;
    y[off + e] = v;
  }
}

template <class Z>
int nyq_apply(hfb_ctx_s* c, int nst, int nneut, const double* field, const double* scale, const Z* x, Z* y,
              cudaStream_t st) {
  const int n = c->n;
  double k[3];
  for (int ax = 0; ax < 3; ++ax) k[ax] = -(M_PI / c->d[ax]) * (M_PI / c->d[ax]) / n;
  nyq_apply_x_kernel<Z><<<2u * nst * (n * n / 32), kVjThreads, 0, st>>>(n, nneut, k[0], field, scale, x, y);
  HFB_CHECK_LAUNCH();
  nyq_apply_yz_kernel<Z><<<2u * nst * n, kVjThreads, 0, st>>>(n, nneut, k[1], k[2], field, scale, x, y);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

}  // namespace
}  // namespace hfb

using namespace hfb;

extern "C" int hfb_nyquist_pair(hfb_ctx_t ctx, int prec, int nst, int nneut, const void* a, const void* b,
                                const double* w, double* field, void* stream) {
  if (!ctx || !a || !b || !w || !field || nst <= 0 || nneut < 0 || nneut > nst) return HFB_ERR_ARG;
  const int n = ctx->n;
  const size_t n2 = (size_t)n * n;
  double* t = (double*)scratch(ctx, hfb_ctx_s::S_VJP, sizeof(double) * 2 * 3 * n2 * (kVjGroups + 1));
  if (!t) return HFB_ERR_ALLOC;
  double* m = t + 2 * 3 * n2 * kVjGroups;
  cudaStream_t st = as_stream(stream);
  VjRuns r;
  for (int iq = 0; iq < 2; ++iq) {
    r.first[iq] = iq ? nneut : 0;
    r.end[iq] = iq ? nst : nneut;
    const int cnt = r.end[iq] - r.first[iq];
    r.run[iq] = (cnt + kVjGroups - 1) / kVjGroups;
    r.groups[iq] = cnt > 0 ? (cnt + r.run[iq] - 1) / r.run[iq] : 0;
  }
  const dim3 grid((n * n + kVjThreads - 1) / kVjThreads, 3, r.groups[0] + r.groups[1]);
  if (prec == HFB_F64)
    nyq_pair_lines_kernel<double2><<<grid, kVjThreads, 0, st>>>(n, r, (const double2*)a, (const double2*)b, w, t);
  else
    nyq_pair_lines_kernel<float2><<<grid, kVjThreads, 0, st>>>(n, r, (const float2*)a, (const float2*)b, w, t);
  HFB_CHECK_LAUNCH();
  nyq_pair_sum_kernel<<<dim3((3 * n * n + kVjThreads - 1) / kVjThreads, 2), kVjThreads, 0, st>>>(n * n, r, t, m);
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
  if (prec == HFB_F64)
    return nyq_apply(ctx, nst, nneut, field, scale, (const double2*)x, (double2*)y, as_stream(stream));
  return nyq_apply(ctx, nst, nneut, field, scale, (const float2*)x, (float2*)y, as_stream(stream));
}
