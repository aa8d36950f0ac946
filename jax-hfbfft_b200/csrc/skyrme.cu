// Mean fields from densities (skyrme, meanfield.py:164-391) and the Coulomb
// potential by FFT on the doubled grid (coulomb.py:14-75).  All FP64.
//
// Derivatives of densities use the dense spectral matrices der1/der2 along
// each axis exactly as the reference's einsums do (an O(n^4) matrix apply;
// small next to the per-state work).
#include <mutex>
#include "diag.cuh"
#include "fields.cuh"

namespace hfb {

// out = sum over the axes of coef * D along the axis applied to in (null: no
// term), so divergences, curls and Laplacians are single jobs and one launch
// runs many jobs without write conflicts.
struct DerivJob {
  const double* in[3];
  double coef[3];
  int der;      // 1 or 2
  double* out;
};
constexpr int kMaxJobs = 24;
struct DerivJobs {
  DerivJob j[kMaxJobs];
};
// Derivative matrices of the x axis; those of another axis are the same times
// scale[der - 1][axis], (dx / d_axis)^der.
struct DerivMats {
  const double* d[2];
  double scale[2][3];
};

// A block takes one plane of one job.  Pass 0: the y-plane, whose x and z
// lines are products of the n x n plane with the derivative matrix from the
// left and from the right; pass 1: the x-plane with its y lines, added to
// pass 0 (fixed order).  Both products run on the FP64 tensor cores, one warp
// per 8 rows; operands staged in shared memory with rows of n + 4 doubles
// (fragment loads then fall on distinct banks).  What bounds it is the latency
// of the staging (54 kB a block at 48^3, three blocks an SM) and the products
// after it.  One pass per term
// on CUDA cores, bound by shared-memory loads, took 130 us for the fields of
// skyrme at 48^3; the two passes take 41 us.
template <int N> struct DerivGeo {
  static constexpr int LD = N + 4, THREADS = 4 * N;
  static constexpr size_t SMEM = sizeof(double) * 3 * N * LD;   // D and the two planes
};

template <int N, bool Y>
__global__ void __launch_bounds__(DerivGeo<N>::THREADS) deriv_pass_kernel(DerivJobs jobs, DerivMats mats) {
  using G = DerivGeo<N>;
  constexpr int LD = G::LD, NB = N / 8;
  constexpr size_t N2 = (size_t)N * N;
  extern __shared__ __align__(16) double deriv_smem[];
  const DerivJob& jb = jobs.j[blockIdx.y];
  const int plane = blockIdx.x;
  // term 0: from the left (x or y lines), term 1: from the right (z lines)
  const double* in[2] = {jb.in[Y ? 1 : 0], Y ? nullptr : jb.in[2]};
  const double* sc = mats.scale[jb.der - 1];
  const double coef[2] = {jb.coef[Y ? 1 : 0] * sc[Y ? 1 : 0], jb.coef[2] * sc[2]};
  double* D = deriv_smem;
  if (!in[0] && !in[1]) return;
  const size_t base = Y ? plane * N2 : (size_t)plane * N, pitch = Y ? N : N2;
  auto cp = [&](double* dst, const double* src, size_t sp) {
    for (int e = threadIdx.x; e < N * N / 2; e += G::THREADS) {
      const int r = e / (N / 2), q = 2 * (e % (N / 2));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * LD + q)),
                   "l"(src + r * sp + q)
                   : "memory");
    }
  };
  // (the fields come from the caller: a base that is only 8-byte aligned is copied by element)
  auto cp8 = [&](double* dst, const double* src, size_t sp) {
    for (int e = threadIdx.x; e < N * N; e += G::THREADS) dst[(e / N) * LD + e % N] = src[(e / N) * sp + e % N];
  };
  cp(D, mats.d[jb.der - 1], N);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (!in[t]) continue;
    const double* src = in[t] + base;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) cp(D + (1 + t) * N * LD, src, pitch);
    else cp8(D + (1 + t) * N * LD, src, pitch);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, fr = lane >> 2, fk = lane & 3;
  double out[NB][2];
#pragma unroll
  for (int v = 0; v < NB; ++v) out[v][0] = out[v][1] = 0.0;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (!in[t]) continue;
    const double* F = D + (1 + t) * N * LD;
    const double* A = (t == 0 ? D : F) + (8 * warp + fr) * LD + fk;
    double acc[NB][2];
#pragma unroll
    for (int v = 0; v < NB; ++v) acc[v][0] = acc[v][1] = 0.0;
#pragma unroll 4
    for (int k = 0; k < N; k += 4) {
      const double a = A[k];
#pragma unroll
      for (int v = 0; v < NB; ++v)
        gd_mma(acc[v], a, t == 0 ? F[(k + fk) * LD + 8 * v + fr] : D[(8 * v + fr) * LD + k + fk]);
    }
#pragma unroll
    for (int v = 0; v < NB; ++v)
#pragma unroll
      for (int c = 0; c < 2; ++c) out[v][c] += coef[t] * acc[v][c];
  }
  const bool add = Y && (jb.in[0] || jb.in[2]);
  double2* o = reinterpret_cast<double2*>(jb.out + base + (8 * warp + fr) * pitch + 2 * fk);   // library scratch
#pragma unroll
  for (int v = 0; v < NB; ++v) {
    const double2 was = add ? o[4 * v] : make_double2(0.0, 0.0);
    o[4 * v] = make_double2(was.x + out[v][0], was.y + out[v][1]);
  }
}

static int run_jobs(hfb_ctx_s* c, const DerivJobs& jobs, int nj, cudaStream_t st) {
  if (nj <= 0) return HFB_OK;
  DerivMats m;
  m.d[0] = c->der1[0];
  m.d[1] = c->der2[0];
  for (int ax = 0; ax < 3; ++ax) {
    const double r = c->d[0] / c->d[ax];
    m.scale[0][ax] = r;
    m.scale[1][ax] = r * r;
  }
  return dispatch_n(c->n, [&](auto nn) -> int {
    constexpr int N = decltype(nn)::value;
    using G = DerivGeo<N>;
    allow_max_dynamic_smem(deriv_pass_kernel<N, false>);
    allow_max_dynamic_smem(deriv_pass_kernel<N, true>);
    deriv_pass_kernel<N, false><<<dim3(N, nj), G::THREADS, G::SMEM, st>>>(jobs, m);
    HFB_CHECK_LAUNCH();
    deriv_pass_kernel<N, true><<<dim3(N, nj), G::THREADS, G::SMEM / 3 * 2, st>>>(jobs, m);
    HFB_CHECK_LAUNCH();
    return HFB_OK;
  });
}

static DerivJob job1(const double* in, int axis, double* out) {
  DerivJob j{};
  j.in[axis] = in; j.coef[axis] = 1.0; j.der = 1; j.out = out;
  return j;
}
static DerivJob jobdiv(const double* v /*[3][n3]*/, size_t n3, double* out) {
  DerivJob j{};
  for (int a = 0; a < 3; ++a) { j.in[a] = v + a * n3; j.coef[a] = 1.0; }
  j.der = 1; j.out = out;
  return j;
}
static DerivJob joblap(const double* f, double* out) {
  DerivJob j{};
  for (int a = 0; a < 3; ++a) { j.in[a] = f; j.coef[a] = 1.0; }
  j.der = 2; j.out = out;
  return j;
}
// component k of curl v: d_a v_b - d_b v_a with (a, b) = (y, z), (z, x), (x, y)
static DerivJob jobcurl(const double* v /*[3][n3]*/, size_t n3, int k, double* out) {
  const int a = (k + 1) % 3, b = (k + 2) % 3;
  DerivJob j{};
  j.in[a] = v + (size_t)b * n3; j.coef[a] = 1.0;
  j.in[b] = v + (size_t)a * n3; j.coef[b] = -1.0;
  j.der = 1; j.out = out;
  return j;
}

int density_derivatives(hfb_ctx_s* c, const double* rho, const double* cur, const double* sd, const double* so,
                        bool mean_field, double** dv_out, cudaStream_t st) {
  const size_t n3 = (size_t)c->n * c->n * c->n;
  double* dv = (double*)scratch(c, hfb_ctx_s::S_DERIV, sizeof(double) * (size_t)2 * kNDeriv * n3);
  if (!dv) return HFB_ERR_ALLOC;
  *dv_out = dv;
  DerivJobs jobs;
  int nj = 0;
  for (int iq = 0; iq < 2; ++iq) {
    double* o = dv + (size_t)iq * kNDeriv * n3;
    const double *r = rho + (size_t)iq * n3, *j3 = cur + (size_t)iq * 3 * n3;
    jobs.j[nj++] = jobdiv(so + (size_t)iq * 3 * n3, n3, o);
    jobs.j[nj++] = joblap(r, o + n3);
    for (int k = 0; k < 3; ++k) {
      if (mean_field) {
        jobs.j[nj++] = job1(r, k, o + (2 + k) * n3);
        jobs.j[nj++] = jobcurl(sd + (size_t)iq * 3 * n3, n3, k, o + (5 + k) * n3);
      }
      jobs.j[nj++] = jobcurl(j3, n3, k, o + (8 + k) * n3);
    }
    if (mean_field) jobs.j[nj++] = jobdiv(j3, n3, o + 11 * n3);
  }
  return run_jobs(c, jobs, nj, st);
}

// ------------------------------------------------------ doubled-grid FFT --
// The Green's function at context creation: in-place forward line FFTs along
// one axis of a complex n2^3 array, lines ordered with the contiguous
// transverse index fastest.
template <int N2, int AXIS>
__global__ void __launch_bounds__(128) coul_fft_kernel(double2* a) {
  constexpr int P = PencilSplit<double, N2>::P;
  constexpr int M = N2 / P, T = (M + P - 1) / P, L = 128 / P, NB = Pencil<double, N2, P>::XB;
  using PC = Pencil<double, N2, P>;
  __shared__ __align__(16) double2 xball[L * NB];
  __shared__ double2 tw[N2];
  fill_twiddles<double>(tw, N2);
  __syncthreads();
  const int lg = threadIdx.x / P, p = threadIdx.x % P;
  const int line_raw = blockIdx.x * L + lg;
  const bool active = line_raw < N2 * N2;
  const int line = active ? line_raw : 0;
  const int u = line / N2, v = line % N2;
  constexpr size_t S2 = (size_t)N2 * N2;
  size_t base, stride;
  if (AXIS == 2) { base = (size_t)u * S2 + (size_t)v * N2; stride = 1; }
  else if (AXIS == 1) { base = (size_t)u * S2 + v; stride = N2; }
  else { base = (size_t)u * N2 + v; stride = S2; }
  double2 vv[M];
  double2 f[T][P];
#pragma unroll
  for (int m = 0; m < M; ++m) vv[m] = a[base + (size_t)(p + P * m) * stride];
  PC::forward(vv, f, xball + lg * NB, tw, p, 0xffffffffu);
  if (!active) return;
#pragma unroll
  for (int t = 0; t < T; ++t)
    if (PC::valid(p, t)) {
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) a[base + (size_t)PC::freq(p, t, k1) * stride] = f[t][k1];
    }
}

template <int N2, int AXIS>
static int coul_pass(double2* a) {
  constexpr int L = 128 / PencilSplit<double, N2>::P;
  coul_fft_kernel<N2, AXIS><<<(unsigned)((N2 * N2 + L - 1) / L), 128>>>(a);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

template <class F>
static int dispatch_n2(int n2, F&& fn) {
  switch (n2) {
    case 8: return fn(std::integral_constant<int, 8>{});
    case 16: return fn(std::integral_constant<int, 16>{});
    case 24: return fn(std::integral_constant<int, 24>{});
    case 32: return fn(std::integral_constant<int, 32>{});
    case 40: return fn(std::integral_constant<int, 40>{});
    case 48: return fn(std::integral_constant<int, 48>{});
    case 64: return fn(std::integral_constant<int, 64>{});
    case 80: return fn(std::integral_constant<int, 80>{});
    case 96: return fn(std::integral_constant<int, 96>{});
    default: return HFB_ERR_UNSUPPORTED_GRID;
  }
}

// q(r) on the doubled grid (coulomb.py:31-47): 1/|r| with wrapped indices,
// the r = 0 cell 2.84 / dV^(1/3); periodic: 1/k^2 with q(0) = 0.
__global__ void coul_green_kernel(double2* q, int n2, double dx, double dy, double dz, int periodic) {
  const size_t tot = (size_t)n2 * n2 * n2;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= tot) return;
  int ix = (int)(i / ((size_t)n2 * n2)), iy = (int)((i / n2) % n2), iz = (int)(i % n2);
  ix = ix <= n2 / 2 ? ix : ix - n2;
  iy = iy <= n2 / 2 ? iy : iy - n2;
  iz = iz <= n2 / 2 ? iz : iz - n2;
  double v;
  if (periodic) {
    const double kx = 2.0 * kPi * ix / (n2 * dx), ky = 2.0 * kPi * iy / (n2 * dy), kz = 2.0 * kPi * iz / (n2 * dz);
    const double s = kx * kx + ky * ky + kz * kz;
    v = (i == 0) ? 0.0 : 1.0 / s;
  } else {
    const double s = (dx * ix) * (dx * ix) + (dy * iy) * (dy * iy) + (dz * iz) * (dz * iz);
    v = (i == 0) ? 2.84 / cbrt(dx * dy * dz) : 1.0 / sqrt(s);
  }
  q[i] = make_double2(v, 0.0);
}

int coulomb_init(hfb_ctx_s* c) {
  const size_t tot = (size_t)c->n2 * c->n2 * c->n2;
  coul_green_kernel<<<(unsigned)((tot + 255) / 256), 256>>>(c->coul_q, c->n2, c->d[0], c->d[1], c->d[2], c->periodic);
  HFB_CHECK_LAUNCH();
  if (c->periodic) return HFB_OK;
  return dispatch_n2(c->n2, [&](auto nn) -> int {
    constexpr int N2 = decltype(nn)::value;
    int r = coul_pass<N2, 2>(c->coul_q);
    if (r == HFB_OK) r = coul_pass<N2, 1>(c->coul_q);
    if (r == HFB_OK) r = coul_pass<N2, 0>(c->coul_q);
    return r;
  });
}

// The doubled-grid solve in three launches.  The density is real, so only
// kz = 0 .. n2 / 2 is kept, and it fills n of n2 points per axis, so only the
// lines that can differ from zero (forward) or are wanted (inverse) are
// transformed:
//   1. per x < n:  z lines (y < n) of the density, then y lines, in shared
//                  memory;
//   2. per (ky, kz): x line, times the Green's function, back to x < n;
//   3. per x < n:  y lines back to y < n, then z lines, in shared memory.
// The work array is [x < n][ky][kz].  (As nine launches over all of the n2^3
// complex array: 90 us at n2 = 96, 45 us here.)
template <int N2> struct CoulGeo {
  static constexpr int P = PencilSplit<double, N2>::P, M = N2 / P, T = (M + P - 1) / P;
  static constexpr int THREADS = 256, L = THREADS / P, NB = Pencil<double, N2, P>::XB;
  static constexpr int NZ = N2 / 2 + 1;
  static constexpr size_t SMEM = sizeof(double2) * ((size_t)N2 * NZ + L * NB + N2);
};

template <int N2>
__global__ void __launch_bounds__(CoulGeo<N2>::THREADS) coul_zy_kernel(const double* __restrict__ rho, double2* a, int n) {
  using G = CoulGeo<N2>;
  constexpr int P = G::P, M = G::M, T = G::T, L = G::L, NZ = G::NZ;
  using PC = Pencil<double, N2, P>;
  extern __shared__ __align__(16) double2 coul_smem[];
  double2* S = coul_smem;                 // [N2 y / ky][NZ kz]
  double2* xball = S + (size_t)N2 * NZ;
  double2* tw = xball + L * G::NB;
  fill_twiddles<double>(tw, N2);
  __syncthreads();
  const int lg = threadIdx.x / P, p = threadIdx.x % P, x = blockIdx.x;
  double2* xb = xball + lg * G::NB;
  double2 vv[M];
  double2 f[T][P];
  for (int l0 = 0; l0 < n; l0 += L) {
    const int y = l0 + lg;
    const bool active = y < n;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int z = p + P * m;
      vv[m] = make_double2(active && z < n ? rho[((size_t)x * n + y) * n + z] : 0.0, 0.0);
    }
    PC::forward(vv, f, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (PC::valid(p, t)) {
#pragma unroll
          for (int k1 = 0; k1 < P; ++k1) {
            const int k = PC::freq(p, t, k1);
            if (k < NZ) S[y * NZ + k] = f[t][k1];
          }
        }
    }
  }
  __syncthreads();
  for (int l0 = 0; l0 < NZ; l0 += L) {
    const int kz = l0 + lg;
    const bool active = kz < NZ;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int y = p + P * m;
      vv[m] = active && y < n ? S[y * NZ + kz] : make_double2(0.0, 0.0);
    }
    PC::forward(vv, f, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (PC::valid(p, t)) {
#pragma unroll
          for (int k1 = 0; k1 < P; ++k1) S[PC::freq(p, t, k1) * NZ + kz] = f[t][k1];
        }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < N2 * NZ; e += G::THREADS) a[(size_t)x * N2 * NZ + e] = S[e];
}

// coulomb.py:68-71: periodic 4 pi e2 Re(q); else e2 wxyz q
template <int N2>
__global__ void __launch_bounds__(128) coul_x_kernel(double2* a, const double2* __restrict__ q, int n, double fac,
                                                     int periodic) {
  using G = CoulGeo<N2>;
  constexpr int P = G::P, M = G::M, T = G::T, L = 128 / P, NZ = G::NZ;
  using PC = Pencil<double, N2, P>;
  __shared__ __align__(16) double2 xball[L * G::NB];
  __shared__ double2 tw[N2];
  fill_twiddles<double>(tw, N2);
  __syncthreads();
  const int lg = threadIdx.x / P, p = threadIdx.x % P;
  double2* xb = xball + lg * G::NB;
  const int line_raw = blockIdx.x * L + lg;
  const bool active = line_raw < N2 * NZ;
  const int line = active ? line_raw : 0;
  const int ky = line / NZ, kz = line % NZ;
  double2 vv[M];
  double2 f[T][P], g[T][P];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int x = p + P * m;
    vv[m] = x < n ? a[(size_t)x * N2 * NZ + line] : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int t = 0; t < T; ++t)
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1)
      if (PC::valid(p, t)) g[t][k1] = q[((size_t)PC::freq(p, t, k1) * N2 + ky) * N2 + kz];
  PC::forward(vv, f, xb, tw, p, 0xffffffffu);
#pragma unroll
  for (int t = 0; t < T; ++t)
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1)
      if (PC::valid(p, t)) {
        const double2 v = f[t][k1], w = make_double2(fac * g[t][k1].x, periodic ? 0.0 : fac * g[t][k1].y);
        f[t][k1] = cmul(w, v);
      }
  PC::inverse(f, vv, xb, tw, p, 0xffffffffu);
  if (!active) return;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int x = p + P * m;
    if (x < n) a[(size_t)x * N2 * NZ + line] = vv[m];
  }
}

template <int N2>
__global__ void __launch_bounds__(CoulGeo<N2>::THREADS) coul_yz_kernel(const double2* __restrict__ a, double* w, int n,
                                                                       double scale) {
  using G = CoulGeo<N2>;
  constexpr int P = G::P, M = G::M, T = G::T, L = G::L, NZ = G::NZ;
  using PC = Pencil<double, N2, P>;
  extern __shared__ __align__(16) double2 coul_smem[];
  double2* S = coul_smem;                 // [N2 ky / y][NZ kz]
  double2* xball = S + (size_t)N2 * NZ;
  double2* tw = xball + L * G::NB;
  const int lg = threadIdx.x / P, p = threadIdx.x % P, x = blockIdx.x;
  fill_twiddles<double>(tw, N2);
  for (int e = threadIdx.x; e < N2 * NZ; e += G::THREADS) S[e] = a[(size_t)x * N2 * NZ + e];
  __syncthreads();
  double2* xb = xball + lg * G::NB;
  double2 vv[M];
  double2 f[T][P];
  for (int l0 = 0; l0 < NZ; l0 += L) {
    const int kz = l0 + lg;
    const bool active = kz < NZ;
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1)
        f[t][k1] = active && PC::valid(p, t) ? S[PC::freq(p, t, k1) * NZ + kz] : make_double2(0.0, 0.0);
    PC::inverse(f, vv, xb, tw, p, 0xffffffffu);
    __syncwarp();
    if (active) {
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (p + P * m < n) S[(p + P * m) * NZ + kz] = vv[m];
    }
  }
  __syncthreads();
  for (int l0 = 0; l0 < n; l0 += L) {
    const int y = l0 + lg;
    const bool active = y < n;
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        f[t][k1] = make_double2(0.0, 0.0);
        if (active && PC::valid(p, t)) {   // real result: the bins above n2 / 2 are conjugates
          const int k = PC::freq(p, t, k1);
          const double2 v = S[y * NZ + (k < NZ ? k : N2 - k)];
          f[t][k1] = make_double2(v.x, k < NZ ? v.y : -v.y);
        }
      }
    PC::inverse(f, vv, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (p + P * m < n) w[((size_t)x * n + y) * n + p + P * m] = scale * vv[m].x;
    }
  }
}

// Elements of the work array, n n2 (n2 / 2 + 1) < n2^3; every one is written
// before it is read, so it may hold anything on entry.
static size_t poisson_work(const hfb_ctx_s* c) { return (size_t)c->n * c->n2 * (c->n2 / 2 + 1); }

static int poisson_solve(const hfb_ctx_s* c, const double* rho_p, double* wcoul, double2* a, cudaStream_t st) {
  const double e2 = 1.4399784085965135;
  const double fac = c->periodic ? 4.0 * kPi * e2 : e2 * c->wxyz;
  return dispatch_n2(c->n2, [&](auto nn) -> int {
    constexpr int N2 = decltype(nn)::value;
    using G = CoulGeo<N2>;
    allow_max_dynamic_smem(coul_zy_kernel<N2>);
    allow_max_dynamic_smem(coul_yz_kernel<N2>);
    coul_zy_kernel<N2><<<c->n, G::THREADS, G::SMEM, st>>>(rho_p, a, c->n);
    HFB_CHECK_LAUNCH();
    constexpr int L = 128 / G::P;
    coul_x_kernel<N2><<<(N2 * G::NZ + L - 1) / L, 128, 0, st>>>(a, c->coul_q, c->n, fac, c->periodic);
    HFB_CHECK_LAUNCH();
    coul_yz_kernel<N2><<<c->n, G::THREADS, G::SMEM, st>>>(a, wcoul, c->n, 1.0 / ((double)N2 * N2 * N2));
    HFB_CHECK_LAUNCH();
    return HFB_OK;
  });
}

int poisson_launch(hfb_ctx_s* c, const double* rho_p, double* wcoul, cudaStream_t st) {
  double2* a = (double2*)scratch(c, hfb_ctx_s::S_POIS, poisson_work(c) * sizeof(double2));
  if (!a) return HFB_ERR_ALLOC;
  return poisson_solve(c, rho_p, wcoul, a, st);
}

// ----------------------------------------------------- potential assembly --
// Steps 1-13 of skyrme (meanfield.py:176-385) at one grid point, the packed
// hpsi potentials pot[iq][field] in precision R (upot, bmass, v_pair, aq,
// spot, wlspot) included.  div aq and grad bmass (steps 11-12) are the same
// linear combinations of div j and grad rho that aq and bmass are of j and
// rho: the derivative matrices of different axes commute, so div curl s = 0,
// and D applied to the constant h2m is 0.
template <class R>
__global__ void skyrme_assemble_kernel(hfb_force f, int tcoul, size_t n3, const double* rho, const double* tau,
                                       const double* chi, const double* cur, const double* dv, const double* wcoul,
                                       double* upot, double* bmass, double* divaq, double* v_pair, double* aq,
                                       double* spot, double* wlspot, double* dbmass, R* pot, double* rearr_out,
                                       double* ecorrp) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n3) return;
  const double r0 = rho[i], r1 = rho[n3 + i];
  const double rt = r0 + r1;
  const double rtp = pow(rt, f.power);
  const double* d0 = dv;
  const double* d1 = dv + (size_t)kNDeriv * n3;
  double rearr = 0.0;
  if (f.ipair == 6)
    rearr = (f.v0neut / f.rho0pr) * chi[i] * chi[i] + (f.v0prot / f.rho0pr) * chi[n3 + i] * chi[n3 + i];
  for (int iq = 0; iq < 2; ++iq) {
    const int ic = 1 - iq;
    const double* dq = iq == 0 ? d0 : d1;
    const double* dc = iq == 0 ? d1 : d0;
    const double rq = rho[iq * n3 + i], rc = rho[ic * n3 + i];
    double u = rtp * ((f.b3 * (f.power + 2.0) / 3.0 - 2.0 * f.b3p / 3.0) * rq + f.b3 * (f.power + 2.0) / 3.0 * rc -
                      (f.b3p * f.power / 3.0) * (r0 * r0 + r1 * r1) / (rt + 1.0e-25));
    u += -(f.b4 + f.b4p) * dq[i] - f.b4 * dc[i];
    if (tcoul && iq == 1) {
      u += wcoul[i];
      if (f.ex != 0) u += -f.slate * cbrt(r1);
    }
    u += (f.b0 - f.b0p) * rq + f.b0 * rc + (f.b1 - f.b1p) * tau[iq * n3 + i] + f.b1 * tau[ic * n3 + i] -
         (f.b2 - f.b2p) * dq[n3 + i] - f.b2 * dc[n3 + i];
    u += rearr;
    const double bm = f.h2m[iq] + (f.b1 - f.b1p) * rq + f.b1 * rc;
    const double v0 = iq == 1 ? f.v0prot : f.v0neut;
    const double vpr = f.ipair == 6 ? v0 * chi[iq * n3 + i] * (1.0 - rt / f.rho0pr) : v0 * chi[iq * n3 + i];
    upot[iq * n3 + i] = u;
    bmass[iq * n3 + i] = bm;
    v_pair[iq * n3 + i] = vpr;
    divaq[iq * n3 + i] = -2.0 * (f.b1 - f.b1p) * dq[11 * n3 + i] - 2.0 * f.b1 * dc[11 * n3 + i];
    R* po = pot ? pot + (size_t)iq * 12 * n3 + i : nullptr;
    if (pot) {
      po[0] = (R)u;
      po[n3] = (R)bm;
      po[2 * n3] = (R)vpr;
    }
    for (int k = 0; k < 3; ++k) {
      const size_t o = ((size_t)iq * 3 + k) * n3 + i;
      const double gq = dq[(2 + k) * n3 + i], gc = dc[(2 + k) * n3 + i];
      const double wl = (f.b4 + f.b4p) * gq + f.b4 * gc;
      const double a = -2.0 * (f.b1 - f.b1p) * cur[((size_t)iq * 3 + k) * n3 + i] -
                       2.0 * f.b1 * cur[((size_t)ic * 3 + k) * n3 + i] - (f.b4 + f.b4p) * dq[(5 + k) * n3 + i] -
                       f.b4 * dc[(5 + k) * n3 + i];
      const double sp = -(f.b4 + f.b4p) * dq[(8 + k) * n3 + i] - f.b4 * dc[(8 + k) * n3 + i];
      wlspot[o] = wl;
      aq[o] = a;
      spot[o] = sp;
      dbmass[o] = (f.b1 - f.b1p) * gq + f.b1 * gc;
      if (pot) {
        po[(3 + k) * n3] = (R)a;
        po[(6 + k) * n3] = (R)sp;
        po[(9 + k) * n3] = (R)wl;
      }
    }
  }
  if (f.ipair == 6) rearr_out[i] = rt * rearr;
  else if (i == 0) *ecorrp = 0.0;
}

// ecorrp = -sum(rho_tot * rearr) * wxyz / 2 (meanfield.py:364) with
// density-dependent pairing, one block.
__global__ void ecorrp_kernel(size_t n3, const double* t, double wxyz, double* out) {
  __shared__ double red[32];
  double s = 0.0;
  for (size_t i = threadIdx.x; i < n3; i += blockDim.x) s += t[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int k = 0; k < (int)(blockDim.x / 32); ++k) a += red[k];
    out[0] = -a * wxyz / 2.0;
  }
}

// pot[iq][field][i] from the field arrays (null: zero).
struct PackIn {
  const double* f[6];   // upot, bmass, v_pair, aq, spot, wlspot
};
template <class R>
__global__ void pack_pot_kernel(size_t n3, PackIn in, R* pot) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n3) return;
  const int k = blockIdx.y % 12, iq = blockIdx.y / 12;
  const int a = k < 3 ? k : 3 + (k - 3) / 3;
  const size_t row = k < 3 ? iq : iq * 3 + (k - 3) % 3;
  pot[blockIdx.y * n3 + i] = in.f[a] ? (R)in.f[a][row * n3 + i] : R(0);
}

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_pack_pot(hfb_ctx_t ctx, int prec, const double* upot, const double* bmass, const double* v_pair,
                            const double* aq, const double* spot, const double* wlspot, void* pot, void* stream) {
  if (!ctx || !pot) return HFB_ERR_ARG;
  const size_t n3 = (size_t)ctx->n * ctx->n * ctx->n;
  const dim3 grid((unsigned)((n3 + 255) / 256), 24);
  const PackIn in{{upot, bmass, v_pair, aq, spot, wlspot}};
  if (prec == HFB_F64) pack_pot_kernel<double><<<grid, 256, 0, as_stream(stream)>>>(n3, in, (double*)pot);
  else pack_pot_kernel<float><<<grid, 256, 0, as_stream(stream)>>>(n3, in, (float*)pot);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

extern "C" int hfb_poisson(hfb_ctx_t ctx, const double* rho_p, double* wcoul, void* stream) {
  if (!ctx || !rho_p || !wcoul) return HFB_ERR_ARG;
  return poisson_launch(ctx, rho_p, wcoul, as_stream(stream));
}

extern "C" int hfb_skyrme(hfb_ctx_t ctx, const hfb_force* f, int tcoul, const double* rho, const double* tau,
                          const double* chi, const double* current, const double* sdens, const double* sodens,
                          double* upot, double* bmass, double* divaq, double* v_pair, double* aq, double* spot,
                          double* wlspot, double* dbmass, double* wcoul, double* ecorrp, int prec, void* pot,
                          void* stream) {
  if (!ctx || !f || !rho || !tau || !chi || !current || !sdens || !sodens || !upot || !bmass || !divaq || !v_pair ||
      !aq || !spot || !wlspot || !dbmass || !ecorrp)
    return HFB_ERR_ARG;
  if (tcoul && !wcoul) return HFB_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  const size_t n3 = (size_t)ctx->n * ctx->n * ctx->n;
  double* dv = nullptr;
  // the Coulomb solve needs rho_p only: on the side stream, beside the
  // derivatives of the densities
  const bool fork = tcoul && ctx->side;
  int r;
  if (fork) {
    cudaEventRecord(ctx->ev_fork, st);
    cudaStreamWaitEvent(ctx->side, ctx->ev_fork, 0);
    r = poisson_launch(ctx, rho + n3, wcoul, ctx->side);
    if (r) return r;
    cudaEventRecord(ctx->ev_join, ctx->side);
  }
  r = density_derivatives(ctx, rho, current, sdens, sodens, true, &dv, st);
  if (r) return r;
  if (fork) {
    cudaStreamWaitEvent(st, ctx->ev_join, 0);
  } else if (tcoul) {
    r = poisson_launch(ctx, rho + n3, wcoul, st);
    if (r) return r;
  }
  double* tmp = (double*)scratch(ctx, hfb_ctx_s::S_MAT, sizeof(double) * n3);
  if (!tmp) return HFB_ERR_ALLOC;
  const unsigned nblk = (unsigned)((n3 + 127) / 128);
  if (prec == HFB_F64)
    skyrme_assemble_kernel<double><<<nblk, 128, 0, st>>>(*f, tcoul, n3, rho, tau, chi, current, dv, wcoul, upot, bmass,
                                                         divaq, v_pair, aq, spot, wlspot, dbmass, (double*)pot, tmp,
                                                         ecorrp);
  else
    skyrme_assemble_kernel<float><<<nblk, 128, 0, st>>>(*f, tcoul, n3, rho, tau, chi, current, dv, wcoul, upot, bmass,
                                                        divaq, v_pair, aq, spot, wlspot, dbmass, (float*)pot, tmp,
                                                        ecorrp);
  HFB_CHECK_LAUNCH();
  if (f->ipair == 6) {
    ecorrp_kernel<<<1, 1024, 0, st>>>(n3, tmp, ctx->wxyz, ecorrp);
    HFB_CHECK_LAUNCH();
  }
  return HFB_OK;
}

// --------------------------------------------- Poisson without allocation --
// A second entry point for the Coulomb solve, for callers that cannot let
// the library allocate device memory when they call it: applications whose
// device memory is entirely owned by their own pool allocator (a cudaMalloc
// behind its back can fail or fragment the pool), and latency-critical loops
// where an allocation, with the synchronisation it implies, would stall.
// Its work buffer is a fixed array in the library's device image instead of
// the context's growable scratch arena.
namespace hfb {

// Its size is that of the work array (poisson_work) of the largest Coulomb grid
// served, n2 = 64 (2n non-periodic: n <= 32; every periodic grid a context
// accepts, n2 = n <= 48, fits): 32 x 64 x 33 complex doubles, 1 MiB.  The larger
// non-periodic grids (3.4 MiB at n = 48) are left to hfb_poisson: every GPU that
// loads the library holds the array until the process exits.
constexpr int kNoAllocN2 = 64;
constexpr size_t kNoAllocWork = (size_t)(kNoAllocN2 / 2) * kNoAllocN2 * (kNoAllocN2 / 2 + 1);
static_assert(kNoAllocWork >= (size_t)48 * 48 * (48 / 2 + 1), "the periodic grids");
static __device__ __align__(256) double2 g_poisson_noalloc[kNoAllocWork];

// Device address of g_poisson_noalloc per device ordinal, looked up on the
// first call made on that device (the array's host-side name is only a
// stand-in and must never be passed to a kernel).
static std::mutex g_noalloc_mu;
static void* g_noalloc_addr[64] = {nullptr};

static int noalloc_buffer(int dev, double2** out) {
  if (dev < 0 || dev >= 64) return HFB_ERR_CUDA;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_poisson_noalloc) != cudaSuccess || !p) {
      cudaGetLastError();
      return HFB_ERR_CUDA;
    }
    g_noalloc_addr[dev] = p;
  }
  *out = (double2*)g_noalloc_addr[dev];
  return HFB_OK;
}

}  // namespace hfb

extern "C" int hfb_poisson_noalloc(hfb_ctx_t ctx, const double* rho_p, double* wcoul, void* stream) {
  using namespace hfb;
  if (!ctx || !rho_p || !wcoul) return HFB_ERR_ARG;
  if (ctx->n2 > kNoAllocN2) return HFB_ERR_UNSUPPORTED_GRID;   // the work array is not sized for this grid
  // the buffer is looked up on the current device; the context's Green's
  // function lives on the device it was created on: they must be the same
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return HFB_ERR_CUDA;
  }
  if (dev != ctx->device) return HFB_ERR_ARG;
  double2* a = nullptr;
  const int r = noalloc_buffer(dev, &a);
  if (r) return r;
  // the solve writes every element before it reads it, so nothing left by an
  // earlier call leaks into this one
  return poisson_solve(ctx, rho_p, wcoul, a, as_stream(stream));
}
