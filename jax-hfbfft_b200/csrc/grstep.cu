// Damped-gradient step: grstep / grstep_helper / e0dmp_gt_zero of
// static.py:93-259, and the k-space preconditioner laplace of
// levels.py:398-437.
//
// The preconditioner is a 3-D FFT, a division by
//   (max(wg,.1) (E0 + h2ma k^2) + 0.5 max(wguv,.1) vmax) * Ntot
// and an inverse 3-D FFT.  It runs as three plane kernels:
//   A (x-plane):  v = ps1 - lagrange (or - <h> psi), norms for efluct, z and y
//                 forward line FFTs;
//   B (y-plane):  x forward FFT, divide, x inverse FFT (stays in registers);
//   C (x-plane):  y and z inverse line FFTs, psi -= x0 * result.
#include "hfb_ctx.cuh"
#include "hpsi.cuh"

namespace hfb {

template <class R, int N>
struct PlaneGeo {
  static constexpr int P = PencilSplit<R, N>::P;
  static constexpr int M = N / P;
  static constexpr int T = (M + P - 1) / P;
  static constexpr int LD = N + 4;
  static constexpr int NB = Pencil<R, N, P>::XB;
  static constexpr int THREADS = ((N * P + 31) / 32) * 32;
  static constexpr int LINES = THREADS / P;
  static constexpr size_t SMEM = sizeof(cplx<R>) * (size_t)(2 * N * LD + LINES * NB + N);
};

// Forward (DIR = -1) or inverse (+1) transform of every line of one staged
// component ``pl`` ([N][LD]); data stays in natural order in the plane.
template <class R, int N, bool ROW, int DIR>
__device__ __forceinline__ void plane_lines(cplx<R>* pl, cplx<R>* xb, const cplx<R>* tw, int line, int p,
                                            bool active) {
  using G = PlaneGeo<R, N>;
  using PC = Pencil<R, N, G::P>;
  using Z = cplx<R>;
  constexpr int M = G::M, T = G::T, P = G::P;
  auto at = [&](int j) -> Z& { return ROW ? pl[line * G::LD + j] : pl[j * G::LD + line]; };
  Z v[M];
  Z f[T][P];
  if (DIR < 0) {
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = at(p + P * m);
    PC::forward(v, f, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (PC::valid(p, t)) {
#pragma unroll
          for (int k1 = 0; k1 < P; ++k1) at(PC::freq(p, t, k1)) = f[t][k1];
        }
    }
  } else {
#pragma unroll
    for (int t = 0; t < T; ++t) {
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) f[t][k1] = PC::valid(p, t) ? at(PC::freq(p, t, k1)) : czero<Z>();
    }
    PC::inverse(f, v, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int m = 0; m < M; ++m) at(p + P * m) = v[m];
    }
  }
}

template <class R>
__device__ __forceinline__ void block_sum2(double& a, double& b, double (*red)[32]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0) { red[0][w] = a; red[1][w] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0, y = 0;
    for (int i = 0; i < (int)(blockDim.x / 32); ++i) { x += red[0][i]; y += red[1][i]; }
    a = x;
    b = y;
  }
}

// A: x-plane, build v and transform along z and y.
template <class R, int N>
__global__ void __launch_bounds__(PlaneGeo<R, N>::THREADS)
precond_a_kernel(const cplx<R>* __restrict__ src, const cplx<R>* __restrict__ lag, int use_lag,
                 const cplx<R>* __restrict__ psi, const double* __restrict__ coef, cplx<R>* tmp, double* fluct) {
  using G = PlaneGeo<R, N>;
  using Z = cplx<R>;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[2][32];
  Z* plane = reinterpret_cast<Z*>(smem_raw);
  Z* xball = plane + 2 * N * G::LD;
  Z* tw = xball + G::LINES * G::NB;
  const int x0 = blockIdx.x, s = blockIdx.y;
  fill_twiddles<R>(tw, N);
  const size_t off = (size_t)s * 2 * N3 + (size_t)x0 * N2;
  const R cf = coef ? (R)coef[s] : R(0);
  double n1 = 0, n2 = 0;
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    size_t g = off + (size_t)c * N3 + r;
    Z v = src[g];
    if (psi) {
      Z ps = psi[g];
      Z lg = lag ? lag[g] : czero<Z>();
      Z hp = cf * ps;
      v = use_lag ? v - lg : v - hp;
      if (fluct) {
        Z e2 = lg - hp;
        n1 += (double)v.x * v.x + (double)v.y * v.y;
        n2 += (double)e2.x * e2.x + (double)e2.y * e2.y;
      }
    }
    plane[(c * N + r / N) * G::LD + r % N] = v;
  }
  if (fluct) {
    block_sum2<R>(n1, n2, red);
    if (threadIdx.x == 0) {
      fluct[((size_t)s * N + x0) * 2 + 0] = n1;
      fluct[((size_t)s * N + x0) * 2 + 1] = n2;
    }
  }
  __syncthreads();
  const int line_raw = threadIdx.x / G::P, p = threadIdx.x % G::P;
  const bool active = line_raw < N;
  const int line = active ? line_raw : 0;
  Z* xb = xball + line_raw * G::NB;
  for (int c = 0; c < 2; ++c) plane_lines<R, N, true, -1>(plane + c * N * G::LD, xb, tw, line, p, active);
  __syncthreads();
  for (int c = 0; c < 2; ++c) plane_lines<R, N, false, -1>(plane + c * N * G::LD, xb, tw, line, p, active);
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    tmp[off + (size_t)c * N3 + r] = plane[(c * N + r / N) * G::LD + r % N];
  }
}

// B: y-plane (fixed ky), transform along x, divide, transform back.
template <class R, int N>
__global__ void __launch_bounds__(PlaneGeo<R, N>::THREADS)
precond_b_kernel(cplx<R>* tmp, int nneut, const double* __restrict__ wg, const double* __restrict__ wu,
                 const double* __restrict__ vmax_dev, double vmax_host, double e0, double h2ma, double kfx, double kfy,
                 double kfz) {
  using G = PlaneGeo<R, N>;
  using PC = Pencil<R, N, G::P>;
  using Z = cplx<R>;
  constexpr int M = G::M, T = G::T, P = G::P;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z* plane = reinterpret_cast<Z*>(smem_raw);
  Z* xball = plane + 2 * N * G::LD;
  Z* tw = xball + G::LINES * G::NB;
  const int y0 = blockIdx.x, s = blockIdx.y;
  const int iq = s >= nneut ? 1 : 0;
  fill_twiddles<R>(tw, N);
  const size_t off = (size_t)s * 2 * N3 + (size_t)y0 * N;
  // compile-time trip count, unrolled: several loads in flight per thread
#pragma unroll 8
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    int a = r / N, b = r % N;
    plane[(c * N + a) * G::LD + b] = tmp[off + (size_t)c * N3 + (size_t)a * N2 + b];
  }
  __syncthreads();
  const int line_raw = threadIdx.x / P, p = threadIdx.x % P;
  const bool active = line_raw < N;
  const int line = active ? line_raw : 0;  // line = kz
  Z* xb = xball + line_raw * G::NB;
  const double wgm = fmax(wg ? wg[s] : 1.0, 0.1);
  const double wum = fmax(wu ? wu[s] : 0.0, 0.1);
  const double vm = vmax_dev ? vmax_dev[iq] : vmax_host;
  const int kyi = signed_k(y0, N), kzi = signed_k(line, N);
  const double kyz2 = (kyi * kfy) * (kyi * kfy) + (kzi * kfz) * (kzi * kfz);
  const double shift = wgm * e0 + 0.5 * wum * vm;
  for (int c = 0; c < 2; ++c) {
    Z* pl = plane + c * N * G::LD;
    Z v[M];
    Z f[T][P];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = pl[(p + P * m) * G::LD + line];
    PC::forward(v, f, xb, tw, p, 0xffffffffu);
#pragma unroll
    for (int t = 0; t < T; ++t) {
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        int kxi = signed_k(PC::freq(p, t, k1), N);
        double k2 = (kxi * kfx) * (kxi * kfx) + kyz2;
        double den = (shift + wgm * h2ma * k2) * (double)N3;
        f[t][k1] = (R)(1.0 / den) * f[t][k1];
      }
    }
    PC::inverse(f, v, xb, tw, p, 0xffffffffu);
    if (active) {
#pragma unroll
      for (int m = 0; m < M; ++m) pl[(p + P * m) * G::LD + line] = v[m];
    }
  }
  __syncthreads();
  // compile-time trip count, unrolled: several loads in flight per thread
#pragma unroll 8
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    int a = r / N, b = r % N;
    tmp[off + (size_t)c * N3 + (size_t)a * N2 + b] = plane[(c * N + a) * G::LD + b];
  }
}

// C: x-plane, inverse along y and z, then write or update.
template <class R, int N>
__global__ void __launch_bounds__(PlaneGeo<R, N>::THREADS)
precond_c_kernel(const cplx<R>* tmp, int mode, double x0, const double* x0_dev, cplx<R>* dst) {
  using G = PlaneGeo<R, N>;
  using Z = cplx<R>;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z* plane = reinterpret_cast<Z*>(smem_raw);
  Z* xball = plane + 2 * N * G::LD;
  Z* tw = xball + G::LINES * G::NB;
  const int xp = blockIdx.x, s = blockIdx.y;
  fill_twiddles<R>(tw, N);
  const size_t off = (size_t)s * 2 * N3 + (size_t)xp * N2;
  // compile-time trip count, unrolled: several loads in flight per thread
#pragma unroll 8
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    plane[(c * N + r / N) * G::LD + r % N] = tmp[off + (size_t)c * N3 + r];
  }
  __syncthreads();
  const int line_raw = threadIdx.x / G::P, p = threadIdx.x % G::P;
  const bool active = line_raw < N;
  const int line = active ? line_raw : 0;
  Z* xb = xball + line_raw * G::NB;
  for (int c = 0; c < 2; ++c) plane_lines<R, N, false, +1>(plane + c * N * G::LD, xb, tw, line, p, active);
  __syncthreads();
  for (int c = 0; c < 2; ++c) plane_lines<R, N, true, +1>(plane + c * N * G::LD, xb, tw, line, p, active);
  __syncthreads();
  const R xr = (R)(x0_dev ? *x0_dev : x0);
  // compile-time trip count, unrolled: several loads in flight per thread
#pragma unroll 8
  for (int e = threadIdx.x; e < 2 * N * N; e += G::THREADS) {
    int c = e / (N * N), r = e - c * N * N;
    size_t g = off + (size_t)c * N3 + r;
    Z v = plane[(c * N + r / N) * G::LD + r % N];
    if (mode == 0) dst[g] = v;
    else dst[g] = dst[g] - xr * v;
  }
}

template <class R, int N>
int precond_launch_t(hfb_ctx_s* c, int ns, int nneut, const void* src, const void* lag, int use_lag, const void* psi,
                     const double* coef, const double* wg, const double* wu, const double* vmax_dev, double vmax_host,
                     double e0, double h2ma, int mode, double x0, void* tmp, void* dst, double* fluct,
                     cudaStream_t st, const double* x0_dev) {
  using G = PlaneGeo<R, N>;
  using Z = cplx<R>;
  if (ns <= 0) return HFB_OK;
  allow_max_dynamic_smem(precond_a_kernel<R, N>);
  allow_max_dynamic_smem(precond_b_kernel<R, N>);
  allow_max_dynamic_smem(precond_c_kernel<R, N>);
  dim3 grid(N, ns);
  precond_a_kernel<R, N><<<grid, G::THREADS, G::SMEM, st>>>((const Z*)src, (const Z*)lag, use_lag, (const Z*)psi,
                                                            coef, (Z*)tmp, fluct);
  HFB_CHECK_LAUNCH();
  const double kf[3] = {2.0 * kPi / (c->d[0] * N), 2.0 * kPi / (c->d[1] * N), 2.0 * kPi / (c->d[2] * N)};
  precond_b_kernel<R, N><<<grid, G::THREADS, G::SMEM, st>>>((Z*)tmp, nneut, wg, wu, vmax_dev, vmax_host, e0, h2ma,
                                                            kf[0], kf[1], kf[2]);
  HFB_CHECK_LAUNCH();
  precond_c_kernel<R, N><<<grid, G::THREADS, G::SMEM, st>>>((const Z*)tmp, mode, x0, x0_dev, (Z*)dst);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

int precond_launch(hfb_ctx_s* c, int prec, int ns, int nneut, const void* src, const void* lag, int use_lag,
                   const void* psi, const double* coef, const double* wg, const double* wu, const double* vmax_dev,
                   double vmax_host, double e0, double h2ma, int mode, double x0, void* tmp, void* dst,
                   double* fluct, cudaStream_t st, const double* x0_dev) {
  return dispatch_n(c->n, [&](auto nn) -> int {
    constexpr int N = decltype(nn)::value;
    if (prec == HFB_F64)
      return precond_launch_t<double, N>(c, ns, nneut, src, lag, use_lag, psi, coef, wg, wu, vmax_dev, vmax_host, e0,
                                         h2ma, mode, x0, tmp, dst, fluct, st, x0_dev);
    return precond_launch_t<float, N>(c, ns, nneut, src, lag, use_lag, psi, coef, wg, wu, vmax_dev, vmax_host, e0,
                                      h2ma, mode, x0, tmp, dst, fluct, st, x0_dev);
  });
}

// ------------------------------------------------------ gradient-step glue --
// Per-state weights (static.py:152-170, 125-136) -- hpsi weights and the
// preconditioner weights -- and max(v_pair[iq]) over the grid, in one launch.
// The maximum reads 2 n^3 doubles: kVmaxBlocks blocks per isospin leave each
// block a few kB (one block per isospin took 116 us at 40^3, bound by one
// SM's loads in flight; 3 us here).  The last block to finish combines the
// blocks' maxima and returns the counter to zero for the next launch.
constexpr int kVmaxBlocks = 64;

__global__ void __launch_bounds__(256)
grstep_weights_kernel(int ns, int tbcs, const double* wocc, const double* wguv, const double* pairwg,
                      const double* wstates, double* wt, double* wu, double* lw, double* lu, const double* v_pair,
                      size_t n3, double* vpart, int* counter, double* vmax) {
  const int blk = blockIdx.x + gridDim.x * blockIdx.y;
  for (int s = blk * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * gridDim.y * blockDim.x) {
    if (tbcs) {
      wt[s] = 1.0; wu[s] = 0.0; lw[s] = 1.0; lu[s] = 0.0;
    } else {
      wt[s] = wstates[s] * wocc[s];
      wu[s] = wstates[s] * wguv[s] * pairwg[s];
      lw[s] = wocc[s];
      lu[s] = wguv[s] * pairwg[s];
    }
  }
  if (!v_pair) {
    if (blk == 0 && threadIdx.x < 2) vmax[threadIdx.x] = 0.0;
    return;
  }
  __shared__ double red[8];
  __shared__ int last;
  const double* v = v_pair + blockIdx.y * n3;
  double m = -1.0e300;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n3; i += (size_t)gridDim.x * blockDim.x)
    m = fmax(m, v[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) m = fmax(m, red[i]);
    vpart[blk] = m;
    __threadfence();
    last = atomicAdd(counter, 1) == (int)(gridDim.x * gridDim.y) - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 64) {
    const int iq = threadIdx.x / 32;
    double r = -1.0e300;
    for (int i = threadIdx.x % 32; i < (int)gridDim.x; i += 32) r = fmax(r, __ldcg(vpart + iq * gridDim.x + i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (threadIdx.x % 32 == 0) vmax[iq] = r;
  }
  if (threadIdx.x == 0) *counter = 0;
}

// Per-state sums of the overlap partials, spe[s] and hexp[s] = scale *
// sum_j part[s][j][0 / 1]: one warp per state, both sums from one read of
// the pairs (fixed order).
__global__ void __launch_bounds__(128)
state_reduce_kernel(int ns, int nparts, const double2* __restrict__ part, double scale, double* spe, double* hexp) {
  const int s = blockIdx.x * 4 + threadIdx.x / 32, lane = threadIdx.x % 32;
  if (s >= ns) return;
  double a = 0.0, b = 0.0;
  for (int j = lane; j < nparts; j += 32) {
    const double2 v = part[(size_t)s * nparts + j];
    a += v.x;
    b += v.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    spe[s] = scale * a;
    hexp[s] = scale * b;
  }
}

// Simple damped step when e0dmp <= 0 (static.py:181-185).
template <class R>
__global__ void simple_step_kernel(int ns, size_t n3, const double* spe_new, const double* spe_old, double x0h,
                                   const double* x0_dev, const cplx<R>* ps1, cplx<R>* psi) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t tot = (size_t)ns * 2 * n3;
  if (i >= tot) return;
  const double x0 = x0_dev ? *x0_dev : x0h;
  int s = (int)(i / (2 * n3));
  R a = (R)(1.0 + x0 * (spe_new[s] - spe_old[s]));
  psi[i] = a * psi[i] - (R)x0 * ps1[i];
}

// Finalise efluct, denerg and the running sums (static.py:110-111, 211, 251-257).
// One block: a warp per state for the plane partials, then one warp's
// fixed-order sums over the states (a thread per state and one thread's
// sums took 61 us for 236 states of 48 planes, a serial chain of L2
// latencies; 6 us here).
__global__ void __launch_bounds__(1024)
grstep_finish_kernel(int ns, int do_fluct, int nplanes, const double2* __restrict__ fl, double wxyz,
                     const double* spe_new, const double* wocc, const double* wstates, double* sp_energy, double* ef1,
                     double* ef2, double* sums) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (do_fluct)
    for (int s = warp; s < ns; s += 32) {
      double a = 0.0, b = 0.0;
      for (int j = lane; j < nplanes; j += 32) {
        const double2 v = fl[(size_t)s * nplanes + j];
        a += v.x;
        b += v.y;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
      if (lane == 0) {
        ef1[s] = sqrt(wxyz * a);
        ef2[s] = sqrt(wxyz * b);
      }
    }
  __syncthreads();
  if (warp != 0) return;
  double sf = 0.0, sd = 0.0;
  for (int s = lane; s < ns; s += 32) {
    const double e = spe_new[s];
    sf += ef1[s];
    sd += wocc[s] * wstates[s] * ((sp_energy[s] - e) / fabs(e));
    sp_energy[s] = e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sf += __shfl_xor_sync(0xffffffffu, sf, o);
    sd += __shfl_xor_sync(0xffffffffu, sd, o);
  }
  if (lane == 0) {
    sums[0] = sf;
    sums[1] = sd;
  }
}

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_laplace(hfb_ctx_t ctx, int prec, int nsp, const void* psin, const double* wg, const double* wguv,
                           double v_pairmax, double e0inv, double h2ma, void* psout, void* stream) {
  if (!ctx || !psin || !psout || nsp < 0) return HFB_ERR_ARG;
  return precond_launch(ctx, prec, nsp, 1 << 30, psin, nullptr, 0, nullptr, nullptr, wg, wguv, nullptr, v_pairmax,
                        e0inv, h2ma, 0, 0.0, psout, psout, nullptr, as_stream(stream));
}

extern "C" int hfb_grstep(hfb_ctx_t ctx, int prec, const hfb_grstep_args* a, void* stream) {
  if (!ctx || !a || !a->psi || !a->hampsi || !a->hmfpsi || !a->pot || !a->sp_energy) return HFB_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  const int ns = a->nst, n = ctx->n;
  if (ns <= 0) return HFB_OK;
  const size_t n3 = (size_t)n * n * n;
  const int nov = hpsi_ovl_parts(ctx, prec);
  double* part = (double*)scratch(ctx, hfb_ctx_s::S_PART, sizeof(double) * (size_t)ns * (nov + n) * 2);
  double* vec = (double*)scratch(ctx, hfb_ctx_s::S_SMALL, sizeof(double) * ((size_t)ns * 6 + 8 + 2 * kVmaxBlocks));
  if (!part || !vec) return HFB_ERR_ALLOC;
  double* ovl = part;
  double* fl = part + (size_t)ns * nov * 2;
  double *wt = vec, *wu = vec + ns, *lw = vec + 2 * ns, *lu = vec + 3 * ns, *spe_new = vec + 4 * ns,
         *hexp = vec + 5 * ns, *vmax = vec + 6 * ns;
  double* vpart = vmax + 8;
  const double* vp = a->tbcs ? nullptr : a->v_pair;
  grstep_weights_kernel<<<vp ? dim3(kVmaxBlocks, 2) : dim3((ns + 255) / 256, 1), 256, 0, st>>>(
      ns, a->tbcs, a->wocc, a->wguv, a->pairwg, a->wstates, wt, wu, lw, lu, vp, n3, vpart, ctx->counters, vmax);
  HFB_CHECK_LAUNCH();
  // 1) h psi_old: ps1 (weighted) into hmfpsi (scratch), h psi into hampsi
  int r = hpsi_launch(ctx, prec, a->pot, 0, ns, a->nneut, a->psi, wt, wu, a->hampsi, a->hmfpsi, a->hampsi, nullptr,
                      ovl, st);
  if (r) return r;
  state_reduce_kernel<<<(ns + 3) / 4, 128, 0, st>>>(ns, nov, (const double2*)ovl, a->wxyz, spe_new, hexp);
  HFB_CHECK_LAUNCH();
  // 2) damped step
  if (a->e0dmp > 0.0) {
    r = precond_launch(ctx, prec, ns, a->nneut, a->hmfpsi, a->lagrange, a->use_lagrange, a->psi, hexp, lw, lu, vmax,
                       0.0, a->e0dmp, a->h2ma, 1, a->x0dmp, a->hmfpsi, a->psi, a->do_fluct ? fl : nullptr, st,
                       a->x0dmp_dev);
    if (r) return r;
  } else {
    size_t tot = (size_t)ns * 2 * n3;
    if (prec == HFB_F64)
      simple_step_kernel<double><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(
          ns, n3, spe_new, a->sp_energy, a->x0dmp, a->x0dmp_dev, (const double2*)a->hmfpsi, (double2*)a->psi);
    else
      simple_step_kernel<float><<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(
          ns, n3, spe_new, a->sp_energy, a->x0dmp, a->x0dmp_dev, (const float2*)a->hmfpsi, (float2*)a->psi);
    HFB_CHECK_LAUNCH();
  }
  grstep_finish_kernel<<<1, 1024, 0, st>>>(ns, a->do_fluct && a->e0dmp > 0.0, n, (const double2*)fl, a->wxyz, spe_new, a->wocc,
                                          a->wstates, a->sp_energy, a->sp_efluct1, a->sp_efluct2, a->sums);
  HFB_CHECK_LAUNCH();
  // 3) h psi_new into hmfpsi (and v_pair psi_new into delpsi when requested)
  return hpsi_launch(ctx, prec, a->pot, 0, ns, a->nneut, a->psi, wt, wu, a->hmfpsi, nullptr, a->hmfpsi, a->delpsi,
                     nullptr, st);
}
