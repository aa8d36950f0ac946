// Damped-gradient step: grstep / grstep_helper / e0dmp_gt_zero of
// static.py:93-259, and the k-space preconditioner laplace of
// levels.py:398-437.
//
// The preconditioner is a 3-D FFT, a division by
//   (max(wg,.1) (E0 + h2ma k^2) + 0.5 max(wguv,.1) vmax) * Ntot
// and an inverse 3-D FFT.  It runs as three kernels over planes of one
// component of a state:
//   A (x-plane):  v = ps1 - lagrange (or - <h> psi), norms for efluct, z and y
//                 forward line FFTs;
//   B (y-plane):  x forward FFT, divide, x inverse FFT (stays in registers);
//   C (x-plane):  y and z inverse line FFTs, psi -= x0 * result.
// Bound by the latency of the lines' exchanges: what helps is more of them in
// flight.  So a plane is in shared memory only between its two line passes
// (z lines start or end in global memory, rows of it; y lines columns), its
// rows double as the lines' exchange buffers, and B needs no plane at all:
// 44 kB a CTA at 48^3 FP64 against 123 kB with both components staged on the
// way in and out (one CTA per SM).  Pb208 (236 states, 48^3), A + B + C: FP64
// 1.29 + 0.97 + 1.27 ms before, 0.70 + 0.63 + 0.57 ms here; FP32 0.46 + 0.32 + 0.49 ms
// before, 0.37 + 0.19 + 0.25 ms here (the bytes alone: 0.51 + 0.26 + 0.38 and
// half of that).
#include "hfb_ctx.cuh"
#include "hpsi.cuh"

namespace hfb {

template <class R, int N>
struct PlaneGeo {
  static constexpr int P = PencilSplit<R, N>::P;
  static constexpr int M = N / P;
  static constexpr int T = (M + P - 1) / P;
  static constexpr int THREADS = ((N * P + 31) / 32) * 32;
  static constexpr int LINES = THREADS / P;
  static constexpr int XB = Pencil<R, N, P>::XB;
  // Row pitch of the plane: a row holds a line's exchange buffer, and the
  // lanes that share a memory transaction (8 in FP64, 16 in FP32: consecutive
  // lines of P lanes) fall on distinct banks in column reads and, for P = 8 and
  // FP32, in the exchange.
  static constexpr int Q = sizeof(R) == 8 ? 8 : 16, WANT = P == 8 ? 1 : sizeof(R) == 8 && P == 4 ? 2 : 4;
  static constexpr int NEED = XB > N ? XB : N;
  static constexpr int LD = NEED + (Q + WANT - NEED % Q) % Q;
  // 36 warps an SM for A (56 registers): FP64 0.70 ms at 48^3 against 0.81 with
  // what the compiler takes, equal at 32^3, 15 % slower at 24^3; B and C equal
  static constexpr int A_CTAS = N >= 32 ? 1152 / THREADS : 1;
  static constexpr size_t SMEM = sizeof(cplx<R>) * (size_t)(LINES * LD + N);
  static constexpr size_t SMEM_B = sizeof(cplx<R>) * (size_t)(LINES * XB + N);
};

// A thread's line and place in it; threads past the last line (n = 8) work on
// line 0 in a buffer of their own and store nothing.
template <class R, int N>
struct LinePlace {
  int raw, p, line;
  bool active;
  __device__ __forceinline__ LinePlace() {
    raw = threadIdx.x / PlaneGeo<R, N>::P;
    p = threadIdx.x % PlaneGeo<R, N>::P;
    active = raw < N;
    line = active ? raw : 0;
  }
};

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

// A: x-plane of one component, build v and transform along z and y.
template <class R, int N>
__global__ void __launch_bounds__(PlaneGeo<R, N>::THREADS, PlaneGeo<R, N>::A_CTAS)
precond_a_kernel(const cplx<R>* src, const cplx<R>* __restrict__ lag, int use_lag, const cplx<R>* __restrict__ psi,
                 const double* __restrict__ coef, cplx<R>* tmp, double* fluct) {
  using G = PlaneGeo<R, N>;
  using PC = Pencil<R, N, G::P>;
  using Z = cplx<R>;
  constexpr int M = G::M, T = G::T, P = G::P, LD = G::LD;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[2][32];
  Z* plane = reinterpret_cast<Z*>(smem_raw);
  Z* tw = plane + G::LINES * LD;
  const int x0 = blockIdx.x % N, sc = blockIdx.x / N;   // sc = 2 state + component
  const LinePlace<R, N> l;
  const size_t off = (size_t)sc * N3 + (size_t)x0 * N2;
  const R cf = coef ? (R)coef[sc / 2] : R(0);
  const bool use_ps = psi && (!use_lag || fluct), use_lg = psi && lag && (use_lag || fluct);
  double n1 = 0, n2 = 0;
  Z v[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const size_t g = off + (size_t)l.line * N + l.p + P * m;
    v[m] = src[g];
    const Z lg = use_lg ? lag[g] : czero<Z>();
    const Z hp = use_ps ? cf * psi[g] : czero<Z>();
    if (psi) {
      v[m] = use_lag ? v[m] - lg : v[m] - hp;
      if (fluct && l.active) {
        const Z e2 = lg - hp;
        n1 += (double)v[m].x * v[m].x + (double)v[m].y * v[m].y;
        n2 += (double)e2.x * e2.x + (double)e2.y * e2.y;
      }
    }
  }
  fill_twiddles<R>(tw, N);
  __syncthreads();
  Z* row = plane + l.raw * LD;
  {
    Z f[T][P];
    PC::forward(v, f, row, tw, l.p, 0xffffffffu);
#pragma unroll
    for (int t = 0; t < T; ++t)
      if (PC::valid(l.p, t)) {
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) row[PC::freq(l.p, t, k1)] = f[t][k1];
      }
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = plane[(l.p + P * m) * LD + l.line];
  if (fluct) {
    block_sum2<R>(n1, n2, red);   // (its barrier also ends the column reads)
    if (threadIdx.x == 0) {
      double* o = fluct + (((size_t)(sc / 2) * 2 + sc % 2) * N + x0) * 2;
      o[0] = n1;
      o[1] = n2;
    }
  } else {
    __syncthreads();
  }
  Z f[T][P];
  PC::forward(v, f, row, tw, l.p, 0xffffffffu);
  if (!l.active) return;
#pragma unroll
  for (int t = 0; t < T; ++t)
    if (PC::valid(l.p, t)) {
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) tmp[off + (size_t)PC::freq(l.p, t, k1) * N + l.line] = f[t][k1];
    }
}

// B: y-plane (fixed ky) of one component, transform along x, divide, transform
// back; lines are independent.
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
  Z* xball = reinterpret_cast<Z*>(smem_raw);
  Z* tw = xball + G::LINES * G::XB;
  const int y0 = blockIdx.x % N, sc = blockIdx.x / N, s = sc / 2;
  const int iq = s >= nneut ? 1 : 0;
  const LinePlace<R, N> l;  // line = kz
  Z* io = tmp + (size_t)sc * N3 + (size_t)y0 * N + l.line;
  Z v[M];
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = io[(size_t)(l.p + P * m) * N2];
  fill_twiddles<R>(tw, N);
  __syncthreads();
  Z* xb = xball + l.raw * G::XB;
  const double wgm = fmax(wg ? wg[s] : 1.0, 0.1);
  const double wum = fmax(wu ? wu[s] : 0.0, 0.1);
  const double vm = vmax_dev ? vmax_dev[iq] : vmax_host;
  const int kyi = signed_k(y0, N), kzi = signed_k(l.line, N);
  const double kyz2 = (kyi * kfy) * (kyi * kfy) + (kzi * kfz) * (kzi * kfz);
  const double shift = wgm * e0 + 0.5 * wum * vm;
  Z f[T][P];
  PC::forward(v, f, xb, tw, l.p, 0xffffffffu);
#pragma unroll
  for (int t = 0; t < T; ++t) {
    if (!PC::valid(l.p, t)) continue;
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      int kxi = signed_k(PC::freq(l.p, t, k1), N);
      double k2 = (kxi * kfx) * (kxi * kfx) + kyz2;
      double den = (shift + wgm * h2ma * k2) * (double)N3;
      f[t][k1] = (R)(1.0 / den) * f[t][k1];
    }
  }
  PC::inverse(f, v, xb, tw, l.p, 0xffffffffu);
  if (!l.active) return;
#pragma unroll
  for (int m = 0; m < M; ++m) io[(size_t)(l.p + P * m) * N2] = v[m];
}

// C: x-plane of one component, inverse along y and z, then write or update.
template <class R, int N>
__global__ void __launch_bounds__(PlaneGeo<R, N>::THREADS)
precond_c_kernel(const cplx<R>* tmp, int mode, double x0, const double* x0_dev, cplx<R>* dst) {
  using G = PlaneGeo<R, N>;
  using PC = Pencil<R, N, G::P>;
  using Z = cplx<R>;
  constexpr int M = G::M, T = G::T, P = G::P, LD = G::LD;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z* plane = reinterpret_cast<Z*>(smem_raw);
  Z* tw = plane + G::LINES * LD;
  const int xp = blockIdx.x % N, sc = blockIdx.x / N;
  const LinePlace<R, N> l;
  const size_t off = (size_t)sc * N3 + (size_t)xp * N2;
  Z f[T][P], v[M];
#pragma unroll
  for (int t = 0; t < T; ++t)
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1)
      f[t][k1] = PC::valid(l.p, t) ? tmp[off + (size_t)PC::freq(l.p, t, k1) * N + l.line] : czero<Z>();
  fill_twiddles<R>(tw, N);
  __syncthreads();
  Z* row = plane + l.raw * LD;
  PC::inverse(f, v, row, tw, l.p, 0xffffffffu);
  __syncthreads();
  if (l.active) {
#pragma unroll
    for (int m = 0; m < M; ++m) plane[(l.p + P * m) * LD + l.line] = v[m];
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < T; ++t)
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) f[t][k1] = PC::valid(l.p, t) ? row[PC::freq(l.p, t, k1)] : czero<Z>();
  __syncwarp();
  PC::inverse(f, v, row, tw, l.p, 0xffffffffu);
  if (!l.active) return;
  const R xr = (R)(x0_dev ? *x0_dev : x0);
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const size_t g = off + (size_t)l.line * N + l.p + P * m;
    if (mode == 0) dst[g] = v[m];
    else dst[g] = dst[g] - xr * v[m];
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
  const unsigned grid = 2u * ns * N;
  precond_a_kernel<R, N><<<grid, G::THREADS, G::SMEM, st>>>((const Z*)src, (const Z*)lag, use_lag, (const Z*)psi,
                                                            coef, (Z*)tmp, fluct);
  HFB_CHECK_LAUNCH();
  const double kf[3] = {2.0 * kPi / (c->d[0] * N), 2.0 * kPi / (c->d[1] * N), 2.0 * kPi / (c->d[2] * N)};
  precond_b_kernel<R, N><<<grid, G::THREADS, G::SMEM_B, st>>>((Z*)tmp, nneut, wg, wu, vmax_dev, vmax_host, e0, h2ma,
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
// latencies; 20 us here for 236 states of 96 planes).
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
  if (!hpsi_aligned(ctx, prec, a->psi, a->hampsi) || !hpsi_aligned(ctx, prec, a->psi, a->hmfpsi)) return HFB_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  const int ns = a->nst, n = ctx->n;
  if (ns <= 0) return HFB_OK;
  const size_t n3 = (size_t)n * n * n;
  const int nov = hpsi_ovl_parts(ctx, prec);
  double* part = (double*)scratch(ctx, hfb_ctx_s::S_PART, sizeof(double) * (size_t)ns * (nov + 2 * n) * 2);
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
  grstep_finish_kernel<<<1, 1024, 0, st>>>(ns, a->do_fluct && a->e0dmp > 0.0, 2 * n, (const double2*)fl, a->wxyz, spe_new, a->wocc,
                                          a->wstates, a->sp_energy, a->sp_efluct1, a->sp_efluct2, a->sums);
  HFB_CHECK_LAUNCH();
  // 3) h psi_new into hmfpsi (and v_pair psi_new into delpsi when requested)
  return hpsi_launch(ctx, prec, a->pot, 0, ns, a->nneut, a->psi, wt, wu, a->hmfpsi, nullptr, a->hmfpsi, a->delpsi,
                     nullptr, st);
}
