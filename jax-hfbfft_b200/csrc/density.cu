// Occupation-weighted densities (add_density, densities.py:177-330), the
// single-particle kinetic energy of sp_properties (inout.py:64-150) and the
// pair densities of two sets of states.
//
// Every density term is local or bilinear in psi and ONE first derivative
// d_d psi (cderv d00).  A work unit is one state on a tile of lines along one
// axis d: the lines are transformed, d_d psi formed and the terms added to
// FP64 accumulators in registers (no atomics).  P lanes own a line of one
// spinor component and P neighbouring lanes the same line of the other one,
// so a lane accumulates the terms that start from its own derivative and
// takes the partner component's value by one shuffle; sums and differences
// over the two components are taken once, when a tile is written.  The local
// densities ride on axes x and y, so that no axis has more than five
// accumulators per point.
//
// Units are numbered axis, isospin, tile, state; a CTA (128 threads) takes
// an equal run of consecutive units whatever the state counts, and writes
// one partial tile per (axis, isospin, tile) it meets.  Partial tile (CTA k,
// tile t) lies at k + t: along the units k or t or both step on, so no two
// share a place, and the buffer holds one tile per CTA and one per tile,
// whatever the state counts.  A combine kernel adds
// the partials in order and applies the density mixing of
// static.py:1820-1823.  (With both components and up to nine accumulators per
// point in a thread, one CTA per SM, equal chunks of unequal isospins in three
// launches and bank conflicts in the transforms' exchange: 670 us for 90 + 60
// single-precision states at 40^3, 2.32 ms for 236 double-precision ones at
// 48^3; 480 us and 1.72 ms here.  Both components in a thread on this scheme:
// 550 us, the registers leave half the warps.)  What bounds it is issue: the
// transforms, and FP64 accumulation with its conversions.
//
// Kinetic energy: with the unnormalised FFT and Parseval,
//   sum_k k_d^2 |psi_k|^2 / Ntot = sum_r |D_d psi|^2
//                                 + (pi/h_d)^2 / n * sum_lines |psi_hat_d(n/2)|^2
// where D_d is the Nyquist-zeroed derivative and psi_hat_d(n/2) the 1-D FFT
// of the line at the Nyquist bin; sp_kinetic = wxyz h2m_q sum_d (...).
#include "hfb_ctx.cuh"

namespace hfb {

namespace {

template <class R, int N>
struct DensGeo {
  static constexpr int P = (N >= 32) ? 8 : (N >= 16 ? 4 : 2);
  static constexpr int M = N / P;
  static constexpr int T = (M + P - 1) / P;
  static constexpr int THREADS = 128;
  static constexpr int L = THREADS / (2 * P);   // lines per tile
  static constexpr int NB = Pencil<R, N, P>::XB;
  static constexpr int NTILE = N * N / L;
  static constexpr int WARPS = THREADS / 32;
  static_assert(N * N % L == 0, "whole tiles");
};

// Fields of a partial tile.  Axis x: tau, current, J parts (two), rho, chi,
// s_z; axis y: tau, current, J parts (two), s_x, s_y; axis z: tau, current,
// J parts (two).
constexpr int kDensFields = 7;
constexpr int kDensPerSm = 4;   // CTAs of an SM that write partial tiles, at most

// How the units are cut up, and where a partial tile lies.
struct DensCut {
  int nq;                   // isospin blocks that have states
  int iq[2], s0[2], cnt[2]; // isospin, first state, states of each
  int ntile, nst;
  long units, run;          // all units; units per CTA
};
// number of (axis, block, tile) among all tiles
__host__ __device__ __forceinline__ long dens_tile(const DensCut& c, int axis, int q, int tile) {
  return ((long)axis * c.nq + q) * c.ntile + tile;
}
// and its first unit
__host__ __device__ __forceinline__ long dens_first(const DensCut& c, int axis, int q, int tile) {
  return (long)axis * c.ntile * c.nst + (q ? (long)c.ntile * c.cnt[0] : 0) + (long)tile * c.cnt[q];
}
__device__ __forceinline__ void dens_decode(const DensCut& c, long u, int& axis, int& q, int& tile, int& s) {
  const long per = (long)c.ntile * c.nst;
  axis = (int)(u / per);
  long r = u - axis * per;
  q = c.nq > 1 && r >= (long)c.ntile * c.cnt[0];
  if (q) r -= (long)c.ntile * c.cnt[0];
  tile = (int)(r / c.cnt[q]);
  s = (int)(r - (long)tile * c.cnt[q]);
}

enum { DENS_KINETIC = 0, DENS_FIELDS = 1, DENS_PAIR = 2 };   // kinetic energies only; densities; pair densities

struct DensArgs {
  const void *psi, *psi2;   // psi2: the second set of a pair density
  const double *wocc, *wguv, *pairwg, *wstates;
  double ks[3], nf[3];
  double* part;
  double* kin;              // [state][axis][tile][warp], or null
  DensCut cut;
};

// States sa..sb of one block on one tile of one axis.
template <class R, int N, int AXIS, int KIND>
__device__ __forceinline__ void dens_segment(const DensArgs& a, int tile, int sa, int sb, double* out,
                                             cplx<R>* xb, const cplx<R>* tw, const R* sk) {
  using G = DensGeo<R, N>;
  using PC = Pencil<R, N, G::P>;
  using Z = cplx<R>;
  constexpr int P = G::P, M = G::M, T = G::T;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  constexpr bool PAIR = KIND == DENS_PAIR, FIELDS = KIND != DENS_KINETIC;
  constexpr int NA = !FIELDS ? 1 : AXIS == 0 ? 5 : 4;
  const int lg = threadIdx.x / (2 * P), c = (threadIdx.x / P) & 1, p = threadIdx.x % P;
  const int line = tile * G::L + lg, u = line / N, v = line % N;
  // line -> transverse coordinates with the contiguous one fastest
  size_t base, stride;
  if (AXIS == 2) { base = (size_t)u * N2 + (size_t)v * N; stride = 1; }        // (x, y) fixed
  else if (AXIS == 1) { base = (size_t)u * N2 + v; stride = N; }               // (x, z) fixed
  else { base = (size_t)u * N + v; stride = N2; }                             // (y, z) fixed
  base += c * N3 + p * stride;
  double acc[NA][M];
#pragma unroll
  for (int f = 0; f < NA; ++f)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[f][m] = 0.0;
  const Z* src = (const Z*)a.psi + base + (size_t)sa * 2 * N3;
  const Z* src2 = (const Z*)a.psi2 + base + (size_t)sa * 2 * N3;
  // the line values of the next state are loaded while this one is
  // transformed and accumulated (not for pairs: the registers are needed)
  Z xn[M];
  if (!PAIR) {
#pragma unroll
    for (int m = 0; m < M; ++m) xn[m] = src[m * (P * stride)];
  }
  // wave numbers of this lane's frequencies
  const R* skl = sk + AXIS * N + p;
  // D_d of a line (cderv d00: k = 0 and Nyquist zeroed)
  auto diff = [&](const Z (&x)[M], Z (&d)[M], double& nyq) {
    Z vv[M];
    Z f[T][P];
#pragma unroll
    for (int m = 0; m < M; ++m) vv[m] = x[m];
    PC::forward(vv, f, xb, tw, p, 0xffffffffu);
    nyq = p == 0 ? (double)f[0][P / 2].x * f[0][P / 2].x + (double)f[0][P / 2].y * f[0][P / 2].y : 0.0;
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        const R sc = PC::valid(p, t) ? skl[P * t + M * k1] : R(0);
        const Z z = f[t][k1];
        f[t][k1] = mk<R>(-sc * z.y, sc * z.x);
      }
    PC::inverse(f, d, xb, tw, p, 0xffffffffu);
  };
  auto partner = [&](Z x) {
    Z y;
    y.x = __shfl_xor_sync(0xffffffffu, x.x, P);
    y.y = __shfl_xor_sync(0xffffffffu, x.y, P);
    return y;
  };
  for (int s = sa; s < sb; ++s) {
    double w = 0.0, wu = 0.0;
    if (FIELDS) {
      const double ws = PAIR ? 1.0 : a.wstates[s];
      w = a.wocc[s] * ws;
      if (AXIS == 0) wu = PAIR ? a.wguv[s] : a.wguv[s] * a.pairwg[s] * ws;
    }
    Z x[M], d[M];
    double nyq;
    if (PAIR) {
      Z y[M], e[M];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        x[m] = src[m * (P * stride)];
        y[m] = src2[m * (P * stride)];
      }
      src += 2 * N3;
      src2 += 2 * N3;
      diff(x, d, nyq);
      diff(y, e, nyq);
      const double h = 0.5 * w;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const Z px = partner(x[m]), py = partner(y[m]);
        const double xr = x[m].x, xi = x[m].y, yr = y[m].x, yi = y[m].y;
        const double dr = d[m].x, di = d[m].y, er = e[m].x, ei = e[m].y;
        const double pr = px.x, pi = px.y, qr = py.x, qi = py.y;
        acc[0][m] += w * (dr * er + di * ei);
        acc[1][m] += h * (di * yr - dr * yi + ei * xr - er * xi);
        if (AXIS != 1) acc[2][m] += h * (dr * qr + di * qi + er * pr + ei * pi);
        if (AXIS != 0) acc[AXIS == 2 ? 3 : 2][m] += h * (di * qr - dr * qi + ei * pr - er * pi);
        if (AXIS == 0) {
          const double xy = xr * yr + xi * yi;
          acc[3][m] += w * xy;
          acc[4][m] += wu * xy;
        }
        if (AXIS == 1)
          acc[3][m] += h * (c == 0 ? xr * qr + xi * qi + yr * pr + yi * pi : pr * yi - pi * yr + qr * xi - qi * xr);
      }
    } else {
#pragma unroll
      for (int m = 0; m < M; ++m) x[m] = xn[m];
      src += 2 * N3;
      if (s + 1 < sb) {
#pragma unroll
        for (int m = 0; m < M; ++m) xn[m] = src[m * (P * stride)];
      }
      diff(x, d, nyq);
      double kin = 0.0;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const double xr = x[m].x, xi = x[m].y, dr = d[m].x, di = d[m].y;
        const double dd = dr * dr + di * di;
        kin += dd;
        if (FIELDS) {
          const Z px = partner(x[m]);
          const double pr = px.x, pi = px.y, wr = w * dr, wi = w * di;
          acc[0][m] += w * dd;
          acc[1][m] += wi * xr;                                  // Im(d conj(x))
          acc[1][m] -= wr * xi;
          if (AXIS != 1) {
            acc[2][m] += wr * pr;                                // Re(d conj(partner))
            acc[2][m] += wi * pi;
          }
          if (AXIS != 0) {
            acc[AXIS == 2 ? 3 : 2][m] += wi * pr;                // Im(d conj(partner))
            acc[AXIS == 2 ? 3 : 2][m] -= wr * pi;
          }
          if (AXIS == 0) {
            const double xx = xr * xr + xi * xi;
            acc[3][m] += w * xx;
            acc[4][m] += wu * xx;
          }
          // Re(conj(up) down) in the lanes of the up component, Im in the others
          if (AXIS == 1) acc[3][m] += w * (c == 0 ? xr * pr + xi * pi : pr * xi - pi * xr);
        }
      }
      if (a.kin) {
        // per-warp partials, summed in a fixed order by kinetic_reduce_kernel
        kin += a.nf[AXIS] * nyq;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) kin += __shfl_xor_sync(0xffffffffu, kin, o);
        if ((threadIdx.x & 31) == 0)
          a.kin[(((size_t)s * 3 + AXIS) * G::NTILE + tile) * G::WARPS + threadIdx.x / 32] = kin;
      }
    }
  }
  if (!FIELDS) return;
  // sums over the components; the two lanes write alternate points
#pragma unroll
  for (int m = 0; m < M && FIELDS; ++m) {
    double up[NA], dn[NA];
#pragma unroll
    for (int f = 0; f < NA; ++f) {
      const double o = __shfl_xor_sync(0xffffffffu, acc[f][m], P);
      up[f] = c == 0 ? acc[f][m] : o;
      dn[f] = c == 0 ? o : acc[f][m];
    }
    if ((m & 1) != c) continue;
    const int j = p + P * m;
    double* w = out + (AXIS == 2 ? lg * N + j : j * G::L + lg);
    constexpr int FS = G::L * N;
    w[0] = up[0] + dn[0];
    w[FS] = up[1] + dn[1];
    if (AXIS == 0) {
      w[2 * FS] = -(up[1] - dn[1]);            // J_y, x part (densities.py:270-273)
      w[3 * FS] = -(dn[2] - up[2]);            // J_z, x part (274-277)
      w[4 * FS] = up[3] + dn[3];
      w[5 * FS] = 0.5 * (up[4] + dn[4]);
      w[6 * FS] = up[3] - dn[3];
    } else if (AXIS == 1) {
      w[2 * FS] = up[1] - dn[1];               // J_x, y part (289-292)
      w[3 * FS] = -(dn[2] + up[2]);            // J_z, y part (293-296)
      w[4 * FS] = 2.0 * up[3];
      w[5 * FS] = 2.0 * dn[3];
    } else {
      w[2 * FS] = dn[2] - up[2];               // J_x, z part (308-311)
      w[3 * FS] = dn[3] + up[3];               // J_y, z part (312-315)
    }
  }
}

template <class R, int N, int KIND>
__global__ void __launch_bounds__(DensGeo<R, N>::THREADS, sizeof(R) == 8 || KIND == DENS_PAIR ? 2 : N > 40 ? 3 : 4)
density_kernel(const __grid_constant__ DensArgs a) {
  using G = DensGeo<R, N>;
  __shared__ __align__(16) cplx<R> xball[G::THREADS / G::P * G::NB];
  __shared__ cplx<R> tw[N];
  __shared__ R sk[3 * N];   // k of each axis, 0 at k = 0 and at the Nyquist mode
  fill_twiddles<R>(tw, N);
  for (int e = threadIdx.x; e < 3 * N; e += G::THREADS) {
    const int k = e % N;
    sk[e] = (k == 0 || 2 * k == N) ? R(0) : (R)(signed_k(k, N) * a.ks[e / N]);
  }
  __syncthreads();
  cplx<R>* xb = xball + (threadIdx.x / G::P) * G::NB;
  const DensCut& cut = a.cut;
  long u = (long)blockIdx.x * cut.run;
  const long end = min(cut.units, u + cut.run);
  while (u < end) {
    int axis, q, tile, s;
    dens_decode(cut, u, axis, q, tile, s);
    const int n = (int)min((long)(cut.cnt[q] - s), end - u);
    const int sa = cut.s0[q] + s;
    double* out = a.part + (blockIdx.x + (size_t)dens_tile(cut, axis, q, tile)) * kDensFields * G::L * N;
    if (axis == 0) dens_segment<R, N, 0, KIND>(a, tile, sa, sa + n, out, xb, tw, sk);
    else if (axis == 1) dens_segment<R, N, 1, KIND>(a, tile, sa, sa + n, out, xb, tw, sk);
    else dens_segment<R, N, 2, KIND>(a, tile, sa, sa + n, out, xb, tw, sk);
    u += n;
  }
}

// Sum the partial tiles of the three axes into the reference's density
// arrays; rho, tau, chi are mixed as mix*new + (1-mix)*old.
template <int N, int L>
__global__ void __launch_bounds__(128)
density_combine_kernel(DensCut cut, const double* __restrict__ part, double mix, double* rho, double* chi, double* tau,
                       double* cur, double* sd, double* so) {
  constexpr size_t N2 = (size_t)N * N, n3 = N2 * N;
  constexpr int FS = L * N;
  const size_t i = blockIdx.x * (size_t)128 + threadIdx.x;
  const int iq = blockIdx.y;
  if (i >= n3) return;
  const int x = (int)(i / N2), y = (int)((i / N) % N), z = (int)(i % N);
  double f[3][kDensFields];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax)
#pragma unroll
    for (int k = 0; k < kDensFields; ++k) f[ax][k] = 0.0;
  for (int q = 0; q < cut.nq; ++q) {
    if (cut.iq[q] != iq) continue;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      const int line = ax == 0 ? y * N + z : ax == 1 ? x * N + z : x * N + y;
      const int j = ax == 0 ? x : ax == 1 ? y : z;
      const int tile = line / L, l = line % L;
      const int off = ax == 2 ? l * N + j : j * L + l;
      const long u0 = dens_first(cut, ax, q, tile), u1 = u0 + cut.cnt[q];
      const long id = dens_tile(cut, ax, q, tile);
      for (long k = u0 / cut.run; k <= (u1 - 1) / cut.run; ++k) {
        const double* p = part + (size_t)(k + id) * kDensFields * FS + off;
        constexpr int NF[3] = {7, 6, 4};
#pragma unroll
        for (int g = 0; g < NF[ax]; ++g) f[ax][g] += p[g * FS];
      }
    }
  }
  const double tnew = f[2][0] + f[1][0] + f[0][0];
  const size_t o = (size_t)iq * n3 + i;
  if (mix < 1.0) {
    rho[o] = mix * f[0][4] + (1.0 - mix) * rho[o];
    chi[o] = mix * f[0][5] + (1.0 - mix) * chi[o];
    tau[o] = mix * tnew + (1.0 - mix) * tau[o];
  } else {
    rho[o] = f[0][4];
    chi[o] = f[0][5];
    tau[o] = tnew;
  }
  const size_t v = (size_t)iq * 3 * n3 + i;
  sd[v] = f[1][4];
  sd[v + n3] = f[1][5];
  sd[v + 2 * n3] = f[0][6];
  cur[v] = f[0][1];
  cur[v + n3] = f[1][1];
  cur[v + 2 * n3] = f[2][1];
  so[v] = f[1][2] + f[2][2];
  so[v + n3] = f[0][2] + f[2][3];
  so[v + 2 * n3] = f[0][3] + f[1][3];
}

// sp_kinetic[s] = wxyz h2m_q times the ``np`` partials of the state, in a
// fixed order; one block per state.
__global__ void __launch_bounds__(128) kinetic_reduce_kernel(int nneut, int np, const double* __restrict__ kin,
                                                             double wxyz, double h2m_n, double h2m_p, double* out) {
  __shared__ double red[4];
  const int s = blockIdx.x;
  double t = 0;
  for (int j = threadIdx.x; j < np; j += 128) t += kin[(size_t)s * np + j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = t;
  __syncthreads();
  if (threadIdx.x == 0) out[s] = wxyz * (s >= nneut ? h2m_p : h2m_n) * (red[0] + red[1] + red[2] + red[3]);
}

struct DensOut {
  double mix;
  double *rho, *chi, *tau, *cur, *sd, *so;   // rho null: kinetic energies only
  const double* h2m;
  double* sp_kinetic;
};

template <class R, int N, int KIND>
int density_launch_t(hfb_ctx_s* c, DensArgs a, int nst, int nneut, const DensOut& o, cudaStream_t st) {
  using G = DensGeo<R, N>;
  // CTAs that are resident together (those that write partial tiles never
  // exceed kDensPerSm: their registers)
  static const int per_sm = [] {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, density_kernel<R, N, KIND>, G::THREADS, 0) != cudaSuccess)
      cudaGetLastError();
    return n < 1 ? 1 : KIND != DENS_KINETIC && n > kDensPerSm ? kDensPerSm : n;
  }();
  DensCut cut{};
  nneut = nneut < 0 ? 0 : nneut > nst ? nst : nneut;
  const int cnt[2] = {nneut, nst - nneut};
  for (int iq = 0; iq < 2; ++iq)
    if (cnt[iq] > 0) {
      cut.iq[cut.nq] = iq;
      cut.s0[cut.nq] = iq ? nneut : 0;
      cut.cnt[cut.nq++] = cnt[iq];
    }
  cut.ntile = G::NTILE;
  cut.nst = nst;
  cut.units = 3L * G::NTILE * nst;
  // one run per resident CTA; at least two units, below which a CTA's start
  // and its partial tiles cost more than the balance gives
  const long places = (long)per_sm * c->sms;
  cut.run = (cut.units + places - 1) / places;
  if (cut.run < 2) cut.run = 2;
  const long ctas = (cut.units + cut.run - 1) / cut.run;
  a.cut = cut;
  a.part = nullptr;
  if (KIND != DENS_KINETIC) {
    // one size for all state counts, precisions and kinds: the buffer is not
    // moved under a captured graph
    const size_t tiles = (size_t)kDensPerSm * c->sms + 3 * 2 * G::NTILE;
    a.part = (double*)scratch(c, hfb_ctx_s::S_DENS, sizeof(double) * tiles * kDensFields * G::L * N);
    if (!a.part) return HFB_ERR_ALLOC;
  }
  a.kin = nullptr;
  if (o.sp_kinetic) {
    a.kin = (double*)scratch(c, hfb_ctx_s::S_RED, sizeof(double) * (size_t)3 * nst * G::NTILE * G::WARPS);
    if (!a.kin) return HFB_ERR_ALLOC;
  }
  for (int ax = 0; ax < 3; ++ax) {
    a.ks[ax] = 2.0 * kPi / (c->d[ax] * N) / N;
    a.nf[ax] = (kPi / c->d[ax]) * (kPi / c->d[ax]) / N;
  }
  density_kernel<R, N, KIND><<<(unsigned)ctas, G::THREADS, 0, st>>>(a);
  HFB_CHECK_LAUNCH();
  if (KIND != DENS_KINETIC) {
    const dim3 g2((unsigned)(((size_t)N * N * N + 127) / 128), 2);
    density_combine_kernel<N, G::L><<<g2, 128, 0, st>>>(cut, a.part, o.mix, o.rho, o.chi, o.tau, o.cur, o.sd, o.so);
    HFB_CHECK_LAUNCH();
  }
  if (o.sp_kinetic) {
    kinetic_reduce_kernel<<<nst, 128, 0, st>>>(nneut, 3 * G::NTILE * G::WARPS, a.kin, c->wxyz, o.h2m[0], o.h2m[1],
                                               o.sp_kinetic);
    HFB_CHECK_LAUNCH();
  }
  return HFB_OK;
}

template <int KIND>
int density_launch(hfb_ctx_s* c, int prec, const DensArgs& a, int nst, int nneut, const DensOut& o, cudaStream_t st) {
  return dispatch_n(c->n, [&](auto nn) -> int {
    constexpr int N = decltype(nn)::value;
    if (prec == HFB_F64) return density_launch_t<double, N, KIND>(c, a, nst, nneut, o, st);
    return density_launch_t<float, N, KIND>(c, a, nst, nneut, o, st);
  });
}

}  // namespace

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_add_density(hfb_ctx_t ctx, int prec, int nst, int nneut, const void* psi, const double* wocc,
                               const double* wguv, const double* pairwg, const double* wstates, double mix,
                               double* rho, double* chi, double* tau, double* current, double* sdens, double* sodens,
                               const double* h2m, double* sp_kinetic, void* stream) {
  if (!ctx || !psi || !wocc || !wguv || !pairwg || !wstates || !rho || !chi || !tau || !current || !sdens || !sodens)
    return HFB_ERR_ARG;
  if (sp_kinetic && !h2m) return HFB_ERR_ARG;
  if (nst <= 0) return HFB_ERR_ARG;
  DensArgs a{};
  a.psi = psi;
  a.wocc = wocc; a.wguv = wguv; a.pairwg = pairwg; a.wstates = wstates;
  return density_launch<DENS_FIELDS>(ctx, prec, a, nst, nneut,
                               DensOut{mix, rho, chi, tau, current, sdens, sodens, h2m, sp_kinetic}, as_stream(stream));
}

extern "C" int hfb_sp_kinetic(hfb_ctx_t ctx, int prec, int nst, int nneut, const void* psi, const double* h2m,
                              double* sp_kinetic, void* stream) {
  if (!ctx || !psi || !h2m || !sp_kinetic || nst <= 0) return HFB_ERR_ARG;
  // weights are not read when no fields are accumulated
  DensArgs a{};
  a.psi = psi;
  DensOut o{};
  o.h2m = h2m;
  o.sp_kinetic = sp_kinetic;
  return density_launch<DENS_KINETIC>(ctx, prec, a, nst, nneut, o, as_stream(stream));
}

extern "C" int hfb_pair_density(hfb_ctx_t ctx, int prec, int nst, int nneut, const void* a, const void* b,
                                const double* w, const double* wu, double* rho, double* chi, double* tau,
                                double* current, double* sdens, double* sodens, void* stream) {
  if (!ctx || !a || !b || !w || !wu || !rho || !chi || !tau || !current || !sdens || !sodens || nst <= 0)
    return HFB_ERR_ARG;
  DensArgs d{};
  d.psi = a;
  d.psi2 = b;
  d.wocc = w; d.wguv = wu;
  return density_launch<DENS_PAIR>(ctx, prec, d, nst, nneut,
                              DensOut{1.0, rho, chi, tau, current, sdens, sodens, nullptr, nullptr}, as_stream(stream));
}
