// Double-precision hpsi (hpsi01, meanfield.py:41-159) on the FP64 tensor
// cores (mma.sync m8n8k4 .f64).
//
// The algebra is the matrix form of the FFT path (hpsi.cu): along each axis d
//     out_d = L_d(D x) + D(L_d x - B D x) + Nyquist term,
// D the real n x n first-derivative matrix with its k = 0 and n/2 bins zero,
// B the effective mass, L_d the pointwise 2x2 current / spin-orbit operator
// of the axis and the Nyquist term (pi/d)^2 mean_line(B) (-1)^j
// sum_l (-1)^l x_l / n of cderv02 (levels.py:314-330).
//
// D changes sign when both its indices are reversed (j -> n-1-j), so with
// x-[l] = x[l] - x[n-1-l], x+[l] = x[l] + x[n-1-l] for l < n/2,
//     (D x)[j] = (Dm x-)[j] + (Dp x+)[j],  (D x)[n-1-j] = (Dm x-)[j] - (Dp x+)[j],
//     Dm[j][l] = (D[j][l] - D[j][n-1-l]) / 2,  Dp[j][l] = (D[j][l] + D[j][n-1-l]) / 2,
// two products with (n/2) x (n/2) matrices: half the MMAs of D itself.
//
// A warp owns one MMA tile of a staged plane, 8 points j < n/2 and their
// mirrors on 8 lines, both spinor components: after GEMM 1 a thread holds
// D x at 4 (point, line) positions in both components, does the pointwise
// step on them, stores w+- for GEMM 2 and gets the same positions back.
//
// Two kernels: X (x-planes: z lines with the local terms, then y lines; what
// the z lines give waits in the w buffer, at the thread's own positions) and
// Y (y-planes: x lines, the final weights and overlaps).  Both are
// persistent: the derivative matrices stay in shared memory, and the next
// plane is copied in (cp.async) from the moment the plane's last reader has
// passed, behind GEMM 2.  In the z pass only the warps of the same lines wait
// for one another, so that some warps' MMAs run beside others' pointwise
// step.  (A warp of its own for the copies took registers from the others:
// 2.0 ms for X at 48^3 against 1.5.)  Planes are stored without padding, 16-byte elements
// XOR-swizzled by row so that fragment loads along rows and columns hit
// distinct banks.
//
// Bound by the tensor pipe and the pointwise FP64 work in turn.  Pb208 (236
// states, 48^3): 4.87 ms a call with the full D, eight warps on five rounds
// of tiles and the partial sums in global memory; 2.5 ms here.
#include <math.h>
#include <vector>
#include "diag.cuh"
#include "hpsi.cuh"

namespace hfb {

namespace {

template <int N>
struct HdGeo {
  static constexpr int H = N / 2;                     // points of a half line
  static constexpr int MB = (H + 7) / 8;              // 8-point blocks of it
  static constexpr int LG = N / 8;                    // 8-line groups of a plane
  static constexpr int WARPS = MB * LG, THREADS = 32 * WARPS;   // one warp per tile
  static constexpr int KS = H / 4;                    // MMA k steps
  static constexpr int HP = 8 * MB;                   // rows of Dm, Dp (zero past H)
  static constexpr int LDH = H % 16 == 4 || H % 16 == 12 ? H : H + 4;   // row stride: rows on distinct banks
  static constexpr int DSZ = 2 * HP * LDH;            // doubles of Dm, Dp of one axis
  static constexpr size_t PLANE = (size_t)2 * N * N;  // complex elements of a plane
  static constexpr size_t smem(int axes) { return sizeof(double2) * (2 * PLANE + axes * 2 * N) + sizeof(double) * axes * (DSZ + N); }
  // CTAs per SM that shared memory and the registers allow for
  static constexpr int CTAS = N >= 40 ? 1 : N == 32 ? 2 : N == 24 ? 4 : 8;
  static_assert(N % 8 == 0 && (LDH % 16 == 4 || LDH % 16 == 12), "grid size");
};

// Element (component, row, column) of a plane.
template <int N>
__device__ __forceinline__ int hd_el(int c, int row, int col) {
  return (c * N + row) * N + (col ^ (((row & 1) * 5) | (row & 2)));
}
// A "line" of a pass runs along the columns (ROW) or along the rows; pt is
// the position along it.
template <int N, bool ROW>
__device__ __forceinline__ int hd_at(int c, int line, int pt) {
  return ROW ? hd_el<N>(c, line, pt) : hd_el<N>(c, pt, line);
}

// A thread's place in its warp's tile: point j (mirror N-1-j), lines l and
// l + 1; fragment row / line fr, k index fk.
struct HdTile {
  int j0, l0, fr, fk, j, l;
  bool on;    // j is a point (not padding)
};
template <int N>
__device__ __forceinline__ HdTile hd_tile() {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  HdTile t;
  t.fr = lane >> 2;
  t.fk = lane & 3;
  t.j0 = 8 * (warp % HdGeo<N>::MB);
  t.l0 = 8 * (warp / HdGeo<N>::MB);
  t.j = t.j0 + t.fr;
  t.l = t.l0 + 2 * t.fk;
  t.on = t.j < HdGeo<N>::H;
  return t;
}

// d[half][line][component] = D applied along the lines; S holds the values
// themselves (PLAIN; ``alt`` then gets sum (-1)^l x_l of line l0 + fr) or
// their +- combinations at positions l and N-1-l.
template <int N, bool ROW, bool PLAIN>
__device__ __forceinline__ void hd_gemm(const double2* S, const double* Dm, const HdTile& t, double2 (&d)[2][2][2],
                                        double2 (&alt)[2]) {
  using G = HdGeo<N>;
  const double* am = Dm + t.j * G::LDH + t.fk;
  const double* ap = am + G::HP * G::LDH;
  double m[4][2], p[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) m[i][0] = m[i][1] = p[i][0] = p[i][1] = 0.0;
  if (PLAIN) alt[0] = alt[1] = make_double2(0.0, 0.0);
#pragma unroll
  for (int ks = 0; ks < G::KS; ++ks) {
    const int pt = 4 * ks + t.fk, line = t.l0 + t.fr;
    const double a = am[4 * ks], b = ap[4 * ks];
    double2 u[2], v[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      u[c] = S[hd_at<N, ROW>(c, line, pt)];
      v[c] = S[hd_at<N, ROW>(c, line, N - 1 - pt)];
      if (PLAIN) {
        const double2 s = u[c] + v[c], r = u[c] - v[c];
        u[c] = s;
        v[c] = r;
        alt[c] = alt[c] + r;
      }
    }
    gd_mma(m[0], a, v[0].x);
    gd_mma(p[0], b, u[0].x);
    gd_mma(m[1], a, v[0].y);
    gd_mma(p[1], b, u[0].y);
    gd_mma(m[2], a, v[1].x);
    gd_mma(p[2], b, u[1].x);
    gd_mma(m[3], a, v[1].y);
    gd_mma(p[3], b, u[1].y);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      d[0][u][c] = make_double2(m[2 * c][u] + p[2 * c][u], m[2 * c + 1][u] + p[2 * c + 1][u]);
      d[1][u][c] = make_double2(m[2 * c][u] - p[2 * c][u], m[2 * c + 1][u] - p[2 * c + 1][u]);
    }
  if (PLAIN) {
    // (-1)^l = (-1)^fk, the mirror's sign is opposite; sum over the four k lanes
    const double sg = (t.fk & 1) ? -1.0 : 1.0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      alt[c] = sg * alt[c];
#pragma unroll
      for (int o = 1; o <= 2; o *= 2) {
        alt[c].x += __shfl_xor_sync(0xffffffffu, alt[c].x, o);
        alt[c].y += __shfl_xor_sync(0xffffffffu, alt[c].y, o);
      }
    }
  }
}

// The pointwise step of an axis at one point: q = L_d e (+ local terms) and
// n = L_d a (w without its -B e).
template <int AXIS, bool LOCAL>
__device__ __forceinline__ void hd_point(const double* pot, size_t n3, size_t g, const double2 (&a)[2],
                                         const double2 (&e)[2], double2 (&q)[2], double2 (&w)[2]) {
  const double h = 0.5;
  const double bm = pot[1 * n3 + g], aq = pot[(3 + AXIS) * n3 + g];
  const double v0 = AXIS != 0 ? pot[9 * n3 + g] : 0.0, v1 = AXIS != 1 ? pot[10 * n3 + g] : 0.0,
               v2 = AXIS != 2 ? pot[11 * n3 + g] : 0.0;
  q[0] = q[1] = make_double2(0.0, 0.0);
  if (LOCAL) {
    // upot psi + sigma.spot psi (meanfield.py:47-58)
    const double up = pot[g], s0 = pot[6 * n3 + g], s1 = pot[7 * n3 + g], s2 = pot[8 * n3 + g];
    q[0] = (up + s2) * a[0] + cmulri(s0, -s1, a[1]);
    q[1] = (up - s2) * a[1] + cmulri(s0, s1, a[0]);
  }
  if (AXIS == 0) {
    // meanfield.py:63-83
    q[0] = q[0] + cmulri(0.0, -(h * aq - h * v1), e[0]) - (h * v2) * e[1];
    q[1] = q[1] + cmulri(0.0, -(h * aq + h * v1), e[1]) + (h * v2) * e[0];
    w[0] = cmulri(0.0, -h * (aq - v1), a[0]) - (h * v2) * a[1];
    w[1] = cmulri(0.0, -h * (aq + v1), a[1]) + (h * v2) * a[0];
  } else if (AXIS == 1) {
    // meanfield.py:92-112
    q[0] = q[0] + cmulri(0.0, -(h * aq + h * v0), e[0]) + cmulri(0.0, h * v2, e[1]);
    q[1] = q[1] + cmulri(0.0, -(h * aq - h * v0), e[1]) + cmulri(0.0, h * v2, e[0]);
    w[0] = cmulri(0.0, -h * (aq + v0), a[0]) + cmulri(0.0, h * v2, a[1]);
    w[1] = cmulri(0.0, -h * (aq - v0), a[1]) + cmulri(0.0, h * v2, a[0]);
  } else {
    // meanfield.py:121-141
    q[0] = q[0] + cmulri(0.0, -(h * aq), e[0]) + cmulri(h * v0, -(h * v1), e[1]);
    q[1] = q[1] + cmulri(0.0, -(h * aq), e[1]) + cmulri(-(h * v0), -(h * v1), e[0]);
    w[0] = cmulri(0.0, -h * aq, a[0]) + cmulri(h * v0, -(h * v1), a[1]);
    w[1] = cmulri(0.0, -h * aq, a[1]) + cmulri(-(h * v0), -(h * v1), a[0]);
  }
  w[0] = w[0] - bm * e[0];
  w[1] = w[1] - bm * e[1];
}

// First half of an axis pass: GEMM 1, the lines' alternating sums into alts,
// the pointwise step and w+- into W; out[half][line][component] = L_d D x
// (+ local terms) (+ what W held at the thread's positions, ADD).  The point
// (line, pt) of the plane is element base + line * sl + pt * sp of a field.
template <int N, int AXIS, bool ROW, bool LOCAL, bool ADD>
__device__ __forceinline__ void hd_first(const double2* X, double2* W, const double* Dm, double2* alts, const HdTile& t,
                                         const double* pot, size_t base, size_t sl, size_t sp,
                                         double2 (&out)[2][2][2]) {
  constexpr size_t N3 = (size_t)N * N * N;
  double2 e[2][2][2], alt[2];
  hd_gemm<N, ROW, true>(X, Dm, t, e, alt);
  if (t.j0 == 0 && t.fk == 0) {
    alts[t.l0 + t.fr] = alt[0];
    alts[N + t.l0 + t.fr] = alt[1];
  }
  if (!t.on) return;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int line = t.l + u;
    double2 w[2][2];
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const int pt = f ? N - 1 - t.j : t.j;
      const double2 a[2] = {X[hd_at<N, ROW>(0, line, pt)], X[hd_at<N, ROW>(1, line, pt)]};
      hd_point<AXIS, LOCAL>(pot, N3, base + line * sl + pt * sp, a, e[f][u], out[f][u], w[f]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (ADD) out[f][u][c] = out[f][u][c] + W[hd_at<N, ROW>(c, line, pt)];
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      W[hd_at<N, ROW>(c, line, t.j)] = w[0][c] + w[1][c];
      W[hd_at<N, ROW>(c, line, N - 1 - t.j)] = w[0][c] - w[1][c];
    }
  }
}

// Second half: GEMM 2 on w+-, and the Nyquist term, added to out; bb is the
// line mean of B of the plane's lines, nq = (pi/d)^2 / n.
template <int N, bool ROW>
__device__ __forceinline__ void hd_second(const double2* W, const double* Dm, const double2* alts, const double* bb,
                                          double nq, const HdTile& t, double2 (&out)[2][2][2]) {
  double2 r[2][2][2], none[2];
  hd_gemm<N, ROW, false>(W, Dm, t, r, none);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const double sg = ((t.j & 1) ? -nq : nq) * bb[t.l + u];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double2 al = sg * alts[c * N + t.l + u];   // the mirror's sign is opposite
      out[0][u][c] = out[0][u][c] + r[0][u][c] + al;
      out[1][u][c] = out[1][u][c] + r[1][u][c] - al;
    }
  }
}

// Barrier of the warps of a line group (tiles of the same lines).
template <int N>
__device__ __forceinline__ void hd_sync_group() {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x >> 5) / HdGeo<N>::MB), "n"(32 * HdGeo<N>::MB) : "memory");
}
// Start the copy of a plane: rows of N elements ``pitch`` apart, components
// N^3 apart.
template <int N>
__device__ __forceinline__ void hd_stage(double2* X, const double2* src, size_t pitch) {
  for (int e = threadIdx.x; e < 2 * N * N; e += HdGeo<N>::THREADS) {
    const int c = e / (N * N), r = e / N % N, q = e % N;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(X + hd_el<N>(c, r, q))),
                 "l"(src + (size_t)c * N * N * N + r * pitch + q)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
// The line means of B of the plane's lines: from the launch's table, or, when
// a CTA has few planes, from the plane of B (element b[line * sl + i * sp]).
template <int N>
__device__ __forceinline__ void hd_means(double* dst, const double* __restrict__ table, const double* __restrict__ b,
                                         size_t sl, size_t sp, int tid) {
  for (int line = tid; line >= 0 && line < N; line += HdGeo<N>::THREADS) {
    double m = 0.0;
    if (table) {
      m = table[line];
    } else {
#pragma unroll 8
      for (int i = 0; i < N; ++i) m += b[line * sl + i * sp];
      m /= N;
    }
    dst[line] = m;
  }
}
__device__ __forceinline__ void hd_staged() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

struct HdArgs {
  const double* pot;
  const double* bbar;      // [iq][axis][line], or null
  const double2* psi;
  double2* acc;
  int s0, ns, nneut;
  const double* dmat;      // [axis][Dm, Dp]
  double nq[3];
  const double *weight, *weightuv;
  double2 *pout, *pout_mf, *pout_del;
  double* ovl;
};

// X: an x-plane of a state; z lines with the local terms, then y lines.
template <int N>
__global__ void __launch_bounds__(HdGeo<N>::THREADS, HdGeo<N>::CTAS) hpsi_dmma_x_kernel(const __grid_constant__ HdArgs a) {
  using G = HdGeo<N>;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char hd_smem[];
  double2* X = reinterpret_cast<double2*>(hd_smem);
  double2* W = X + G::PLANE;
  double* dz = reinterpret_cast<double*>(W + G::PLANE);
  double* dy = dz + G::DSZ;
  double* bz = dy + G::DSZ;
  double* by = bz + N;
  double2* az = reinterpret_cast<double2*>(by + N);
  double2* ay = az + 2 * N;
  const HdTile t = hd_tile<N>();
  const int items = a.ns * N;
  auto source = [&](int it) { return a.psi + (size_t)(a.s0 + it / N) * 2 * N3 + (size_t)(it % N) * N2; };
  int it = blockIdx.x;
  hd_stage<N>(X, source(it), N);
  for (int e = threadIdx.x; e < G::DSZ; e += G::THREADS) {
    dz[e] = a.dmat[2 * G::DSZ + e];
    dy[e] = a.dmat[G::DSZ + e];
  }
  for (; it < items; it += gridDim.x) {
    const int s = a.s0 + it / N, x0 = it % N, iq = s >= a.nneut ? 1 : 0;
    const double* pot = a.pot + (size_t)iq * 12 * N3;
    {
      const double* tb = a.bbar ? a.bbar + (size_t)iq * 3 * N2 + (size_t)x0 * N : nullptr;
      hd_means<N>(bz, tb ? tb + 2 * N2 : nullptr, pot + N3 + (size_t)x0 * N2, N, 1, threadIdx.x);
      hd_means<N>(by, tb ? tb + N2 : nullptr, pot + N3 + (size_t)x0 * N2, 1, N, (int)threadIdx.x - G::THREADS / 2);
    }
    hd_staged();
    double2 out[2][2][2];
    hd_first<N, 2, true, true, false>(X, W, dz, az, t, pot, (size_t)x0 * N2, N, 1, out);
    hd_sync_group<N>();
    hd_second<N, true>(W, dz, az, bz, a.nq[2], t, out);
    hd_sync_group<N>();
    if (t.on) {
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int c = 0; c < 2; ++c) W[hd_at<N, true>(c, t.l + u, f ? N - 1 - t.j : t.j)] = out[f][u][c];
    }
    __syncthreads();
    hd_first<N, 1, false, false, true>(X, W, dy, ay, t, pot, (size_t)x0 * N2, 1, N, out);
    __syncthreads();
    if (it + (int)gridDim.x < items) hd_stage<N>(X, source(it + gridDim.x), N);
    hd_second<N, false>(W, dy, ay, by, a.nq[1], t, out);
    if (t.on) {
      double2* dst = a.acc + (size_t)s * 2 * N3 + (size_t)x0 * N2 + t.l;
#pragma unroll
      for (int f = 0; f < 2; ++f)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int u = 0; u < 2; ++u) dst[c * N3 + (size_t)(f ? N - 1 - t.j : t.j) * N + u] = out[f][u][c];
    }
    __syncthreads();   // the means are rewritten
  }
}

// Y: a y-plane of a state; x lines, then pout = weight * h psi - weightuv *
// v_pair psi, pout_del = v_pair psi and the plane's overlaps.
template <int N>
__global__ void __launch_bounds__(HdGeo<N>::THREADS, HdGeo<N>::CTAS) hpsi_dmma_y_kernel(const __grid_constant__ HdArgs a) {
  using G = HdGeo<N>;
  constexpr size_t N2 = (size_t)N * N, N3 = N2 * N;
  extern __shared__ __align__(16) unsigned char hd_smem[];
  __shared__ double red[2][G::WARPS];
  double2* X = reinterpret_cast<double2*>(hd_smem);   // row x, column z
  double2* W = X + G::PLANE;
  double* dx = reinterpret_cast<double*>(W + G::PLANE);
  double* bx = dx + G::DSZ;
  double2* ax = reinterpret_cast<double2*>(bx + N);
  const HdTile t = hd_tile<N>();
  const int items = a.ns * N;
  auto source = [&](int it) { return a.psi + (size_t)(a.s0 + it / N) * 2 * N3 + (size_t)(it % N) * N; };
  int it = blockIdx.x;
  hd_stage<N>(X, source(it), N2);
  for (int e = threadIdx.x; e < G::DSZ; e += G::THREADS) dx[e] = a.dmat[e];
  for (; it < items; it += gridDim.x) {
    const int s = a.s0 + it / N, y0 = it % N, iq = s >= a.nneut ? 1 : 0;
    const double* pot = a.pot + (size_t)iq * 12 * N3;
    hd_means<N>(bx, a.bbar ? a.bbar + (size_t)iq * 3 * N2 + (size_t)y0 * N : nullptr, pot + N3 + (size_t)y0 * N, 1, N2,
                threadIdx.x);
    hd_staged();
    double2 out[2][2][2];
    hd_first<N, 0, false, false, false>(X, W, dx, ax, t, pot, (size_t)y0 * N, 1, N2, out);
    __syncthreads();
    if (it + (int)gridDim.x < items) hd_stage<N>(X, source(it + gridDim.x), N2);
    hd_second<N, false>(W, dx, ax, bx, a.nq[0], t, out);
    const double wt = a.weight ? a.weight[s] : 1.0, wu = a.weightuv ? a.weightuv[s] : 0.0;
    double ov_mf = 0.0, ov_po = 0.0;
    if (t.on) {
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const size_t g = (size_t)y0 * N + (size_t)(f ? N - 1 - t.j : t.j) * N2 + t.l, gs = (size_t)s * 2 * N3 + g;
        double2 ps[2][2], pm[2][2];
        double vp[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          vp[u] = pot[2 * N3 + g + u];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            ps[u][c] = a.psi[gs + c * N3 + u];   // the plane itself may be gone
            pm[u][c] = a.acc[gs + c * N3 + u];
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const size_t gi = gs + c * N3 + u;
            const double2 mf = pm[u][c] + out[f][u][c];
            const double2 dl = vp[u] * ps[u][c];
            const double2 po = wt * mf - wu * dl;
            if (a.pout_mf) a.pout_mf[gi] = mf;
            if (a.pout) a.pout[gi] = po;
            if (a.pout_del) a.pout_del[gi] = dl;
            ov_mf += ps[u][c].x * mf.x + ps[u][c].y * mf.y;
            ov_po += ps[u][c].x * po.x + ps[u][c].y * po.y;
          }
      }
    }
    if (a.ovl) {
      // fixed order: warp shuffles, then one thread per sum
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ov_mf += __shfl_xor_sync(0xffffffffu, ov_mf, o);
        ov_po += __shfl_xor_sync(0xffffffffu, ov_po, o);
      }
      if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x / 32] = ov_mf;
        red[1][threadIdx.x / 32] = ov_po;
      }
    }
    __syncthreads();   // red is complete; the means are rewritten
    if (a.ovl && threadIdx.x < 2) {
      double p = 0.0;
      for (int i = 0; i < G::WARPS; ++i) p += red[threadIdx.x][i];
      a.ovl[((size_t)(s - a.s0) * N + y0) * 2 + threadIdx.x] = p;
    }
  }
}

// bbar[iq][axis][line] = mean of B along the line; lines numbered by their two
// other coordinates in increasing order.
__global__ void __launch_bounds__(128) hd_bbar_kernel(int n, const double* __restrict__ pot, double* __restrict__ bbar) {
  const int n2 = n * n, line = blockIdx.x * 128 + threadIdx.x, ax = blockIdx.y, iq = blockIdx.z;
  if (line >= n2) return;
  const int u = line / n, v = line % n;
  const double* b = pot + ((size_t)iq * 12 + 1) * n2 * n + (ax == 0 ? (size_t)line : ax == 1 ? (size_t)u * n2 + v : (size_t)line * n);
  const size_t st = ax == 0 ? n2 : ax == 1 ? n : 1;
  double s = 0.0;
#pragma unroll 8
  for (int j = 0; j < n; ++j) s += b[j * st];
  bbar[((size_t)iq * 3 + ax) * n2 + line] = s / n;
}

template <int N>
int hpsi_dmma_launch_t(hfb_ctx_s* c, HdArgs a, cudaStream_t st) {
  using G = HdGeo<N>;
  if (a.ns <= 0) return HFB_OK;
  for (int ax = 0; ax < 3; ++ax) a.nq[ax] = (M_PI / c->d[ax]) * (M_PI / c->d[ax]) / N;
  allow_max_dynamic_smem(hpsi_dmma_x_kernel<N>);
  allow_max_dynamic_smem(hpsi_dmma_y_kernel<N>);
  const long items = (long)a.ns * N, places = (long)G::CTAS * c->sms;
  const unsigned grid = (unsigned)(items < places ? items : places);
  // a table of the line means (one launch, about 8 us with its gap) pays from
  // a few planes a CTA on (about 1 us each without it).  It lies behind the
  // derivative matrices: in the arena's slot, which the single-precision
  // kernels grow, it could move under a captured graph.
  a.bbar = nullptr;
  if (items > 8 * places) {
    double* bbar = c->hpsi_d64 + 3 * G::DSZ;
    hd_bbar_kernel<<<dim3((N * N + 127) / 128, 3, 2), 128, 0, st>>>(N, a.pot, bbar);
    HFB_CHECK_LAUNCH();
    a.bbar = bbar;
  }
  hpsi_dmma_x_kernel<N><<<grid, G::THREADS, G::smem(2), st>>>(a);
  HFB_CHECK_LAUNCH();
  hpsi_dmma_y_kernel<N><<<grid, G::THREADS, G::smem(1), st>>>(a);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

}  // namespace

// Dm and Dp of each axis, rows padded and strided as the kernels read them,
// from D (levels.py:132-189 as a matrix): D[j][l] = -(2 kf / n)
// sum_{k=1}^{n/2-1} k sin(2 pi k (j - l) / n), kf = 2 pi / (n d), in double.
int hpsi_dmma_prepare(hfb_ctx_s* c) {
  c->hpsi_d64 = nullptr;
  return dispatch_n(c->n, [&](auto nn) -> int {
    constexpr int N = decltype(nn)::value;
    using G = HdGeo<N>;
    std::vector<double> d((size_t)3 * G::DSZ, 0.0);
    for (int ax = 0; ax < 3; ++ax) {
      const double kf = 2.0 * M_PI / (N * c->d[ax]);
      auto el = [&](int j, int l) {
        double v = 0.0;
        for (int k = 1; k < N / 2; ++k) {
          const int ph = (((k * (j - l)) % N) + N) % N;
          v += k * sin(2.0 * M_PI * ph / N);
        }
        return -2.0 * kf / N * v;
      };
      for (int j = 0; j < G::H; ++j)
        for (int l = 0; l < G::H; ++l) {
          const double p = el(j, l), q = el(j, N - 1 - l);
          d[(size_t)ax * G::DSZ + j * G::LDH + l] = 0.5 * (p - q);
          d[(size_t)ax * G::DSZ + (G::HP + j) * G::LDH + l] = 0.5 * (p + q);
        }
    }
    // and room for the line means of a launch, [2][3][n^2]
    if (cudaMalloc(&c->hpsi_d64, (d.size() + 6 * N * N) * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      c->hpsi_d64 = nullptr;
      return HFB_ERR_ALLOC;
    }
    if (cudaMemcpy(c->hpsi_d64, d.data(), d.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
      return HFB_ERR_CUDA;
    return HFB_OK;
  });
}

bool hpsi_dmma_available(hfb_ctx_s* c, int prec) { return prec == HFB_F64 && c->f64_hpsi == 1 && c->hpsi_d64; }

int hpsi_dmma_launch(hfb_ctx_s* c, const void* pot, int s0, int ns, int nneut, const void* psi, const double* weight,
                     const double* weightuv, void* acc, void* pout, void* pout_mf, void* pout_del, double* ovl,
                     cudaStream_t st) {
  HdArgs a{};
  a.pot = (const double*)pot;
  a.psi = (const double2*)psi;
  a.acc = (double2*)acc;
  a.s0 = s0; a.ns = ns; a.nneut = nneut;
  a.dmat = c->hpsi_d64;
  a.weight = weight; a.weightuv = weightuv;
  a.pout = (double2*)pout; a.pout_mf = (double2*)pout_mf; a.pout_del = (double2*)pout_del;
  a.ovl = ovl;
  return dispatch_n(c->n, [&](auto nn) -> int { return hpsi_dmma_launch_t<decltype(nn)::value>(c, a, st); });
}

}  // namespace hfb
