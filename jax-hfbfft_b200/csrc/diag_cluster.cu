// The small-matrix chains of the diagonalisation step (static.py:261-577),
// one thread-block cluster per isospin and one launch per chain:
//   loewdin_kernel    S^-1/2 by the coupled Newton-Schulz iteration
//   refine_kernel     eigenpairs of a nearly diagonal Hermitian matrix
//   construct_kernel  U = S^-1/2 V, U^H H U, lambda, the outputs of
//                     construct_hfb_matrices, and U lambda
//
// The matrices (n <= 256, a few hundred kB) stay in L2 and the products are
// short, so what bounds these chains is the number of dependent steps.  As
// separate launches (51 products and 16 convergence checks for S^-1/2 alone,
// most of them retired on the device after convergence) they cost 2 us of
// launch gap each; here a step is a barrier of the cluster (below 1 us) and
// the loop ends when it has converged.  A warp owns 16 x 16 output blocks on
// the FP64 tensor cores with both operands read from L2; Hermitian results
// are computed on the upper blocks and mirrored.  A block's sum runs in the
// same order whatever the cluster size.
// S^-1/2 of two matrices, as separate launches and here: n = 10: 190 us with
// the gaps -> 26 us; n = 61: 240 us -> 75 us; construct n = 61: 60 -> 37 us.
#include <math.h>
#include "diag.cuh"

namespace hfb {

namespace {

constexpr int kClThreads = 256;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClMax = 16;     // CTAs per cluster at most (8 portable, 16 opted in to)
constexpr int kTile = 16;      // output block of a warp

__device__ __forceinline__ int cl_rank() {
  int r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ int cl_size() {
  int r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// All threads of the cluster; global writes before it are visible to reads
// through L2 (__ldcg) after it.
__device__ __forceinline__ void cl_sync() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// What a thread needs to know about its place in the cluster.
struct Place {
  int b;        // isospin
  int rank, size;
  int warp;     // cluster-wide warp index, consecutive warps on different SMs
  int nwarp;
  int tid, nthr;
};
__device__ __forceinline__ Place place() {
  Place p;
  p.rank = cl_rank();
  p.size = cl_size();
  p.b = blockIdx.x / p.size;
  p.warp = (threadIdx.x / 32) * p.size + p.rank;
  p.nwarp = kClWarps * p.size;
  p.tid = p.rank * kClThreads + threadIdx.x;
  p.nthr = kClThreads * p.size;
  return p;
}

// Sum or maximum of NV values over the cluster.  ``slots``: 2 x NV x kClMax
// doubles of global memory; ``turn`` alternates between the two halves, so
// that one barrier per call is enough.
template <int NV, bool MAX>
__device__ void cl_reduce(const Place& p, double (&v)[NV], double* slots, int& turn) {
  __shared__ double red[NV][kClWarps];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = MAX ? fmax(v[k], w) : v[k] + w;
    }
    if (threadIdx.x % 32 == 0) red[k][threadIdx.x / 32] = v[k];
  }
  __syncthreads();
  double* s = slots + turn * NV * kClMax;
  if (threadIdx.x < NV) {
    double t = red[threadIdx.x][0];
    for (int w = 1; w < kClWarps; ++w) t = MAX ? fmax(t, red[threadIdx.x][w]) : t + red[threadIdx.x][w];
    s[threadIdx.x * kClMax + p.rank] = t;
  }
  cl_sync();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = __ldcg(s + k * kClMax);
    for (int r = 1; r < p.size; ++r) {
      const double w = __ldcg(s + k * kClMax + r);
      v[k] = MAX ? fmax(v[k], w) : v[k] + w;
    }
  }
  turn ^= 1;
}

// One 16 x 16 block of A B (HA false) or A^H B (HA true), n x n complex
// matrices read through L2.  With k' running over (Re, Im) of each k,
//   Re C = sum_k' A'[i][k'] (Re B, -Im B),  Im C = sum_k' A'[i][k'] (Im B, Re B).
// The thread holds rows i0 + 8 m + lane / 4, columns j0 + 8 v + 2 (lane % 4) + c.
struct Block16 {
  double re[2][2][2], im[2][2][2];
};

template <bool HA>
__device__ void block_product(int n, const double2* A, int lda, const double2* B, int ldb, int i0, int j0,
                              Block16& o) {
  const int lane = threadIdx.x % 32, fr = lane >> 2, part = lane & 1, kh = (lane >> 1) & 1;
  const double* Ad = reinterpret_cast<const double*>(A);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int v = 0; v < 2; ++v) o.re[m][v][0] = o.re[m][v][1] = o.im[m][v][0] = o.im[m][v][1] = 0.0;
  // KS MMA steps (of two complex k) are in registers, the next KS on their way
  constexpr int KS = 4;
  double a[2][KS][2];
  double2 bb[2][KS][2];
  auto load = [&](int k0, double (&an)[KS][2], double2 (&bn)[KS][2]) {
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      const int k = k0 + 2 * s + kh;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int i = i0 + 8 * m + fr;
        an[s][m] = 0.0;
        if (k < n && i < n) an[s][m] = __ldcg(Ad + 2 * (HA ? (size_t)k * lda + i : (size_t)i * lda + k) + part);
      }
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int j = j0 + 8 * v + fr;
        bn[s][v] = make_double2(0.0, 0.0);
        if (k < n && j < n) bn[s][v] = __ldcg(B + (size_t)k * ldb + j);
      }
    }
  };
  auto mul = [&](const double (&ac)[KS][2], const double2 (&bc)[KS][2]) {
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const double br = part ? -bc[s][v].y : bc[s][v].x, bi = part ? bc[s][v].x : bc[s][v].y;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const double x = HA && part ? -ac[s][m] : ac[s][m];
          gd_mma(o.re[m][v], x, br);
          gd_mma(o.im[m][v], x, bi);
        }
      }
  };
  load(0, a[0], bb[0]);
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += 4 * KS) {
    load(k0 + 2 * KS, a[1], bb[1]);
    mul(a[0], bb[0]);
    if (k0 + 2 * KS >= n) break;
    load(k0 + 4 * KS, a[0], bb[0]);
    mul(a[1], bb[1]);
  }
}

// f(i, j, re, im) for the elements of a block that lie in the matrix.
template <class F>
__device__ __forceinline__ void block_each(int n, int i0, int j0, const Block16& o, F&& f) {
  const int lane = threadIdx.x % 32;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int i = i0 + 8 * m + (lane >> 2), j = j0 + 8 * v + 2 * (lane & 3) + c;
        if (i < n && j < n) f(i, j, o.re[m][v][c], o.im[m][v][c]);
      }
}

// t-th block on or above the diagonal of an nt x nt arrangement.
__device__ __forceinline__ void upper_block(int t, int nt, int& ti, int& tj) {
  ti = 0;
  while (t >= nt - ti) {
    t -= nt - ti;
    ++ti;
  }
  tj = ti + t;
}

// C = alpha A' B + dadd I, Hermitian by construction; returns max |C - I|
// over the elements this thread formed.
template <bool HA>
__device__ double product_herm(int n, int nt, int t, const double2* A, int lda, const double2* B, int ldb, double2* C,
                               int ldc, double alpha, double dadd) {
  int ti, tj;
  upper_block(t, nt, ti, tj);
  Block16 o;
  block_product<HA>(n, A, lda, B, ldb, ti * kTile, tj * kTile, o);
  double mx = 0.0;
  block_each(n, ti * kTile, tj * kTile, o, [&](int i, int j, double re, double im) {
    if (i > j) return;
    const double2 v = make_double2(alpha * re + (i == j ? dadd : 0.0), i == j ? 0.0 : alpha * im);
    C[(size_t)i * ldc + j] = v;
    if (i != j) C[(size_t)j * ldc + i] = make_double2(v.x, -v.y);
    mx = fmax(mx, hypot(v.x - (i == j ? 1.0 : 0.0), v.y));
  });
  return mx;
}

// Block t (row-major) of C = A' B.
template <bool HA>
__device__ void product_full(int n, int nt, int t, const double2* A, int lda, const double2* B, int ldb, double2* C,
                             int ldc) {
  const int i0 = (t / nt) * kTile, j0 = (t % nt) * kTile;
  Block16 o;
  block_product<HA>(n, A, lda, B, ldb, i0, j0, o);
  block_each(n, i0, j0, o, [&](int i, int j, double re, double im) { C[(size_t)i * ldc + j] = make_double2(re, im); });
}

// ------------------------------------------------- Loewdin by Newton-Schulz --
// S^-1/2 from the coupled Newton-Schulz iteration on A = S / c, with c the
// largest absolute row sum (so the spectrum of A lies in (0, 1]):
//   T = (3 I - Z Y) / 2,  Y <- Y T,  Z <- T Z,   Y -> A^1/2, Z -> A^-1/2.
// This is the matrix the reference forms as V diag(w^-1/2) V^H
// (static.py:470-480) whenever no eigenvalue of S falls below its floor
// max(1e-12, eps max(w) n); S is then positive definite with condition far
// from that floor.  All three are polynomials of S, so Hermitian.  The step
// at which max |T - I| over the isospin's block is below 1e-9 is the last: it
// squares that error to rounding.
constexpr int kNSMaxIt = 16;   // S is close to I after a gradient step: 4-6 steps in practice

struct LoewdinWork {
  double2 *Y[2], *Z[2], *T;
  double* slots;
};

__global__ void __launch_bounds__(kClThreads, 1) loewdin_kernel(LoewdinArgs a, LoewdinWork w) {
  const Place p = place();
  const int n = a.nper.v[p.b], ld = a.ld, nt = (n + kTile - 1) / kTile, nu = nt * (nt + 1) / 2;
  const size_t sm = (size_t)ld * ld;
  const double2* S = a.S + p.b * a.sS;
  double2* Y[2] = {w.Y[0] + p.b * sm, w.Y[1] + p.b * sm};
  double2* Z[2] = {w.Z[0] + p.b * sm, w.Z[1] + p.b * sm};
  double2* T = w.T + p.b * sm;
  double* slots = w.slots + p.b * 2 * kClMax;
  int turn = 0;
  const int lane = threadIdx.x % 32;
  double c[1] = {0.0};
  for (int i = p.warp; i < n; i += p.nwarp) {
    double rs = 0.0;
    for (int j = lane; j < n; j += 32) {
      const double2 v = S[(size_t)i * ld + j];
      rs += hypot(v.x, v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
    c[0] = fmax(c[0], rs);
  }
  for (int k = p.tid; k < n; k += p.nthr) a.sp_norm[a.off.v[p.b] + k] = S[(size_t)k * ld + k].x;
  cl_reduce<1, true>(p, c, slots, turn);
  const double ci = 1.0 / c[0];
  // first step: Z = I, so T needs no product and Z <- T
  double mx[1] = {0.0};
  for (int e = p.tid; e < n * n; e += p.nthr) {
    const int i = e / n, j = e % n;
    const size_t g = (size_t)i * ld + j;
    const double2 s = S[g];
    const double2 y = make_double2(s.x * ci, s.y * ci);
    const double2 t = make_double2((i == j ? 1.5 : 0.0) - 0.5 * y.x, -0.5 * y.y);
    Y[0][g] = y;
    T[g] = t;
    Z[1][g] = t;
    mx[0] = fmax(mx[0], hypot(t.x - (i == j ? 1.0 : 0.0), t.y));
  }
  int k = 0;
  bool done = false;
  for (;; ++k) {
    cl_reduce<1, true>(p, mx, slots, turn);
    done = mx[0] < 1e-9;
    const int cur = k & 1, nxt = cur ^ 1;
    // Y is not needed any more after the last step
    const int ny = done ? 0 : nu, nz = k == 0 ? 0 : nu;
    for (int t = p.warp; t < ny + nz; t += p.nwarp) {
      if (t < nz) product_herm<false>(n, nt, t, T, ld, Z[cur], ld, Z[nxt], ld, 1.0, 0.0);
      else product_herm<false>(n, nt, t - nz, Y[cur], ld, T, ld, Y[nxt], ld, 1.0, 0.0);
    }
    cl_sync();
    if (done || k + 1 == kNSMaxIt) break;
    mx[0] = 0.0;
    for (int t = p.warp; t < nu; t += p.nwarp)
      mx[0] = fmax(mx[0], product_herm<false>(n, nt, t, Z[nxt], ld, Y[nxt], ld, T, ld, -0.5, 1.5));
  }
  if (!done && p.tid == 0) latch_error(a.status, HFB_ERR_NO_CONVERGENCE);
  const double2* Zf = Z[(k & 1) ^ 1];
  const double sc = sqrt(ci);
  double2* U = a.U + p.b * sm;
  for (int e = p.tid; e < n * n; e += p.nthr) {
    const size_t g = (size_t)(e / n) * ld + e % n;
    const double2 v = __ldcg(Zf + g);
    U[g] = make_double2(v.x * sc, v.y * sc);
  }
}

// ------------------------------------------ Hermitian eigen refinement ----
// Eigenpairs of a Hermitian matrix that is already nearly diagonal in the
// current basis (lambda after a gradient step: the states are the previous
// eigenvectors), by the iterative refinement of Ogita and Aishima (Japan J.
// Indust. Appl. Math. 35, 2018; clustered eigenvalues: 36, 2019).  From X
// (start I):
//   R = I - X^H X,  S = X^H A X,  l_i = Re S_ii / (1 - Re R_ii),
//   d = 2 (||S - diag(l)||_F + ||A||_F ||R||_F),
//   E_ij = (S_ij + l_j R_ij) / (l_j - l_i)  if |l_i - l_j| > d,  R_ij / 2 else,
//   X <- X (I + E),
// quadratically convergent for the pairs separated by more than d.  The
// pairs the last step left coupled (Kramers pairs, accidental
// near-degeneracies) form clusters that are diagonalised exactly as small
// blocks of the final X^H A X; the eigenpairs are sorted ascending and
// accepted only if V^H A V is diagonal and V^H V = I to the requested
// accuracy.  When the refinement has not converged after kRefMaxIt steps, a
// cluster has more than kClusterMax members or the acceptance test fails,
// the fallback flags are set and the caller's Jacobi solver, gated on them,
// runs instead: the choice needs no host round trip.
constexpr int kRefMaxIt = 6;
constexpr int kClusterMax = 16;   // a j = 15/2 shell of a near-spherical nucleus
constexpr int kRefMaxN = 256;

struct RefineWork {
  double2 *Ah, *X0, *X1, *AX, *S, *R, *Q;   // [nb][ld][ld] each; Q [nb][ld][kClusterMax]
  double *ev, *slots;                       // [nb][ld], [12 kClMax]
  int* cinfo;                               // [nb][ld][4]
};

// The clusters of the sorted l (consecutive values closer than tau), each
// block of S diagonalised by serial cyclic Jacobi (one thread per cluster).
// Output per eigenpair P (sorted position of its cluster start s plus local
// index): ev[P] and cinfo[P] = (s, size, local, original index of sorted
// position P).  One CTA.
__device__ void refine_clusters(int n, int ld, const double2* S, const double* l, double tau, double2* Qb, double* ev,
                                int* ci, int* fallback) {
  __shared__ double dg[kRefMaxN];
  __shared__ int idx[kRefMaxN], cstart[kRefMaxN];
  for (int i = threadIdx.x; i < n; i += blockDim.x) dg[i] = l[i];
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int r = 0;
    for (int j = 0; j < n; ++j) r += (dg[j] < dg[i]) || (dg[j] == dg[i] && j < i);
    idx[r] = i;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int s0 = 0;
    for (int p = 0; p < n; ++p) {
      if (p > 0 && dg[idx[p]] - dg[idx[p - 1]] > tau) s0 = p;
      cstart[p] = s0;
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    if (cstart[p] != p) continue;            // one thread per cluster start
    int c = 1;
    while (p + c < n && cstart[p + c] == p) ++c;
    if (c > kClusterMax) {
      *fallback = 1;
      continue;
    }
    double2 a[kClusterMax][kClusterMax], q[kClusterMax][kClusterMax];
    double nrm = 0.0;
    for (int r = 0; r < c; ++r)
      for (int t = 0; t < c; ++t) {
        a[r][t] = __ldcg(S + (size_t)idx[p + r] * ld + idx[p + t]);
        q[r][t] = make_double2(r == t ? 1.0 : 0.0, 0.0);
        nrm += a[r][t].x * a[r][t].x + a[r][t].y * a[r][t].y;
      }
    nrm = sqrt(nrm);
    for (int sweep = 0; sweep < 40 && c > 1; ++sweep) {
      bool any = false;
      for (int r = 0; r < c; ++r)
        for (int t = r + 1; t < c; ++t) {
          const double2 apq = a[r][t];
          const double mag = hypot(apq.x, apq.y);
          if (mag <= 1e-300 || mag <= 2.220446049250313e-16 * 1e-2 * nrm) continue;
          any = true;
          const double app = a[r][r].x, aqq = a[t][t].x;
          const double theta = (aqq - app) / (2.0 * mag);
          double tt = 1.0 / (fabs(theta) + sqrt(theta * theta + 1.0));
          if (theta < 0.0) tt = -tt;
          const double cs = 1.0 / sqrt(tt * tt + 1.0), sn = tt * cs;
          // apq = mag e^{i phi}; G = [[cs, sn], [-sn e^{-i phi}, cs e^{-i phi}]] on (r, t)
          const double2 om = make_double2(apq.x / mag, -apq.y / mag);
          for (int u = 0; u < c; ++u) {          // A <- A G, Q <- Q G (columns r, t)
            const double2 x0 = a[u][r], x1 = cmul(a[u][t], om);
            a[u][r] = make_double2(cs * x0.x - sn * x1.x, cs * x0.y - sn * x1.y);
            a[u][t] = make_double2(sn * x0.x + cs * x1.x, sn * x0.y + cs * x1.y);
            const double2 y0 = q[u][r], y1 = cmul(q[u][t], om);
            q[u][r] = make_double2(cs * y0.x - sn * y1.x, cs * y0.y - sn * y1.y);
            q[u][t] = make_double2(sn * y0.x + cs * y1.x, sn * y0.y + cs * y1.y);
          }
          const double2 oc = make_double2(om.x, -om.y);
          for (int u = 0; u < c; ++u) {          // A <- G^H A (rows r, t)
            const double2 x0 = a[r][u], x1 = cmul(oc, a[t][u]);
            a[r][u] = make_double2(cs * x0.x - sn * x1.x, cs * x0.y - sn * x1.y);
            a[t][u] = make_double2(sn * x0.x + cs * x1.x, sn * x0.y + cs * x1.y);
          }
          a[r][t] = make_double2(0.0, 0.0);
          a[t][r] = make_double2(0.0, 0.0);
        }
      if (!any) break;
    }
    for (int k = 0; k < c; ++k) {
      ev[p + k] = a[k][k].x;
      int* cp = ci + (size_t)(p + k) * 4;
      cp[0] = p;
      cp[1] = c;
      cp[2] = k;
      for (int m = 0; m < c; ++m) Qb[(size_t)(p + m) * kClusterMax + k] = q[m][k];
    }
  }
  for (int p = threadIdx.x; p < n; p += blockDim.x) ci[(size_t)p * 4 + 3] = idx[p];
}

// Both matrices in one cluster: they share the number of steps and the
// choice of the solver.  (Solved apart, the two isospins of a nucleus changed
// solver at different iterations, which moves the bases of degenerate pairs
// and with them max |lambda_asym|, the step-size rule's measure.)
__global__ void __launch_bounds__(kClThreads, 1) refine_kernel(RefineArgs a, RefineWork w, int nb) {
  __shared__ double lam[2][kRefMaxN];
  __shared__ int opos[kRefMaxN];
  const Place p = place();
  const int ld = a.ld;
  const size_t sm = (size_t)ld * ld;
  int n[2], nt[2], nu[2];
  int full = 0, upper = 0;     // blocks of all matrices
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    n[b] = b < nb ? a.nper.v[b] : 0;
    nt[b] = (n[b] + kTile - 1) / kTile;
    nu[b] = nt[b] * (nt[b] + 1) / 2;
    full += nt[b] * nt[b];
    upper += nu[b];
  }
  double* slots = w.slots;
  int turn = 0, turn4 = 0;
  // C = A' B on all blocks / on the upper blocks of all matrices
  auto each_full = [&](auto&& f) {
    for (int t = p.warp; t < full; t += p.nwarp) {
      const int b = t >= nt[0] * nt[0];
      f(b, b ? t - nt[0] * nt[0] : t);
    }
  };
  auto each_upper = [&](int first, auto&& f) {
    for (int t = p.warp; t < first + upper; t += p.nwarp) {
      if (t < first) continue;
      const int u = t - first, b = u >= nu[0];
      f(b, b ? u - nu[0] : u);
    }
  };
  auto gram = [&](const double2* X, double2* R, int first) {   // R = I - X^H X
    each_upper(first, [&](int b, int t) {
      product_herm<true>(n[b], nt[b], t, X + b * sm, ld, X + b * sm, ld, R + b * sm, ld, -1.0, 1.0);
    });
  };
  auto times_a = [&](const double2* X, size_t sX, double2* AX) {
    each_full([&](int b, int t) { product_full<false>(n[b], nt[b], t, w.Ah + b * sm, ld, X + b * sX, ld, AX + b * sm, ld); });
  };
  auto rotated = [&](const double2* X, size_t sX, const double2* AX, double2* S) {
    each_upper(0, [&](int b, int t) {
      product_herm<true>(n[b], nt[b], t, X + b * sX, ld, AX + b * sm, ld, S + b * sm, ld, 1.0, 0.0);
    });
  };
  if (p.tid < nb) a.fallback[p.tid] = 0;
  // A = the Hermitian matrix of the lower triangle (the diagonal's imaginary
  // part dropped, as eigh with UPLO='L')
  double f2[2] = {0.0, 0.0};
  for (int b = 0; b < nb; ++b) {
    const double2* A0 = a.A + b * a.sA;
    for (int e = p.tid; e < n[b] * n[b]; e += p.nthr) {
      const int i = e / n[b], j = e % n[b];
      double2 v = i >= j ? A0[(size_t)i * ld + j] : A0[(size_t)j * ld + i];
      if (i < j) v.y = -v.y;
      if (i == j) v.y = 0.0;
      w.Ah[b * sm + (size_t)i * ld + j] = v;
      f2[b] += v.x * v.x + v.y * v.y;
    }
  }
  cl_reduce<2, false>(p, f2, slots, turn);
  const double an[2] = {sqrt(f2[0]), sqrt(f2[1])};
  // Step k: X[k & 1] -> X[1 - (k & 1)].  The first one starts from X = I, so
  // S = A and R = 0 without a product and X <- I + E.
  double2* X[2] = {w.X0, w.X1};
  int k = 0;
  bool conv = false;
  double d[2] = {0.0, 0.0};
  for (; k < kRefMaxIt; ++k) {
    const double2* Xc = X[k & 1];
    double2* Xn = X[(k & 1) ^ 1];
    const double2* Sk = k == 0 ? w.Ah : w.S;
    if (k > 0) {
      times_a(Xc, sm, w.AX);
      gram(Xc, w.R, full % p.nwarp);
      cl_sync();
      rotated(Xc, sm, w.AX, w.S);
      cl_sync();
    }
    auto rk = [&](size_t g) { return k == 0 ? make_double2(0.0, 0.0) : __ldcg(w.R + g); };
    double o2[2] = {0.0, 0.0}, r2[2] = {0.0, 0.0}, nc2[2] = {0.0, 0.0};
    for (int b = 0; b < nb; ++b)
      for (int i = threadIdx.x; i < n[b]; i += blockDim.x) {
        const size_t g = b * sm + (size_t)i * ld + i;
        lam[b][i] = __ldcg(Sk + g).x / (1.0 - rk(g).x);
      }
    __syncthreads();
    for (int b = 0; b < nb; ++b)
      for (int e = p.tid; e < n[b] * n[b]; e += p.nthr) {
        const int i = e / n[b], j = e % n[b];
        const size_t g = b * sm + (size_t)i * ld + j;
        const double2 sv = __ldcg(Sk + g), rv = rk(g);
        const double dx = i == j ? sv.x - lam[b][i] : sv.x;
        o2[b] += dx * dx + sv.y * sv.y;
        r2[b] += rv.x * rv.x + rv.y * rv.y;
      }
    double s4[4] = {o2[0], o2[1], r2[0], r2[1]};
    cl_reduce<4, false>(p, s4, slots + 4 * kClMax, turn4);
    conv = true;
#pragma unroll
    for (int b = 0; b < 2; ++b) d[b] = 2.0 * (sqrt(s4[b]) + an[b] * sqrt(s4[2 + b]));
    // I + E goes where A X was (k > 0), or is X itself
    double2* E = k == 0 ? Xn : w.AX;
    for (int b = 0; b < nb; ++b)
      for (int e = p.tid; e < n[b] * n[b]; e += p.nthr) {
        const int i = e / n[b], j = e % n[b];
        const size_t g = b * sm + (size_t)i * ld + j;
        const double2 sv = __ldcg(Sk + g), rv = rk(g);
        double2 ev;
        if (i == j) {
          ev = make_double2(1.0 + 0.5 * rv.x, 0.5 * rv.y);
        } else if (fabs(lam[b][i] - lam[b][j]) > d[b]) {
          const double den = lam[b][j] - lam[b][i];
          ev = make_double2((sv.x + lam[b][j] * rv.x) / den, (sv.y + lam[b][j] * rv.y) / den);
          nc2[b] += sv.x * sv.x + sv.y * sv.y;
        } else {
          ev = make_double2(0.5 * rv.x, 0.5 * rv.y);
        }
        E[g] = ev;
      }
    cl_reduce<2, false>(p, nc2, slots, turn);
    // ||I - X^H X||_F cannot go below the rounding of the n-term sums
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (b < nb) conv = conv && sqrt(nc2[b]) <= a.tol * an[b] && sqrt(s4[2 + b]) <= fmax(a.tol, 1e-11);
    if (k > 0) {
      each_full([&](int b, int t) {
        product_full<false>(n[b], nt[b], t, Xc + b * sm, ld, w.AX + b * sm, ld, Xn + b * sm, ld);
      });
      cl_sync();
    }
    if (conv) break;
  }
  if (!conv) {
    if (p.tid < nb) a.fallback[p.tid] = 1;
    return;
  }
  const double2* Xf = X[(k & 1) ^ 1];
  times_a(Xf, sm, w.AX);
  cl_sync();
  rotated(Xf, sm, w.AX, w.S);
  cl_sync();
  if (p.rank < nb) {
    const int b = p.rank;
    refine_clusters(n[b], ld, w.S + b * sm, lam[b], d[b], w.Q + (size_t)b * ld * kClusterMax, w.ev + (size_t)b * ld,
                    w.cinfo + (size_t)b * ld * 4, a.fallback);
  }
  if (nb > 1 && p.size == 1) {
    __syncthreads();
    refine_clusters(n[1], ld, w.S + sm, lam[1], d[1], w.Q + (size_t)ld * kClusterMax, w.ev + ld, w.cinfo + (size_t)ld * 4,
                    a.fallback);
  }
  cl_sync();
  if (__ldcg(a.fallback)) {
    if (p.tid < nb) a.fallback[p.tid] = 1;
    return;
  }
  // V[:, o(P)] = sum_m Xf[:, idx[s + m]] Q[s + m][l], w[o(P)] = ev[P], with o
  // the ascending order of ev (ties by P)
  for (int b = 0; b < nb; ++b) {
    const double* ev = w.ev + (size_t)b * ld;
    const int* ci = w.cinfo + (size_t)b * ld * 4;
    const double2 *Qb = w.Q + (size_t)b * ld * kClusterMax, *Xb = Xf + b * sm;
    double* W = a.W + b * a.sW;
    double2* V = a.V + b * a.sV;
    __syncthreads();
    for (int P = threadIdx.x; P < n[b]; P += blockDim.x) {
      int r = 0;
      const double e = __ldcg(ev + P);
      for (int q = 0; q < n[b]; ++q) {
        const double eq = __ldcg(ev + q);
        r += (eq < e) || (eq == e && q < P);
      }
      opos[P] = r;
      if (p.rank == 0) W[r] = e;
    }
    __syncthreads();
    for (int e = p.tid; e < n[b] * n[b]; e += p.nthr) {
      const int row = e / n[b], P = e % n[b];
      const int s0 = __ldcg(ci + P * 4), c = __ldcg(ci + P * 4 + 1), l = __ldcg(ci + P * 4 + 2);
      double re = 0.0, im = 0.0;
      for (int m = 0; m < c; ++m) {
        const int col = __ldcg(ci + (s0 + m) * 4 + 3);
        const double2 x = __ldcg(Xb + (size_t)row * ld + col), q = __ldcg(Qb + (size_t)(s0 + m) * kClusterMax + l);
        re += x.x * q.x - x.y * q.y;
        im += x.x * q.y + x.y * q.x;
      }
      V[(size_t)row * ld + opos[P]] = make_double2(re, im);
    }
  }
  cl_sync();
  // acceptance: with S = V^H A V and R = I - V^H V, no off-diagonal |S_ij| or
  // diagonal |S_ii - w_i| above tol_s ||A||_F and no |R_ij| above tol_s
  times_a(a.V, a.sV, w.AX);
  each_upper(full % p.nwarp, [&](int b, int t) {
    product_herm<true>(n[b], nt[b], t, a.V + b * a.sV, ld, a.V + b * a.sV, ld, w.R + b * sm, ld, -1.0, 1.0);
  });
  cl_sync();
  rotated(a.V, a.sV, w.AX, w.S);
  cl_sync();
  const double tol_s = fmax(1e3 * a.tol, 1e-11);
  int bad = 0;
  for (int b = 0; b < nb; ++b)
    for (int e = p.tid; e < n[b] * n[b]; e += p.nthr) {
      const int i = e / n[b], j = e % n[b];
      const size_t g = b * sm + (size_t)i * ld + j;
      double2 sv = __ldcg(w.S + g);
      if (i == j) sv.x -= __ldcg(a.W + b * a.sW + i);
      const double2 rv = __ldcg(w.R + g);
      if (!(hypot(sv.x, sv.y) <= tol_s * an[b]) || !(hypot(rv.x, rv.y) <= tol_s)) bad = 1;
    }
  if (bad)
    for (int b = 0; b < nb; ++b) a.fallback[b] = 1;
}

// ------------------------------------------------- construct_hfb_matrices --
// U = S^-1/2 V (or S^-1/2), H = U^H H_old U and G likewise, lambda and the
// outputs of static.py:511-575, and L = U lambda for the Lagrange fields.
// With tbcs only the diagonal of G is kept (static.py:542-544).
struct ConstructWork {
  double2 *TH, *TG;
  double* slots;
};

__global__ void __launch_bounds__(kClThreads, 1) construct_kernel(ConstructArgs a, ConstructWork w) {
  const Place p = place();
  const int n = a.nper.v[p.b], o = a.off.v[p.b], ld = a.ld, nmax = a.nmax;
  const int nt = (n + kTile - 1) / kTile, nu = nt * (nt + 1) / 2;
  const size_t sm = (size_t)ld * ld, mm = (size_t)p.b * nmax * nmax;
  const double2* Ur = a.Ur + p.b * sm;
  double2* U = a.U + p.b * sm;
  int turn = 0;
  if (a.diagonalize) {
    for (int t = p.warp; t < nt * nt; t += p.nwarp)
      product_full<false>(n, nt, t, Ur, ld, a.Vl + p.b * sm, ld, U, ld);
  } else {
    for (int e = p.tid; e < n * n; e += p.nthr) {
      const size_t g = (size_t)(e / n) * ld + e % n;
      U[g] = Ur[g];
    }
  }
  cl_sync();
  if (a.construct) {
    double2 *TH = w.TH + p.b * sm, *TG = w.TG + p.b * sm;
    const int nfull = nt * nt;
    for (int t = p.warp; t < (a.ipair ? 2 : 1) * nfull; t += p.nwarp) {
      if (t < nfull) product_full<false>(n, nt, t, a.H + p.b * a.sG, ld, U, ld, TH, ld);
      else product_full<false>(n, nt, t - nfull, a.G + p.b * a.sG, ld, U, ld, TG, ld);
    }
    cl_sync();
    double mx[1] = {0.0}, s2[1] = {0.0};
    for (int t = p.warp; t < nu; t += p.nwarp) {
      int ti, tj;
      upper_block(t, nt, ti, tj);
      Block16 h, g;
      block_product<true>(n, U, ld, TH, ld, ti * kTile, tj * kTile, h);
      const bool have_g = a.ipair && (!a.tbcs || ti == tj);
      if (have_g) block_product<true>(n, U, ld, TG, ld, ti * kTile, tj * kTile, g);
      const int lane = threadIdx.x % 32;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int v = 0; v < 2; ++v)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int i = ti * kTile + 8 * m + (lane >> 2), j = tj * kTile + 8 * v + 2 * (lane & 3) + c;
            if (i > j || j >= n) continue;
            const double hr = h.re[m][v][c], hi = i == j ? 0.0 : h.im[m][v][c];
            const bool keep = have_g && (!a.tbcs || i == j);
            const double gr = keep ? g.re[m][v][c] : 0.0, gi = keep && i != j ? g.im[m][v][c] : 0.0;
            // lambda_ij = w_j h_ij - u_j g_ij; its symmetric and antisymmetric parts
            const double wi = a.wocc[o + i] * a.wstates[o + i], wj = a.wocc[o + j] * a.wstates[o + j];
            const double ui = a.wguv[o + i] * a.pairwg[o + i] * a.wstates[o + i];
            const double uj = a.wguv[o + j] * a.pairwg[o + j] * a.wstates[o + j];
            const double2 l = make_double2(wj * hr - uj * gr, wj * hi - uj * gi);
            const double2 lt = make_double2(wi * hr - ui * gr, wi * hi - ui * gi);   // conj(lambda_ji)
            const double2 as = make_double2(0.5 * (l.x - lt.x), 0.5 * (l.y - lt.y));
            const double2 sy = make_double2(0.5 * (l.x + lt.x), 0.5 * (l.y + lt.y));
            const size_t e = mm + (size_t)i * nmax + j, et = mm + (size_t)j * nmax + i;
            a.hmat[e] = make_double2(hr, hi);
            a.gmat[e] = make_double2(gr, gi);
            a.symc[e] = as;
            a.lsave[e] = sy;
            if (i != j) {
              a.hmat[et] = make_double2(hr, -hi);
              a.gmat[et] = make_double2(gr, -gi);
              a.symc[et] = make_double2(-as.x, as.y);
              a.lsave[et] = make_double2(sy.x, -sy.y);
            } else {
              a.sp_energy[o + i] = hr;
              if (a.ipair) a.deltaf[o + i] = gr * a.pairwg[o + i];
            }
            const double ab = hypot(as.x, as.y);
            mx[0] = fmax(mx[0], ab);
            s2[0] += (i == j ? 1.0 : 2.0) * ab * ab;
          }
    }
    double* slots = w.slots + p.b * 4 * kClMax;
    cl_reduce<1, true>(p, mx, slots, turn);
    turn = 0;
    cl_reduce<1, false>(p, s2, slots + 2 * kClMax, turn);
    if (p.tid == 0) {
      a.efluct[p.b] = mx[0];
      a.efluct[2 + p.b] = sqrt(s2[0] / ((double)n * n));
    }
  }
  for (int t = p.warp; t < nt * nt; t += p.nwarp)
    product_full<false>(n, nt, t, U, ld, a.lsave + mm, nmax, a.L + p.b * sm, ld);
}

// CTAs per matrix: one warp per output block of the largest product phase
// and no more than one such warp on each of an SM's four tensor pipes, as
// far as a portable cluster goes (n = 10: 1 CTA, 32: 2, 48: 4, 61: 8).
int cluster_size(int n, int most = 8) {
  const int nt = (n + kTile - 1) / kTile;
  int c = 1;
  while (c < most && c * 4 < nt * (nt + 1)) c *= 2;
  return c;
}

// ``begun`` (optional) is recorded once every CTA of the launch runs.
template <class... KA, class... A>
int cluster_launch(void (*kern)(KA...), int nb, int size, cudaEvent_t begun, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(nb * size));
  cfg.blockDim = dim3(kClThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (begun) {
    at[1].id = cudaLaunchAttributeLaunchCompletionEvent;
    at[1].val.launchCompletionEvent.event = begun;
    at[1].val.launchCompletionEvent.flags = 0;
    cfg.numAttrs = 2;
  }
  count_launch();
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    note_cuda_error((int)e);
    return HFB_ERR_CUDA;
  }
  return HFB_OK;
}

int max2(Pair2 n) { return n.v[0] > n.v[1] ? n.v[0] : n.v[1]; }

}  // namespace

size_t loewdin_bytes(int ld) { return sizeof(double2) * 2 * 5 * (size_t)ld * ld + sizeof(double) * 4 * kClMax; }

int loewdin_launch(const LoewdinArgs& a, void* work, bool alone, cudaStream_t st) {
  const size_t sm = 2 * (size_t)a.ld * a.ld;
  double2* m = (double2*)work;
  LoewdinWork w;
  w.Y[0] = m; w.Y[1] = m + sm; w.Z[0] = m + 2 * sm; w.Z[1] = m + 3 * sm; w.T = m + 4 * sm;
  w.slots = (double*)(m + 5 * sm);
  return cluster_launch(loewdin_kernel, 2, alone ? cluster_size(max2(a.nper)) : 1, nullptr, st, a, w);
}

size_t refine_bytes(int nb, int ld) {
  return sizeof(double2) * (6 * (size_t)nb * ld * ld + (size_t)nb * ld * kClusterMax) +
         sizeof(double) * ((size_t)nb * ld + 12 * kClMax) + sizeof(int) * (size_t)nb * ld * 4;
}

// Largest cluster of the refinement on the context's device: 16 CTAs, which the
// kernel has to be allowed on each device, or 8 where those are refused or no
// 16 SMs of a cluster are free to the process.  Asked once per context.
static int refine_widest(hfb_ctx_s* c) {
  if (c->refine_ctas) return c->refine_ctas;
  c->refine_ctas = 8;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kClMax;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(kClMax);
  cfg.blockDim = dim3(kClThreads);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int places = 0;
  if (cudaFuncSetAttribute(refine_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&places, refine_kernel, &cfg) != cudaSuccess)
    cudaGetLastError();
  else if (places > 0)
    c->refine_ctas = kClMax;
  return c->refine_ctas;
}

int refine_launch(hfb_ctx_s* c, int nb, const RefineArgs& a, void* work, cudaEvent_t begun, cudaStream_t st) {
  if (a.ld > kRefMaxN) return HFB_ERR_UNSUPPORTED_GRID;
  const size_t sm = (size_t)nb * a.ld * a.ld;
  double2* m = (double2*)work;
  RefineWork w;
  w.Ah = m; w.X0 = m + sm; w.X1 = m + 2 * sm; w.AX = m + 3 * sm; w.S = m + 4 * sm; w.R = m + 5 * sm;
  w.Q = m + 6 * sm;
  double* d = (double*)(w.Q + (size_t)nb * a.ld * kClusterMax);
  w.ev = d; w.slots = d + (size_t)nb * a.ld;
  w.cinfo = (int*)(w.slots + 12 * kClMax);
  const int n = nb > 1 ? max2(a.nper) : a.nper.v[0];
  int size = cluster_size(n, kClMax);
  if (size > 8) size = refine_widest(c);
  return cluster_launch(refine_kernel, 1, size, begun, st, a, w, nb);
}

size_t construct_bytes(int ld) { return sizeof(double2) * 2 * 2 * (size_t)ld * ld + sizeof(double) * 2 * 4 * kClMax; }

int construct_launch(const ConstructArgs& a, void* work, cudaStream_t st) {
  const size_t sm = 2 * (size_t)a.ld * a.ld;
  ConstructWork w;
  w.TH = (double2*)work;
  w.TG = w.TH + sm;
  w.slots = (double*)(w.TG + sm);
  return cluster_launch(construct_kernel, 2, cluster_size(max2(a.nper)), nullptr, st, a, w);
}

}  // namespace hfb
