// Diagonalisation step: diagstep (static.py:261-461), loewdin_orthonormalize
// (463-482) and construct_hfb_matrices (484-577).
//
//  * Gram contractions C_a = wxyz Psi^H X_a (X = psi, hampsi, hmfpsi,
//    v_pair psi) over K = 2 n^3: one launch over the output tiles of all
//    requested matrices; split-K partials are summed in a fixed order.  On the
//    tensor cores in gram_tc.cu (FP32) and contract_f64.cu (FP64); the kernel on
//    CUDA cores here serves what those do not.
//  * Hermitian eigensolver: cyclic two-sided Jacobi in one CTA on the folded
//    lower triangle held in shared memory (round-robin ordering, n/2 disjoint
//    rotations per round); the rotations are recorded and replayed onto the
//    eigenvector matrix by a row-parallel kernel.  Eigenvalues ascending.
//  * the small-matrix chains (S^-1/2, eigen refinement, U^H H U, U lambda) as
//    one cluster launch each (diag_cluster.cu).
//  * rotation [psi_new | lagrange] = psi [U | U lambda_sym] as one GEMM pass.
#include <math.h>
#include "diag.cuh"

namespace hfb {

// ================================================================ Gram ====
// C = wxyz Psi^H X for X in {psi, hampsi, hmfpsi, v_pair psi} (mask bits 0-3)
// over K = 2 n^3.  Work is a list of 48 x 48 output tiles, one matrix per
// tile; S, H and G are Hermitian (Gram matrices of one set of vectors, h
// and v_pair Hermitian) so only tiles with ti <= tj are computed and the
// reduction mirrors them.  Split-K partials are summed in a fixed order.
// 48-state tiles keep the padding of the usual neutron/proton counts small
// (140 -> 144, 96 -> 96); 192 threads (16 x 12) hold 4 x 3 outputs each.
constexpr int GT = 48;        // tile edge (states)
constexpr int GKS = 8;        // k per shared-memory stage
constexpr int GCHUNK = 8192;  // k per split-K chunk (at most; shorter when the grid would be small)
constexpr int GTHREADS = 192;
constexpr int kGramMaxTiles = 160;

struct GramTile {
  unsigned char b, a, ti, tj;   // block (isospin), matrix, tile row, tile column
};
struct GramJob {
  int ntile;
  GramTile t[kGramMaxTiles];
  int s0[2], ns[2];              // state range of each block
  const double* vp[2];           // v_pair for each block (X = v psi)
  int herm_mask;                 // matrices computed on upper tiles only
};

template <class R>
__global__ void __launch_bounds__(GTHREADS)
gram_kernel(GramJob job, size_t K, size_t n3, const cplx<R>* __restrict__ psi, const cplx<R>* __restrict__ hampsi,
            const cplx<R>* __restrict__ hmfpsi, double2* part, int nchunk, int kchunk) {
  using Z = cplx<R>;
  __shared__ Z As[2][GKS][GT + 1];
  __shared__ Z Bs[2][GKS][GT + 1];
  const GramTile tl = job.t[blockIdx.x];
  const int b = tl.b, am = tl.a;
  const int ns = job.ns[b];
  const int i0 = tl.ti * GT, j0 = tl.tj * GT;
  const cplx<R>* P = psi + (size_t)job.s0[b] * K;
  const cplx<R>* X = am == 1 ? hampsi + (size_t)job.s0[b] * K : am == 2 ? hmfpsi + (size_t)job.s0[b] * K : P;
  const double* vp = job.vp[b];
  const size_t k0 = (size_t)blockIdx.y * kchunk;
  const size_t k1 = min(K, k0 + (size_t)kchunk);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;   // rows ty + 12 u, columns tx + 16 v
  R acc[4][3][2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 3; ++v) acc[u][v][0] = acc[u][v][1] = R(0);
  // loader: 48 states x 8 k per operand = 384 elements, two per thread
  auto load = [&](int buf, size_t kb) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = threadIdx.x + GTHREADS * h;
      const int st_ = e / GKS, kk = e % GKS;
      const size_t k = kb + kk;
      const bool okk = k < k1;
      const int gi = i0 + st_, gj = j0 + st_;
      As[buf][kk][st_] = (okk && gi < ns) ? P[(size_t)gi * K + k] : czero<Z>();
      Z v = czero<Z>();
      if (okk && gj < ns) {
        v = X[(size_t)gj * K + k];
        if (am == 3) v = (R)vp[k % n3] * v;
      }
      Bs[buf][kk][st_] = v;
    }
  };
  load(0, k0);
  __syncthreads();
  int buf = 0;
  for (size_t kb = k0; kb < k1; kb += GKS) {
    if (kb + GKS < k1) load(buf ^ 1, kb + GKS);
#pragma unroll
    for (int kk = 0; kk < GKS; ++kk) {
      Z av[4], bv[3];
#pragma unroll
      for (int u = 0; u < 4; ++u) av[u] = As[buf][kk][ty + 12 * u];
#pragma unroll
      for (int v = 0; v < 3; ++v) bv[v] = Bs[buf][kk][tx + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          // conj(a) * b
          acc[u][v][0] += av[u].x * bv[v].x + av[u].y * bv[v].y;
          acc[u][v][1] += av[u].x * bv[v].y - av[u].y * bv[v].x;
        }
    }
    __syncthreads();
    buf ^= 1;
  }
  double2* o = part + ((size_t)blockIdx.x * nchunk + blockIdx.y) * GT * GT;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 3; ++v)
      o[(ty + 12 * u) * GT + tx + 16 * v] = make_double2((double)acc[u][v][0], (double)acc[u][v][1]);
}

struct GramOut {
  double2* p[8];   // [block * 4 + matrix]
};

// out_a[b][i][j] = wxyz * sum over chunks (fixed order); Hermitian matrices
// take the lower triangle from the upper one.
__global__ void gram_reduce_kernel(GramJob job, int nchunk, const double2* part, double scale, GramOut outs,
                                   int ldo) {
  const int t = blockIdx.y;
  const GramTile tl = job.t[t];
  const int b = tl.b, am = tl.a;
  const int ns = job.ns[b];
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= GT * GT) return;
  const int li = e / GT, lj = e % GT;
  const int i = tl.ti * GT + li, j = tl.tj * GT + lj;
  if (i >= ns || j >= ns) return;
  double re = 0, im = 0;
  const double2* p = part + (size_t)t * nchunk * GT * GT + e;
  for (int c = 0; c < nchunk; ++c) {
    const double2 v = p[(size_t)c * GT * GT];
    re += v.x;
    im += v.y;
  }
  double2* out = outs.p[b * 4 + am];
  const bool herm = (job.herm_mask >> am) & 1;
  if (herm && i > j) return;           // written from the mirrored element below
  out[(size_t)i * ldo + j] = make_double2(scale * re, scale * im);
  if (herm && i != j) out[(size_t)j * ldo + i] = make_double2(scale * re, -scale * im);
}

int gram_tc_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const int* masks, const void* psi,
                   const void* hampsi, const void* hmfpsi, const double* const* vp, double wxyz,
                   double2* const* outs_host, int ldo, int leave, cudaStream_t st);   // gram_tc.cu

// One launch for the requested matrices of up to two state blocks.
// outs[b * 4 + a] receives matrix a of block b (leading dimension ldo); the
// tensor-core launches stay off ``leave`` SMs.

int gram_launch(hfb_ctx_s* c, int prec, int nblk, const int* s0, const int* ns, const int* masks, const void* psi,
                const void* hampsi, const void* hmfpsi, const double* const* vp, double wxyz, double2* const* outs_host,
                int ldo, cudaStream_t st, int leave = 0) {
  // single precision: tensor cores (three-term tf32) unless disabled for this context
  if (prec != HFB_F64 && c->use_tcgen05) {
    const int r = gram_tc_launch(c, nblk, s0, ns, masks, psi, hampsi, hmfpsi, vp, wxyz, outs_host, ldo, leave, st);
    if (r != HFB_ERR_UNSUPPORTED_GRID) return r;
  }
  const size_t n3 = (size_t)c->n * c->n * c->n, K = 2 * n3;
  int kchunk = GCHUNK;   // set below from the tile count
  GramJob job{};
  job.herm_mask = 1 | 4 | 8;
  for (int b = 0; b < nblk; ++b) {
    job.s0[b] = s0[b];
    job.ns[b] = ns[b];
    job.vp[b] = vp ? vp[b] : nullptr;
    const int nt = (ns[b] + GT - 1) / GT;
    for (int a = 0; a < 4; ++a) {
      if (!(masks[b] & (1 << a)) || ns[b] <= 0) continue;
      const bool herm = (job.herm_mask >> a) & 1;
      for (int ti = 0; ti < nt; ++ti)
        for (int tj = herm ? ti : 0; tj < nt; ++tj) {
          if (job.ntile >= kGramMaxTiles) return HFB_ERR_ARG;
          job.t[job.ntile++] = GramTile{(unsigned char)b, (unsigned char)a, (unsigned char)ti, (unsigned char)tj};
        }
    }
  }
  if (job.ntile == 0) return HFB_OK;
  if (prec == HFB_F64 && c->f64_mma)
    return gram_f64_launch(c, nblk, s0, ns, masks, psi, hampsi, hmfpsi, vp, wxyz, outs_host, ldo, leave, st);
  // split K so that the grid has about two CTAs per SM even for few tiles
  // and short K (small grids): chunks a multiple of 64 elements, at most
  // GCHUNK
  {
    const size_t want = (size_t)(2 * 148 + job.ntile - 1) / job.ntile;
    size_t kc = (K + want - 1) / want;
    kc = (kc + 63) / 64 * 64;
    if (kc < 256) kc = 256;
    if (kc > (size_t)GCHUNK) kc = GCHUNK;
    kchunk = (int)kc;
  }
  const int nchunk = (int)((K + kchunk - 1) / kchunk);
  double2* part = (double2*)scratch(c, hfb_ctx_s::S_GRAM, sizeof(double2) * (size_t)job.ntile * nchunk * GT * GT);
  if (!part) return HFB_ERR_ALLOC;
  GramOut ot;
  for (int q = 0; q < 8; ++q) ot.p[q] = outs_host[q];
  dim3 grid(job.ntile, nchunk);
  if (prec == HFB_F64)
    gram_kernel<double><<<grid, GTHREADS, 0, st>>>(job, K, n3, (const double2*)psi, (const double2*)hampsi,
                                              (const double2*)hmfpsi, part, nchunk, kchunk);
  else
    gram_kernel<float><<<grid, GTHREADS, 0, st>>>(job, K, n3, (const float2*)psi, (const float2*)hampsi,
                                             (const float2*)hmfpsi, part, nchunk, kchunk);
  HFB_CHECK_LAUNCH();
  dim3 g2((GT * GT + 255) / 256, job.ntile);
  gram_reduce_kernel<<<g2, 256, 0, st>>>(job, nchunk, part, wxyz, ot, ldo);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

// ============================================================== Jacobi ====
// The strict lower triangle of a Hermitian matrix of even size m folded into
// m - 1 rows of h = m / 2: columns l < h below one another, the rest of the
// triangle transposed into the corner that they leave free.  Walks along rows
// and along columns are contiguous or ``ld`` apart (odd where it fits), so the
// lanes of a warp fall on distinct banks; packed row by row, column walks
// collided.
struct Folded {
  double2* p;
  int h, ld;
  __device__ __forceinline__ double2& at(int k, int l) const {   // k > l
    return l < h ? p[(k - 1) * ld + l] : p[(l - h) * ld + k - h];
  }
  __device__ __forceinline__ double2 get(int k, int l) const {
    if (k > l) return at(k, l);
    const double2 v = at(l, k);
    return make_double2(v.x, -v.y);
  }
  __device__ __forceinline__ void set(int k, int l, double2 v) const {
    if (k > l) at(k, l) = v;
    else at(l, k) = make_double2(v.x, -v.y);
  }
};
// Row and column of entry e of a packed lower triangle with its diagonal.
__device__ __forceinline__ void unpack_lower(int e, int& k, int& l) {
  k = (int)((sqrt(8.0 * e + 1.0) - 1.0) / 2.0);
  while (k * (k + 1) / 2 > e) --k;
  while ((k + 1) * (k + 2) / 2 <= e) ++k;
  l = e - k * (k + 1) / 2;
}

// Round-robin tournament: round r < m - 1 (m even), pair index q < m / 2.
__device__ __forceinline__ void rr_pair(int m, int r, int q, int& a, int& b) {
  a = r + q;
  b = q == 0 ? m - 1 : r + m - 1 - q;
  if (a >= m - 1) a -= m - 1;
  if (q != 0 && b >= m - 1) b -= m - 1;
  if (a > b) { int t = a; a = b; b = t; }
}

struct JacRot {
  double cs, sn;   // sn == 0: the identity
  double2 om;      // exp(-i phi)
};

constexpr int kJacMaxSweeps = 40;
constexpr int kEighMax = 4;     // matrices per batched launch
constexpr int kJacThreads = 1024, kJacSmall = 512;
constexpr int kJacBlk = 4;      // 2x2 blocks per thread: 84 * 85 / 2 over 928 threads
constexpr int kJacMaxN = 168;   // what shared memory holds
constexpr int kJacAhead = 32;   // pairs from which a round's rotations are computed in the round before

// One batched solve: up to kEighMax independent matrices, one CTA each.
struct EighBatch {
  int nb;
  int n[kEighMax];
  int lda[kEighMax];
  const double2* a[kEighMax];
  double* w[kEighMax];
  double2* v[kEighMax];
  int vblk0[kEighMax + 1];     // prefix of row blocks for the vector replay
  int* sweeps;                 // optional device output [nb]: sweeps used
  double tol_rel;              // off-diagonal threshold relative to ||A||_F (0: double eps)
  int stage_half;              // rotations per round in the replay's staging buffer (set by eigh_batch)
  const int* gate;             // optional device flags [nb]: matrix b is solved only when gate[b] != 0
};

// One CTA per matrix: cyclic two-sided Jacobi on the folded lower triangle and
// the diagonal.  Each round applies n/2 disjoint rotations (round-robin
// pairing) as updates of the 2x2 blocks (pair q1 rows x pair q2 columns, q1 >
// q2), and skips a block when both of its rotations are the identity.  A
// round's own latency is its rotations (hypot, roots and quotients one after
// the other, for one pair per thread), so from kJacAhead pairs on the first
// warps compute the next round's behind the update: the elements that pair up next lie in blocks
// (1, 0), (q + 1, q - 1) and (half - 1, half - 2), which these warps update
// first.  With fewer pairs the update is as short as that part of it.  The
// other threads own fixed blocks for the whole solve.  Rotations are recorded for
// the eigenvector replay.  Lambda of Pb208 (140 + 96 states): 2.46 ms with
// the rotations between two block barriers, 1.88 ms here (single-precision
// threshold 1.51, 1.20).
// TH: the block's largest size (up to kJacSmall threads the loop keeps out of
// local memory: 32 + 32 states 150 us against 172).
template <int TH>
__global__ void __launch_bounds__(TH)
jacobi_kernel(EighBatch eb, JacRot* rot, int* nrounds_out, int* status, size_t rot_stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int b = blockIdx.x;
  if (eb.gate && eb.gate[b] == 0) return;
  const int n = eb.n[b], lda = eb.lda[b];
  const int m = n + (n & 1);   // pad odd sizes with a decoupled index
  const int half = m / 2;
  const Folded a{reinterpret_cast<double2*>(smem_raw), half, m == kJacMaxN ? half : half | 1};
  double2* rcs = a.p + (size_t)(m - 1) * a.ld;                 // (cs, sn) [2][half], by the round's parity
  double2* rom = rcs + 2 * half;                               // om
  double* dg = reinterpret_cast<double*>(rom + 2 * half);      // diagonal
  const bool ahead = half >= kJacAhead;
  __shared__ int any_rot;
  __shared__ int round_rot[2];   // a rotation in round r (parity r & 1)
  const double2* Ab = eb.a[b];
  JacRot* rotb = rot + (size_t)b * rot_stride;
  // the lower triangle (eigh with symmetrize_input=False reads only it; the
  // diagonal's imaginary part is ignored as by LAPACK heevd)
  for (int e = threadIdx.x; e < m * (m + 1) / 2; e += blockDim.x) {
    int k, l;
    unpack_lower(e, k, l);
    const double2 v = k < n && l < n ? Ab[(size_t)k * lda + l] : make_double2(0.0, 0.0);
    if (k == l) dg[k] = v.x;
    else a.at(k, l) = v;
  }
  // Frobenius norm (invariant under the rotations): an off-diagonal element
  // below eps ||A||_F is at the rounding-noise level the rotations
  // themselves create, so it is not rotated (the eigenvalue error this
  // leaves is second order in it).  Summed as by kJacThreads threads whatever
  // the block's size.
  __shared__ double red_f[kJacThreads / 32];
  __shared__ double tol_abs;
  for (int w = threadIdx.x / 32; w < kJacThreads / 32; w += blockDim.x / 32) {
    double f2 = 0.0;
    for (int e = 32 * w + threadIdx.x % 32; e < m * (m + 1) / 2; e += kJacThreads) {
      int k, l;
      unpack_lower(e, k, l);
      double v = 0.0;
      if (k < n && l < n) {
        const double2 x = Ab[(size_t)k * lda + l];
        v = (k == l ? x.x * x.x : 2.0 * (x.x * x.x + x.y * x.y));
      }
      f2 += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f2 += __shfl_xor_sync(0xffffffffu, f2, o);
    if ((threadIdx.x & 31) == 0) red_f[w] = f2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kJacThreads / 32; ++w) t += red_f[w];
    tol_abs = (eb.tol_rel > 0.0 ? eb.tol_rel : 2.220446049250313e-16) * sqrt(t);
  }
  const int rotators = (half + 31) / 32 * 32;   // threads of the rotating warps
  // the other threads' blocks (round independent)
  const int nblk = half * (half + 1) / 2;
  int blk[kJacBlk];   // q1 << 8 | q2, or -1
#pragma unroll
  for (int j = 0; j < kJacBlk; ++j) {
    const int e = (int)threadIdx.x - rotators + j * ((int)blockDim.x - rotators);
    blk[j] = -1;
    if ((int)threadIdx.x >= rotators && e < nblk) {
      int q1, q2;
      unpack_lower(e, q1, q2);
      const bool next = q1 - q2 == 2 || (q1 == 1 && q2 == 0) || (q1 == half - 1 && q2 == half - 2);
      if (q1 != q2 && !(ahead && next)) blk[j] = q1 << 8 | q2;
    }
  }
  __syncthreads();
  int rounds = 0;
  int sweep = 0;
  auto negligible = [&](double app, double aqq, double mag) {
    // off-diagonal element at the noise level or negligible beside both
    // diagonal entries
    return mag <= tol_abs || (fabs(app) + 100.0 * mag == fabs(app) && fabs(aqq) + 100.0 * mag == fabs(aqq));
  };
  // rotation of pair q of round r, number ``at`` of the record; what it does to
  // the pair itself follows in diagonal(), beside the update of other blocks
  struct { double cs, sn, app, aqq, mag; } mine;
  auto rotation = [&](int r, int q, int at) {
    int p_, q_;
    rr_pair(m, r, q, p_, q_);
    JacRot g;
    g.cs = 1.0; g.sn = 0.0; g.om = make_double2(1.0, 0.0);
    const double app = dg[p_], aqq = dg[q_];
    const double2 apq = a.get(p_, q_);
    const double mag = hypot(apq.x, apq.y);
    if (!negligible(app, aqq, mag)) {
      const double theta = (aqq - app) / (2.0 * mag);
      double t = 1.0 / (fabs(theta) + sqrt(theta * theta + 1.0));
      if (theta < 0.0) t = -t;
      g.cs = 1.0 / sqrt(t * t + 1.0);
      g.sn = t * g.cs;
      g.om = make_double2(apq.x / mag, -apq.y / mag);
      any_rot = 1;
      round_rot[r & 1] = 1;
    }
    mine.cs = g.cs; mine.sn = g.sn; mine.app = app; mine.aqq = aqq; mine.mag = mag;
    rcs[(r & 1) * half + q] = make_double2(g.cs, g.sn);
    rom[(r & 1) * half + q] = g.om;
    rotb[(size_t)at * half + q] = g;
  };
  auto diagonal = [&](int r, int q) {
    if (mine.sn == 0.0) return;
    int p_, q_;
    rr_pair(m, r, q, p_, q_);
    const double u = mine.sn / mine.cs;
    dg[p_] = mine.app - u * mine.mag;
    dg[q_] = mine.aqq + u * mine.mag;
    a.set(q_, p_, make_double2(0.0, 0.0));
  };
  // block (q1, q2) under the rotations of round r
  auto update = [&](int r, int q1, int q2) {
    const int o = (r & 1) * half;
    const double2 s1 = rcs[o + q1], s2 = rcs[o + q2];
    const bool a1 = s1.y != 0.0, a2 = s2.y != 0.0;
    if (!a1 && !a2) return;
    int k0, k1, l0, l1;
    rr_pair(m, r, q1, k0, k1);
    rr_pair(m, r, q2, l0, l1);
    // G = [[cs, sn], [-sn om, cs om]] (rows: old index, cols: new index)
    const JacRot g1{s1.x, s1.y, rom[o + q1]}, g2{s2.x, s2.y, rom[o + q2]};
    double2 B00 = a.get(k0, l0), B01 = a.get(k0, l1), B10 = a.get(k1, l0), B11 = a.get(k1, l1);
    auto cm = [](double2 x, double2 y) { return make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x); };
    if (a2) {   // right multiply by G2 (columns l0, l1)
      const double2 t10 = cm(B01, g2.om), t11 = cm(B11, g2.om);
      const double2 c00 = make_double2(g2.cs * B00.x - g2.sn * t10.x, g2.cs * B00.y - g2.sn * t10.y);
      const double2 c01 = make_double2(g2.sn * B00.x + g2.cs * t10.x, g2.sn * B00.y + g2.cs * t10.y);
      const double2 c10 = make_double2(g2.cs * B10.x - g2.sn * t11.x, g2.cs * B10.y - g2.sn * t11.y);
      const double2 c11 = make_double2(g2.sn * B10.x + g2.cs * t11.x, g2.sn * B10.y + g2.cs * t11.y);
      B00 = c00; B01 = c01; B10 = c10; B11 = c11;
    }
    if (a1) {   // left multiply by G1^H = [[cs, -sn conj(om)], [sn, cs conj(om)]] (rows k0, k1)
      const double2 oc = make_double2(g1.om.x, -g1.om.y);
      const double2 u0 = cm(B10, oc), u1 = cm(B11, oc);
      const double2 d00 = make_double2(g1.cs * B00.x - g1.sn * u0.x, g1.cs * B00.y - g1.sn * u0.y);
      const double2 d01 = make_double2(g1.cs * B01.x - g1.sn * u1.x, g1.cs * B01.y - g1.sn * u1.y);
      const double2 d10 = make_double2(g1.sn * B00.x + g1.cs * u0.x, g1.sn * B00.y + g1.cs * u0.y);
      const double2 d11 = make_double2(g1.sn * B01.x + g1.cs * u1.x, g1.sn * B01.y + g1.cs * u1.y);
      B00 = d00; B01 = d01; B10 = d10; B11 = d11;
    }
    a.set(k0, l0, B00);
    a.set(k0, l1, B01);
    a.set(k1, l0, B10);
    a.set(k1, l1, B11);
  };
  for (; sweep < kJacMaxSweeps; ++sweep) {
    if (threadIdx.x == 0) any_rot = 0;
    __syncthreads();
    // a sweep in which every pair is negligible at its start rotates nothing
    // (the matrix never changes), so it is skipped after one parallel check
    // of all pairs instead of being run round by round
    {
      int need = 0;
      for (int e = threadIdx.x; e < m * (m - 1) / 2 && !need; e += blockDim.x) {
        int p_, q_;
        unpack_lower(e, p_, q_);
        ++p_;   // p_ > q_
        const double2 apq = a.at(p_, q_);
        if (!negligible(dg[p_], dg[q_], hypot(apq.x, apq.y))) need = 1;
      }
      if (need) any_rot = 1;
      __syncthreads();
      const int go = any_rot;
      __syncthreads();
      if (!go) break;
    }
    if (threadIdx.x == 0) any_rot = round_rot[0] = 0;
    __syncthreads();
    if (!ahead) {
      for (int r = 0; r < m - 1; ++r, ++rounds) {
        const int q = threadIdx.x;
        // the next round's flag is cleared here; no thread reads it before
        // this round's barrier
        if (q == 0) round_rot[(r + 1) & 1] = 0;
        if (q < half) rotation(r, q, rounds);
        __syncthreads();
        // a round without rotations leaves the matrix as it is: no update
        // pass and no second barrier
        if (!round_rot[r & 1]) continue;
        if (q < half) diagonal(r, q);
#pragma unroll
        for (int j = 0; j < kJacBlk; ++j)
          if (blk[j] >= 0) update(r, blk[j] >> 8, blk[j] & 255);
        __syncthreads();
      }
      const int cont = any_rot;
      __syncthreads();
      if (!cont) break;
      continue;
    }
    if ((int)threadIdx.x < half) rotation(0, threadIdx.x, rounds);
    __syncthreads();
    for (int r = 0; r < m - 1; ++r, ++rounds) {
      // a round without rotations leaves the matrix as it is
      const int on = round_rot[r & 1];
      if ((int)threadIdx.x < rotators) {
        const int q = threadIdx.x;
        if (q == 0) round_rot[(r + 1) & 1] = 0;   // all have read the last round's
        if (on && q < half) {
          diagonal(r, q);
          update(r, q == half - 1 ? q : q + 1, q == 0 ? 0 : q - 1);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(rotators) : "memory");
        if (q < half && r + 1 < m - 1) rotation(r + 1, q, rounds + 1);
      } else if (on) {
#pragma unroll
        for (int j = 0; j < kJacBlk; ++j)
          if (blk[j] >= 0) update(r, blk[j] >> 8, blk[j] & 255);
      }
      __syncthreads();
    }
    const int cont = any_rot;
    __syncthreads();
    if (!cont) break;
  }
  if (threadIdx.x == 0) {
    nrounds_out[b] = rounds;
    if (eb.sweeps) eb.sweeps[b] = sweep + 1;
    if (sweep >= kJacMaxSweeps) latch_error(status, HFB_ERR_NO_CONVERGENCE);
  }
  double* wb = eb.w[b];
  for (int k = threadIdx.x; k < n; k += blockDim.x) wb[k] = dg[k];
}

// Replay V = I G_1 G_2 ... onto blocks of kVecRows rows, then order the
// columns by ascending eigenvalue (stable for ties).  The recorded rotations
// are streamed through shared memory kVecChunk rounds at a time with
// cp.async double buffering, so each round costs one block barrier instead
// of one global-memory latency.
constexpr int kVecRows = 2;   // Pb208 (236 states): 8 rows 0.46 ms, 4 0.33 ms, 2 0.22 ms
constexpr int kVecChunk = 8;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

__global__ void __launch_bounds__(256)
jacobi_vectors_kernel(EighBatch eb, const JacRot* __restrict__ rot, const int* __restrict__ nrounds,
                      size_t rot_stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int b = 0;
  while (b + 1 < eb.nb && (int)blockIdx.x >= eb.vblk0[b + 1]) ++b;
  if (eb.gate && eb.gate[b] == 0) return;
  const int rb = blockIdx.x - eb.vblk0[b];
  const int n = eb.n[b], lda = eb.lda[b];
  const int m = n + (n & 1), half = m / 2;
  JacRot* stage = reinterpret_cast<JacRot*>(smem_raw);                      // [2][kVecChunk][hmax]
  const int hmax = eb.stage_half;
  double2* v = reinterpret_cast<double2*>(stage + 2 * kVecChunk * hmax);    // [kVecRows][m]
  int* order = reinterpret_cast<int*>(v + (size_t)kVecRows * m);
  const int r0 = rb * kVecRows;
  for (int e = threadIdx.x; e < kVecRows * m; e += blockDim.x) {
    const int i = e / m, j = e % m;
    v[e] = make_double2((r0 + i) == j ? 1.0 : 0.0, 0.0);
  }
  const JacRot* rb_ = rot + (size_t)b * rot_stride;
  const int nr = nrounds[b];
  const int nchunk = (nr + kVecChunk - 1) / kVecChunk;
  auto stage_load = [&](int c) {
    if (c < nchunk) {
      const int rs = c * kVecChunk;
      const int cnt = (nr - rs < kVecChunk ? nr - rs : kVecChunk) * half;   // rotations in this chunk
      const char* src = reinterpret_cast<const char*>(rb_ + (size_t)rs * half);
      char* dst = reinterpret_cast<char*>(stage + (size_t)(c & 1) * kVecChunk * hmax);
      for (int e = threadIdx.x; e < 2 * cnt; e += blockDim.x) cp_async16(dst + 16 * e, src + 16 * e);
    }
    cp_async_commit();
  };
  stage_load(0);
  for (int c = 0; c < nchunk; ++c) {
    stage_load(c + 1);
    cp_async_wait1();
    __syncthreads();
    const JacRot* sg = stage + (size_t)(c & 1) * kVecChunk * hmax;
    const int rs = c * kVecChunk;
    const int re = nr - rs < kVecChunk ? nr : rs + kVecChunk;
    for (int r = rs; r < re; ++r) {
      const int rr_ = r % (m - 1);
      const JacRot* gr = sg + (size_t)(r - rs) * half;
      for (int e = threadIdx.x; e < kVecRows * half; e += blockDim.x) {
        const int i = e / half, q = e % half;
        const JacRot g = gr[q];
        if (g.sn == 0.0) continue;
        int p_, q_;
        rr_pair(m, rr_, q, p_, q_);
        const double2 vp = v[i * m + p_], vq = v[i * m + q_];
        const double2 t = make_double2(vq.x * g.om.x - vq.y * g.om.y, vq.x * g.om.y + vq.y * g.om.x);
        v[i * m + p_] = make_double2(g.cs * vp.x - g.sn * t.x, g.cs * vp.y - g.sn * t.y);
        v[i * m + q_] = make_double2(g.sn * vp.x + g.cs * t.x, g.sn * vp.y + g.cs * t.y);
      }
      __syncthreads();
    }
  }
  const double* wb = eb.w[b];
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    int rank = 0;
    const double wj = wb[j];
    for (int k = 0; k < n; ++k) {
      const double wk = wb[k];
      rank += (wk < wj) || (wk == wj && k < j);
    }
    order[rank] = j;
  }
  __syncthreads();
  double2* Vb = eb.v[b];
  for (int e = threadIdx.x; e < kVecRows * n; e += blockDim.x) {
    const int i = e / n, c = e % n;
    if (r0 + i < n) Vb[(size_t)(r0 + i) * lda + c] = v[i * m + order[c]];
  }
}

__global__ void sort_values_kernel(EighBatch eb) {
  const int b = blockIdx.x;
  if (eb.gate && eb.gate[b] == 0) return;
  const int n = eb.n[b];
  extern __shared__ double tmpw[];
  double* wb = eb.w[b];
  for (int j = threadIdx.x; j < n; j += blockDim.x) tmpw[j] = wb[j];
  __syncthreads();
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    int rank = 0;
    const double wj = tmpw[j];
    for (int k = 0; k < n; ++k) rank += (tmpw[k] < wj) || (tmpw[k] == wj && k < j);
    wb[rank] = wj;
  }
}

// Batched Hermitian eigensolver over the matrices of ``eb`` (all concurrent).
int eigh_batch(hfb_ctx_s* c, EighBatch eb, cudaStream_t st) {
  if (eb.nb <= 0) return HFB_OK;
  int mmax = 0, nmax = 0;
  eb.vblk0[0] = 0;
  for (int i = 0; i < eb.nb; ++i) {
    if (eb.n[i] <= 0 || eb.lda[i] < eb.n[i]) return HFB_ERR_ARG;
    const int m = eb.n[i] + (eb.n[i] & 1);
    mmax = m > mmax ? m : mmax;
    nmax = eb.n[i] > nmax ? eb.n[i] : nmax;
    eb.vblk0[i + 1] = eb.vblk0[i] + (eb.n[i] + kVecRows - 1) / kVecRows;
  }
  const int half = mmax / 2;
  if (mmax > kJacMaxN) return HFB_ERR_ARG;
  const size_t smem = sizeof(double2) * (size_t)(mmax - 1) * (mmax == kJacMaxN ? half : half | 1) +
                      sizeof(JacRot) * 2 * half + sizeof(double) * mmax;
  // a thread per block of the largest matrix beside the rotating warps
  const int want = (half + 31) / 32 * 32 + (half * (half + 1) / 2 + 31) / 32 * 32;
  const int threads = want < kJacThreads ? want : kJacThreads;
  const size_t rot_stride = (size_t)kJacMaxSweeps * (mmax - 1) * half;
  char* buf = (char*)scratch(c, hfb_ctx_s::S_MAT, sizeof(JacRot) * rot_stride * eb.nb + sizeof(int) * kEighMax + 64);
  if (!buf) return HFB_ERR_ALLOC;
  JacRot* rot = (JacRot*)buf;
  int* nr = (int*)(buf + sizeof(JacRot) * rot_stride * eb.nb);
  const auto kernel = threads <= kJacSmall ? jacobi_kernel<kJacSmall> : jacobi_kernel<kJacThreads>;
  allow_max_dynamic_smem(kernel);
  kernel<<<eb.nb, threads, smem, st>>>(eb, rot, nr, c->dev_status, rot_stride);
  HFB_CHECK_LAUNCH();
  eb.stage_half = half;
  const size_t smem2 =
      sizeof(JacRot) * 2 * kVecChunk * half + sizeof(double2) * kVecRows * mmax + sizeof(int) * mmax;
  allow_max_dynamic_smem(jacobi_vectors_kernel);
  jacobi_vectors_kernel<<<eb.vblk0[eb.nb], 256, smem2, st>>>(eb, rot, nr, rot_stride);
  HFB_CHECK_LAUNCH();
  sort_values_kernel<<<eb.nb, 256, sizeof(double) * nmax, st>>>(eb);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

// nb matrices a[nb][n][lda] -> w[nb][n] ascending, v[nb][n][lda].
int eigh_launch(hfb_ctx_s* c, int nb, int n, int lda, const double2* a, double* w, double2* v, int* sweeps,
                cudaStream_t st) {
  for (int b0 = 0; b0 < nb; b0 += kEighMax) {
    EighBatch eb{};
    eb.sweeps = sweeps ? sweeps + b0 : nullptr;
    eb.nb = nb - b0 < kEighMax ? nb - b0 : kEighMax;
    for (int i = 0; i < eb.nb; ++i) {
      eb.n[i] = n;
      eb.lda[i] = lda;
      eb.a[i] = a + (size_t)(b0 + i) * n * lda;
      eb.w[i] = w + (size_t)(b0 + i) * n;
      eb.v[i] = v + (size_t)(b0 + i) * n * lda;
    }
    int r = eigh_batch(c, eb, st);
    if (r) return r;
  }
  return HFB_OK;
}

// ========================================================= small GEMMs ====
// C = A' B' with A' = A or A^H, B' = B or B^H; n x n, leading dim ld.
__global__ void zgemm_small_kernel(int n, int ld, int ta, int tb, const double2* A, const double2* B, double2* C) {
  __shared__ double2 As[16][17], Bs[16][17];
  const int i = blockIdx.y * 16 + threadIdx.y, j = blockIdx.x * 16 + threadIdx.x;
  double re = 0, im = 0;
  for (int k0 = 0; k0 < n; k0 += 16) {
    const int ka = k0 + threadIdx.x, kb = k0 + threadIdx.y;
    double2 av = make_double2(0, 0), bv = make_double2(0, 0);
    if (i < n && ka < n) {
      if (ta) { av = A[(size_t)ka * ld + i]; av.y = -av.y; }
      else av = A[(size_t)i * ld + ka];
    }
    if (j < n && kb < n) {
      if (tb) { bv = B[(size_t)j * ld + kb]; bv.y = -bv.y; }
      else bv = B[(size_t)kb * ld + j];
    }
    As[threadIdx.y][threadIdx.x] = av;
    Bs[threadIdx.y][threadIdx.x] = bv;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const double2 x = As[threadIdx.y][k], y = Bs[k][threadIdx.x];
      re += x.x * y.x - x.y * y.y;
      im += x.x * y.y + x.y * y.x;
    }
    __syncthreads();
  }
  if (i < n && j < n) C[(size_t)i * ld + j] = make_double2(re, im);
}

// One n x n product C = A' B' (A' = A or A^H, B' = B or B^H), leading
// dimension ld, for other translation units.
int zgemm_small_one(int n, int ld, int ta, int tb, const double2* A, const double2* B, double2* C, cudaStream_t st) {
  const unsigned g = (unsigned)((n + 15) / 16);
  zgemm_small_kernel<<<dim3(g, g), dim3(16, 16), 0, st>>>(n, ld, ta, tb, A, B, C);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

// Eigenpairs of up to two nearly diagonal Hermitian matrices (lower
// triangles at A + b sA, leading dimension ld): w ascending at W + b sW,
// eigenvectors in the columns of V + b sV, by refinement (diag_cluster.cu);
// Jacobi for the matrices it does not apply to.  ``jacobi`` (optional, device
// [nb]) receives 1 where that was so, else 0.
static int eigh_refine(hfb_ctx_s* c, int nb, Pair2 nper, int ld, const double2* A, size_t sA, double* W, size_t sW,
                       double2* V, size_t sV, double tol_rel, cudaStream_t st,
                       cudaEvent_t begun = nullptr, int* jacobi = nullptr) {
  const size_t wb = (refine_bytes(nb, ld) + 15) / 16 * 16;
  char* buf = (char*)scratch(c, hfb_ctx_s::S_EIG, wb + sizeof(int) * nb);
  if (!buf) return HFB_ERR_ALLOC;
  int* fallback = jacobi ? jacobi : (int*)(buf + wb);
  const RefineArgs a{nper, ld, A, sA, W, sW, V, sV, tol_rel > 0.0 ? tol_rel : 1e-13, fallback};
  const int r = refine_launch(c, nb, a, buf, begun, st);
  if (r) return r;
  EighBatch eb{};
  eb.tol_rel = tol_rel;
  eb.gate = fallback;
  for (int b = 0; b < nb; ++b) {
    eb.n[eb.nb] = nper.v[b];
    eb.lda[eb.nb] = ld;
    eb.a[eb.nb] = A + b * sA;
    eb.w[eb.nb] = W + b * sW;
    eb.v[eb.nb] = V + b * sV;
    ++eb.nb;
  }
  return eigh_batch(c, eb, st);
}

// ============================================================== rotate ====
// out1_j = sum_i psi_i U_ij, out2_j = sum_i psi_i L_ij for the states of one
// block: a (K x ns) by (ns x 2 ns) GEMM.  64 (k) x 64 (j) tile per CTA, 256
// threads with 4 x 4 outputs each, double-buffered 8-state stages.
template <class R>
__global__ void __launch_bounds__(256)
rotate_kernel(int ns, size_t K, const cplx<R>* __restrict__ psi, const double2* __restrict__ U,
              const double2* __restrict__ L, int ld, cplx<R>* out1, cplx<R>* out2) {
  using Z = cplx<R>;
  constexpr int KT = 64, JT = 64, IT = 8;
  __shared__ Z Ps[2][IT][KT + 1];
  __shared__ Z Ws[2][IT][JT + 1];
  const int njt = (2 * ns + JT - 1) / JT;
  const int jt = blockIdx.x % njt;
  const size_t k0 = (size_t)(blockIdx.x / njt) * KT;
  const int j0 = jt * JT;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;   // tx -> k (4), ty -> j (4)
  R acc[4][4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v][0] = acc[u][v][1] = R(0);
  auto load = [&](int buf, int i0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = threadIdx.x + 256 * h;
      const int ii = e / KT, kk = e % KT;
      const size_t k = k0 + kk;
      Ps[buf][ii][kk] = (i0 + ii < ns && k < K) ? psi[(size_t)(i0 + ii) * K + k] : czero<Z>();
      const int ii2 = e / JT, jj = e % JT;
      const int j = j0 + jj;
      double2 w = make_double2(0, 0);
      if (i0 + ii2 < ns && j < 2 * ns)
        w = j < ns ? U[(size_t)(i0 + ii2) * ld + j] : L[(size_t)(i0 + ii2) * ld + (j - ns)];
      Ws[buf][ii2][jj] = mk<R>((R)w.x, (R)w.y);
    }
  };
  load(0, 0);
  __syncthreads();
  int buf = 0;
  for (int i0 = 0; i0 < ns; i0 += IT) {
    if (i0 + IT < ns) load(buf ^ 1, i0 + IT);
#pragma unroll
    for (int ii = 0; ii < IT; ++ii) {
      Z pv[4], wv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) pv[u] = Ps[buf][ii][tx + 16 * u];
#pragma unroll
      for (int v = 0; v < 4; ++v) wv[v] = Ws[buf][ii][ty + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          acc[u][v][0] += pv[u].x * wv[v].x - pv[u].y * wv[v].y;
          acc[u][v][1] += pv[u].x * wv[v].y + pv[u].y * wv[v].x;
        }
    }
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const int j = j0 + ty + 16 * v;
    if (j >= 2 * ns) continue;
    Z* o = j < ns ? out1 + (size_t)j * K : out2 + (size_t)(j - ns) * K;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t k = k0 + tx + 16 * u;
      if (k < K) o[k] = mk<R>(acc[u][v][0], acc[u][v][1]);
    }
  }
}

// Single-precision variant with a larger register tile: 128 (k) x 96 (j)
// per CTA, 256 threads holding 8 x 6 complex accumulators each (48
// independent chains), 8 states per double-buffered shared-memory stage.
// The 96-wide j tile keeps the padding of 2 ns columns small (280 -> 288,
// 192 -> 192).
constexpr int kRotKT = 128, kRotJT = 96, kRotIT = 8;

__global__ void __launch_bounds__(256, 1)
rotate_f32_kernel(int ns, size_t K, const float2* __restrict__ psi, const double2* __restrict__ U,
                  const double2* __restrict__ L, int ld, float2* out1, float2* out2) {
  __shared__ __align__(16) float2 Ps[2][kRotIT][kRotKT];
  __shared__ __align__(16) float2 Ws[2][kRotIT][kRotJT];
  const int njt = (2 * ns + kRotJT - 1) / kRotJT;
  const int jt = blockIdx.x % njt;
  const size_t k0 = (size_t)(blockIdx.x / njt) * kRotKT;
  const int j0 = jt * kRotJT;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;   // k = tx + 16 u (u < 8), j = ty + 16 v (v < 6)
  float acc[8][6][2];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 6; ++v) acc[u][v][0] = acc[u][v][1] = 0.f;
  // stage loads into registers first so the next stage's global reads
  // overlap this stage's arithmetic
  float4 pr[2];
  float2 wr[3];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = threadIdx.x + 256 * h;          // 512 float4 = 8 states x 64 pairs
      const int ii = e / (kRotKT / 2), kk = 2 * (e % (kRotKT / 2));
      const size_t k = k0 + kk;
      pr[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i0 + ii < ns && k < K) {
        if (k + 2 <= K) pr[h] = *reinterpret_cast<const float4*>(psi + (size_t)(i0 + ii) * K + k);
        else { const float2 a = psi[(size_t)(i0 + ii) * K + k]; pr[h] = make_float4(a.x, a.y, 0.f, 0.f); }
      }
    }
#pragma unroll
    for (int h = 0; h < 3; ++h) {
      const int e = threadIdx.x + 256 * h;          // 768 = 8 states x 96 columns
      const int ii = e / kRotJT, jj = e % kRotJT;
      const int j = j0 + jj;
      double2 w = make_double2(0.0, 0.0);
      if (i0 + ii < ns && j < 2 * ns)
        w = j < ns ? U[(size_t)(i0 + ii) * ld + j] : L[(size_t)(i0 + ii) * ld + (j - ns)];
      wr[h] = make_float2((float)w.x, (float)w.y);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = threadIdx.x + 256 * h;
      const int ii = e / (kRotKT / 2), kk = 2 * (e % (kRotKT / 2));
      *reinterpret_cast<float4*>(&Ps[buf][ii][kk]) = pr[h];
    }
#pragma unroll
    for (int h = 0; h < 3; ++h) {
      const int e = threadIdx.x + 256 * h;
      Ws[buf][e / kRotJT][e % kRotJT] = wr[h];
    }
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int i0 = 0; i0 < ns; i0 += kRotIT) {
    const bool more = i0 + kRotIT < ns;
    if (more) fetch(i0 + kRotIT);
#pragma unroll
    for (int ii = 0; ii < kRotIT; ++ii) {
      float2 pv[8], wv[6];
#pragma unroll
      for (int u = 0; u < 8; ++u) pv[u] = Ps[buf][ii][tx + 16 * u];
#pragma unroll
      for (int v = 0; v < 6; ++v) wv[v] = Ws[buf][ii][ty + 16 * v];
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int v = 0; v < 6; ++v) {
          acc[u][v][0] = fmaf(pv[u].x, wv[v].x, fmaf(-pv[u].y, wv[v].y, acc[u][v][0]));
          acc[u][v][1] = fmaf(pv[u].x, wv[v].y, fmaf(pv[u].y, wv[v].x, acc[u][v][1]));
        }
    }
    if (more) stash(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int v = 0; v < 6; ++v) {
    const int j = j0 + ty + 16 * v;
    if (j >= 2 * ns) continue;
    float2* o = j < ns ? out1 + (size_t)j * K : out2 + (size_t)(j - ns) * K;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const size_t k = k0 + tx + 16 * u;
      if (k < K) o[k] = make_float2(acc[u][v][0], acc[u][v][1]);
    }
  }
}

int rotate_tc_launch(hfb_ctx_s* c, int ns, const void* psi, const double2* U, const double2* L, int ld, void* out1,
                     void* out2, cudaStream_t st, int pre);   // rotate_tc.cu
int rotate_tc_transpose(hfb_ctx_s* c, int which, int ns, const void* psi, cudaStream_t st);

// ``pre`` (single precision on the tensor cores): 0 or 1 when the states were
// transposed already by rotate_tc_transpose into that rotation's buffer.
int rotate_launch(hfb_ctx_s* c, int prec, int s0, int ns, const void* psi, const double2* U, const double2* L, int ld,
                  void* out1, void* out2, cudaStream_t st, int pre) {
  if (ns <= 0) return HFB_OK;
  if (prec == HFB_F64 && c->f64_mma)
    return rotate_f64_launch(c, 1, &s0, &ns, psi, &U, &L, ld, out1, out2, st);
  if (prec != HFB_F64 && c->use_tcgen05) {
    const size_t Kc = (size_t)2 * c->n * c->n * c->n, offc = (size_t)s0 * Kc;
    const int r = rotate_tc_launch(c, ns, (const float2*)psi + offc, U, L, ld, (float2*)out1 + offc,
                                   (float2*)out2 + offc, st, pre);
    if (r != HFB_ERR_UNSUPPORTED_GRID) return r;
  }
  const size_t K = (size_t)2 * c->n * c->n * c->n;
  const int njt = (2 * ns + 63) / 64;
  const size_t nkt = (K + 63) / 64;
  const size_t off = (size_t)s0 * K;
  if (prec == HFB_F64)
    rotate_kernel<double><<<(unsigned)(nkt * njt), 256, 0, st>>>(ns, K, (const double2*)psi + off, U, L, ld,
                                                                 (double2*)out1 + off, (double2*)out2 + off);
  else {
    const int njt2 = (2 * ns + kRotJT - 1) / kRotJT;
    const size_t nkt2 = (K + kRotKT - 1) / kRotKT;
    rotate_f32_kernel<<<(unsigned)(nkt2 * njt2), 256, 0, st>>>(ns, K, (const float2*)psi + off, U, L, ld,
                                                               (float2*)out1 + off, (float2*)out2 + off);
  }
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

}  // namespace hfb

using namespace hfb;

extern "C" int hfb_gram(hfb_ctx_t ctx, int prec, int s0, int ns, int mask, const void* psi, const void* hampsi,
                        const void* hmfpsi, const double* v_pair_iq, double wxyz, double* out, void* stream) {
  if (!ctx || !psi || !out || ns <= 0) return HFB_ERR_ARG;
  if (((mask & 2) && !hampsi) || ((mask & 4) && !hmfpsi) || ((mask & 8) && !v_pair_iq)) return HFB_ERR_ARG;
  if ((ns + GT - 1) / GT > 255) return HFB_ERR_ARG;
  double2* o = (double2*)out;
  double2* outs[8] = {o, o + (size_t)ns * ns, o + 2 * (size_t)ns * ns, o + 3 * (size_t)ns * ns,
                      nullptr, nullptr, nullptr, nullptr};
  const double* vp[2] = {v_pair_iq, nullptr};
  mask &= 15;
  return gram_launch(ctx, prec, 1, &s0, &ns, &mask, psi, hampsi, hmfpsi, vp, wxyz, outs, ns, as_stream(stream));
}

extern "C" int hfb_eigh(hfb_ctx_t ctx, int nb, int n, int lda, const double* a, double* w, double* v, int* sweeps,
                        void* stream) {
  if (!ctx || !a || !w || !v || n <= 0 || lda < n) return HFB_ERR_ARG;
  return eigh_launch(ctx, nb, n, lda, (const double2*)a, w, (double2*)v, sweeps, as_stream(stream));
}

extern "C" int hfb_eigh_near_diagonal(hfb_ctx_t ctx, int nb, int n, int lda, const double* a, double* w,
                                      double* v, void* stream) {
  return hfb_eigh_near_diagonal_info(ctx, nb, n, lda, a, w, v, nullptr, stream);
}

extern "C" int hfb_eigh_near_diagonal_info(hfb_ctx_t ctx, int nb, int n, int lda, const double* a, double* w,
                                           double* v, int* jacobi, void* stream) {
  if (!ctx || !a || !w || !v || n <= 0 || lda < n || nb <= 0) return HFB_ERR_ARG;
  if (lda > 256) return HFB_ERR_UNSUPPORTED_GRID;
  cudaStream_t st = as_stream(stream);
  const size_t mstride = (size_t)n * lda;
  for (int b0 = 0; b0 < nb; b0 += 2) {
    const int cnt = nb - b0 < 2 ? nb - b0 : 2;
    Pair2 nper;
    nper.v[0] = n;
    nper.v[1] = cnt > 1 ? n : 0;
    int r = eigh_refine(ctx, cnt, nper, lda, (const double2*)a + b0 * mstride, mstride, w + (size_t)b0 * n, n,
                        (double2*)v + b0 * mstride, mstride, 0.0, st, nullptr, jacobi ? jacobi + b0 : nullptr);
    if (r) return r;
  }
  return HFB_OK;
}

extern "C" int hfb_diagstep(hfb_ctx_t ctx, int prec, const hfb_diag_args* a, void* stream) {
  if (!ctx || !a || !a->psi || !a->psi_out || a->psi_out == a->psi || !a->lagrange || !a->sp_norm || !a->lambda_save) return HFB_ERR_ARG;
  if (a->diagonalize && !a->hampsi) return HFB_ERR_ARG;
  if (a->construct && (!a->hmfpsi || !a->sp_energy || !a->hmatrix || !a->gapmatrix || !a->symcond || !a->efluct))
    return HFB_ERR_ARG;
  if (a->construct && a->ipair && (!a->v_pair || !a->deltaf)) return HFB_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  const int n0 = a->npsi[0], n1 = a->npsi[1];
  const int ld = n0 > n1 ? n0 : n1;
  const size_t sm = (size_t)ld * ld;
  const size_t n3 = (size_t)ctx->n * ctx->n * ctx->n;
  // workspace per isospin: 4 Gram matrices, S^-1/2, the eigenvectors of
  // lambda, U and U lambda; then the eigenvalues and the chains' own work
  const size_t wl = loewdin_bytes(ld), wc = construct_bytes(ld);
  char* ws = (char*)scratch(ctx, hfb_ctx_s::S_SMALL,
                            sizeof(double2) * 16 * sm + sizeof(double) * 2 * ld + (wl > wc ? wl : wc));
  if (!ws) return HFB_ERR_ALLOC;
  double2* gm = (double2*)ws;                 // [iq][4][ld][ld]: S, Lambda, H_old, G_old
  double2* Ur = gm + 8 * sm;                  // S^-1/2
  double2* Vl = Ur + 2 * sm;                  // eigenvectors of lambda
  double2* U = Vl + 2 * sm;                   // total transform
  double2* Lw = U + 2 * sm;                   // U lambda
  double* w = (double*)(Lw + 2 * sm);         // [iq][ld] eigenvalues of lambda
  void* work = w + 2 * ld;                    // loewdin, then construct
  Pair2 nper, off;
  nper.v[0] = n0; nper.v[1] = n1;
  off.v[0] = 0; off.v[1] = n0;
  const int nq[2] = {n0, n1}, so[2] = {0, n0};
  int r;
  // The eigensolve of lambda and S^-1/2 need the first Gram launch only.  H
  // and G are needed only by the construct step, so when they are asked for,
  // the first launch computes S and lambda and the H, G launch runs beside
  // the two chains (HFB_GRAM_SPLIT=0: one launch).  A kernel of a chain that
  // found every SM in use would wait for the launch to drain (2.9 ms on
  // Pb208 FP64; stream priority did not help, no CTA of the launch ends
  // early), so the H, G launch comes last and leaves four SMs alone: two for
  // the Jacobi solver, one for each isospin's S^-1/2.  The refinement, which
  // is short, takes its SMs before the launch: its launch completion event
  // starts the other stream (from a common event the Gram's CTAs sometimes came
  // first, and the refinement waited 2.6 ms for them); the launch's CTAs that
  // do not fit at once follow it.  Pb208 FP64 iteration: 34.7 ms with the H, G
  // launch first, 32.2 ms with it last, 26.5 ms with contract_f64.cu and the
  // free SMs (27.8 ms without them).
  int mask = 1;
  if (a->diagonalize) mask |= 2 | kGramLowerLambda;   // the eigensolver reads the lower triangle
  if (a->construct) mask |= 4;
  if (a->construct && a->ipair) mask |= 8;
  const bool beside = a->diagonalize && ctx->side && ctx->side2;
  const bool split = beside && a->construct && ctx->gram_split;
  const bool refine = a->diagonalize && ctx->lambda_refine && prec == HFB_F64;
  const double* vp[2] = {a->v_pair, a->v_pair ? a->v_pair + n3 : nullptr};
  double2* outs[8];
  for (int iq = 0; iq < 2; ++iq)
    for (int m = 0; m < 4; ++m) outs[iq * 4 + m] = gm + ((size_t)iq * 4 + m) * sm;
  {
    const int m1 = split ? (mask & (3 | kGramLowerLambda)) : mask;
    const int masks[2] = {m1, m1};
    r = gram_launch(ctx, prec, 2, so, nq, masks, a->psi, a->hampsi, a->hmfpsi, vp, a->wxyz, outs, ld, st);
    if (r) return r;
  }
  cudaStream_t nst = st;
  if (beside) {
    cudaEventRecord(ctx->ev_fork, st);
    cudaStreamWaitEvent(ctx->side2, ctx->ev_fork, 0);
    if (split && !refine) cudaEventRecord(ctx->ev_fork2, ctx->side2);
    nst = ctx->side2;
  }
  r = loewdin_launch(LoewdinArgs{nper, off, ld, gm, 4 * sm, Ur, a->sp_norm, ctx->dev_status}, work, !split, nst);
  if (r) return r;
  if (a->diagonalize) {
    // single-precision states carry rounding noise of 2^-24 relative in
    // lambda; converging below that level refines nothing
    const double tol_rel = prec != HFB_F64 ? 5.9604644775390625e-08 : 0.0;
    // FP64: refinement (measured 1 ms per Pb208 iteration faster than the
    // Jacobi sweeps near convergence); FP32: the looser Jacobi threshold
    // converges in a few sweeps and measured faster (11.4 ms against 12.0
    // ms per Pb208 iteration: in the bulk the refinement's acceptance test
    // fails and the Jacobi runs after it)
    if (refine) {
      r = eigh_refine(ctx, 2, nper, ld, gm + sm, 4 * sm, w, ld, Vl, sm, tol_rel, st, split ? ctx->ev_fork2 : nullptr);
    } else {
      EighBatch eb{};
      eb.tol_rel = tol_rel;
      for (int iq = 0; iq < 2; ++iq) {
        eb.n[eb.nb] = nq[iq];
        eb.lda[eb.nb] = ld;
        eb.a[eb.nb] = gm + (size_t)iq * 4 * sm + sm;
        eb.w[eb.nb] = w + (size_t)iq * ld;
        eb.v[eb.nb] = Vl + (size_t)iq * sm;
        ++eb.nb;
      }
      r = eigh_batch(ctx, eb, st);
    }
    if (r) return r;
  }
  if (split) {
    cudaStreamWaitEvent(ctx->side, ctx->ev_fork2, 0);
    const int m2 = mask & 12;
    const int masks[2] = {m2, m2};
    r = gram_launch(ctx, prec, 2, so, nq, masks, a->psi, a->hampsi, a->hmfpsi, vp, a->wxyz, outs, ld, ctx->side, 4);
    if (r) return r;
    cudaEventRecord(ctx->ev_join, ctx->side);
  }
  // the rotation's transposes of the states depend on psi only: they follow
  // S^-1/2 on the second side stream
  int pre[2] = {-1, -1};
  if (split && prec != HFB_F64 && ctx->use_tcgen05) {
    const size_t Kc = (size_t)2 * n3;
    for (int iq = 0; iq < 2; ++iq) {
      r = rotate_tc_transpose(ctx, iq, nq[iq], (const float2*)a->psi + (size_t)so[iq] * Kc, nst);
      if (r == HFB_OK) pre[iq] = iq;
      else if (r != HFB_ERR_UNSUPPORTED_GRID) return r;
    }
  }
  if (beside) {
    cudaEventRecord(ctx->ev_join2, ctx->side2);
    cudaStreamWaitEvent(st, ctx->ev_join2, 0);
  }
  if (split) cudaStreamWaitEvent(st, ctx->ev_join, 0);
  r = construct_launch(
      ConstructArgs{nper, off, ld, a->nmax, a->diagonalize, a->construct, a->ipair, a->tbcs, Ur, Vl, U, gm + 2 * sm,
                    gm + 3 * sm, 4 * sm, Lw, a->wocc, a->wguv, a->pairwg, a->wstates, (double2*)a->hmatrix,
                    (double2*)a->gapmatrix, (double2*)a->symcond, (double2*)a->lambda_save, a->sp_energy, a->deltaf,
                    a->efluct},
      work, st);
  if (r) return r;
  if (prec == HFB_F64 && ctx->f64_mma) {
    const double2 *Us[2] = {U, U + sm}, *Ls[2] = {Lw, Lw + sm};
    return rotate_f64_launch(ctx, 2, so, nq, a->psi, Us, Ls, ld, a->psi_out, a->lagrange, st);
  }
  for (int iq = 0; iq < 2; ++iq) {
    r = rotate_launch(ctx, prec, so[iq], nq[iq], a->psi, U + (size_t)iq * sm, Lw + (size_t)iq * sm, ld, a->psi_out,
                      a->lagrange, st, pre[iq]);
    if (r) return r;
  }
  return HFB_OK;
}
