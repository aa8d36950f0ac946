// The two large FP64 contractions of the diagonalisation step on the FP64
// tensor cores (mma.sync m8n8k4 .f64, 37.1 TFLOP/s measured on this part with
// 8 or more warps per SM):
//   Gram      C_a = wxyz Psi^H X_a over K = 2 n^3 grid points
//   rotation  [psi U | psi L] over the states
// Both are bound by the tensor pipe once it is fed, so what counts is the work
// done for padding and the balance of the last wave.
#include "diag.cuh"

namespace hfb {

namespace {

__device__ __forceinline__ void cp16(void* smem, const void* gmem, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp8(void* smem, const void* gmem, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ================================================================ Gram ====
// Over the interleaved storage, with k' running over (Re, Im) of each k,
//   Re C_ij = sum_k' a_ik' b_jk',   a = psi_i, b = x_j,
//   Im C_ij = sum_k' a_ik' bt_jk',  bt = (Im x, -Re x) per element,
// so each 8 x 8 output block takes two real MMAs per four k'; bt is b with
// the partner lane's value (one shuffle).  Work is a list of output tiles,
// one matrix per tile, and a CTA (4 warps) takes one tile over one K slice;
// split-K partials are summed in a fixed order.  S, H and G are Hermitian
// (Gram matrices of one set of vectors, h and v_pair Hermitian): tiles on and
// above the diagonal, mirrored by the reduction.  lambda is needed on and
// below the diagonal only when it goes to the eigensolver.  On the diagonal
// the 8 x 8 blocks of the other triangle are skipped.
//
// Tile edge: 48 (four quadrants of 24 x 24, one per warp), 32 (quadrants of
// 16 x 16), 24 and 16 (every warp the whole tile over its share of a stage,
// added up in shared memory), by the smallest work over the two state counts:
// 10 states in 48-state tiles are 23 times the work, 61 states 2.5 times.
// A group of four warps takes one tile over one K slice at a time from a
// ticket; a CTA is four groups, one CTA per SM, so a launch on fewer CTAs
// than SMs leaves whole SMs to what runs beside it.  The slices are short
// enough for about four tickets a group (fewer on small grids, where a slice
// would fall below 1024 points and its start-up show); they do not depend on
// which matrices a launch computes, so neither does any sum's order.  S + lambda
// of 140 states at 48^3 alone with 1, 2, 4 and 8 tickets: 2.76, 2.10, 2.08, 1.95
// ms; of 61 states 654, 495, 468, 448 us; at 32^3 2 to 8 are equal.  (The S +
// lambda, H + G launches of a Pb208 iteration are equal with 4 and 6.)
// Measured, S + lambda of Pb208 (140 + 96 states, 48^3): 3.8 ms with 594
// equal CTAs on 592 places and all of lambda, 2.1 ms here (30 TFLOP/s).  G's
// factor v_pair is applied at the fragment loads (multiplied on the way into
// shared memory, its tiles could not be copied ahead: H + G on 144 SMs 3.3 ms,
// 2.4 ms here).
enum { GF_FULL = 0, GF_UPPER = 1, GF_LOWER = 2 };

struct GfGroup {
  int b, a, type, nt, first;   // isospin, matrix, triangle, tiles per edge, first tile
};
struct GfJob {
  int ngroup, ntile;
  GfGroup g[8];
  int s0[2], ns[2];
  const double* vp[2];
};

__device__ __forceinline__ GfGroup gf_tile(const GfJob& job, int t, int& ti, int& tj) {
  int q = 0;
  while (q + 1 < job.ngroup && t >= job.g[q + 1].first) ++q;
  const GfGroup g = job.g[q];
  int u = t - g.first;
  if (g.type == GF_FULL) {
    ti = u / g.nt;
    tj = u % g.nt;
  } else {
    ti = 0;
    while (u >= g.nt - ti) {
      u -= g.nt - ti;
      ++ti;
    }
    tj = ti + u;
    if (g.type == GF_LOWER) {
      const int x = ti;
      ti = tj;
      tj = x;
    }
  }
  return g;
}

constexpr int GF_THREADS = 128;   // of a group
constexpr int GF_GROUPS = 4;      // per CTA

template <int GT> struct GfGeo {
  static constexpr int WG = GT >= 32 ? 2 : 1;       // warps per tile edge
  static constexpr int MB = GT / (8 * WG);          // 8-blocks per warp and edge
  static constexpr int WK = 4 / (WG * WG);          // warps sharing a tile along K
  static constexpr int KB = WG == 2 ? 16 : 32;      // complex k per stage
  static constexpr int LD = KB + 1;                 // rows fall on distinct bank groups
  static constexpr size_t STAGES = sizeof(double2) * 2 * 2 * GT * LD;
  static constexpr size_t SMEM = STAGES + sizeof(double) * 2 * KB;   // and v_pair of each stage
  static_assert(WK == 1 || sizeof(double2) * WK * GT * GT <= STAGES, "warp sums reuse the stages");
};

template <int GT>
__device__ __forceinline__ void gf_item(const GfJob& job, size_t K, size_t n3, const double2* __restrict__ psi,
                                        const double2* __restrict__ hampsi, const double2* __restrict__ hmfpsi,
                                        double2* part, int nchunk, int kchunk, int item, double2* gf_smem, int tid,
                                        int bar) {
  using G = GfGeo<GT>;
  constexpr int MB = G::MB, KB = G::KB, LD = G::LD, RS = GF_THREADS / KB, NL = GT / RS;
  auto sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(GF_THREADS) : "memory"); };
  double2* As = gf_smem;                 // [2][GT][LD]
  double2* Bs = gf_smem + 2 * GT * LD;
  double* vs = reinterpret_cast<double*>(Bs + 2 * GT * LD);   // [2][KB]
  const int tile = item % job.ntile, chunk = item / job.ntile;
  int ti, tj;
  const GfGroup gr = gf_tile(job, tile, ti, tj);
  const int b = gr.b, am = gr.a, ns = job.ns[b];
  const int i0 = ti * GT, j0 = tj * GT;
  const size_t base = (size_t)job.s0[b] * K;
  const double2* P = psi + base;
  const double2* X = am == 1 ? hampsi + base : am == 2 ? hmfpsi + base : P;
  const double* vp = job.vp[b];
  const bool scaled = am == 3;             // by v_pair, at the fragment loads
  const bool same = (am == 0 || scaled) && ti == tj;   // both operands are the same rows
  const size_t k0 = (size_t)chunk * kchunk;
  const size_t k1 = min(K, k0 + (size_t)kchunk);
  const int lane = tid & 31;
  // the quadrants that are idle on a diagonal tile go to different warps
  // (so to different tensor pipes) from item to item
  const int role = ((tid >> 5) + tile + chunk) & 3;
  const int rw = G::WG == 2 ? role >> 1 : 0, cw = G::WG == 2 ? role & 1 : 0;
  const int fr = lane >> 2, fk = lane & 3;   // fragment row (A) / column (B), k' within the 4
  const bool tri = gr.type != GF_FULL && ti == tj;
  const bool idle = tri && (gr.type == GF_UPPER ? rw > cw : rw < cw);
  const int half = !tri || rw != cw ? 0 : gr.type;
  double accR[MB][MB][2], accI[MB][MB][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < MB; ++j) accR[i][j][0] = accR[i][j][1] = accI[i][j][0] = accI[i][j][1] = 0.0;
  // one stage: GT rows x KB elements of each operand, consecutive threads on
  // consecutive elements of a row
  const int lr = tid / KB, lk = tid % KB;
  auto load = [&](int buf, size_t kb) {
    const size_t k = kb + lk;
    const bool okk = k < k1;
    double2* da = As + ((size_t)buf * GT + lr) * LD + lk;
    double2* db = Bs + ((size_t)buf * GT + lr) * LD + lk;
#pragma unroll
    for (int h = 0; h < NL; ++h) {
      const int gi = i0 + lr + h * RS;
      const bool ok = okk && gi < ns;
      cp16(da + h * RS * LD, ok ? P + (size_t)gi * K + k : P, ok);
    }
    if (!same) {
#pragma unroll
      for (int h = 0; h < NL; ++h) {
        const int gj = j0 + lr + h * RS;
        const bool ok = okk && gj < ns;
        cp16(db + h * RS * LD, ok ? X + (size_t)gj * K + k : X, ok);
      }
    }
    if (scaled && lr == 0) cp8(vs + buf * KB + lk, okk ? vp + (k < n3 ? k : k - n3) : vp, okk);
    cp_commit();
  };
  auto stage = [&](int buf, auto tc) {
    constexpr int T = decltype(tc)::value;
    const double* A = reinterpret_cast<const double*>(As + (size_t)buf * GT * LD);
    const double* V = vs + buf * KB;
    const double* B = same ? A : reinterpret_cast<const double*>(Bs + (size_t)buf * GT * LD);
    constexpr int NS = KB / 2 / G::WK;
    const int ks0 = G::WK == 1 ? 0 : (tid >> 5) * NS;
#pragma unroll 4
    for (int ks = ks0; ks < ks0 + NS; ++ks) {
      const int kd = 4 * ks + fk;      // double index of k' in the row
      double a[MB], bv[MB], bt[MB];
#pragma unroll
      for (int m = 0; m < MB; ++m) a[m] = A[(8 * (MB * rw + m) + fr) * (2 * LD) + kd];
#pragma unroll
      for (int v = 0; v < MB; ++v) {
        bv[v] = B[(8 * (MB * cw + v) + fr) * (2 * LD) + kd];
        if (scaled) bv[v] *= V[kd >> 1];
        const double o = __shfl_xor_sync(0xffffffffu, bv[v], 1);
        bt[v] = (fk & 1) ? -o : o;
      }
#pragma unroll
      for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int v = 0; v < MB; ++v) {
          if ((T == GF_UPPER && m > v) || (T == GF_LOWER && m < v)) continue;
          gd_mma(accR[m][v], a[m], bv[v]);
          gd_mma(accI[m][v], a[m], bt[v]);
        }
    }
  };
  load(0, k0);
  int buf = 0;
  for (size_t kb = k0; kb < k1; kb += KB) {
    if (kb + KB < k1) {
      load(buf ^ 1, kb + KB);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    sync();
    if (!idle) {
      if (half == 0) stage(buf, std::integral_constant<int, GF_FULL>{});
      else if (half == GF_UPPER) stage(buf, std::integral_constant<int, GF_UPPER>{});
      else stage(buf, std::integral_constant<int, GF_LOWER>{});
    }
    sync();
    buf ^= 1;
  }
  double2* o = part + ((size_t)tile * nchunk + chunk) * GT * GT;
  // (blocks of the other triangle keep zeros; the reduction does not read them)
  double2* dst = G::WK == 1 ? o : gf_smem + (tid >> 5) * GT * GT;
#pragma unroll
  for (int m = 0; m < MB; ++m)
#pragma unroll
    for (int v = 0; v < MB; ++v)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        dst[(8 * (MB * rw + m) + fr) * GT + 8 * (MB * cw + v) + 2 * fk + c] = make_double2(accR[m][v][c], accI[m][v][c]);
  if (G::WK > 1) {
    sync();
    for (int e = tid; e < GT * GT; e += GF_THREADS) {
      double2 s = gf_smem[e];
#pragma unroll
      for (int w = 1; w < G::WK; ++w) {
        const double2 t = gf_smem[w * GT * GT + e];
        s.x += t.x;
        s.y += t.y;
      }
      o[e] = s;
    }
    sync();   // the next item's stages overwrite the sums
  }
}

template <int GT>
__global__ void __launch_bounds__(GF_THREADS* GF_GROUPS, 1)
gram_f64_kernel(GfJob job, size_t K, size_t n3, const double2* __restrict__ psi, const double2* __restrict__ hampsi,
                const double2* __restrict__ hmfpsi, double2* part, int nchunk, int kchunk, int* ticket) {
  extern __shared__ double2 gf_smem[];
  __shared__ int next[GF_GROUPS];
  const int group = threadIdx.x / GF_THREADS, tid = threadIdx.x % GF_THREADS, bar = 1 + group;
  const int items = job.ntile * nchunk;
  for (;;) {
    if (tid == 0) next[group] = atomicAdd(ticket, 1);
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(GF_THREADS) : "memory");
    const int item = next[group];
    if (item >= items) return;
    gf_item<GT>(job, K, n3, psi, hampsi, hmfpsi, part, nchunk, kchunk, item,
                gf_smem + group * (GfGeo<GT>::SMEM / sizeof(double2)), tid, bar);
  }
}

struct GfOut {
  double2* p[8];   // [block * 4 + matrix]
};

// out_a[b][i][j] = wxyz * sum over slices (fixed order: eight interleaved
// partial sums per element, then those in turn); Hermitian matrices take the
// lower triangle from the upper one.
template <int GT>
__global__ void __launch_bounds__(256) gram_f64_reduce_kernel(GfJob job, int nchunk, const double2* __restrict__ part,
                                                              double scale, GfOut outs, int ldo, int* ticket) {
  __shared__ double2 red[8][33];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *ticket = 0;   // for the next launch
  int ti, tj;
  const GfGroup gr = gf_tile(job, blockIdx.y, ti, tj);
  const int ns = job.ns[gr.b], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  const int i = ti * GT + e / GT, j = tj * GT + e % GT;
  const bool want = i < ns && j < ns && !(gr.type == GF_UPPER && i > j) && !(gr.type == GF_LOWER && i < j);
  double re = 0.0, im = 0.0;
  if (want) {
    const double2* p = part + (size_t)blockIdx.y * nchunk * GT * GT + e;
#pragma unroll 4
    for (int c = w; c < nchunk; c += 8) {
      const double2 v = p[(size_t)c * GT * GT];
      re += v.x;
      im += v.y;
    }
  }
  red[w][lane] = make_double2(re, im);
  __syncthreads();
  if (w != 0 || !want) return;
#pragma unroll
  for (int q = 1; q < 8; ++q) {
    re += red[q][lane].x;
    im += red[q][lane].y;
  }
  double2* out = outs.p[gr.b * 4 + gr.a];
  out[(size_t)i * ldo + j] = make_double2(scale * re, scale * im);
  if (gr.type == GF_UPPER && i != j) out[(size_t)j * ldo + i] = make_double2(scale * re, -scale * im);
}

template <int GT>
int gram_f64_run(hfb_ctx_s* c, const GfJob& job, size_t K, const double2* psi, const double2* ham, const double2* hmf,
                 double wxyz, const GfOut& ot, int ldo, int nchunk, int kchunk, int sms, cudaStream_t st) {
  double2* part = (double2*)scratch(c, hfb_ctx_s::S_GRAM, sizeof(double2) * (size_t)job.ntile * nchunk * GT * GT);
  if (!part) return HFB_ERR_ALLOC;
  int* ticket = c->counters + 1;
  const int need = (job.ntile * nchunk + GF_GROUPS - 1) / GF_GROUPS;
  allow_max_dynamic_smem(gram_f64_kernel<GT>);
  gram_f64_kernel<GT><<<need < sms ? need : sms, GF_THREADS * GF_GROUPS, GF_GROUPS * GfGeo<GT>::SMEM, st>>>(
      job, K, K / 2, psi, ham, hmf, part, nchunk, kchunk, ticket);
  HFB_CHECK_LAUNCH();
  gram_f64_reduce_kernel<GT><<<dim3(GT * GT / 32, job.ntile), 256, 0, st>>>(job, nchunk, part, wxyz, ot, ldo, ticket);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

// ============================================================== rotate ====
// With the state index interleaved with (Re, Im), i' = 2 i + part,
//   A'[k][i'] = (Re, Im) psi_i(k),
//   Re out_j(k) = sum_i' A'[k][i'] Br[i'][j],  Br = (Re W_ij, -Im W_ij),
//   Im out_j(k) = sum_i' A'[k][i'] Bi[i'][j],  Bi = (Im W_ij,  Re W_ij),
// W = [U | L].  A CTA (8 warps, 16 grid points each) computes 128 points x
// 8 JB outputs, the states in three cp.async stages of 8, two CTAs per SM.
// (With stages loaded through registers each stage waited for its loads:
// 14 TFLOP/s.)  JB = 1..6 is the one with the least padding of the 2 ns
// columns of both isospins (280 and 192: JB = 5 and 6 cost the same, 64: 4);
// a tile costs its columns and about a third of a block for its points.
// Pb208 (140 + 96 states, 48^3): 7.2 ms before, 3.6 ms here (28 TFLOP/s).
constexpr int RF_KT = 128, RF_IT = 8, RF_ST = 3, RF_THREADS = 256;
constexpr int RF_PP = RF_KT + 4;   // row pitches: the two rows a load touches fall on distinct banks

template <int JB> struct RfGeo {
  static constexpr int JT = 8 * JB, WP = JT + 2;
  static constexpr size_t STAGE = (size_t)RF_IT * (RF_PP + WP);
  static constexpr size_t SMEM = sizeof(double2) * RF_ST * STAGE;
};

struct RfJob {
  int s0[2], ns[2], njt[2];
  int blk1;                         // first CTA of the second isospin
  const double2 *U[2], *L[2];
};

template <int JB>
__global__ void __launch_bounds__(RF_THREADS, 2)
rotate_f64_kernel(RfJob job, size_t K, const double2* __restrict__ psi, int ld, double2* out1, double2* out2) {
  using G = RfGeo<JB>;
  constexpr int JT = G::JT, WP = G::WP;
  extern __shared__ double2 rf_smem[];
  const int b = (int)blockIdx.x >= job.blk1;
  const int blk = blockIdx.x - (b ? job.blk1 : 0);
  const int ns = job.ns[b], jt = blk % job.njt[b], j0 = jt * JT;
  const size_t k0 = (size_t)(blk / job.njt[b]) * RF_KT, base = (size_t)job.s0[b] * K;
  const double2* P = psi + base;
  const double2 *U = job.U[b], *L = job.L[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int fr = lane >> 2, fk = lane & 3;
  const bool im = fk & 1;
  double accR[2][JB][2], accI[2][JB][2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < JB; ++v) accR[u][v][0] = accR[u][v][1] = accI[u][v][0] = accI[u][v][1] = 0.0;
  const int lk = threadIdx.x % RF_KT, li = threadIdx.x / RF_KT;   // loader: 2 states x 128 points at a time
  const bool okk = k0 + lk < K;
  auto load = [&](int s) {
    double2* Ps = rf_smem + (s % RF_ST) * G::STAGE;
    double2* Ws = Ps + RF_IT * RF_PP;
    const int i0 = s * RF_IT;
    if (i0 < ns) {
#pragma unroll
      for (int h = 0; h < RF_IT / 2; ++h) {
        const int i = i0 + li + 2 * h;
        const bool ok = okk && i < ns;
        cp16(Ps + (li + 2 * h) * RF_PP + lk, ok ? P + (size_t)i * K + k0 + lk : P, ok);
      }
      for (int e = threadIdx.x; e < RF_IT * JT; e += RF_THREADS) {
        const int ii = e / JT, jj = e % JT, i = i0 + ii, j = j0 + jj;
        const bool ok = i < ns && j < 2 * ns;
        const double2* w = !ok ? U : j < ns ? U + (size_t)i * ld + j : L + (size_t)i * ld + (j - ns);
        cp16(Ws + ii * WP + jj, w, ok);
      }
    }
    cp_commit();
  };
  const int nst = (ns + RF_IT - 1) / RF_IT;
  load(0);
  load(1);
  for (int s = 0; s < nst; ++s) {
    cp_wait<1>();
    __syncthreads();
    load(s + 2);     // into the stage every warp has left
    const double* Pd = reinterpret_cast<const double*>(rf_smem + (s % RF_ST) * G::STAGE);
    const double2* Ws = rf_smem + (s % RF_ST) * G::STAGE + RF_IT * RF_PP;
#pragma unroll
    for (int kk = 0; kk < RF_IT / 2; ++kk) {
      const int ii = 2 * kk + (fk >> 1);     // state of this lane's k' within the step
      double a[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) a[u] = Pd[2 * (ii * RF_PP + 16 * warp + 8 * u + fr) + (fk & 1)];
#pragma unroll
      for (int v = 0; v < JB; ++v) {
        const double2 w = Ws[ii * WP + 8 * v + fr];
        const double br = im ? -w.y : w.x, bi = im ? w.x : w.y;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          gd_mma(accR[u][v], a[u], br);
          gd_mma(accI[u][v], a[u], bi);
        }
      }
    }
  }
  cp_wait<0>();
  // the thread holds rows k = 16 warp + 8 u + fr, columns j = 8 v + 2 fk + c
#pragma unroll
  for (int v = 0; v < JB; ++v)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int j = j0 + 8 * v + 2 * fk + c;
      if (j >= 2 * ns) continue;
      double2* o = (j < ns ? out1 + (size_t)j * K : out2 + (size_t)(j - ns) * K) + base;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const size_t k = k0 + 16 * warp + 8 * u + fr;
        if (k < K) o[k] = make_double2(accR[u][v][c], accI[u][v][c]);
      }
    }
}

template <int JB>
int rotate_f64_run(RfJob job, size_t K, const double2* psi, int ld, double2* out1, double2* out2, cudaStream_t st) {
  const size_t nkt = (K + RF_KT - 1) / RF_KT;
  for (int b = 0; b < 2; ++b) job.njt[b] = (2 * job.ns[b] + 8 * JB - 1) / (8 * JB);
  job.blk1 = (int)(nkt * job.njt[0]);
  const size_t blocks = nkt * (job.njt[0] + job.njt[1]);
  allow_max_dynamic_smem(rotate_f64_kernel<JB>);
  rotate_f64_kernel<JB><<<(unsigned)blocks, RF_THREADS, RfGeo<JB>::SMEM, st>>>(job, K, psi, ld, out1, out2);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

}  // namespace

int gram_f64_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const int* masks, const void* psi,
                    const void* hampsi, const void* hmfpsi, const double* const* vp, double wxyz,
                    double2* const* outs, int ldo, int leave, cudaStream_t st) {
  const size_t K = (size_t)2 * c->n * c->n * c->n;
  // tile edge by the MMA work of Hermitian matrices; the smaller edges have
  // fewer MMAs per fragment load.  Time at the same work against edge 48 at
  // 48^3, S + H: 140 states, edge 32 1.09, 24 1.02, 16 1.11; 48 states, 24 1.05,
  // 16 1.17.  With these factors the choice is the fastest edge or within 5 % of
  // it for 10 to 140 states from 24^3 to 48^3 (with all of lambda, whose work is
  // not halved, up to 20 % off at 48 states)
  const int edge[4] = {48, 32, 24, 16};
  const double slow[4] = {1.0, 1.05, 1.1, 1.25};
  int gt = 48, tiles = 0;
  double best = 0.0;
  for (int q = 0; q < 4; ++q) {
    int n = 0;
    for (int b = 0; b < nblk; ++b) {
      const int t = (ns[b] + edge[q] - 1) / edge[q];
      n += t * (t + 1) / 2;
    }
    const double cost = slow[q] * n * edge[q] * edge[q];
    if (q == 0 || cost < best) {
      best = cost;
      gt = edge[q];
      tiles = n;
    }
  }
  GfJob job{};
  GfOut ot{};
  for (int b = 0; b < nblk; ++b) {
    job.s0[b] = s0[b];
    job.ns[b] = ns[b];
    job.vp[b] = vp ? vp[b] : nullptr;
    const int nt = (ns[b] + gt - 1) / gt;
    for (int a = 0; a < 4; ++a) {
      ot.p[b * 4 + a] = outs[b * 4 + a];
      if (!(masks[b] & (1 << a)) || ns[b] <= 0) continue;
      const int type = a != 1 ? GF_UPPER : (masks[b] & kGramLowerLambda) ? GF_LOWER : GF_FULL;
      job.g[job.ngroup++] = GfGroup{b, a, type, nt, job.ntile};
      job.ntile += type == GF_FULL ? nt * nt : nt * (nt + 1) / 2;
    }
  }
  if (job.ntile == 0) return HFB_OK;
  const int kb = gt >= 32 ? 16 : 32;
  auto slice = [&](int tickets) {
    const int n = tickets * GF_GROUPS * c->sms / (2 * tiles);
    const size_t kc = (K + (n < 1 ? 1 : n) - 1) / (n < 1 ? 1 : n);
    return (int)((kc + kb - 1) / kb * kb);
  };
  int tickets = 4;
  while (tickets > 1 && slice(tickets) < 1024) --tickets;
  int kchunk = slice(tickets);
  if (kchunk < 128) kchunk = 128;
  const int nchunk = (int)((K + kchunk - 1) / kchunk);
  const int sms = c->sms - leave;
  const double2 *p = (const double2*)psi, *h = (const double2*)hampsi, *m = (const double2*)hmfpsi;
  switch (gt) {
    case 48: return gram_f64_run<48>(c, job, K, p, h, m, wxyz, ot, ldo, nchunk, kchunk, sms, st);
    case 32: return gram_f64_run<32>(c, job, K, p, h, m, wxyz, ot, ldo, nchunk, kchunk, sms, st);
    case 24: return gram_f64_run<24>(c, job, K, p, h, m, wxyz, ot, ldo, nchunk, kchunk, sms, st);
    default: return gram_f64_run<16>(c, job, K, p, h, m, wxyz, ot, ldo, nchunk, kchunk, sms, st);
  }
}

int rotate_f64_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const void* psi, const double2* const* U,
                      const double2* const* L, int ld, void* out1, void* out2, cudaStream_t st) {
  const size_t K = (size_t)2 * c->n * c->n * c->n;
  RfJob job{};
  for (int b = 0; b < nblk; ++b) {
    job.s0[b] = s0[b];
    job.ns[b] = ns[b];
    job.U[b] = U[b];
    job.L[b] = L[b];
  }
  int jb = 6;
  double best = 0.0;
  for (int q = 6; q >= 1; --q) {
    double cost = 0.0;
    for (int b = 0; b < nblk; ++b) cost += ((2 * ns[b] + 8 * q - 1) / (8 * q)) * (q + 0.35);
    if (q == 6 || cost < best) {
      best = cost;
      jb = q;
    }
  }
  if (job.ns[0] <= 0 && job.ns[1] <= 0) return HFB_OK;
  const double2* p = (const double2*)psi;
  double2 *o1 = (double2*)out1, *o2 = (double2*)out2;
  switch (jb) {
    case 6: return rotate_f64_run<6>(job, K, p, ld, o1, o2, st);
    case 5: return rotate_f64_run<5>(job, K, p, ld, o1, o2, st);
    case 4: return rotate_f64_run<4>(job, K, p, ld, o1, o2, st);
    case 3: return rotate_f64_run<3>(job, K, p, ld, o1, o2, st);
    case 2: return rotate_f64_run<2>(job, K, p, ld, o1, o2, st);
    default: return rotate_f64_run<1>(job, K, p, ld, o1, o2, st);
  }
}

}  // namespace hfb
