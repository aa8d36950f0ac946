// Single-precision Gram matrices on the tcgen05 tensor cores.
//
// C_a[i][j] = wxyz <psi_i | x_j> (X = psi, hampsi, hmfpsi, v_pair psi;
// static.py:283-290, 380-387 and construct_hfb_matrices 484-577) for complex64
// states.  Operands are split as x = hi + lo with hi = tf32(x), lo = x - hi
// (exact, left unrounded: the MMA takes its tf32 part) and D accumulates
// hi*hi + hi*lo + lo*hi (the three-term tf32 scheme, about 21 significant
// bits per product).
//
// A unit is 128 rows x_j (the requested matrices' vectors j, interleaved) by
// up to 144 columns psi_i of one isospin.  Producers store real and imaginary
// parts of 16 points side by side in a 128-byte row, so one staged block
// serves both
//   D_re = x_r psi_r + x_i psi_i   and   D_im = x_i psi_r - x_r psi_i
// (the minus sign is the descriptor's).  Only one triangle is computed: i >= j
// of S and of lambda (the eigensolver reads its lower triangle; all of lambda
// when the caller wants it), i <= j of H and G, whose rows go by descending j.
// The columns of a block start or end at its first row's j, which leaves 56 %
// of them for two matrices of 140 states.
//
// Work items are (K slice, unit), handed out by a ticket to one CTA per SM
// (fewer when the launch is to leave SMs to what runs beside it).  The slices
// depend on the grid alone, so no sum's order depends on which matrices are
// computed together.
//   warps 0-5   split a block of 16 points of the rows from the raw ring into
//               a 128-byte-swizzled stage (two of them);
//   warp 6      fills the raw ring by TMA, 16 rows a copy (two blocks and up
//               in flight: rows lie a state apart, 1.8 MB at 48^3, so every
//               row of a block is another page and a block takes 1.4 us to
//               arrive; a block ahead in registers left the MMAs waiting);
//   warp 7      issues the MMAs (M = 128, N = columns, K = 8) into TMEM
//               accumulators, three in rotation for D_re and D_im, which start
//               from zero every four blocks;
//   warps 8-15  drain the finished accumulator into fp32 registers, four warps
//               D_re and four D_im, so the tensor core's own fp32 accumulation
//               spans at most 48 MMAs and the sum over drains is rounded to
//               nearest.
// Per-slice partial sums are added in fp64 in a fixed order by a second
// kernel, which also writes the mirrored elements.
// A row that is also a column (S, G) is loaded once and stored twice.
// Pb208 (140 + 96 states, 48^3), S + lambda and H + G: 3.04 ms with the real
// and imaginary rows in units of their own (each loaded and split separately),
// 2.4 ms with the rows loaded through registers, 1.37 ms here; Zr90 (61 + 47
// states, 40^3, S + H + G): 329, 337, 262 us.
// Every wait is bounded; a timeout latches HFB_ERR_CUDA, drains the MMAs
// in flight and releases TMEM before returning.
#include <math.h>
#include <algorithm>
#include "diag.cuh"
#include "tc_sm100.cuh"

namespace hfb {

namespace {

constexpr int kTcSplitWarps = 6, kTcLoadWarp = 6, kTcMmaWarp = 7, kTcEpilogueWarps = 8;
constexpr int kTcThreads = 32 * (kTcMmaWarp + 1 + kTcEpilogueWarps);
// registers: 512 x 128 at launch, then 256 x 72 + 256 x 184
constexpr int kTcProducerRegs = 72, kTcEpilogueRegs = 184;
constexpr int kTcStages = 2, kTcMaxRaw = 8;   // split and raw stages
constexpr int kTcMaxNp = 160;           // padded states per isospin handled here
constexpr int kTcMaxCols = 144;         // columns of a unit: the epilogue's accumulator registers
constexpr int kTcMaxUnits = 32;
constexpr int kTcBoxRows = 16, kTcBoxBytes = kTcBoxRows * 128;
constexpr int kTcMaxBoxes = 18;         // columns, rows among them or not, other rows: 9 + 8 at most
constexpr int kTcItems = 6;             // 32-byte row quarters per splitting thread and block
static_assert(kTcItems * kTcSplitWarps * 32 >= 4 * kTcBoxRows * kTcMaxBoxes, "splitters' share");
constexpr int kTcTmemCols = 512, kTcAccCols = 160;   // three accumulators
// up to this many states hi*(hi|lo) is one MMA of twice the columns, which is
// what an accumulator holds; by the states of the isospin, not the columns of
// the unit, so that it depends on nothing else.  16 states at 48^3 (S + lambda)
// 171 us against 179 apart, 48 states 220 and 222, 80 states 269 and 265; all
// four matrices at 40^3: 16 states 171 and 173, 61 states 251 and 247
constexpr int kTcPairCols = kTcAccCols / 2;
constexpr uint32_t kTcABytes = 128 * 128;   // 128 rows x 128 bytes
constexpr long long kTcWaitLimit = 2000000000LL;
// Blocks accumulated in TMEM between drains into registers: 4 measured 6 %
// faster than 1 and stays inside the 3e-6 bar of the single-precision Gram
// test
constexpr int kTcDrain = 4;
// K slices: enough that the last wave of items is short, at least six drains
constexpr int kTcMaxSlices = 148, kTcMinSlice = 24;
constexpr int kTcMaxWin = 48 * 48 * 48 / 8 / kTcMaxSlices + 1;   // blocks of a slice of the largest grid
constexpr size_t kTcVps = sizeof(float) * 16 * kTcMaxWin;
constexpr size_t kTcSmem = 226 * 1024;   // the rings take what they get
static_assert(kTcMaxWin > 2 * kTcMinSlice, "slices of small grids");

constexpr uint32_t kNone = 0xffffffffu;
enum TcGroup { TC_LOWER = 0, TC_UPPER = 1, TC_FULL = 2, TC_GROUPS = 3 };   // S and lambda; H and G; lambda

struct TcUnit {
  unsigned char b, group;      // isospin, TcGroup
  short row0, col0, cols;      // first stacked row; first column and padded count
  short extra0, extra_n;       // psi rows of S or G that are not columns
  short x0, x_n, xmap;         // rows of lambda or H, and their array
  int off;                     // of its sums among a slice's: [re, im][128][cols]
  __host__ __device__ int boxes() const {
    return cols / kTcBoxRows + (extra_n + kTcBoxRows - 1) / kTcBoxRows + (x_n + kTcBoxRows - 1) / kTcBoxRows;
  }
};
struct TcMaps {
  CUtensorMap m[2][3];         // [isospin][psi, hampsi, hmfpsi]
};
struct TcJob {
  int nunit, slices, kb_total, n3, slice_sums;
  uint32_t stage_bytes, raw_bytes;
  int raw_stages;
  TcUnit u[kTcMaxUnits];
  int s0[2], ns[2];
  int nm[2][TC_GROUPS];        // [isospin][group] matrices stacked
  unsigned char mat[2][TC_GROUPS][2];   // their numbers
  const double* vp[2];
};

__device__ __forceinline__ void tc_sync_all() { asm volatile("bar.sync 1, %0;" ::"n"(kTcThreads) : "memory"); }

__global__ void __launch_bounds__(kTcThreads, 1)
gram_tc_kernel(const __grid_constant__ TcJob job, const __grid_constant__ TcMaps maps, float* __restrict__ part,
               int* ticket, int* status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[kTcStages], empty[kTcStages], rfull[kTcMaxRaw], rempty[kTcMaxRaw], dfull[3], dempty[3], fin;
  __shared__ uint32_t tbase;
  __shared__ volatile int abort_flag;
  __shared__ volatile int next[2];

  unsigned char* raw = smem + kTcStages * job.stage_bytes;
  float* vps = reinterpret_cast<float*>(raw + job.raw_stages * job.raw_bytes);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31;
  const int items = job.nunit * job.slices;
  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(&full[s], kTcSplitWarps);
      tc::mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < kTcMaxRaw; ++s) {
      tc::mbar_init(&rfull[s], 1);
      tc::mbar_init(&rempty[s], kTcSplitWarps);
    }
    for (int d = 0; d < 3; ++d) {
      tc::mbar_init(&dfull[d], 1);
      tc::mbar_init(&dempty[d], kTcEpilogueWarps / 2);
    }
    tc::mbar_init(&fin, 1);
    abort_flag = 0;
    next[0] = atomicAdd(ticket, 1);
  }
  if (warp == kTcMmaWarp) {
    tc::tmem_alloc(&tbase, kTcTmemCols);
    tc::tmem_relinquish();
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tbase;

  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    if (tc::mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!tc::mbar_try_wait(bar, parity)) {
      if (abort_flag) return false;
      if (clock64() - t0 > kTcWaitLimit) {
        abort_flag = 1;
        latch_error(status, HFB_ERR_CUDA);
        return false;
      }
    }
    return true;
  };
  // The next item, or -1; every role calls it once per item, after its part of
  // the last one.  The first block of the slice in kb0, their number in nwin.
  auto take = [&](int it, int& kb0, int& nwin) -> int {
    tc_sync_all();
    const int item = next[it & 1];
    if (item >= items || abort_flag) return -1;
    const int slice = item / job.nunit;
    kb0 = (int)((long long)job.kb_total * slice / job.slices);
    nwin = (int)((long long)job.kb_total * (slice + 1) / job.slices) - kb0;
    return item;
  };
  int kb0, nwin;

  if (warp <= kTcMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcProducerRegs));
    if (warp < kTcSplitWarps) {
      // -------------------------------------------------------- splitters
      const int q = tid & 3;                              // 32-byte quarter of the row
      int w = 0;                                          // blocks since the start
      for (int it = 0;; ++it) {
        const int item = take(it, kb0, nwin);
        if (item < 0) break;
        if (tid == 0) next[(it + 1) & 1] = atomicAdd(ticket, 1);
        const TcUnit U = job.u[item % job.nunit];
        const int b = U.b, n = job.ns[b], nm = job.nm[b][U.group];
        const int cb = U.cols, eb = (U.extra_n + kTcBoxRows - 1) / kTcBoxRows * kTcBoxRows;
        const int count = (U.boxes() * kTcBoxRows * 4 + kTcSplitWarps * 32 - 1) / (kTcSplitWarps * 32);
        const bool upper = U.group == TC_UPPER, sg = job.mat[b][U.group][upper ? nm - 1 : 0] == (upper ? 3 : 0);
        // place of row j of S or G / of lambda or H among the stacked rows
        auto row_sg = [&](int j) { return (upper ? (n - 1 - j) * nm + nm - 1 : j * nm) - U.row0; };
        auto row_x = [&](int j) { return (upper ? (n - 1 - j) * nm : j * nm + nm - 1) - U.row0; };
        uint32_t dst[kTcItems], dup[kTcItems];   // place, and for a column that is also a row, that place
        unsigned gmask = 0;
        auto raw_row = [&](int p) {
          // eight threads take rows r and r ^ 5: both the raw chunks and the
          // split ones fall on distinct banks
          const int e = (p * kTcSplitWarps * 32 + tid) >> 2;
          return (e & ~7) | (((e & 7) >> 1) ^ ((e & 1) * 5));
        };
#pragma unroll
        for (int p = 0; p < kTcItems; ++p) {
          const int r = raw_row(p);
          dst[p] = dup[p] = kNone;
          if (r < cb) {
            const int i = U.col0 + r, g = row_sg(i);
            if (i < n) {
              dst[p] = 2 * kTcABytes + tc::sw128_offset(r, q);
              if (sg && g >= 0 && g < 128) dup[p] = tc::sw128_offset(g, q);
            }
          } else if (r < cb + eb) {
            const int k = r - cb, j = U.extra0 + k;
            if (k < U.extra_n && !(j >= U.col0 && j < U.col0 + U.cols)) {
              dst[p] = tc::sw128_offset(row_sg(j), q);
              if (upper) gmask |= 1u << p;
            }
          } else {
            const int k = r - cb - eb;
            if (k < U.x_n) dst[p] = tc::sw128_offset(row_x(U.x0 + k), q);
          }
        }
        if (upper && sg) {   // v_pair of the slice
          const double* vp = job.vp[b];
          for (int e = tid; e < 16 * nwin; e += 32 * kTcSplitWarps)
            vps[e] = (float)vp[((size_t)kb0 * 16 + e) % (size_t)job.n3];
          asm volatile("bar.sync 2, %0;" ::"n"(32 * kTcSplitWarps) : "memory");
        }
        auto scale = [&](float4 (&x)[2], int i) {
          const float4 v = *reinterpret_cast<const float4*>(vps + 16 * i + 4 * q);
          x[0] = make_float4(v.x * x[0].x, v.x * x[0].y, v.y * x[0].z, v.y * x[0].w);
          x[1] = make_float4(v.z * x[1].x, v.z * x[1].y, v.w * x[1].z, v.w * x[1].w);
        };
        auto put = [&](unsigned char* st, uint32_t at, uint32_t lo, const float4 (&x)[2]) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {   // real parts, imaginary parts
            float4 h, l;
            tc::split_tf32(c ? x[0].y : x[0].x, h.x, l.x);
            tc::split_tf32(c ? x[0].w : x[0].z, h.y, l.y);
            tc::split_tf32(c ? x[1].y : x[1].x, h.z, l.z);
            tc::split_tf32(c ? x[1].w : x[1].z, h.w, l.w);
            unsigned char* t = st + (at ^ (c ? 64u : 0u));
            *reinterpret_cast<float4*>(t) = h;
            *reinterpret_cast<float4*>(t + lo) = l;
          }
        };
        for (int i = 0; i < nwin; ++i, ++w) {
          const int s = w % kTcStages, rs = w % job.raw_stages;
          if (!wait(&rfull[rs], (uint32_t)((w / job.raw_stages) & 1))) break;
          if (w >= kTcStages && !wait(&empty[s], (uint32_t)((w / kTcStages - 1) & 1))) break;
          unsigned char* st = smem + (size_t)s * job.stage_bytes;
          const unsigned char* rw = raw + (size_t)rs * job.raw_bytes;
#pragma unroll
          for (int h = 0; h < kTcItems; h += 3) {
            float4 d[3][2];
#pragma unroll
            for (int k = 0; k < 3; ++k)
              if (h + k < count) {
                const int r = raw_row(h + k);
                d[k][0] = *reinterpret_cast<const float4*>(rw + tc::sw128_offset(r, 2 * q));
                d[k][1] = *reinterpret_cast<const float4*>(rw + tc::sw128_offset(r, 2 * q + 1));
              }
            if (h + 3 >= kTcItems) {
              __syncwarp();
              if (lane == 0) tc::mbar_arrive(&rempty[rs]);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const int p = h + k;
              if (p >= count || dst[p] == kNone) continue;
              if ((gmask >> p) & 1) scale(d[k], i);
              put(st, dst[p], dst[p] >= 2 * kTcABytes ? (uint32_t)U.cols * 128 : kTcABytes, d[k]);
              if (dup[p] != kNone) {
                if (upper) scale(d[k], i);
                put(st, dup[p], kTcABytes, d[k]);
              }
            }
          }
          tc::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&full[s]);
        }
      }
    } else if (warp == kTcLoadWarp) {
      // ------------------------------------------------------------ loads
      int w = 0;
      for (int it = 0;; ++it) {
        const int item = take(it, kb0, nwin);
        if (item < 0) break;
        const TcUnit U = job.u[item % job.nunit];
        const int boxes = U.boxes(), cbox = U.cols / kTcBoxRows, ebox = (U.extra_n + kTcBoxRows - 1) / kTcBoxRows;
        // this lane's box: its array and first row (rows past the last read as zero)
        const CUtensorMap* map = &maps.m[U.b][lane < cbox + ebox ? 0 : U.xmap];
        const int y = lane < cbox          ? U.col0 + kTcBoxRows * lane
                      : lane < cbox + ebox ? U.extra0 + kTcBoxRows * (lane - cbox)
                                           : U.x0 + kTcBoxRows * (lane - cbox - ebox);
        for (int i = 0; i < nwin; ++i, ++w) {
          const int rs = w % job.raw_stages;
          if (w >= job.raw_stages && !wait(&rempty[rs], (uint32_t)((w / job.raw_stages - 1) & 1))) break;
          if (lane == 0) tc::mbar_arrive_expect_tx(&rfull[rs], (uint32_t)(boxes * kTcBoxBytes));
          __syncwarp();
          if (lane < boxes)
            tc::tma_load_2d(raw + (size_t)rs * job.raw_bytes + lane * kTcBoxBytes, map, (kb0 + i) * 32, y, &rfull[rs]);
          __syncwarp();
        }
      }
      // no copy is in flight when the CTA ends
      for (int k = w > job.raw_stages ? w - job.raw_stages : 0; k < w; ++k)
        if (!tc::mbar_wait(&rfull[k % job.raw_stages], (uint32_t)((k / job.raw_stages) & 1), kTcWaitLimit))
          latch_error(status, HFB_ERR_CUDA);
    } else {
      // -------------------------------------------------------------- MMA
      int w = 0, grp = 0, nfin = 0;
      const bool one = tc::elect_one();
      const uint64_t stage0 = tc::sw128_desc(tc::smem_u32(smem));
      for (int it = 0;; ++it) {
        const int item = take(it, kb0, nwin);
        if (item < 0) break;
        // the whole warp runs the loop, so that descriptors stay uniform
        const uint32_t cols = __shfl_sync(0xffffffffu, (uint32_t)job.u[item % job.nunit].cols, 0);
        const uint32_t idesc = tc::idesc_tf32(128, cols), ineg = idesc | tc::kNegateA, lob = (cols * 128) >> 4;
        constexpr uint64_t loa = kTcABytes >> 4;
        const bool pair = __shfl_sync(0xffffffffu, job.ns[job.u[item % job.nunit].b], 0) <= kTcPairCols;
        const uint32_t idpair = tc::idesc_tf32(128, 2 * cols) - tc::idesc_tf32(128, cols);
        bool ok = true;
        for (int i = 0; i < nwin && ok; ++i, ++w) {
          const int s = w % kTcStages, er = 2 * grp, ei = er + 1;
          const bool first = i % kTcDrain == 0, last = i % kTcDrain == kTcDrain - 1 || i == nwin - 1;
          ok = wait(&full[s], (uint32_t)((w / kTcStages) & 1));
          if (first && er >= 3 && ok) ok = wait(&dempty[er % 3], (uint32_t)((er / 3 - 1) & 1));
          if (!ok) break;
          tc::fence_after();
          const uint64_t da = stage0 + (uint64_t)((uint32_t)s * (job.stage_bytes >> 4)), db = da + 2 * loa;
          const uint32_t dr = tmem + (uint32_t)(er % 3) * kTcAccCols, di = tmem + (uint32_t)(ei % 3) * kTcAccCols;
          auto mma3 = [&](uint32_t dt, int ka, int kb, uint32_t id, uint32_t acc) {
            if (pair) {
              tc::mma_tf32(dt, da + 2 * ka, db + 2 * kb, id + idpair, acc);
            } else {
              tc::mma_tf32(dt, da + 2 * ka, db + 2 * kb, id, acc);
              tc::mma_tf32(dt, da + 2 * ka, db + lob + 2 * kb, id, 1);
            }
            tc::mma_tf32(dt, da + loa + 2 * ka, db + 2 * kb, id, 1);
          };
          // k steps 0, 1 of a row: real parts, 2, 3: imaginary parts
          if (one) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mma3(dr, k, k, idesc, k > 0 || !first);
            if (last) tc::mma_commit(&dfull[er % 3]);
          }
          __syncwarp();
          if (first && ei >= 3) ok = wait(&dempty[ei % 3], (uint32_t)((ei / 3 - 1) & 1));
          if (!ok) break;
          tc::fence_after();
          if (one) {
#pragma unroll
            for (int k = 0; k < 2; ++k) mma3(di, 2 + k, k, idesc, k > 0 || !first);
#pragma unroll
            for (int k = 0; k < 2; ++k) mma3(di, k, 2 + k, ineg, 1);
            tc::mma_commit(&empty[s]);
            if (last) tc::mma_commit(&dfull[ei % 3]);
          }
          __syncwarp();
          if (last) ++grp;
        }
        // every MMA issued above has completed once this arrives
        if (one) tc::mma_commit(&fin);
        __syncwarp();
        if (!tc::mbar_wait(&fin, (uint32_t)(nfin & 1), kTcWaitLimit)) {
          abort_flag = 1;
          latch_error(status, HFB_ERR_CUDA);
        }
        ++nfin;
        __syncwarp();
      }
    }
  } else {
    // ----------------------------------------------------------- epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcEpilogueRegs));
    const int qd = warp & 3;                              // TMEM lane quarter of this warp
    const int im = (warp - kTcMmaWarp - 1) / 4;     // D_re or D_im
    int grp = 0;
    for (int it = 0;; ++it) {
      const int item = take(it, kb0, nwin);
      if (item < 0) break;
      const int ng = job.u[item % job.nunit].cols / 16;
      const bool pair = job.ns[job.u[item % job.nunit].b] <= kTcPairCols;
      float acc[kTcMaxCols / 16][16];
#pragma unroll
      for (int g = 0; g < kTcMaxCols / 16; ++g)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[g][i] = 0.f;
      bool ok = true;
      for (int i = 0; i < nwin; i += kTcDrain, ++grp) {
        const int e = 2 * grp + im;
        if (!wait(&dfull[e % 3], (uint32_t)((e / 3) & 1))) { ok = false; break; }
        tc::fence_after();
        const uint32_t ta = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(e % 3) * kTcAccCols;
#pragma unroll
        for (int g = 0; g < kTcMaxCols / 16; ++g)
          if (g < ng) {
            float v[16];
            tc::tmem_ld16(ta + (uint32_t)(g * 16), v);
#pragma unroll
            for (int c = 0; c < 16; ++c) acc[g][c] += v[c];
            if (pair) {
              tc::tmem_ld16(ta + (uint32_t)((ng + g) * 16), v);
#pragma unroll
              for (int c = 0; c < 16; ++c) acc[g][c] += v[c];
            }
          }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&dempty[e % 3]);
      }
      if (ok && !abort_flag) {
        const TcUnit& U = job.u[item % job.nunit];
        float* o = part + (size_t)(item / job.nunit) * job.slice_sums + U.off + (im * 128 + qd * 32 + lane) * U.cols;
#pragma unroll
        for (int g = 0; g < kTcMaxCols / 16; ++g)
          if (g < ng) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              *reinterpret_cast<float4*>(o + g * 16 + i) =
                  make_float4(acc[g][i], acc[g][i + 1], acc[g][i + 2], acc[g][i + 3]);
          }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == kTcMmaWarp) {
    tc::fence_after();
    tc::tmem_dealloc(tmem, kTcTmemCols);
  }
}

struct TcOut {
  double2* p[8];   // [block * 4 + matrix]
};

// out_a[b][i][j] = wxyz (D_re, D_im)[row of j][column of i], the K slices
// summed in fp64 in a fixed order (six interleaved sums, then those in turn).
// One block per row of a unit: four columns a thread, six threads over the
// slices.  (A launch per matrix and isospin with one thread per element: 73 us
// of a 2.3 ms Zr90 step.)
constexpr int kTcRedLanes = 6, kTcRedCols = kTcMaxCols / 4;
__global__ void __launch_bounds__(kTcRedLanes* kTcRedCols)
gram_tc_reduce_kernel(const __grid_constant__ TcJob job, const float* __restrict__ part, double scale,
                      const __grid_constant__ TcOut outs, int ldo, int* ticket) {
  __shared__ double red[kTcRedLanes][kTcRedCols][8];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *ticket = 0;   // for the next launch
  const TcUnit U = job.u[blockIdx.y];
  const int row = blockIdx.x, b = U.b, n = job.ns[b], nm = job.nm[b][U.group];
  const int g = U.row0 + row;
  if (g >= n * nm) return;
  const int j = U.group == TC_UPPER ? n - 1 - g / nm : g / nm, am = job.mat[b][U.group][g % nm];
  const int c4 = threadIdx.x % kTcRedCols, sl = threadIdx.x / kTcRedCols;
  const bool on = 4 * c4 < U.cols;
  double s[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = 0.0;
  if (on) {
    const float* p = part + U.off + row * U.cols + 4 * c4;
#pragma unroll 4
    for (int c = sl; c < job.slices; c += kTcRedLanes) {
      const float* o = p + (size_t)c * job.slice_sums;
      const float4 re = *reinterpret_cast<const float4*>(o);
      const float4 im = *reinterpret_cast<const float4*>(o + 128 * U.cols);
      s[0] += re.x; s[1] += re.y; s[2] += re.z; s[3] += re.w;
      s[4] += im.x; s[5] += im.y; s[6] += im.z; s[7] += im.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) red[sl][c4][i] = s[i];
  }
  __syncthreads();
  if (sl != 0 || !on) return;
#pragma unroll
  for (int q = 1; q < kTcRedLanes; ++q)
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] += red[q][c4][i];
  double2* out = outs.p[b * 4 + am];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = U.col0 + 4 * c4 + k;
    if (i >= n || (U.group == TC_LOWER && i < j) || (U.group == TC_UPPER && i > j)) continue;
    out[(size_t)i * ldo + j] = make_double2(scale * s[k], scale * s[4 + k]);
    if (am != 1 && i != j) out[(size_t)j * ldo + i] = make_double2(scale * s[k], -scale * s[4 + k]);
  }
}

}  // namespace

// Returns HFB_ERR_UNSUPPORTED_GRID when a block exceeds kTcMaxNp states or its
// arrays have no tensor map (base not 16-byte aligned)
// (the caller then uses the CUDA-core kernel).
int gram_tc_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const int* masks, const void* psi,
                   const void* hampsi, const void* hmfpsi, const double* const* vp, double wxyz,
                   double2* const* outs_host, int ldo, int leave, cudaStream_t st) {
  TcJob job{};
  job.n3 = c->n * c->n * c->n;
  job.kb_total = job.n3 / 8;
  TcMaps maps{};
  int boxes = 0, widest = 0;
  for (int b = 0; b < nblk; ++b) {
    if (ns[b] <= 0) continue;
    const int n = ns[b];
    job.s0[b] = s0[b];
    job.ns[b] = n;
    job.vp[b] = vp ? vp[b] : nullptr;
    if ((n + 15) / 16 * 16 > kTcMaxNp) return HFB_ERR_UNSUPPORTED_GRID;
    for (int a = 0; a < 4; ++a) {
      if (!(masks[b] & (1 << a))) continue;
      const int g = a >= 2 ? TC_UPPER : a == 1 && !(masks[b] & kGramLowerLambda) ? TC_FULL : TC_LOWER;
      job.mat[b][g][job.nm[b][g]++] = (unsigned char)a;
    }
    const void* arrays[3] = {psi, hampsi, hmfpsi};
    for (int a = 0; a < 3; ++a)
      if (a == 0 || (masks[b] & (1 << a))) {
        const float* base = (const float*)arrays[a] + (size_t)s0[b] * 4 * job.n3;
        // (the CUDA-core kernel takes any alignment)
        if (!encode_fp32_rows_map(&maps.m[b][a], base, 4 * (uint64_t)job.n3, n, kTcBoxRows))
          return HFB_ERR_UNSUPPORTED_GRID;
      }
    for (int g = 0; g < TC_GROUPS; ++g) {
      const int nm = job.nm[b][g];
      for (int row0 = 0; row0 < n * nm; row0 += 128) {
        const int first = g == TC_LOWER ? row0 / nm / 16 * 16 : 0, end = g == TC_UPPER ? n - row0 / nm : n;
        const int all = (end - first + 15) / 16 * 16;
        const int parts = (all + kTcMaxCols - 1) / kTcMaxCols, cols = (all / 16 + parts - 1) / parts * 16;
        for (int col0 = first; col0 < end; col0 += cols) {
          if (job.nunit >= kTcMaxUnits) return HFB_ERR_UNSUPPORTED_GRID;
          TcUnit u{(unsigned char)b, (unsigned char)g, (short)row0, (short)col0,
                   (short)std::min(cols, (end - col0 + 15) / 16 * 16), 0, 0, 0, 0, 0, 0};
          // the vectors j of the block's rows
          const int ja = row0 / nm, jb = (std::min(row0 + 128, n * nm) - 1) / nm;
          const int j0 = g == TC_UPPER ? n - 1 - jb : ja, jn = jb - ja + 1;
          for (int m = 0; m < nm; ++m) {
            const int a = job.mat[b][g][m];
            if (a == 1 || a == 2) {
              u.x0 = (short)j0;
              u.x_n = (short)jn;
              u.xmap = (short)a;
            } else if (j0 < col0 || j0 + jn > std::min(col0 + u.cols, n)) {
              u.extra0 = (short)j0;
              u.extra_n = (short)jn;
            }
          }
          if (u.boxes() > kTcMaxBoxes) return HFB_ERR_UNSUPPORTED_GRID;
          boxes = std::max(boxes, u.boxes());
          widest = std::max(widest, (int)u.cols);
          job.u[job.nunit++] = u;
        }
      }
    }
  }
  if (job.nunit == 0) return HFB_OK;
  // the widest units first, so that the last items of a launch are short
  std::stable_sort(job.u, job.u + job.nunit, [](const TcUnit& x, const TcUnit& y) { return x.cols > y.cols; });
  for (int u = 0; u < job.nunit; ++u) {
    job.u[u].off = job.slice_sums;
    job.slice_sums += 2 * 128 * job.u[u].cols;
  }
  job.slices = std::max(1, std::min(kTcMaxSlices, job.kb_total / kTcMinSlice));
  const int items = job.nunit * job.slices, sms = c->sms - leave;
  float* part = (float*)scratch(c, hfb_ctx_s::S_GRAM, sizeof(float) * (size_t)job.slices * job.slice_sums);
  if (!part) return HFB_ERR_ALLOC;
  int* ticket = c->counters + 1;
  allow_max_dynamic_smem(gram_tc_kernel);
  job.stage_bytes = 2 * kTcABytes + 2 * widest * 128;
  job.raw_bytes = (uint32_t)(boxes * kTcBoxBytes);
  job.raw_stages = std::min<int>(kTcMaxRaw, (kTcSmem - 1024 - kTcVps - kTcStages * job.stage_bytes) / job.raw_bytes);
  gram_tc_kernel<<<std::min(items, sms), kTcThreads, kTcSmem, st>>>(job, maps, part, ticket, c->dev_status);
  HFB_CHECK_LAUNCH();
  TcOut ot;
  for (int q = 0; q < 8; ++q) ot.p[q] = outs_host[q];
  gram_tc_reduce_kernel<<<dim3(128, job.nunit), kTcRedLanes * kTcRedCols, 0, st>>>(job, part, wxyz, ot, ldo, ticket);
  HFB_CHECK_LAUNCH();
  return HFB_OK;
}

}  // namespace hfb
