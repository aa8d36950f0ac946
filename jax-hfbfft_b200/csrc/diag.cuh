// Shared by the translation units of the diagonalisation step.
#pragma once
#include "hfb_ctx.cuh"

namespace hfb {

struct Pair2 {
  int v[2];
};

// D += A B on the FP64 tensor cores, 8 x 8 x 4.
__device__ __forceinline__ void gd_mma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// ---- contract_f64.cu: Gram and rotation on the FP64 tensor cores -----------
// Mask bits 0-3 ask for S, lambda, H, G; with kGramLowerLambda matrix 1 is
// written on and below its diagonal only; ``leave`` SMs stay free.
constexpr int kGramLowerLambda = 16;
int gram_f64_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const int* masks, const void* psi,
                    const void* hampsi, const void* hmfpsi, const double* const* vp, double wxyz,
                    double2* const* outs, int ldo, int leave, cudaStream_t st);
// out1 = psi U, out2 = psi L for up to two blocks of states of one array
int rotate_f64_launch(hfb_ctx_s* c, int nblk, const int* s0, const int* ns, const void* psi, const double2* const* U,
                      const double2* const* L, int ld, void* out1, void* out2, cudaStream_t st);

// ---- diag_cluster.cu: matrix chains of the two isospins, one cluster each --
struct RefineArgs {
  Pair2 nper;
  int ld;
  const double2* A;   // lower triangles at A + b sA, leading dimension ld
  size_t sA;
  double* W;          // ascending eigenvalues at W + b sW
  size_t sW;
  double2* V;         // eigenvectors in the columns of V + b sV
  size_t sV;
  double tol;         // convergence: coupling relative to ||A||_F
  int* fallback;      // [nb]: set when the refinement does not apply to matrix b
};
size_t refine_bytes(int nb, int ld);
// begun: recorded once every CTA runs (or null)
int refine_launch(hfb_ctx_s* c, int nb, const RefineArgs& a, void* work, cudaEvent_t begun, cudaStream_t st);

struct LoewdinArgs {
  Pair2 nper, off;
  int ld;
  const double2* S;   // overlaps at S + b sS
  size_t sS;
  double2* U;         // S^-1/2 at U + b ld^2
  double* sp_norm;    // diagonal of S, by state
  int* status;
};
size_t loewdin_bytes(int ld);
// ``alone``: nothing else runs beside it, so each matrix may take a cluster of several SMs
int loewdin_launch(const LoewdinArgs& a, void* work, bool alone, cudaStream_t st);

struct ConstructArgs {
  Pair2 nper, off;
  int ld, nmax;
  int diagonalize, construct, ipair, tbcs;
  const double2* Ur;        // S^-1/2
  const double2* Vl;        // eigenvectors of lambda (diagonalize)
  double2* U;               // out: Ur Vl, or a copy of Ur
  const double2 *H, *G;     // old-basis matrices at + b sG
  size_t sG;
  double2* L;               // out: U lambda
  const double *wocc, *wguv, *pairwg, *wstates;
  double2 *hmat, *gmat, *symc, *lsave;
  double *sp_energy, *deltaf, *efluct;
};
size_t construct_bytes(int ld);
int construct_launch(const ConstructArgs& a, void* work, cudaStream_t st);

}  // namespace hfb
