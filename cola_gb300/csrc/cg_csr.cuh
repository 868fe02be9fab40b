// The fused CG of a single CSR operator and one right-hand side over all SMs (cg_csr.cu), called by cg.cu.
#pragma once

#include "common.cuh"

namespace colagb {

template <class T, class S>
struct CsrCgArgs {
  const int32_t* indptr;
  const int32_t* indices;
  const S* vals;
  int n;
  T shift;          // A + shift * I
  const T* dinv;    // Jacobi diagonal or null
  const T* B;
  int64_t ldb;
  T* X;             // x0 on entry, the solution on return
  int64_t ldx;
  T *Z, *P0, *P1;   // exchange buffers of n entries each
  T* part;          // 2 x 2 x nb partial sums
  double tol;
  int max_iters;
  T* hist;
  int* iters;
  unsigned int* count;  // grid barrier counter, zero at launch
  int* err;
  long long spin_limit;
  int smem;         // set by the launch: dynamic shared memory bytes
  int gathers;      // set by the launch: the most CTAs that may lack a column window
  int longest;      // set by the launch: the most entries of a row
  unsigned int* votes;  // CTAs against taking the solve, zero at launch
};

// In *err: the CTAs left after the first barrier because of the pattern (a row longer than `longest`, or more
// than `gathers` CTAs whose columns are too far apart for a window); x is untouched, the general kernel takes it.
constexpr int kCsrLeft = -1;

// CTAs a solve uses (the caller provides 4 partials for each).
int cg_csr_blocks(int64_t n);

// Launches the solve when the problem fits (*ran), else leaves it to the general kernel.
template <class T, class S>
int cg_csr_solve(CsrCgArgs<T, S>& a, int64_t nnz, cudaStream_t st, bool* ran);

}  // namespace colagb
