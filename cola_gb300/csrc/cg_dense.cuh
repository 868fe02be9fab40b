// The one-exchange fused CG of a single Dense operator (cg_dense.cu), called by cg.cu.
#pragma once

#include "common.cuh"

namespace colagb {

template <class T, class S>
struct DenseCgArgs {
  const S* A;
  int64_t lda;
  int n, k;
  T shift;          // A + shift * I
  const T* dinv;    // Jacobi diagonal or null
  const T* B;
  int64_t ldb;
  T* X;             // x0 on entry, the solution on return
  int64_t ldx;
  T* AP;            // two exchange buffers of k * (n rounded up to 4) each
  double tol;
  int max_iters;
  int aligned;      // the rows start at quad boundaries and n % 4 == 0
  int resident;     // set by the launch: a CTA's rows are kept in shared memory
  int wc, few;      // set by the launch: how the warps share a CTA's rows
  T* hist;
  int* iters;
  unsigned int* count;  // grid barrier counter, zero at launch
  int* err;
  long long spin_limit;
};

// Launches the solve when the problem fits (*ran), else leaves it to the general kernel.
template <class T, class S>
int cg_dense_solve(DenseCgArgs<T, S>& a, cudaStream_t st, bool* ran);

}  // namespace colagb
