// pb_cg_small.cuh -- PCG iterations of a short vector in one cooperative launch
// (pb_cg_small.cu).
#pragma once

#include "pb_ilu.cuh"

namespace pb {

template <class T>
struct CgSmallArgs {
  DevMat<T> A;              // natural layout: the diagonal copy or the sliced-ELLPACK copy
  const T* dinv = nullptr;  // point Jacobi, null: no preconditioner
  T *x = nullptr, *r = nullptr, *s = nullptr;   // solution, residual, M^-1 r
  T *p = nullptr, *p2 = nullptr;                // direction, and a second buffer for it
  KState* st = nullptr;     // after EPI_CG_INIT; updated as the epilogues of the kernels do
  double* hist = nullptr;
  double rtol = 0.0;
  int maxit = 0;            // iterations of this launch
  unsigned long long* slots = nullptr;   // cg_small_slots() words, zeroed before the solve
  unsigned tag0 = 0;        // iterations already tagged in the slots
  int* err = nullptr;
};

// CTAs of the launch for n rows with nnz entries, 0 when the separate kernels are for them.
template <class T> int cg_small_grid(int64_t n, int64_t nnz);
constexpr int kCgCopies = 16, kCgLine = 16;   // copies of a grid sum's total, a 128-byte line each
// Words of both sums: at most four per CTA and the total's copies, each.
__host__ __device__ constexpr size_t cg_small_slots(int grid) {
  return 2 * ((((size_t)grid * 4 + kCgLine - 1) & ~(size_t)(kCgLine - 1)) + kCgCopies * kCgLine);
}
template <class T> void cg_small(const CgSmallArgs<T>& a, cudaStream_t st);

}  // namespace pb
