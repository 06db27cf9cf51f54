// Dense FP64 building blocks of the reconstructor and of the Cee/Cvv chain.
#ifndef MOAO_DENSE_H
#define MOAO_DENSE_H

#include <cuda_runtime.h>

#include "moao_internal.h"

namespace moao {

// Which part of the STORED B matrix a GEMM may read (the rest is taken as 0):
// used to multiply by a symmetric matrix held in its lower triangle.
enum TriMode { TRI_FULL = 0, TRI_LOWER = 1, TRI_STRICT_LOWER = 2 };

struct GemmArgs {
  long M = 0, N = 0, K = 0;
  double alpha = 1, beta = 0;
  const double* A = nullptr;  // M x K, column-major, lda
  long lda = 0;
  const double* B = nullptr;  // K x N (transB = false) or N x K (transB = true)
  long ldb = 0;
  bool transB = false;
  TriMode triB = TRI_FULL;
  long tri_off = 0;           // column index of B's first column (triB != TRI_FULL)
  double* C = nullptr;        // M x N, column-major, ldc
  long ldc = 0;
  bool lowerC = false;        // write only C(i, j) with i >= j (SYRK / SYR2K)
  bool chained = false;       // may start beside its predecessor in the stream (dense_f64.cu)
  int cfg = 1;                // tile configuration of the large products (128x64 CTA tiles;
                              // 0: K 16 per stage, 4 stages; 1: K 32, 2 stages (default);
                              // 2: K 32, 3 stages; 3: K 16, 6 stages)
};
constexpr int kGemmConfigs = 4;

// C = alpha * A * op(B) + beta * C in FP64 on the DMMA tensor-core path.
moao_status gemm_f64(const GemmArgs& g, cudaStream_t s, long long* launches);

// The same product on the tiles [tile0, tile0 + tiles) of a 128 x 256-tile walk
// over C (tile_walk.cuh), only when *flag_a or *flag_b (device) is nonzero.
moao_status gemm_f64_guarded(const GemmArgs& g, long tile0, long tiles, const int* flag_a,
                             const int* flag_b, cudaStream_t s, long long* launches);

// Factor the n x n (n <= 64) diagonal block A (lower triangle read) in place:
// A <- L (lower; the upper triangle is left untouched) and Linv <- L^-1 (lower,
// zeros above the diagonal, ldi). On a non-positive pivot the 1-based global
// column (col0 + local column + 1) is stored in *d_info if it is still 0.
moao_status potrf_inv_leaf(double* A, long lda, double* Linv, long ldi, int n, long col0,
                           int* d_info, bool chained, cudaStream_t s, long long* launches);

// Factor and inverse of the nb x nb diagonal block A in one cooperative launch of `ctas`
// CTAs (nb for which diag_block_fits). W: nb^2 doubles, d_sync: one word. A barrier whose
// wait (of `polls` polls, 0: the default, some seconds) ran out raises d_info[1].
bool diag_block_fits(long nb);
moao_status diag_block(double* A, long lda, double* D, long ldd, long nb, long col0, int* d_info,
                       double* W, unsigned* d_sync, int ctas, unsigned polls, cudaStream_t s,
                       long long* launches);

// Elementwise helpers (column-major).
moao_status copy_matrix(const double* src, long lds, double* dst, long ldd, long m, long n,
                        cudaStream_t s, long long* launches = nullptr);
// dst (m x n) = src and the zm x zn block at z = 0, in one launch.
moao_status copy_zero(const double* src, long lds, double* dst, long ldd, long m, long n, double* z,
                      long ldz, long zm, long zn, bool chained, cudaStream_t s,
                      long long* launches);
// Cee <- sym(tril(Cpp)): the net effect of laset('U',0,0) + lacpy('L') +
// geadd('T') + scal(diag, 0.5) in lapack/compute/cee_cvv.cpp:73-92.
moao_status sym_from_lower(const double* Cpp, long ldp, double* Cee, long lde, long n,
                           cudaStream_t s, long long* launches);

}  // namespace moao

#endif  // MOAO_DENSE_H
