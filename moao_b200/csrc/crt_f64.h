// FP64 products on the int8 tensor cores (see crt_f64.cu).
#ifndef MOAO_CRT_F64_H
#define MOAO_CRT_F64_H

#include <cuda_runtime.h>

#include "context.h"
#include "dense.h"

namespace moao {

// One operand of a product: its rows (the M rows of A, or the N columns of
// op(B)) as residues, K entries each.
struct CrtOperand {
  long rows = 0, K = 0, ldq = 0;  // ldq: K rounded up to 128
  int8_t* q = nullptr;            // kCrt64Moduli planes of rows x ldq
  int* erow = nullptr;            // per row: largest biased exponent
  int* flag = nullptr;            // its guard
};

// Whether C (M x N) over K is faster as residue products than on the FP64
// tensor cores (lower: C's lower triangle only).
bool crt64_pays(const moao_ctx* ctx, long M, long N, long K, bool lower);

// Forms of a second operand: CRT_ROWS a column-major rows x K matrix, CRT_COLS the
// columns of a column-major K x rows matrix, CRT_SYM columns of the symmetric K x K
// matrix held in its lower triangle.
enum CrtForm { CRT_ROWS = 0, CRT_COLS = 1, CRT_SYM = 2 };

// Lowers the operands' guard: before the first operand of a product.
moao_status crt64_begin(moao_ctx* ctx);

// The rows of a column-major rows x K matrix as an operand for products with
// itself, in the context's buffers.
moao_status crt64_operand(moao_ctx* ctx, const double* A, long lda, long rows, long K,
                          CrtOperand* out);

// The same operand for a group of panels, in buffers and under a guard of its own: it
// outlives the operands of other products. Reserve: its buffers for up to n rows and K
// columns, and those of its panels of nb, so that nothing is allocated in between.
moao_status crt64_reserve_group(moao_ctx* ctx, long n, long nb, long K);
moao_status crt64_group_operand(moao_ctx* ctx, const double* A, long lda, long rows, long K,
                                CrtOperand* out);

// fp64[0] from the operands' rows [a0, a0 + M) and [b0, b0 + N). Where the guard
// is raised (a non-finite value or an exponent out of range in an operand, or a
// tensor-core wait that ran out) the FP64 tensor cores compute fp64[0..n - 1] in
// turn instead, whose sum of products is the same.
moao_status crt64_product(moao_ctx* ctx, const CrtOperand& A, long a0, const CrtOperand& B, long b0,
                          const GemmArgs* fp64, int n, int max_ctas = 0);

// Scales of the variables that K runs over: A's column k is scaled by 2^(sign e_k)
// and op(B)'s by the inverse, e_k the exponent of diag[k * stride] (half: half of
// it, for a diagonal of variances).
struct CrtBalance {
  const double* diag;
  long stride;
  int half, sign;
};

// g (triB: full) by residue products, operands included. MOAO_ERR_OOM: C is as given.
moao_status crt64_gemm(moao_ctx* ctx, const GemmArgs& g, const CrtBalance* bal);
// C (M x n) = A (M x n) S, S the symmetric n x n matrix in the lower triangle of B.
moao_status crt64_symm(moao_ctx* ctx, long M, long n, const double* A, long lda, const double* B,
                       long ldb, double* C, long ldc);

// Blocks whose update of what lies beyond them is taken together: in the factorisation,
// where longer groups leave less to run beside the diagonal blocks, and in the solves.
constexpr long kFactorGroup = 2, kSolveGroup = 4;

// Device bytes the residue products of an FP64 reconstructor (nmeas n, nmeasts m,
// panel nb) and, with nact > 0, of the Cee/Cvv chain hold on a context.
size_t crt64_bytes(long n, long m, long nb, long nact);

}  // namespace moao

#endif  // MOAO_CRT_F64_H
