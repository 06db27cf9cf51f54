// Orchestration of the FP64 dense stages on one stream.
//
//   potrf_f64        tiled right-looking Cholesky: recursive diagonal blocks
//                    (64-wide leaves factored and inverted in shared memory),
//                    panel solve as a product with the inverse diagonal block,
//                    trailing SYRK on the lower tiles only.
//   solve_right_f64  R = Ctm L^-T L^-1: right-looking forward pass X L^T = Ctm,
//                    then backward pass R L = X, each a sequence of block
//                    products with the stored inverse diagonal blocks.
//   moao_cee_cvv     lapack/compute/cee_cvv.cpp:50-125 step for step.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "context.h"
#include "crt_f64.h"
#include "dense.h"

namespace moao {

constexpr int kLeaf = 64;

moao_status gemm(moao_ctx* ctx, long M, long N, long K, double alpha, const double* A, long lda,
                 const double* B, long ldb, bool transB, double beta, double* C, long ldc,
                 bool lowerC, TriMode tri) {
  GemmArgs g;
  g.M = M; g.N = N; g.K = K; g.alpha = alpha; g.beta = beta;
  g.A = A; g.lda = lda; g.B = B; g.ldb = ldb; g.transB = transB; g.triB = tri;
  g.C = C; g.ldc = ldc; g.lowerC = lowerC;
  g.cfg = ctx->gemm_cfg;
  g.chained = ctx->chained;
  // algorithmic flops: 2MNK, halved when only a triangle of C or of B counts
  double fl = 2.0 * M * N * K;
  if (lowerC) fl = (double)M * N * K + (double)std::min(M, N) * K;
  if (tri != TRI_FULL) fl *= 0.5;
  KernelTimer kt(ctx, "gemm_f64", fl);
  return gemm_f64(g, ctx->stream, &ctx->launches);
}

// Whether a product goes by residues. Under stream capture it does not: their buffers
// cannot be allocated there, and a graph would keep addresses that a later call moves.
static bool by_residues(const moao_ctx* ctx, long M, long N, long K, bool lower) {
  if (!crt64_pays(ctx, M, N, K, lower)) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess) {
    cudaGetLastError();  // the legacy stream while another one captures
    return false;
  }
  return cap == cudaStreamCaptureStatusNone;
}

// The same product by int8 residue products where those are faster (crt_f64.cu);
// the FP64 tensor cores where not, or where their buffers do not fit.
moao_status gemm_long(moao_ctx* ctx, long M, long N, long K, double alpha, const double* A,
                      long lda, const double* B, long ldb, bool transB, double beta, double* C,
                      long ldc, bool lowerC = false, const CrtBalance* bal = nullptr) {
  if (by_residues(ctx, M, N, K, lowerC)) {
    GemmArgs g;
    g.M = M; g.N = N; g.K = K; g.alpha = alpha; g.beta = beta;
    g.A = A; g.lda = lda; g.B = B; g.ldb = ldb; g.transB = transB;
    g.C = C; g.ldc = ldc; g.lowerC = lowerC;
    const moao_status st = crt64_gemm(ctx, g, bal);
    if (st != MOAO_ERR_OOM) return st;
  }
  return gemm(ctx, M, N, K, alpha, A, lda, B, ldb, transB, beta, C, ldc, lowerC);
}

// C (M x n) = A (M x n) S, S the symmetric n x n matrix in the lower triangle of B.
moao_status symm_right(moao_ctx* ctx, long M, long n, const double* A, long lda, const double* B,
                       long ldb, double* C, long ldc) {
  if (by_residues(ctx, M, n, n, false)) {
    const moao_status st = crt64_symm(ctx, M, n, A, lda, B, ldb, C, ldc);
    if (st != MOAO_ERR_OOM) return st;
  }
  MOAO_TRY(gemm(ctx, M, n, n, 1.0, A, lda, B, ldb, false, 0.0, C, ldc, false, TRI_LOWER));
  return gemm(ctx, M, n, n, 1.0, A, lda, B, ldb, true, 1.0, C, ldc, false, TRI_STRICT_LOWER);
}

// The side stream and events of the lookahead (created on first use).
moao_status ensure_lookahead(moao_ctx* ctx) {
  if (ctx->aux) return MOAO_OK;
  int lo = 0, hi = 0;
  MOAO_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&lo, &hi));
  MOAO_CUDA_TRY(cudaStreamCreateWithPriority(&ctx->aux, cudaStreamNonBlocking, hi));
  for (auto& e : ctx->la_ev) MOAO_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return MOAO_OK;
}

int diag_sms(const moao_ctx* ctx, double seconds) {
  // A block of 1,024 takes 0.45 ms (its chain) + 6.6 ms over the SMs, one CTA on each. As
  // many as let it end with the update, 64 at most (0.56 ms).
  // The block's CTAs must not outnumber the SMs left: each would take one of the update's,
  // whose persistent CTA would then start when the block ends (2.2 -> 3.2 ms).
  int sms = ctx->lookahead_sms;
  while (sms < 64 && 0.45e-3 + 6.6e-3 / sms > seconds * 148.0 / (148 - sms))
    sms = std::min(64, sms + std::max(1, sms / 2));
  return sms;
}

moao_status ensure_diag_sync(moao_ctx* ctx) {
  return ctx->chained && !ctx->graph_mode ? ctx->ws_sync.ensure(sizeof(unsigned)) : MOAO_OK;
}

// Factor the nb x nb diagonal block A (lda) and write its inverse into D (ldd).
// W is scratch of nb x nb doubles. One launch (diag_block) on contexts that own the word
// its barrier counts in; launch by launch where there is none (the call without
// allocations, whose scratch is fixed), and under capture, where graphs of several
// instances run side by side and should not wait for SMs to be free all at once.
moao_status potrf_inv_block(moao_ctx* ctx, double* A, long lda, double* D, long ldd, long nb,
                            long col0, int* d_info, double* W) {
  if (ctx->ws_sync.p && !ctx->graph_mode && diag_block_fits(nb)) {
    int nsm = 148;
    MOAO_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    const int ctas = std::min(nsm, std::max(1, ctx->diag_ctas));
    KernelTimer kt(ctx, "diag_block", (double)nb * nb * nb * (2.0 / 3));
    return diag_block(A, lda, D, ldd, nb, col0, d_info, W, ctx->ws_sync.as<unsigned>(), ctas,
                      ctx->diag_polls, ctx->stream, &ctx->launches);
  }
  if (nb <= kLeaf) {
    KernelTimer kt(ctx, "potrf_leaf", (double)nb * nb * nb * (1.0 / 3 + 1.0 / 3));
    return potrf_inv_leaf(A, lda, D, ldd, (int)nb, col0, d_info, ctx->chained, ctx->stream,
                          &ctx->launches);
  }
  const long n1 = kLeaf * ((nb + 2 * kLeaf - 1) / (2 * kLeaf));
  const long n2 = nb - n1;
  double* A11 = A;
  double* A21 = A + n1;
  double* A22 = A + n1 + n1 * lda;
  double* D11 = D;
  double* D21 = D + n1;
  double* D22 = D + n1 + n1 * ldd;
  MOAO_TRY(potrf_inv_block(ctx, A11, lda, D11, ldd, n1, col0, d_info, W));
  // L21 = A21 L11^-T ; D12 = 0
  MOAO_TRY(gemm(ctx, n2, n1, n1, 1.0, A21, lda, D11, ldd, true, 0.0, W, n2));
  MOAO_TRY(copy_zero(W, n2, A21, lda, n2, n1, D + n1 * ldd, ldd, n1, n2, ctx->chained, ctx->stream,
                     &ctx->launches));
  // A22 -= L21 L21^T (lower)
  MOAO_TRY(gemm(ctx, n2, n2, n1, -1.0, A21, lda, A21, lda, true, 1.0, A22, lda, true));
  MOAO_TRY(potrf_inv_block(ctx, A22, lda, D22, ldd, n2, col0 + n1, d_info, W));
  // D21 = -D22 L21 D11
  MOAO_TRY(gemm(ctx, n2, n1, n1, 1.0, A21, lda, D11, ldd, false, 0.0, W, n2));
  MOAO_TRY(gemm(ctx, n2, n1, n2, -1.0, D22, ldd, W, n2, false, 0.0, D21, ldd));
  return MOAO_OK;
}

// The trailing updates of the factorisation by residue products. The blocks of a group
// update only each other's columns; the columns beyond get the whole group's update at
// once, over its K: the combine step and the products' epilogues are then fewer (nmeas
// 29,120, groups of 1, 2 and 4: factorisation 131, 113 and 114 ms, solves 100, 85 and
// 79 ms). The next diagonal block is always factored on the side stream, beside products
// that leave it the context's lookahead SMs: its own columns are updated first, those it
// does not need beside it. So the group's update beyond the next group runs in shares,
// one beside each of that group's blocks. (270 -> 252 ms with groups of one; not beside
// the FP64 tensor cores' update, whose CTAs leave no SM free.)
struct Trailing {
  moao_ctx* ctx;
  double* A;
  long lda, n;
  int max_ctas;
  CrtOperand op;     // rows r0.. of columns [p0, r0): the last whole group
  long p0 = 0, r0 = 0, done = 0;  // its update has reached columns [r0, done)

  // A(c0.., c0..c1) -= its part of the product over o's columns [p, p + K), o's rows from q0 on
  moao_status part(const CrtOperand& o, long q0, long p, long c0, long c1, int ctas) {
    if (c1 <= c0) return MOAO_OK;
    GemmArgs g;
    g.M = n - c0; g.N = c1 - c0; g.K = o.K; g.alpha = -1.0; g.beta = 1.0;
    g.A = g.B = A + c0 + p * lda;
    g.lda = g.ldb = lda;
    g.transB = true;
    g.C = A + c0 + c0 * lda; g.ldc = lda; g.lowerC = true;
    return crt64_product(ctx, o, c0 - q0, o, c0 - q0, &g, 1, ctas);
  }
  // columns up to c of what is due from the last group
  moao_status advance(long c, int ctas) {
    const long c0 = done;
    done = std::max(done, std::min(c, n));
    return part(op, r0, p0, c0, done, ctas);
  }
};

// Columns up to which the first b of q shares of columns [c0, n) reach, equal areas of
// the lower triangle each.
long share(long c0, long n, long b, long q) {
  return b >= q ? n : n - (long)((double)(n - c0) * std::sqrt(1.0 - (double)b / q));
}

moao_status potrf_f64(moao_ctx* ctx, double* A, long lda, long n, double* dinv, int* d_info) {
  const long nb = ctx->nb;
  MOAO_TRY(ctx->ws_w.ensure(sizeof(double) * (size_t)std::max(n, 1L) * nb));
  double* W = ctx->ws_w.as<double>();
  MOAO_TRY(ensure_diag_sync(ctx));
  int nsm = 148;
  Trailing t{ctx, A, lda, n, 0};
  t.done = n;  // nothing is due
  auto diag_block = [&](long k0, cudaStream_t st, int sms = 0) -> moao_status {
    cudaStream_t keep = ctx->stream;
    const int ctas = ctx->diag_ctas;
    if (sms > 0) ctx->diag_ctas = sms;
    ctx->stream = st;  // potrf_inv_block launches on the context's stream
    const moao_status r = potrf_inv_block(ctx, A + k0 + k0 * lda, lda, dinv + k0, n,
                                          std::min(nb, n - k0), k0, d_info, W);
    ctx->stream = keep;
    ctx->diag_ctas = ctas;
    return r;
  };
  // the next diagonal block beside what is launched until join(): updates of columns
  // [c0, c1) over K from the first group and [d0, d1) over L from the last
  auto fork = [&](long k0, long c0, long c1, long K, long d0, long d1, long L) -> moao_status {
    if (ctx->lookahead_sms == 0) return diag_block(k0, ctx->stream);  // the same steps in order
    auto area = [&](long x, long y) { return 0.5 * ((double)(n - x) * (n - x) - (double)(n - y) * (n - y)); };
    const int sms = diag_sms(ctx, 2.0 * 16 / 1.9e15 * (area(c0, c1) * K + area(d0, d1) * L));
    t.max_ctas = std::max(1, nsm - sms);
    MOAO_CUDA_TRY(cudaEventRecord(ctx->la_ev[0], ctx->stream));
    MOAO_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->la_ev[0], 0));
    MOAO_TRY(diag_block(k0, ctx->aux, sms));
    MOAO_CUDA_TRY(cudaEventRecord(ctx->la_ev[1], ctx->aux));
    return MOAO_OK;
  };
  auto join = [&]() -> moao_status {
    if (ctx->lookahead_sms == 0) return MOAO_OK;
    MOAO_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->la_ev[1], 0));
    return MOAO_OK;
  };
  auto ahead_pays = [&](long k1) {  // the update from column k1 on, K = nb
    return k1 + nb < n && crt64_pays(ctx, n - k1 - nb, n - k1 - nb, nb, true);
  };
  bool ahead = ahead_pays(nb);
  if (ahead) {
    if (ctx->lookahead_sms > 0) MOAO_TRY(ensure_lookahead(ctx));
    MOAO_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
    const moao_status st = crt64_reserve_group(ctx, n - nb, nb, kFactorGroup * nb);
    if (st != MOAO_OK && st != MOAO_ERR_OOM) return st;
    ahead = st == MOAO_OK;
  }
  MOAO_TRY(diag_block(0, ctx->stream));
  for (long s0 = 0; s0 < n;) {
    const bool grouped = ahead && ahead_pays(s0 + nb);
    const long s1 = std::min(n, s0 + (grouped ? kFactorGroup : 1) * nb);
    const long nblk = (s1 - s0 + nb - 1) / nb;
    // shares of the last group's update beyond this group, beside this group's blocks;
    // the first was taken with this group's columns
    const long due0 = t.done;
    for (long k0 = s0, b = 0; k0 < s1; k0 += nb, ++b) {
      const long kb = std::min(nb, n - k0), k1 = k0 + kb, rest = n - k1;
      if (rest <= 0) break;
      double* P = A + k1 + k0 * lda;
      // panel: P <- P L_kk^-T
      // (column k of P goes with the variable whose pivot is 1 / Dk(k, k))
      const CrtBalance piv{dinv + k0, n + 1, 0, 1};
      MOAO_TRY(gemm_long(ctx, rest, kb, kb, 1.0, P, lda, dinv + k0, n, true, 0.0, W, rest, false, &piv));
      MOAO_TRY(copy_matrix(W, rest, P, lda, rest, kb, ctx->stream, &ctx->launches));
      if (!grouped) {
        MOAO_TRY(t.advance(n, 0));
        MOAO_TRY(gemm_long(ctx, rest, rest, kb, -1.0, P, lda, P, lda, true, 1.0, A + k1 + k1 * lda, lda, true));
        MOAO_TRY(diag_block(k1, ctx->stream));
        continue;
      }
      if (k1 < s1) {
        CrtOperand o;
        MOAO_TRY(crt64_begin(ctx));
        MOAO_TRY(crt64_operand(ctx, P, lda, rest, kb, &o));
        const long c1 = std::min(s1, k1 + nb);
        MOAO_TRY(t.part(o, k1, k0, k1, c1, 0));
        const long d1 = share(due0, n, b + 1, nblk - 1);
        MOAO_TRY(fork(k1, c1, s1, kb, t.done, d1, t.op.K));
        MOAO_TRY(t.part(o, k1, k0, c1, s1, t.max_ctas));
        MOAO_TRY(t.advance(d1, t.max_ctas));
        MOAO_TRY(join());
      } else {
        MOAO_TRY(t.advance(n, 0));
        t.p0 = s0;
        t.r0 = t.done = s1;
        MOAO_TRY(crt64_group_operand(ctx, A + s1 + s0 * lda, lda, n - s1, s1 - s0, &t.op));
        const long c1 = std::min(n, s1 + nb);
        MOAO_TRY(t.advance(c1, 0));
        // the next group's other columns, and the first share of what is beyond
        const long g = ahead_pays(s1 + nb) ? kFactorGroup : 1;
        const long d1 = g > 1 ? share(std::min(n, s1 + g * nb), n, 1, g) : n;
        MOAO_TRY(fork(s1, n, n, 0, c1, d1, s1 - s0));
        MOAO_TRY(t.advance(d1, t.max_ctas));
        MOAO_TRY(join());
      }
    }
    s0 = s1;
  }
  return MOAO_OK;
}

moao_status solve_right_f64(moao_ctx* ctx, const double* L, long ldl, long n, const double* dinv,
                            double* B, long ldb, long m) {
  const long nb = ctx->nb;
  // groups of blocks, as in the factorisation
  const long group = (crt64_pays(ctx, m, nb, nb, false) ? kSolveGroup : 1) * nb;
  MOAO_TRY(ctx->ws_w.ensure(sizeof(double) * (size_t)std::max(m, 1L) * nb));
  double* W = ctx->ws_w.as<double>();
  // Forward: X L^T = B.
  for (long k0 = 0; k0 < n; k0 += nb) {
    const long kb = std::min(nb, n - k0);
    double* Bk = B + k0 * ldb;
    const CrtBalance piv{dinv + k0, n + 1, 0, 1};
    MOAO_TRY(gemm_long(ctx, m, kb, kb, 1.0, Bk, ldb, dinv + k0, n, true, 0.0, W, m, false, &piv));
    MOAO_TRY(copy_matrix(W, m, Bk, ldb, m, kb, ctx->stream, &ctx->launches));
    // the group's own columns, and at its end the ones beyond with the group's K
    const long k1 = k0 + kb, s0 = k0 / group * group, s1 = std::min(n, s0 + group);
    if (k1 < s1)
      MOAO_TRY(gemm_long(ctx, m, s1 - k1, kb, -1.0, Bk, ldb, L + k1 + k0 * ldl, ldl, true, 1.0,
                         B + k1 * ldb, ldb));
    else if (k1 < n)
      MOAO_TRY(gemm_long(ctx, m, n - k1, k1 - s0, -1.0, B + s0 * ldb, ldb, L + k1 + s0 * ldl, ldl, true,
                         1.0, B + k1 * ldb, ldb));
  }
  // Backward: R L = X.
  const long nblk = (n + nb - 1) / nb;
  for (long b = nblk - 1; b >= 0; --b) {
    const long k0 = b * nb, kb = std::min(nb, n - k0);
    double* Bk = B + k0 * ldb;
    MOAO_TRY(gemm_long(ctx, m, kb, kb, 1.0, Bk, ldb, dinv + k0, n, false, 0.0, W, m));
    MOAO_TRY(copy_matrix(W, m, Bk, ldb, m, kb, ctx->stream, &ctx->launches));
    const long s0 = k0 / group * group, s1 = std::min(n, s0 + group);
    if (k0 > s0) {
      const CrtBalance piv{L + k0 + k0 * ldl, ldl + 1, 0, 1};  // R(:, k) goes with L(k, :)
      MOAO_TRY(gemm_long(ctx, m, k0 - s0, kb, -1.0, Bk, ldb, L + k0 + s0 * ldl, ldl, false, 1.0,
                         B + s0 * ldb, ldb, false, &piv));
    } else if (s0 > 0) {
      const CrtBalance piv{L + s0 + s0 * ldl, ldl + 1, 0, 1};
      MOAO_TRY(gemm_long(ctx, m, s0, s1 - s0, -1.0, B + s0 * ldb, ldb, L + s0, ldl, false, 1.0, B, ldb,
                         false, &piv));
    }
  }
  return MOAO_OK;
}

moao_status await_inputs(moao_ctx* ctx) {
  if (ctx->wait_inputs) {
    MOAO_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->inputs_ready, 0));
    ctx->wait_inputs = false;
  }
  return MOAO_OK;
}

// Column panels of the lower part of the n x n factor (device ld ldCmm) into the
// host buffer (ld host_factor_ld), on the copy stream after the context stream's
// work so far.
moao_status factor_to_host(moao_ctx* ctx, const double* Cmm, long ldCmm, long n) {
  if (ctx->copy_ev.empty()) {
    cudaEvent_t e;
    MOAO_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ctx->copy_ev.push_back(e);
  }
  MOAO_CUDA_TRY(cudaEventRecord(ctx->copy_ev[0], ctx->stream));
  MOAO_CUDA_TRY(cudaStreamWaitEvent(ctx->copy, ctx->copy_ev[0], 0));
  const long w = 512;
  for (long c0 = 0; c0 < n; c0 += w) {
    const long c1 = std::min(n, c0 + w);
    MOAO_CUDA_TRY(cudaMemcpy2DAsync(ctx->host_factor + c0 * ctx->host_factor_ld + c0,
                                    sizeof(double) * ctx->host_factor_ld, Cmm + c0 * ldCmm + c0,
                                    sizeof(double) * ldCmm, sizeof(double) * (n - c0), c1 - c0,
                                    cudaMemcpyDeviceToHost, ctx->copy));
  }
  return MOAO_OK;
}

// FP64 reconstructor: factor Cmm in place, then the solves of targets g0..ngal-1.
moao_status reconstructor_fp64(moao_ctx* ctx, long nmeas, long nmeasts, double* d_Cmm, long ldCmm,
                               double* d_Ctm, long ldCtm, long g0, long ngal,
                               moao_solve_report* r) {
  MOAO_TRY(ctx->ws_dinv.ensure(sizeof(double) * (size_t)nmeas * ctx->nb));
  MOAO_TRY(ctx->ws_info.ensure(3 * sizeof(int)));
  int* d_info = ctx->ws_info.as<int>();
  MOAO_CUDA_TRY(cudaMemsetAsync(d_info, 0, 3 * sizeof(int), ctx->stream));
  cudaEventRecord(ctx->ev[0], ctx->stream);
  MOAO_TRY(potrf_f64(ctx, d_Cmm, ldCmm, nmeas, ctx->ws_dinv.as<double>(), d_info));
  cudaEventRecord(ctx->ev[1], ctx->stream);
  int infos[2] = {0, 0};
  MOAO_CUDA_TRY(cudaMemcpyAsync(infos, d_info, sizeof(infos), cudaMemcpyDeviceToHost, ctx->stream));
  MOAO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (infos[1]) return set_error(MOAO_ERR_TIMEOUT, "dpotrf: bounded wait expired");
  const int info = r->info = infos[0];
  if (info != 0) {
    // The reference prints and returns without solving (reconstructor.cpp:34-38).
    return set_error(MOAO_ERR_NOT_SPD, "dpotrf: non-positive pivot at column " +
                                           std::to_string(info));
  }
  if (ctx->host_factor) {  // the factor is final: back to the host beside the solves
    MOAO_TRY(factor_to_host(ctx, d_Cmm, ldCmm, nmeas));
    ctx->factor_done = true;
  }
  MOAO_TRY(await_inputs(ctx));
  for (long g = g0; g < ngal; ++g) {
    double* Ctm_g = d_Ctm + nmeas * nmeasts * g;
    MOAO_TRY(solve_right_f64(ctx, d_Cmm, ldCmm, nmeas, ctx->ws_dinv.as<double>(), Ctm_g, ldCtm,
                             nmeasts));
  }
  cudaEventRecord(ctx->ev[2], ctx->stream);
  MOAO_CUDA_TRY(cudaEventSynchronize(ctx->ev[2]));
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
  r->ms_factor += ms;
  cudaEventElapsedTime(&ms, ctx->ev[1], ctx->ev[2]);
  r->ms_solve += ms;
  return MOAO_OK;
}

}  // namespace moao

using namespace moao;

extern "C" {

moao_status moao_reconstructor(moao_ctx* ctx, long nmeas, long nmeasts, double* d_Cmm,
                               long ldCmm, double* d_Ctm, long ldCtm, long ngal, moao_prec prec,
                               moao_solve_report* rep) {
  if (!ctx) return set_error(MOAO_ERR_BAD_ARG, "reconstructor: null context");
  if (nmeas < 0 || nmeasts < 0 || ngal < 0 || ldCmm < std::max(1L, nmeas) ||
      ldCtm < std::max(1L, nmeasts) || (nmeas > 0 && (!d_Cmm || !d_Ctm)))
    return set_error(MOAO_ERR_BAD_ARG, "reconstructor: bad sizes or pointers");
  if (prec != MOAO_PREC_FP64 && prec != MOAO_PREC_MIXED)
    return set_error(MOAO_ERR_BAD_ARG, "reconstructor: unknown precision");
  moao_solve_report local{};
  moao_solve_report* r = rep ? rep : &local;
  std::memset(r, 0, sizeof(*r));
  if (nmeas == 0) return MOAO_OK;
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  ctx->factor_done = false;
  if (prec == MOAO_PREC_MIXED) {
    long g = 0;
    for (; g < ngal; ++g) {
      // one factorisation serves every target: later targets reuse it
      MOAO_TRY(reconstructor_mixed(ctx, nmeas, nmeasts, d_Cmm, ldCmm,
                                   d_Ctm + nmeas * nmeasts * g, ldCtm, g > 0, r));
      if (r->fallback) break;
    }
    if (r->fallback) {
      // the mixed estimate missed the accuracy target: this and the remaining
      // targets from the FP64 path (Cmm and their Ctm are still as given)
      ctx->mx_factored_n = -1;
      ctx->rstate_valid = false;
      return reconstructor_fp64(ctx, nmeas, nmeasts, d_Cmm, ldCmm, d_Ctm, ldCtm, g, ngal, r);
    }
    if (!ctx->keep_cmm && !ctx->factor_done) MOAO_TRY(finish_mixed(ctx, nmeas, d_Cmm, ldCmm));
    if (ctx->factor_done) ctx->mx_factored_n = -1;  // A32 no longer matches what finish_mixed leaves
    MOAO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    return MOAO_OK;
  }
  return reconstructor_fp64(ctx, nmeas, nmeasts, d_Cmm, ldCmm, d_Ctm, ldCtm, 0, ngal, r);
}

moao_status moao_cee_cvv(moao_ctx* ctx, long nmeas, long nmeasts, long nact, double* Cmm,
                         long ldCmm, double* Cpp, long ldCpp, double* Cpm, long ldCpm, double* R,
                         long ldR, double* Dx, long ldDx, double* Cee, long ldCee, double* Cvv,
                         long ldCvv, double* Tmp, long ldTmp) {
  return moao_cee_cvv_prec(ctx, nmeas, nmeasts, nact, Cmm, ldCmm, Cpp, ldCpp, Cpm, ldCpm, R, ldR,
                           Dx, ldDx, Cee, ldCee, Cvv, ldCvv, Tmp, ldTmp, MOAO_PREC_FP64);
}

moao_status moao_cee_cvv_prec(moao_ctx* ctx, long nmeas, long nmeasts, long nact, double* Cmm,
                              long ldCmm, double* Cpp, long ldCpp, double* Cpm, long ldCpm,
                              double* R, long ldR, double* Dx, long ldDx, double* Cee, long ldCee,
                              double* Cvv, long ldCvv, double* Tmp, long ldTmp, moao_prec prec) {
  if (!ctx) return set_error(MOAO_ERR_BAD_ARG, "Cee_Cvv: null context");
  if (prec != MOAO_PREC_FP64 && prec != MOAO_PREC_MIXED)
    return set_error(MOAO_ERR_BAD_ARG, "Cee_Cvv: unknown precision");
  if (nmeas < 0 || nmeasts < 0 || nact < 0)
    return set_error(MOAO_ERR_BAD_ARG, "Cee_Cvv: negative size");
  if (ldCmm < std::max(1L, nmeas) || ldCpp < std::max(1L, nmeasts) ||
      ldCpm < std::max(1L, nmeasts) || ldR < std::max(1L, nmeasts) ||
      ldDx < std::max(1L, nact) || ldCee < std::max(1L, nmeasts) ||
      ldCvv < std::max(1L, nact) || ldTmp < std::max(1L, nact))
    return set_error(MOAO_ERR_BAD_ARG, "Cee_Cvv: leading dimension too small");
  if ((nmeas > 0 && (!Cmm || !R)) || (nmeasts > 0 && (!Cpp || !Cpm || !Cee)) ||
      (nact > 0 && (!Dx || !Cvv || !Tmp)))
    return set_error(MOAO_ERR_BAD_ARG, "Cee_Cvv: null matrix pointer");
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  if (prec == MOAO_PREC_MIXED)
    return cee_cvv_mixed(ctx, nmeas, nmeasts, nact, Cmm, ldCmm, Cpp, ldCpp, Cpm, ldCpm, R, ldR, Dx,
                         ldDx, Cee, ldCee, Cvv, ldCvv, Tmp, ldTmp);
  const long nm = nmeas, nt = nmeasts;
  // the measurements' variances: Ctm and R Cmm scale with them, R with their inverse
  const CrtBalance var{Cmm, ldCmm + 1, 1, -1}, var_r{Cmm, ldCmm + 1, 1, 1};
  // (1) Cpp <- Cpp - Cpm R^T - R Cpm^T  (syr2k, lower)
  MOAO_TRY(gemm_long(ctx, nt, nt, nm, -1.0, Cpm, ldCpm, R, ldR, true, 1.0, Cpp, ldCpp, true, &var));
  MOAO_TRY(gemm_long(ctx, nt, nt, nm, -1.0, R, ldR, Cpm, ldCpm, true, 1.0, Cpp, ldCpp, true, &var_r));
  // (2) Cpm <- R Cmm  (symm right, Cmm lower-stored)
  MOAO_TRY(symm_right(ctx, nt, nm, R, ldR, Cmm, ldCmm, Cpm, ldCpm));
  // (3)-(6) Cee <- sym(tril(Cpp))
  MOAO_TRY(sym_from_lower(Cpp, ldCpp, Cee, ldCee, nt, ctx->stream, &ctx->launches));
  // (7) Cee += Cpm R^T
  MOAO_TRY(gemm_long(ctx, nt, nt, nm, 1.0, Cpm, ldCpm, R, ldR, true, 1.0, Cee, ldCee, false, &var));
  // (8) Tmp <- Dx sym(tril(Cee))
  MOAO_TRY(symm_right(ctx, nact, nt, Dx, ldDx, Cee, ldCee, Tmp, ldTmp));
  // (9) Cvv <- Tmp Dx^T
  {
    const CrtBalance err{Cee, ldCee + 1, 1, -1};  // Tmp(:, k) scales with Cee(k, k)
    MOAO_TRY(gemm_long(ctx, nact, nact, nt, 1.0, Tmp, ldTmp, Dx, ldDx, true, 0.0, Cvv, ldCvv, false,
                       &err));
  }
  return MOAO_OK;
}

moao_status moao_dense_potrf_inv(moao_ctx* ctx, long n, double* A, long lda, double* Ainv,
                                 long ldi, int* info) {
  if (!ctx || n < 0 || (n > 0 && (!A || !Ainv)) || lda < std::max(1L, n) ||
      ldi < std::max(1L, n))
    return set_error(MOAO_ERR_BAD_ARG, "dense_potrf_inv: bad sizes or pointers");
  if (info) *info = 0;
  if (n == 0) return MOAO_OK;
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  MOAO_TRY(ctx->ws_w.ensure(sizeof(double) * (size_t)n * n));
  MOAO_TRY(ctx->ws_info.ensure(3 * sizeof(int)));
  int* d_info = ctx->ws_info.as<int>();
  MOAO_CUDA_TRY(cudaMemsetAsync(d_info, 0, 3 * sizeof(int), ctx->stream));
  MOAO_TRY(ensure_diag_sync(ctx));
  MOAO_TRY(potrf_inv_block(ctx, A, lda, Ainv, ldi, n, 0, d_info, ctx->ws_w.as<double>()));
  int hi[2] = {0, 0};
  MOAO_CUDA_TRY(cudaMemcpyAsync(hi, d_info, sizeof(hi), cudaMemcpyDeviceToHost, ctx->stream));
  MOAO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (hi[1]) return set_error(MOAO_ERR_TIMEOUT, "dense_potrf_inv: bounded wait expired");
  const int h = hi[0];
  if (info) *info = h;
  if (h) return set_error(MOAO_ERR_NOT_SPD, "dense_potrf_inv: non-positive pivot at column " +
                                                std::to_string(h));
  return MOAO_OK;
}

moao_status moao_dense_gemm(moao_ctx* ctx, int transB, int lowerC, long M, long N, long K,
                            double alpha, const double* A, long lda, const double* B, long ldb,
                            double beta, double* C, long ldc) {
  if (!ctx) return set_error(MOAO_ERR_BAD_ARG, "dense_gemm: null context");
  if (M < 0 || N < 0 || K < 0) return set_error(MOAO_ERR_BAD_ARG, "dense_gemm: negative size");
  if (M == 0 || N == 0) return MOAO_OK;
  if (!C || (K > 0 && (!A || !B))) return set_error(MOAO_ERR_BAD_ARG, "dense_gemm: null matrix");
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  return gemm(ctx, M, N, K, alpha, A, lda, B, ldb, transB != 0, beta, C, ldc, lowerC != 0);
}

}  // extern "C"
