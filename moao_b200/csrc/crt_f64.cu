// FP64 products on the int8 tensor cores.
//
// Blackwell's FP64 tensor rate is 1/130 of its int8 rate, so a long FP64 product
// C = alpha A B^T + beta C is faster as 16 exact int8 products (the Ozaki scheme
// in its Chinese-remainder form, Ozaki, Uchino and Imamura 2025):
//   operands  the columns k of A and B are balanced against each other by powers of
//             two taken from the system's own diagonal (A's column k times 2^s, B's
//             times 2^-s), so that a diagonal scaling of the system, whose effect on
//             the two cancels in FP64, costs no bits here either; then every row of
//             A and of B is scaled by a power of two and rounded to integers X of
//             `bits` bits (|X| <= 2^bits, bits as large as the moduli allow for this K:
//             57 for K <= 1,024, 53 for K near 2^17), and stored as centred residues
//             modulo 16 pairwise coprime m_i <= 256;
//   product   one int8 GEMM per modulus with exact int32 sums, reduced modulo m_i
//             in its epilogue (tc_gemm, all moduli in one launch);
//   combine   X Y^T from its residues, scaled back and added to C (tc_modz_combine).
// The only roundings are the operands' (elements within 2^4 of their row's
// largest are exact at 57 bits) and the two of the reconstruction, against K
// rounded additions per element on the FP64 tensor cores. The bound is one per row:
// an element of the result is off by up to 2^(1 - bits) K times the largest entries of
// its two rows (balanced), where FP64 sums are off by K 2^-53 times the sum of its own
// terms' absolute values. The two differ where all large entries of a row meet entries
// 2^-50 of their own row's largest.
//
// Measured (B200, against the FP64 tensor cores at 28-31 TF/s): the FP64
// reconstructor at nmeas 29,120 563 -> 190 ms (lookahead and groups included), its Cee/Cvv chain
// 253 -> 81 ms; the int8 products alone run at 1.7 Pop/s over K = 1,024 and 2.2 over
// K = 29,120. Error against an FP64 library's result 1.5e-11 -> 1.3e-11 and 9.9e-12 ->
// 3.9e-12.
//
// Guard: a NaN, an infinity or a magnitude outside 2^-900 .. 2^900 in an operand
// (found with the row exponents) or a tensor-core wait that ran out raises a flag on
// the device; the combine step then writes nothing and the FP64 tensor-core
// kernel computes the product as it always did. No host read is needed.
#include "crt_f64.h"

#include <algorithm>
#include <cmath>

#include "moao_b200_debug.h"
#include "tc_gemm.h"

namespace moao {
namespace {

constexpr int kNM = kCrt64Moduli;
constexpr int kMaxBits = 57;
// Tiles of the product held at once (2 GB of residues). Running the combine step of
// one part beside the products of the next (a second stream, parts of 128 to 1,024
// tiles) was slower at every size: the products lose what the overlap gains.
constexpr long kPartTiles = 4096;
constexpr long kMaxChunks = 4096;
// cf_flag: the operands' guard, one word per part of a product, the group operand's guard
constexpr long kGroupFlag = 1 + kMaxChunks, kFlags = kGroupFlag + 1;
constexpr size_t kOperandBytes = (size_t)6 << 30;  // residues of one operand held at once

// Bits of the scaled operands: |sum of K products| <= K 2^(2 bits) < M / 2.
int bits_for(long K) {
  double lm = 0;
  for (int m : kCrt64Mod) lm += std::log2((double)m);
  return std::min(kMaxBits, (int)std::floor((lm - 1.0 - std::log2((double)K) - 1e-6) / 2));
}

// Exponents are biased (x in [2^(E - 1023), 2^(E - 1022))); kNone marks a row
// without a nonzero element. It is the value of bytes 0x80 (memset).
constexpr int kNone = (int)0x80808080;

__device__ __forceinline__ int exponent_of(double x) {
  return x == 0.0 ? kNone : (__double2hiint(x) >> 20) & 0x7ff;
}
// |x| < 2^exp_of(e) for the elements of a row whose largest exponent is e
__device__ __forceinline__ int exp_of(int e) { return e == kNone ? 0 : e - 1022; }

// Element S(k, j) of a symmetric matrix held in its lower triangle.
__device__ __forceinline__ double sym_at(const double* A, long lda, long k, long j) {
  return k >= j ? A[j * lda + k] : A[k * lda + j];
}

// Largest exponents of a line, offsets (the balance along K) included.
struct ExpMax {
  int m = kNone, raw = kNone;
  __device__ __forceinline__ void add(double x, int off) {
    const int e = exponent_of(x);
    raw = max(raw, e);
    if (e != kNone) m = max(m, e + off);
  }
  __device__ __forceinline__ void store(int* out) const {
    if (m != kNone) atomicMax(out, m);
  }
  __device__ __forceinline__ void check(int* flag) const {  // NaN or infinity
    if (raw == 0x7ff) atomicOr(flag, 1 << 8);
  }
};

// Per row of a column-major nr x nc matrix, over its columns, with offset
// sign off[c] (off null: 0). A thread takes 32 columns of a row.
__global__ void exps_over_cols_kernel(const double* __restrict__ A, long lda, long nr, long nc,
                                      const int* __restrict__ off, int sign, int* __restrict__ out,
                                      int* flag) {
  const long r = blockIdx.x * 32L + threadIdx.x;
  const long c0 = blockIdx.y * 256L + threadIdx.y * 32L;
  if (r >= nr) return;
  ExpMax st;
  const int lim = (int)min(32L, nc - c0);
  const double* a = A + c0 * lda + r;
#pragma unroll
  for (int h = 0; h < 32; h += 16) {
    double v[16];  // all in flight before the first is used
#pragma unroll
    for (int c = 0; c < 16; ++c) v[c] = h + c < lim ? a[(h + c) * lda] : 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c) st.add(v[c], off && h + c < lim ? sign * off[c0 + h + c] : 0);
  }
  st.check(flag);
  st.store(out + r);
}

// Per column, over the rows, with offset sign off[r]. A warp takes 1,024 rows of a
// column (all its lanes reach the reduction).
__global__ void exps_over_rows_kernel(const double* __restrict__ A, long lda, long nr, long nc,
                                      const int* __restrict__ off, int sign, int* __restrict__ out,
                                      int* flag) {
  const long c = blockIdx.x * 8L + threadIdx.y;
  if (c >= nc) return;
  const long r0 = blockIdx.y * 1024L;
  ExpMax st;
#pragma unroll
  for (int h = 0; h < 32; h += 16) {
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const long r = r0 + (h + q) * 32 + threadIdx.x;
      v[q] = r < nr ? A[c * lda + r] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const long r = r0 + (h + q) * 32 + threadIdx.x;
      st.add(v[q], off && r < nr ? sign * off[r] : 0);
    }
  }
  st.check(flag);
  st.m = __reduce_max_sync(0xffffffffu, st.m);
  if (threadIdx.x == 0) st.store(out + c);
}

// Per column c0 .. c0 + nc - 1 of the symmetric K x K matrix held in its lower
// triangle, with offset sign off[k].
__global__ void exps_sym_kernel(const double* __restrict__ A, long lda, long nc, long K, long c0,
                                const int* __restrict__ off, int sign, int* __restrict__ out,
                                int* flag) {
  __shared__ double t[32][33];
  const long j0 = blockIdx.x * 32L, k0 = blockIdx.y * 32L;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool below = k0 >= c0 + j0;  // stored as A(k, j): contiguous in k
  for (int q = ty; q < 32; q += 8) {
    const long k = k0 + (below ? tx : q), j = c0 + j0 + (below ? q : tx);
    const double v = (k < K && j < c0 + nc) ? sym_at(A, lda, k, j) : 0.0;
    if (below) t[q][tx] = v;
    else t[tx][q] = v;
  }
  __syncthreads();
  const int o = (off && k0 + tx < K) ? sign * off[k0 + tx] : 0;
  for (int q = ty; q < 32; q += 8) {
    ExpMax st;
    st.add(t[q][tx], o);
    st.check(flag);
    st.m = __reduce_max_sync(0xffffffffu, st.m);
    if (tx == 0 && j0 + q < nc) st.store(out + j0 + q);
  }
}

// s[k] = the exponent of diag[k * stride] (half of it for a variance), as A's
// column k of the product is to be scaled: times sign.
__global__ void balance_kernel(const double* __restrict__ diag, long stride, int half, int sign,
                               int* __restrict__ s, long K) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= K) return;
  const int e = exponent_of(diag[k * stride]);
  int v = 0;
  if (e != kNone && e != 0x7ff) v = half ? (e - 1023) >> 1 : e - 1023;
  s[k] = sign * max(-400, min(400, v));
}

// Raises the guard for rows whose (balanced) exponent lies outside 2^-900 .. 2^900.
__global__ void check_rows_kernel(const int* __restrict__ e, long rows, int* flag) {
  const long r = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int v = e[r];
  if (v != kNone && (v < 1023 - 900 || v > 1023 + 900)) atomicOr(flag, 1 << 8);
}

// ---- residues of 57-bit integers
// X + 2^58 is a non-negative 59-bit integer; its bytes times 256^k mod m_i (two
// dp4a of unsigned bytes by signed weights) and a multiple of m_i give 0 <= r < 2^20
// congruent to X, here with 0x4b000000 added: the bits of the float 2^23 + r. The
// nearest integer to r / m (m odd, so at least 1 / 2m from a tie, against an error below
// 2^-11) comes from one FP32 fused multiply-add with 1.5 2^23, and r - m q has the
// centred residue in its low byte: both constants' low bytes are zero.
struct ByteWeights {
  int lo[kNM], hi[kNM];  // signed bytes 256^k mod m_i, k = 0..3 and 4..7
  int bias[kNM];         // -(2^58 mod m_i) plus a multiple of m_i above 2^18, plus 0x4b000000
  float inv[kNM];
  int neg[kNM];
};
constexpr ByteWeights byte_weights() {
  ByteWeights b{};
  for (int i = 0; i < kNM; ++i) {
    const int m = kCrt64Mod[i];
    int p = 1 % m;
    unsigned w[2] = {0, 0};
    for (int k = 0; k < 8; ++k) {
      int s = p;
      if (s > m / 2) s -= m;
      if (s > 127) s -= m;  // m = 256: 1, then 0
      w[k / 4] |= ((unsigned)s & 0xffu) << (8 * (k % 4));
      p = p * 256 % m;
    }
    b.lo[i] = (int)w[0];
    b.hi[i] = (int)w[1];
    long long t = 1;
    for (int k = 0; k < 58; ++k) t = t * 2 % m;
    b.bias[i] = (262144 + m - 1) / m * m + m - (int)t + 0x4b000000;
    b.inv[i] = 1.0f / m;
    b.neg[i] = -m;
  }
  return b;
}
__constant__ ByteWeights c_bw = byte_weights();

__device__ __forceinline__ int dp4a_us(uint32_t a, int b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// The residues modulo m_i of four integers (low and high words of X + 2^58), a byte each.
__device__ __forceinline__ uint32_t pack_bytes(const uint32_t (&b)[4]) {
  return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}
__device__ __forceinline__ uint32_t residue_word(const uint32_t* lo, const uint32_t* hi, int i) {
  uint32_t b[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = dp4a_us(lo[q], c_bw.lo[i], dp4a_us(hi[q], c_bw.hi[i], c_bw.bias[i]));
    const float f = fmaf(__int_as_float(r) - 8388608.0f, c_bw.inv[i], 12582912.0f);
    b[q] = (uint32_t)(r + c_bw.neg[i] * __float_as_int(f));
  }
  return pack_bytes(b);
}

// Residues of an operand: tiles of 32 rows x 128 entries through shared memory, each
// thread 16 consecutive entries of a row, so that a modulus is one 16-byte store and a
// row's tile one 128-byte line; entries K..ldq - 1 are zeros. Bound by integer issue
// (~9 slots a residue) and stores: 6.0 ps an entry, 4.0 TB/s, over 3,640 x 29,120 entries
// (7.9 with 32 x 32 tiles, 4-byte stores and a 32-bit multiply-high a residue).
// An entry k of a row is at k + k / 16, rows 137 apart: neither the walk along rows nor
// the one along k conflicts in the banks.
template <int FORM>
__global__ void __launch_bounds__(256)
    residues_kernel(const double* __restrict__ A, long lda, long rows, long K, long c0, int bits,
                    const int* __restrict__ erow, const int* __restrict__ off, int sign,
                    int8_t* __restrict__ out, long ldq, long plane) {
  __shared__ double t[32 * 137];
  const long r0 = blockIdx.x * 32L, k0 = blockIdx.y * 128L;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int h = 0; h < 4; ++h) {  // 32 x 32 parts
    const long kh = k0 + h * 32;
    const bool along_k = FORM == CRT_COLS || (FORM == CRT_SYM && kh >= c0 + r0);
#pragma unroll
    for (int q0 = 0; q0 < 32; q0 += 8) {
      const int q = q0 + ty, kk = along_k ? tx : q, rr = along_k ? q : tx;
      const long k = kh + kk, r = r0 + rr;
      double v = 0.0;
      if (k < K && r < rows) {
        if (FORM == CRT_ROWS) v = A[k * lda + r];
        else if (FORM == CRT_COLS) v = A[r * lda + k];
        else v = sym_at(A, lda, k, c0 + r);
      }
      const int kt = h * 32 + kk;
      t[rr * 137 + kt + (kt >> 4)] = v;
    }
  }
  __syncthreads();
  const int tid = ty * 32 + tx, a = tid >> 3, q16 = (tid & 7) * 16;
  const long r = r0 + a;
  if (r >= rows) return;
  const int e = bits - exp_of(erow[r]);
  uint32_t lo[16], hi[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    // in two steps: the exponent may pass 1,023 by itself
    const long k = k0 + q16 + q;
    const int sh = e + ((off && k < K) ? sign * off[k] : 0), s1 = sh / 2;
    const double m1 = __hiloint2double((s1 + 1023) << 20, 0);
    const double m2 = __hiloint2double((sh - s1 + 1023) << 20, 0);
    const long long x = __double2ll_rn((t[a * 137 + q16 + (q16 >> 4) + q] * m1) * m2);
    const unsigned long long u = (unsigned long long)(x + (1ll << 58));
    lo[q] = (uint32_t)u;
    hi[q] = (uint32_t)(u >> 32);
  }
  int8_t* o = out + r * ldq + k0 + q16;
  static_assert(kCrt64Mod[0] == 256, "its residue is the low byte");
  uint4 w;
  uint32_t b[4][4];
#pragma unroll
  for (int q = 0; q < 16; ++q) b[q >> 2][q & 3] = lo[q];
  w.x = pack_bytes(b[0]);
  w.y = pack_bytes(b[1]);
  w.z = pack_bytes(b[2]);
  w.w = pack_bytes(b[3]);
  *reinterpret_cast<uint4*>(o) = w;
#pragma unroll 3
  for (int i = 1; i < kNM; ++i) {
    w.x = residue_word(lo, hi, i);
    w.y = residue_word(lo + 4, hi + 4, i);
    w.z = residue_word(lo + 8, hi + 8, i);
    w.w = residue_word(lo + 12, hi + 12, i);
    *reinterpret_cast<uint4*>(o + i * plane) = w;
  }
}

long round128(long x) { return (x + 127) / 128 * 128; }

}  // namespace

static long part_tiles(const moao_ctx* ctx) {
  return ctx->cf_part_tiles > 0 ? ctx->cf_part_tiles : kPartTiles;
}
static size_t z_bytes(const moao_ctx* ctx, long tiles) {
  return (size_t)std::min(tiles, part_tiles(ctx)) * kNM * kTcZTile;
}
// Rows of an operand over K whose residues are held at once.
static long part_rows(const moao_ctx* ctx, long K) {
  const size_t bytes = ctx->cf_operand_bytes ? ctx->cf_operand_bytes : kOperandBytes;
  return std::max(256L, (long)(bytes / ((size_t)kNM * round128(K))) / 256 * 256);
}

bool crt64_pays(const moao_ctx* ctx, long M, long N, long K, bool lower) {
  // Below K = 1,024 the combine step (an element of C at a time) costs about what the
  // FP64 product does: at K = 512 35 ps an element on the FP64 tensor cores, 8 + 7 ps
  // here and the operands' share besides.
  if (!ctx->crt_f64 || M < 256 || N < 256 || K < 1024 || K >= (1L << 17)) return false;
  // Measured rates (B200): the FP64 tensor cores 29 TF/s; the residue products
  // 1.9 Pop/s, the combine step 2.4e11 elements/s, the operands 6e10 entries/s,
  // and ~60 us for the extra launches and their last waves.
  const double mnk = (double)M * N * K * (lower ? 0.5 : 1.0);
  const double dmma = 2.0 * mnk / 29e12;
  const double crt = 2.0 * kNM * mnk / 1.9e15 + mnk / K / 2.4e11 +
                     (double)(M + N) * K / 6e10 + 60e-6;
  return crt < dmma;
}

size_t crt64_bytes(long n, long m, long nb, long nact) {
  moao_ctx c;  // the default settings
  size_t qa = 0, qb = 0, z = 0, small = 0;
  auto product = [&](long M, long N, long K, bool lower, int share) {
    if (!crt64_pays(&c, M, N, K, lower)) return;
    const size_t row = (size_t)round128(K) * kNM;
    qa = std::max(qa, std::min(kOperandBytes, row * (size_t)M));
    qb = std::max(qb, std::min(kOperandBytes / share, row * (size_t)N));
    z = std::max(z, z_bytes(&c, tc_tile_count(M, N, lower)));
    small = std::max(small, sizeof(int) * (size_t)(M + N + K + kMaxChunks + 1));
  };
  const long rest = n - nb;
  product(rest, rest, nb, true, 1);
  product(rest, nb, nb, false, 1);
  product(m, nb, nb, false, 1);
  product(m, rest, nb, false, 1);
  size_t qc = 0;
  if (crt64_pays(&c, rest - nb, rest - nb, nb, true)) {
    qc = (size_t)round128(kFactorGroup * nb) * kNM * rest + sizeof(int) * (size_t)rest;
    z = std::max(z, z_bytes(&c, tc_tile_count(rest, rest, true)));
  }
  if (crt64_pays(&c, m, nb, nb, false)) {
    product(m, kSolveGroup * nb, nb, false, 1);
    product(m, std::max(0L, n - kSolveGroup * nb), kSolveGroup * nb, false, 1);
  }
  if (nact > 0) {
    product(m, m, n, true, 1);
    product(m, m, n, false, 1);
    product(m, n, n, false, 8);
    product(nact, m, m, false, 8);
    product(nact, nact, m, false, 1);
  }
  return qa + qb + qc + z + small;
}

moao_status crt64_begin(moao_ctx* ctx) {
  MOAO_TRY(ctx->cf_flag.ensure(sizeof(int) * kFlags));
  MOAO_CUDA_TRY(cudaMemsetAsync(ctx->cf_flag.p, 0, sizeof(int), ctx->stream));
  return MOAO_OK;
}

// Exponents per row and residues of an operand; off (per k, sign +-1): the balance.
static moao_status make_operand(moao_ctx* ctx, int slot, CrtForm form, const double* A, long lda,
                                long rows, long K, long c0, const int* off, int sign,
                                CrtOperand* out) {
  cudaStream_t s = ctx->stream;
  CrtOperand o;
  o.rows = rows;
  o.K = K;
  o.ldq = round128(K);
  DevBuf& qb = slot == 2 ? ctx->cf_c : slot ? ctx->cf_b : ctx->cf_a;
  DevBuf& mb = slot == 2 ? ctx->cf_mc : slot ? ctx->cf_mb : ctx->cf_ma;
  MOAO_TRY(qb.ensure((size_t)kNM * rows * o.ldq));
  MOAO_TRY(mb.ensure(sizeof(int) * (size_t)rows));
  o.q = qb.as<int8_t>();
  o.erow = mb.as<int>();
  int* flag = o.flag = ctx->cf_flag.as<int>() + (slot == 2 ? kGroupFlag : 0);
  KernelTimer kt(ctx, "crt_operand", (double)rows * K);
  MOAO_CUDA_TRY(cudaMemsetAsync(o.erow, 0x80, sizeof(int) * (size_t)rows, s));
  const dim3 blk(32, 8);
  const unsigned rt = (unsigned)((rows + 31) / 32);
  if (form == CRT_ROWS)
    exps_over_cols_kernel<<<dim3(rt, (unsigned)((K + 255) / 256)), blk, 0, s>>>(A, lda, rows, K, off,
                                                                               sign, o.erow, flag);
  else if (form == CRT_COLS)
    exps_over_rows_kernel<<<dim3((unsigned)((rows + 7) / 8), (unsigned)((K + 1023) / 1024)), blk, 0,
                           s>>>(A, lda, K, rows, off, sign, o.erow, flag);
  else
    exps_sym_kernel<<<dim3(rt, (unsigned)((K + 31) / 32)), blk, 0, s>>>(A, lda, rows, K, c0, off, sign,
                                                                       o.erow, flag);
  check_rows_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, s>>>(o.erow, rows, flag);
  const dim3 grid(rt, (unsigned)(o.ldq / 128));
  const long plane = rows * o.ldq;
  const int bits = bits_for(K);
  if (form == CRT_ROWS)
    residues_kernel<CRT_ROWS><<<grid, blk, 0, s>>>(A, lda, rows, K, c0, bits, o.erow, off, sign, o.q,
                                                   o.ldq, plane);
  else if (form == CRT_COLS)
    residues_kernel<CRT_COLS><<<grid, blk, 0, s>>>(A, lda, rows, K, c0, bits, o.erow, off, sign, o.q,
                                                   o.ldq, plane);
  else
    residues_kernel<CRT_SYM><<<grid, blk, 0, s>>>(A, lda, rows, K, c0, bits, o.erow, off, sign, o.q,
                                                  o.ldq, plane);
  ctx->launches += 3;
  MOAO_CUDA_TRY(cudaGetLastError());
  *out = o;
  return MOAO_OK;
}

moao_status crt64_operand(moao_ctx* ctx, const double* A, long lda, long rows, long K,
                          CrtOperand* out) {
  return make_operand(ctx, 0, CRT_ROWS, A, lda, rows, K, 0, nullptr, 0, out);
}

// The balance's exponents into the context's buffer (null where there is none).
static moao_status make_balance(moao_ctx* ctx, const CrtBalance* bal, long K, const int** off) {
  *off = nullptr;
  if (!bal) return MOAO_OK;
  MOAO_TRY(ctx->cf_k.ensure(sizeof(int) * (size_t)K));
  int* sk = ctx->cf_k.as<int>();
  balance_kernel<<<(unsigned)((K + 255) / 256), 256, 0, ctx->stream>>>(bal->diag, bal->stride, bal->half,
                                                                       bal->sign, sk, K);
  ++ctx->launches;
  MOAO_CUDA_TRY(cudaGetLastError());
  *off = sk;
  return MOAO_OK;
}

// Buffers of products of up to rows_a x rows_b over K and `tiles` tiles. A product that
// adds to C takes all it needs here before it writes: MOAO_ERR_OOM then means that C is
// as given, and the caller may compute it another way. rows_b 0: one operand; bal: with
// a balance along K.
static moao_status reserve(moao_ctx* ctx, long rows_a, long rows_b, long K, bool bal, long tiles) {
  MOAO_TRY(ctx->cf_flag.ensure(sizeof(int) * kFlags));
  MOAO_TRY(ctx->cf_a.ensure((size_t)kNM * rows_a * round128(K)));
  MOAO_TRY(ctx->cf_ma.ensure(sizeof(int) * (size_t)rows_a));
  if (rows_b > 0) {
    MOAO_TRY(ctx->cf_b.ensure((size_t)kNM * rows_b * round128(K)));
    MOAO_TRY(ctx->cf_mb.ensure(sizeof(int) * (size_t)rows_b));
  }
  if (bal) MOAO_TRY(ctx->cf_k.ensure(sizeof(int) * (size_t)K));
  return ctx->cf_z.ensure(z_bytes(ctx, tiles));
}

moao_status crt64_reserve_group(moao_ctx* ctx, long n, long nb, long K) {
  const long rows = std::max(1L, n);
  MOAO_TRY(reserve(ctx, rows, 0, nb, false, tc_tile_count(n, n, true)));
  MOAO_TRY(ctx->cf_c.ensure((size_t)kNM * rows * round128(K)));
  return ctx->cf_mc.ensure(sizeof(int) * (size_t)rows);
}

moao_status crt64_group_operand(moao_ctx* ctx, const double* A, long lda, long rows, long K,
                                CrtOperand* out) {
  MOAO_CUDA_TRY(cudaMemsetAsync(ctx->cf_flag.as<int>() + kGroupFlag, 0, sizeof(int), ctx->stream));
  return make_operand(ctx, 2, CRT_ROWS, A, lda, rows, K, 0, nullptr, 0, out);
}

moao_status crt64_product(moao_ctx* ctx, const CrtOperand& A, long a0, const CrtOperand& B, long b0,
                          const GemmArgs* fp64, int n, int max_ctas) {
  const GemmArgs& f = fp64[0];
  const long M = f.M, N = f.N;
  if (A.K != B.K || A.K != f.K || a0 + M > A.rows || b0 + N > B.rows)
    return set_error(MOAO_ERR_BAD_ARG, "crt64: operands do not cover the product");
  cudaStream_t s = ctx->stream;
  int* flag = ctx->cf_flag.as<int>();
  TcTensor ta[kNM], tb[kNM];
  TcGemm g;
  g.kind = kTcI8;
  g.epi = kTcEpiModZ;
  g.nmod = kNM;
  g.moduli = kCrt64Mod;
  g.M = M;
  g.N = N;
  for (int i = 0; i < kNM; ++i) {
    MOAO_TRY(make_tc_map(&ta[i], A.q + (size_t)i * A.rows * A.ldq, kTcI8, A.rows, A.ldq, A.ldq));
    MOAO_TRY(make_tc_map(&tb[i], B.q + (size_t)i * B.rows * B.ldq, kTcI8, B.rows, B.ldq, B.ldq, 256));
    g.A[i] = &ta[i];
    g.B[i] = &tb[i];
  }
  g.nA = g.nB = kNM;
  g.a_row0 = (int)a0;
  g.b_row0 = (int)b0;
  g.seg[0] = TcSegment{0, 0, 0, 0, (int)(A.ldq / 128), 0};
  g.nseg = 1;
  g.lower = f.lowerC ? 1 : 0;
  g.max_ctas = max_ctas;
  g.spin_limit = ctx->cf_polls;
  const long total = tc_tile_count(M, N, f.lowerC);
  const long part = part_tiles(ctx), parts = (total + part - 1) / part;
  if (parts > kMaxChunks) return set_error(MOAO_ERR_UNSUPPORTED, "crt64: product too large");
  MOAO_TRY(ctx->cf_z.ensure(z_bytes(ctx, total)));
  MOAO_CUDA_TRY(cudaMemsetAsync(flag + 1, 0, sizeof(int) * (size_t)parts, s));
  g.C = ctx->cf_z.p;
  TcModz z;
  z.M = M;
  z.N = N;
  z.lower = g.lower;
  z.bits = bits_for(A.K);
  z.ea = A.erow + a0;
  z.eb = B.erow + b0;
  z.Z = ctx->cf_z.as<uint8_t>();
  z.alpha = f.alpha;
  z.beta = f.beta;
  z.C = f.C;
  z.ldc = f.ldc;
  z.skip_a = A.flag;
  for (long c = 0; c < parts; ++c) {
    g.tile0 = z.tile0 = c * part;
    g.tiles = z.tiles = std::min(part, total - c * part);
    g.err = flag + 1 + c;
    z.skip_b = g.err;
    {
      KernelTimer kt(ctx, "crt_int8", 2.0 * kNM * g.tiles * kTcZTile * (double)A.K);
      MOAO_TRY(tc_gemm(g, s, &ctx->launches));
    }
    {
      KernelTimer kt(ctx, "crt_combine", (double)g.tiles * kTcZTile);
      MOAO_TRY(tc_modz_combine(z, s, &ctx->launches));
    }
    for (int i = 0; i < n; ++i)
      MOAO_TRY(gemm_f64_guarded(fp64[i], g.tile0, g.tiles, z.skip_a, z.skip_b, s, &ctx->launches));
  }
  return MOAO_OK;
}

moao_status crt64_gemm(moao_ctx* ctx, const GemmArgs& g, const CrtBalance* bal) {
  // the operands' rows in parts that fit the residue buffers
  const long part = part_rows(ctx, g.K);
  const bool same = g.transB && g.A == g.B && g.lda == g.ldb && g.M == g.N && g.M <= part;
  // the first part is the largest, but of a lower C it is a triangle, and a part below
  // it may hold more tiles
  long tiles = tc_tile_count(std::min(part, g.M), std::min(part, g.N), g.lowerC);
  if (g.lowerC && g.M > part) tiles = std::max(tiles, tc_tile_count(std::min(part, g.M - part), part, false));
  MOAO_TRY(reserve(ctx, std::min(part, g.M), same ? 0 : std::min(part, g.N), g.K, bal && !same, tiles));
  for (long n0 = 0; n0 < g.N; n0 += part) {
    const long nn = std::min(part, g.N - n0);
    for (long m0 = g.lowerC ? n0 : 0; m0 < g.M; m0 += part) {
      const long mm = std::min(part, g.M - m0);
      GemmArgs p = g;
      p.M = mm;
      p.N = nn;
      p.A = g.A + m0;
      p.B = g.transB ? g.B + n0 : g.B + n0 * g.ldb;
      p.C = g.C + m0 + n0 * g.ldc;
      p.lowerC = g.lowerC && m0 == n0;
      MOAO_TRY(crt64_begin(ctx));
      CrtOperand a, b;
      if (same) {
        MOAO_TRY(crt64_operand(ctx, p.A, p.lda, mm, p.K, &a));
        b = a;
      } else {
        const CrtForm form = p.transB ? CRT_ROWS : CRT_COLS;
        const int* off;
        MOAO_TRY(make_balance(ctx, bal, p.K, &off));
        MOAO_TRY(make_operand(ctx, 0, CRT_ROWS, p.A, p.lda, mm, p.K, 0, off, 1, &a));
        MOAO_TRY(make_operand(ctx, 1, form, p.B, p.ldb, nn, p.K, 0, off, -1, &b));
      }
      MOAO_TRY(crt64_product(ctx, a, 0, b, 0, &p, 1));
    }
  }
  return MOAO_OK;
}

moao_status crt64_symm(moao_ctx* ctx, long M, long n, const double* A, long lda, const double* B,
                       long ldb, double* C, long ldc) {
  // columns of S in parts of an eighth of the buffer: their residues are written
  // and read once each
  const long part = part_rows(ctx, n), cpart = std::max(256L, part / 8 / 256 * 256);
  MOAO_TRY(reserve(ctx, std::min(part, M), std::min(cpart, n), n, true,
                   tc_tile_count(std::min(part, M), std::min(cpart, n), false)));
  for (long m0 = 0; m0 < M; m0 += part) {
    const long mm = std::min(part, M - m0);
    MOAO_TRY(crt64_begin(ctx));
    CrtOperand a, b;
    const int* off;
    const CrtBalance bal{B, ldb + 1, 1, 1};  // S's own diagonal: A(:, k) goes with S(k, :)
    MOAO_TRY(make_balance(ctx, &bal, n, &off));
    MOAO_TRY(make_operand(ctx, 0, CRT_ROWS, A + m0, lda, mm, n, 0, off, 1, &a));
    for (long c0 = 0; c0 < n; c0 += cpart) {
      const long cc = std::min(cpart, n - c0);
      MOAO_TRY(make_operand(ctx, 1, CRT_SYM, B, ldb, cc, n, c0, off, -1, &b));
      GemmArgs f[2];
      f[0].M = mm; f[0].N = cc; f[0].K = n;
      f[0].A = A + m0; f[0].lda = lda;
      f[0].B = B + c0 * ldb; f[0].ldb = ldb;
      f[0].triB = TRI_LOWER; f[0].tri_off = c0;
      f[0].C = C + m0 + c0 * ldc; f[0].ldc = ldc;
      f[1] = f[0];
      f[1].beta = 1.0;
      f[1].B = B + c0; f[1].transB = true;
      f[1].triB = TRI_STRICT_LOWER;
      MOAO_TRY(crt64_product(ctx, a, 0, b, 0, f, 2));
    }
  }
  return MOAO_OK;
}

}  // namespace moao

extern "C" moao_status moao_debug_crt64(moao_ctx* ctx, int form, int lower, long M, long N, long K,
                                        double alpha, const double* A, long lda, const double* B,
                                        long ldb, double beta, double* C, long ldc) {
  using namespace moao;
  if (!ctx || !A || !B || !C || form < 0 || form > 2 || M < 1 || N < 1 || K < 1 || K >= (1L << 17) ||
      lda < M || ldb < (form == CRT_ROWS ? N : K) || ldc < M ||
      (lower && (form != CRT_ROWS || M != N)) || (form == CRT_SYM && N != K))
    return set_error(MOAO_ERR_BAD_ARG, "debug_crt64: bad arguments");
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  if (form == CRT_SYM) return crt64_symm(ctx, M, N, A, lda, B, ldb, C, ldc);
  GemmArgs g;
  g.M = M; g.N = N; g.K = K;
  g.alpha = alpha; g.beta = beta;
  g.A = A; g.lda = lda;
  g.B = B; g.ldb = ldb;
  g.transB = form == CRT_ROWS;
  g.C = C; g.ldc = ldc;
  g.lowerC = lower != 0;
  return crt64_gemm(ctx, g, nullptr);
}
