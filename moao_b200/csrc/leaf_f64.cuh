// Leaf Cholesky factorisation fused with the inversion of the factor, for one
// diagonal block of at most 64 columns: a device function run by one CTA of
// 256 threads, shared by the blocked factorisation's leaf kernel and the
// persistent tile-task kernel of batched small instances.
#ifndef MOAO_LEAF_F64_CUH
#define MOAO_LEAF_F64_CUH

namespace moao {

constexpr int LEAF = 64;
constexpr int LEAF_THREADS = 256;
constexpr int LEAF_SB = 16;               // sub-block edge
constexpr int LEAF_NB = LEAF / LEAF_SB;   // sub-blocks per side (4)
// leading dimension of the shared blocks: 4 mod 16 doubles, so the MMA fragment
// reads (gid + tig LD and tig + gid LD) hit distinct banks
constexpr int LEAF_LD = LEAF + 4;
// shared memory of leaf_factor_inverse, bytes: factor, inverse, reciprocal pivots
constexpr int LEAF_SMEM_BYTES = (2 * LEAF * LEAF_LD + LEAF) * 8;

// Bound: the chain of 64 dependent pivots (each the previous column's update of
// one element, then a reciprocal square root), so everything else is kept off
// that chain. The block is walked in four steps of 16 columns:
//   A(p)  warp 0 brings the 16x16 diagonal sub-block p up to date and factors
//         it in registers (lane i = row i; four columns at a time, their 4x4
//         pivot block factored redundantly by every lane, so one exchange
//         serves four pivots); meanwhile warps 1-7 apply step p - 1 to the rest
//         of the trailing block, form the sums of row p of the inverse,
//         T_pj = -sum_k L_pk X_kj (all as m16n8k16 MMAs), and send what is
//         final to global memory;
//   B(p)  one thread per row below solves x L_pp^T = A_ip, one thread per
//         column of the inverse L_pp x = T_pj.
// Every element takes the same operations in the same order as in the plain
// right-looking algorithm by columns, a(i,k) <- fma(-L(i,j), L(k,j), a(i,k))
// with L(i,j) = a(i,j) rsqrt(a(j,j)), and forward substitution by rows, so the
// results are those of that algorithm bit for bit (the mixed path's FP32 factor
// does not depend on how the leaf is arranged). Two CTA barriers per 16 columns
// instead of one per pivot and per inverse row: 53.9 -> 17.2 us per 64 x 64 leaf
// launch (CUDA events; the element-wise form on 1,024 threads before), 11 us of
// it in the CTA.
// A non-positive pivot is reported (first failing global column, 1-based, into
// *info) and replaced by 1 so the kernel finishes without NaNs; rows and
// columns beyond n are an identity block. Only the n x n parts of A (lower) and
// Linv are written. A is read through L2 (ld.global.cg): in the tile-task
// kernel other SMs wrote it moments before.

__device__ __forceinline__ void leaf_mma(double (&c)[4], const double (&a)[8],
                                         const double (&b)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
      "{%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
        "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// c -= P Q (TRANSQ: P Q^T) for a 16 x 8 tile: P 16 x 16 at p, Q 16 x 8 (TRANSQ:
// 8 x 16) at q, both column-major with leading dimension LEAF_LD. The MMA is the
// chain of fused multiply-adds over ascending k.
template <bool TRANSQ>
__device__ __forceinline__ void leaf_tile(double (&c)[4], const double* p, const double* q) {
  const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  double a[8], b[4];
#pragma unroll
  for (int r = 0; r < 8; ++r) a[r] = -p[gid + 8 * (r & 1) + (4 * (r >> 1) + tig) * LEAF_LD];
#pragma unroll
  for (int r = 0; r < 4; ++r)
    b[r] = TRANSQ ? q[gid + (4 * r + tig) * LEAF_LD] : q[4 * r + tig + gid * LEAF_LD];
  leaf_mma(c, a, b);
}

// element h of this lane's part of the 16 x 8 tile at d
__device__ __forceinline__ double* leaf_tile_at(double* d, int h) {
  const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  return d + gid + 8 * (h >> 1) + (2 * tig + (h & 1)) * LEAF_LD;
}

// Columns J..J+3 of a 16 x 16 diagonal sub-block held one row per lane (a, lanes
// 16-31 repeating lanes 0-15): the 4 x 4 pivot block is broadcast and factored
// by every lane for itself, the finished columns go to D and the rest of the
// row is updated from there. n and col0: valid columns from, and global index
// of, the sub-block's first column.
template <int J>
__device__ __forceinline__ void leaf_pivots(double (&a)[LEAF_SB], double* D, double* rinv, int row,
                                            int n, long col0, int* info) {
  const int lane = threadIdx.x & 31;
  double b[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) b[r][c] = __shfl_sync(0xffffffffu, a[J + c], J + r);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const bool bad = !(b[c][c] > 0.0);
    if (bad && lane == 0 && J + c < n) atomicCAS(info, 0, (int)(col0 + J + c + 1));
    b[c][c] = bad ? 1.0 : b[c][c];
    if (row == J + c) a[J + c] = b[c][c];
    const double r = rsqrt(b[c][c]);
    if (lane == J + c) rinv[J + c] = r;
    a[J + c] *= r;
#pragma unroll
    for (int q = c + 1; q < 4; ++q) {
      b[q][c] *= r;
#pragma unroll
      for (int t = c + 1; t <= q; ++t) b[q][t] = fma(-b[q][c], b[t][c], b[q][t]);
    }
#pragma unroll
    for (int q = c + 1; q < 4; ++q) a[J + q] = fma(-a[J + c], b[q][c], a[J + q]);
  }
  if (lane < LEAF_SB) {
#pragma unroll
    for (int c = 0; c < 4; ++c) D[row + (J + c) * LEAF_LD] = J + c <= row ? a[J + c] : 0.0;
  }
  __syncwarp();
#pragma unroll
  for (int k = J + 4; k < LEAF_SB; ++k)
#pragma unroll
    for (int c = 0; c < 4; ++c) a[k] = fma(-a[J + c], D[k + (J + c) * LEAF_LD], a[k]);
}

// Called by all LEAF_THREADS threads of the CTA.
__device__ __forceinline__ void leaf_factor_inverse(double* A, long lda, double* Linv, long ldi,
                                                    int n, long col0, int* info,
                                                    double* leaf_smem) {
  constexpr int LD = LEAF_LD, SB = LEAF_SB;
  double* S = leaf_smem;              // the block, then its factor
  double* X = S + LEAF * LD;          // the inverse (T_pj in its place until finished)
  double* rinv = X + LEAF * LD;       // 1 / L(j,j)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  {
    constexpr int PER = LEAF * LEAF / LEAF_THREADS;
    double v[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = tid + q * LEAF_THREADS, i = e & (LEAF - 1), j = e >> 6;
      v[q] = (i < n && j < n) ? (i >= j ? __ldcg(A + (long)j * lda + i) : 0.0)
                              : (i == j ? 1.0 : 0.0);
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = tid + q * LEAF_THREADS;
      S[(e & (LEAF - 1)) + (e >> 6) * LD] = v[q];
    }
  }
  __syncthreads();
  auto at = [&](double* m, int i, int j) { return m + SB * i + SB * j * LD; };
  // 16 x 8 tile at d -= P Q^T
  auto update = [&](double* d, const double* pp, const double* qq) {
    double c[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) c[h] = *leaf_tile_at(d, h);
    leaf_tile<true>(c, pp, qq);
#pragma unroll
    for (int h = 0; h < 4; ++h) *leaf_tile_at(d, h) = c[h];
  };
  // finished parts to global memory: columns of panel i of the factor, rows of
  // sub-block row i of the inverse, by threads 0..nthr-1
  auto write_out = [&](int i, int t, int nthr) {
    for (int e = t; e < SB * LEAF; e += nthr) {
      const int r = e & (LEAF - 1), c = SB * i + (e >> 6);
      if (r >= c && r < n) A[(long)c * lda + r] = S[r + c * LD];
      const int xr = SB * i + (e & (SB - 1)), xc = e >> 4;
      if (xr < n && xc < n) Linv[(long)xc * ldi + xr] = xr >= xc ? X[xr + xc * LD] : 0.0;
    }
  };
#pragma unroll 1
  for (int p = 0; p < LEAF_NB; ++p) {
    // ---- A(p)
    if (warp == 0) {
      if (p > 0) {
        double c[2][4];
#pragma unroll
        for (int t = 0; t < 8; ++t) c[t >> 2][t & 3] = *leaf_tile_at(at(S, p, p) + 8 * (t >> 2) * LD, t & 3);
#pragma unroll
        for (int t = 0; t < 2; ++t)
          leaf_tile<true>(c[t], at(S, p, p - 1), at(S, p, p - 1) + 8 * t);
#pragma unroll
        for (int t = 0; t < 8; ++t) *leaf_tile_at(at(S, p, p) + 8 * (t >> 2) * LD, t & 3) = c[t >> 2][t & 3];
        __syncwarp();
      }
      double* D = at(S, p, p);
      const int row = lane & (SB - 1);  // lanes 16-31 repeat lanes 0-15
      double a[SB];
#pragma unroll
      for (int k = 0; k < SB; ++k) a[k] = D[row + k * LD];
      const int pc = SB * p;
      leaf_pivots<0>(a, D, rinv + pc, row, n - pc, col0 + pc, info);
      leaf_pivots<4>(a, D, rinv + pc, row, n - pc, col0 + pc, info);
      leaf_pivots<8>(a, D, rinv + pc, row, n - pc, col0 + pc, info);
      leaf_pivots<12>(a, D, rinv + pc, row, n - pc, col0 + pc, info);
    } else if (p > 0) {
      // trailing tiles (i, j) >= p of step p - 1 except (p, p)
      int t = 0;
      for (int j = p; j < LEAF_NB; ++j)
        for (int i = j; i < LEAF_NB; ++i) {
          if (i == p && j == p) continue;
          for (int h = 0; h < 2; ++h, ++t)
            if (t % 7 == warp - 1)
              update(at(S, i, j) + 8 * h * LD, at(S, i, p - 1), at(S, j, p - 1) + 8 * h);
        }
      // T_pj = -sum over k in j..p-1 of L_pk X_kj
      for (int h = 0; h < 2 * p; ++h, ++t)
        if (t % 7 == warp - 1) {
          double c[4] = {};
          for (int k = h >> 1; k < p; ++k)
            leaf_tile<false>(c, at(S, p, k), at(X, k, 0) + 8 * h * LD);
#pragma unroll
          for (int e = 0; e < 4; ++e) *leaf_tile_at(at(X, p, 0) + 8 * h * LD, e) = c[e];
        }
      write_out(p - 1, tid - 32, LEAF_THREADS - 32);
    }
    __syncthreads();
    // ---- B(p)
    const double* D = at(S, p, p);
    const double* rp = rinv + SB * p;
    const int below = LEAF - SB * (p + 1), left = SB * (p + 1);
    const bool rows = tid < below, cols = tid >= 64 && tid < 64 + left;
    if (rows || cols) {
      // a row below: x L_pp^T = its 16 entries; a column of X: L_pp x = its sums
      const int c = tid - 64;
      double* v = rows ? S + left + tid + SB * p * LD : X + SB * p + c * LD;
      const int inc = rows ? LD : 1;
      double x[SB];
#pragma unroll
      for (int j = 0; j < SB; ++j)
        x[j] = (cols && c >= SB * p) ? (j == c - SB * p ? 1.0 : 0.0) : v[j * inc];
#pragma unroll
      for (int j = 0; j < SB; ++j) {
        x[j] *= rp[j];
#pragma unroll
        for (int k = j + 1; k < SB; ++k) x[k] = fma(-x[j], D[k + j * LD], x[k]);
      }
#pragma unroll
      for (int j = 0; j < SB; ++j) v[j * inc] = x[j];
    }
    __syncthreads();
  }
  write_out(LEAF_NB - 1, tid, LEAF_THREADS);
}

}  // namespace moao

#endif  // MOAO_LEAF_F64_CUH
