// FP64 dense kernels for the plain-FP64 reconstructor path.
//
// Blackwell has no FP64 kind for tcgen05.mma, so FP64 contractions run on the
// FP64 DMMA path (mma.sync m16n8k16 .f64), fed by a 4-stage cp.async pipeline of
// 128x64x16 (or 64x64x16) tiles in shared memory (bank-conflict-free padded
// layouts). One kernel template serves every contraction of the path:
//   trailing SYRK of the tiled Cholesky   (transB, lowerC)
//   panel TRSM as a product with the inverse diagonal block
//   the two triangular solves of R        (NN / NT)
//   SYR2K / SYMM / GEMM of the Cee/Cvv chain (triB masks a lower-stored
//   symmetric operand; no symmetric copy is ever materialised)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "chain.cuh"
#include "dense.h"
#include "leaf_f64.cuh"
#include "tile_walk.cuh"

namespace moao {
namespace {

constexpr int PAD_MN = 4;  // doubles of padding on m/n-contiguous rows
constexpr int PAD_K = 4;   // doubles of padding on k-contiguous rows

// CTA tile BM x BN; each warp computes WM x 32 (warps: BM/WM along m, BN/32
// along n). 128x64 (8 warps of 32x32, ~120 registers, two CTAs per SM so one
// CTA's prologue and C epilogue overlap the other's DMMA loop) for large
// products: 26.2 TF/s on the ELT FP64 build against 21.4 for 128x128 tiles with
// one CTA per SM and 24.4 for 128x64 with 4 warps of 64x32. 64x64 (4 warps of
// 32x32) when even that would leave most SMs idle (the small products of the
// diagonal-block recursion). BK (K per pipeline stage, a multiple of 16) and
// STAGES (the cp.async ring) are the other dimensions a configuration sets
// (GemmArgs::cfg, chosen per context: moao_ctx_set_gemm_tile / the autotuner).
template <int BM_, int BN_, int WM_, int BK_ = 16, int STAGES_ = 4, int WN_ = 32>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, BK = BK_, STAGES = STAGES_;
  static constexpr int WARPS_M = BM / WM, WARPS_N = BN / WN;
  static constexpr int NTHREADS = 32 * WARPS_M * WARPS_N;
  static constexpr int MF = WM / 8;             // 8-row fragments per warp
  static constexpr int NF = WN / 8;             // 8-column fragments per warp
  static constexpr int LDA_S = BM + PAD_MN;     // As[k][m]
  static constexpr int LDB_S = BN + PAD_MN;     // Bs[k][n]   (transB)
  static constexpr int LDBT_S = BK + PAD_K;     // Bs[n][k]   (!transB)
  static constexpr int A_STAGE = BK * LDA_S;
  static constexpr int B_STAGE = (BK * LDB_S > BN * LDBT_S) ? BK * LDB_S : BN * LDBT_S;
  static constexpr size_t SMEM_BYTES = (size_t)STAGES * (A_STAGE + B_STAGE) * sizeof(double);
};
using TileL = Tile<128, 64, 32>;
using TileS = Tile<64, 64, 32>;
// 32 x 32 tiles for the products of a handful of 64 x 64 ones: an SM does a
// 64 x 64 x K tile in 64 K cycles (its FP64 rate is 64 multiply-adds a cycle), so
// few large tiles leave a product of the diagonal-block recursion to a few SMs.
using TileXS = Tile<32, 32, 16, 32, 3, 16>;
// alternative large-product configurations (GemmArgs::cfg 1..3)
using TileL32x2 = Tile<128, 64, 32, 32, 2>;   // 102 KB: two CTAs per SM, two k16 steps per barrier
using TileL32x3 = Tile<128, 64, 32, 32, 3>;   // 154 KB: one CTA per SM
using TileL16x6 = Tile<128, 64, 32, 16, 6>;   // 154 KB: one CTA per SM, deeper ring

__device__ __forceinline__ void cp_async(double* smem, const double* gmem, int vec, int valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = valid * 8;
  if (vec == 2) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(bytes));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem),
                 "r"(bytes));
  }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// m16n8k16 FP64 MMA: A 16x16 (8 per thread: rows gid, gid+8; cols tig + 4r),
// B 16x8 (4 per thread: rows tig + 4r, col gid), C 16x8 (rows gid, gid+8;
// cols 2 tig, 2 tig + 1).
__device__ __forceinline__ void dmma16(double& c0, double& c1, double& c2, double& c3,
                                       const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, "
      "{%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c0), "+d"(c1), "+d"(c2), "+d"(c3)
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]),
        "d"(b[0]), "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

struct KParams {
  long M, N, K;
  double alpha, beta;
  const double* A;
  long lda;
  const double* B;
  long ldb;
  double* C;
  long ldc;
  int triB;
  long tri_off;
  int triA = 0;  // A lower triangular (zeros stored above): k <= row only
  // tile order (set by the launcher): bands of group_m row tiles; inside a band
  // the column tiles in turn, the band's row tiles fastest
  int tiles_m, tiles_n, group_m;
};

// Tile v of the launch in band order. Consecutive CTAs share one column strip
// of B and the band's row strips of A stay in L2 while the band sweeps the
// columns: the CTAs resident together touch group_m strips of A and a few of B
// instead of every row strip of A (which, for a 1,024-wide panel of an
// nmeas ~ 15k-48k factorisation, no longer fits in L2). For a lower C the sweep
// of a band stops at the diagonal. Returns false past the last tile.
template <int BM, int BN, bool LOWERC>
__device__ __forceinline__ bool band_tile(const KParams& p, long v, long* m0, long* n0) {
  for (int b0 = 0; b0 < p.tiles_m; b0 += p.group_m) {
    const int rows = min(p.group_m, p.tiles_m - b0);
    long cols = p.tiles_n;
    if (LOWERC) cols = min((long)p.tiles_n, ((long)(b0 + rows) * BM - 1) / BN + 1);
    const long cnt = rows * cols;
    if (v < cnt) {
      *m0 = (long)(b0 + (int)(v % rows)) * BM;
      *n0 = (v / rows) * BN;
      return true;
    }
    v -= cnt;
  }
  return false;
}

// Load one BK-slice of an MN-contiguous operand (A, or B when transB): the tile
// rows r0..r0+R-1 of columns k0..k0+15 of a column-major rows x K matrix, stored
// with row stride LDS (R = BM, LDS = LDA_S for A; R = BN, LDS = LDB_S for B).
template <class TL, int VEC, int R, int LDS>
__device__ __forceinline__ void load_mn_tile(double* s, const double* g, long ld, long rows,
                                             long K, long r0, long k0) {
  constexpr int CH = R / VEC;                // chunks per k column
  constexpr int TOTAL = CH * TL::BK;
  for (int c = threadIdx.x; c < TOTAL; c += TL::NTHREADS) {
    const int kk = c / CH, rr = (c % CH) * VEC;
    const long gr = r0 + rr, gk = k0 + kk;
    int valid = 0;
    if (gk < K && gr < rows) valid = (int)min((long)VEC, rows - gr);
    const double* src = valid ? g + gk * ld + gr : g;
    cp_async(s + kk * LDS + rr, src, VEC, valid);
  }
}

// Load one BK-slice of a K-contiguous operand (B when !transB): rows k0..k0+15
// of columns n0..n0+BN-1 of a column-major K x N matrix, stored Bs[n][k].
template <class TL, int VEC>
__device__ __forceinline__ void load_k_tile(double* s, const double* g, long ld, long N,
                                            long K, long n0, long k0) {
  constexpr int CH = TL::BK / VEC;
  constexpr int TOTAL = CH * TL::BN;
  for (int c = threadIdx.x; c < TOTAL; c += TL::NTHREADS) {
    const int nn = c / CH, kk = (c % CH) * VEC;
    const long gn = n0 + nn, gk = k0 + kk;
    int valid = 0;
    if (gn < N && gk < K) valid = (int)min((long)VEC, K - gk);
    const double* src = valid ? g + gn * ld + gk : g;
    cp_async(s + nn * TL::LDBT_S + kk, src, VEC, valid);
  }
}

// The tile of C at (m0, n0), by all threads of the CTA.
template <class TL, bool TRANSB, bool LOWERC, int VEC, bool MMA16>
__device__ __forceinline__ void gemm_tile(const KParams& p, double* smem, const long m0,
                                          const long n0) {
  constexpr int BM = TL::BM, BN = TL::BN, NTHREADS = TL::NTHREADS, MF = TL::MF, NF = TL::NF;
  constexpr int BK = TL::BK, STAGES = TL::STAGES;
  constexpr int LDA_S = TL::LDA_S, LDB_S = TL::LDB_S, LDBT_S = TL::LDBT_S;
  constexpr int A_STAGE = TL::A_STAGE, B_STAGE = TL::B_STAGE;
  double* As = smem;
  double* Bs = smem + STAGES * A_STAGE;

  // K range (tile aligned); a triangular B limits it.
  long kb = 0, ke = p.K;
  if (p.triB != 0) {
    if (!TRANSB) kb = n0 + p.tri_off;          // B(k, n) with k >= n
    else ke = min(p.K, n0 + p.tri_off + BN);   // B(n, k) with n >= k
  }
  if (p.triA) ke = min(ke, m0 + BM);
  kb = (kb / BK) * BK;
  const int ntiles = (ke > kb) ? (int)((ke - kb + BK - 1) / BK) : 0;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = (warp % TL::WARPS_M) * TL::WM, wn = (warp / TL::WARPS_M) * TL::WN;
  const int gid = lane >> 2, tig = lane & 3;

  // acc[i][j][h]: k4 layout = MF m-frags of 8 rows x NF n-frags x 2;
  // k16 layout = MF/2 m-frags of 16 rows x NF n-frags x 4.
  double acc[MF][NF][2];
#pragma unroll
  for (int i = 0; i < MF; ++i)
#pragma unroll
    for (int j = 0; j < NF; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  auto issue = [&](int stage, int t) {
    const long k0 = kb + (long)t * BK;
    load_mn_tile<TL, VEC, BM, LDA_S>(As + stage * A_STAGE, p.A, p.lda, p.M, p.K, m0, k0);
    if (TRANSB)
      load_mn_tile<TL, VEC, BN, LDB_S>(Bs + stage * B_STAGE, p.B, p.ldb, p.N, p.K, n0, k0);
    else load_k_tile<TL, VEC>(Bs + stage * B_STAGE, p.B, p.ldb, p.N, p.K, n0, k0);
  };

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ntiles) issue(s, s);
    cp_commit();
  }

  for (int t = 0; t < ntiles; ++t) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    const int stage = t % STAGES;
    double* as = As + stage * A_STAGE;
    double* bs = Bs + stage * B_STAGE;
    if (p.triB != 0) {
      // Zero the entries of the stored B outside its lower (or strictly lower)
      // triangle when this slice crosses the diagonal.
      const long k0 = kb + (long)t * BK;
      const long d0 = n0 + p.tri_off;
      const bool crosses = TRANSB ? (k0 + BK - 1 >= d0) : (k0 <= d0 + BN - 1);
      if (crosses) {
        for (int e = threadIdx.x; e < BK * BN; e += NTHREADS) {
          const int kk = e / BN, nn = e % BN;
          const long gk = k0 + kk, gn = d0 + nn;
          // stored row / column of this element
          const long row = TRANSB ? gn : gk, col = TRANSB ? gk : gn;
          const bool keep = (p.triB == 1) ? (row >= col) : (row > col);
          if (!keep) {
            if (TRANSB) bs[kk * LDB_S + nn] = 0.0;
            else bs[nn * LDBT_S + kk] = 0.0;
          }
        }
        __syncthreads();
      }
    }
    {
      const int nt = t + STAGES - 1;
      if (nt < ntiles) issue(nt % STAGES, nt);
      cp_commit();
    }
    if (MMA16) {
#pragma unroll
      for (int k16 = 0; k16 < BK; k16 += 16) {
        double bf[NF][4];
#pragma unroll
        for (int j = 0; j < NF; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int k = k16 + r * 4 + tig, n = wn + j * 8 + gid;
            bf[j][r] = TRANSB ? bs[k * LDB_S + n] : bs[n * LDBT_S + k];
          }
#pragma unroll
        for (int i = 0; i < MF / 2; ++i) {
          double af[8];
#pragma unroll
          for (int r = 0; r < 8; ++r)
            af[r] = as[(k16 + (r >> 1) * 4 + tig) * LDA_S + wm + i * 16 + gid + 8 * (r & 1)];
#pragma unroll
          for (int j = 0; j < NF; ++j)
            dmma16(acc[2 * i][j][0], acc[2 * i][j][1], acc[2 * i + 1][j][0], acc[2 * i + 1][j][1],
                   af, bf[j]);
        }
      }
    } else {
#pragma unroll
      for (int k4 = 0; k4 < BK; k4 += 4) {
        double a[MF], b[NF];
#pragma unroll
        for (int i = 0; i < MF; ++i) a[i] = as[(k4 + tig) * LDA_S + wm + i * 8 + gid];
#pragma unroll
        for (int j = 0; j < NF; ++j) {
          if (TRANSB) b[j] = bs[(k4 + tig) * LDB_S + wn + j * 8 + gid];
          else b[j] = bs[(wn + j * 8 + gid) * LDBT_S + k4 + tig];
        }
#pragma unroll
        for (int i = 0; i < MF; ++i)
#pragma unroll
          for (int j = 0; j < NF; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
      }
    }
  }
  cp_wait<0>();

  // Epilogue through shared memory (the operand ring is free now): the C tile
  // is read with coalesced loads, all in flight (only when beta != 0), each
  // thread combines its accumulators with it in place, and the tile goes back
  // with coalesced stores, lower part only for a lower C. Leading dimension
  // BM + 2 keeps the fragment accesses free of bank conflicts.
  // k4: fragment i covers rows wm + 8 i; k16: acc[2q][j] and acc[2q+1][j] hold
  // the 4 values of m16 fragment q (rows wm + 16 q + gid and + 8).
  constexpr int LDC_S = BM + 2;
  static_assert((size_t)BN * LDC_S * sizeof(double) <= TL::SMEM_BYTES, "C tile exceeds the ring");
  __syncthreads();
  double* Cs = smem;
  const bool read_c = p.beta != 0.0;
  for (int e = threadIdx.x; e < BM * BN; e += NTHREADS) {
    const int rr = e % BM, cc = e / BM;
    const long r = m0 + rr, c = n0 + cc;
    Cs[cc * LDC_S + rr] = (read_c && r < p.M && c < p.N) ? p.C[c * p.ldc + r] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MF; ++i) {
    const int rr = MMA16 ? wm + (i >> 1) * 16 + (i & 1) * 8 + gid : wm + i * 8 + gid;
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc = wn + j * 8 + 2 * tig + h;
        double* d = Cs + cc * LDC_S + rr;
        *d = read_c ? p.alpha * acc[i][j][h] + p.beta * *d : p.alpha * acc[i][j][h];
      }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < BM * BN; e += NTHREADS) {
    const int rr = e % BM, cc = e / BM;
    const long r = m0 + rr, c = n0 + cc;
    if (r < p.M && c < p.N && !(LOWERC && r < c)) p.C[c * p.ldc + r] = Cs[cc * LDC_S + rr];
  }
}

template <class TL, bool TRANSB, bool LOWERC, int VEC, bool MMA16>
__global__ void __launch_bounds__(TL::NTHREADS) gemm_f64_kernel(const KParams p) {
  extern __shared__ __align__(16) double smem[];
  chain_wait();
  long m0 = 0, n0 = 0;
  if (!band_tile<TL::BM, TL::BN, LOWERC>(p, blockIdx.x, &m0, &n0)) return;
  if (LOWERC && m0 + TL::BM <= n0) return;  // tile strictly above the diagonal
  gemm_tile<TL, TRANSB, LOWERC, VEC, MMA16>(p, smem, m0, n0);
}

// The tiles [tile0, tile0 + tiles) of a tensor-core product's walk over C, when
// one of its two guard flags is raised; otherwise the few CTAs leave at once.
template <class TL, bool TRANSB, bool LOWERC, int VEC>
__global__ void __launch_bounds__(TL::NTHREADS)
    gemm_f64_guard_kernel(const KParams p, const __grid_constant__ TileWalk walk, int tile0,
                          int tiles, const int* flag_a, const int* flag_b) {
  extern __shared__ __align__(16) double smem[];
  if (*flag_a == 0 && *flag_b == 0) return;
  constexpr int PER = kWalkTileN / TL::BN;  // columns of this kernel's tiles in one of the walk's
  static_assert(TL::BM == 128, "the walk's tiles are 128 rows");
  for (int v = blockIdx.x; v < tiles * PER; v += gridDim.x) {
    int mt, nt;
    decode_tile(walk, tile0 + v / PER, &mt, &nt);
    const long m0 = (long)mt * TL::BM, n0 = (long)nt * kWalkTileN + (v % PER) * TL::BN;
    if (m0 >= p.M || n0 >= p.N || (LOWERC && m0 + TL::BM <= n0)) continue;
    gemm_tile<TL, TRANSB, LOWERC, VEC, true>(p, smem, m0, n0);
    __syncthreads();  // the C tile in shared memory is stored before the next ring fill
  }
}

// FP64 MMA shape: m16n8k16 unless MOAO_GEMM_MMA=k4 selects m8n8k4.
bool use_mma16() {
  static const bool v = [] {
    const char* e = getenv("MOAO_GEMM_MMA");
    return !(e && e[0] == 'k' && e[1] == '4');
  }();
  return v;
}

template <class TL, bool TRANSB, bool LOWERC, int VEC, bool MMA16>
moao_status launch_gemm_t(const KParams& p, bool chained, cudaStream_t s) {
  static std::atomic<unsigned long long> configured{0};
  auto kern = gemm_f64_kernel<TL, TRANSB, LOWERC, VEC, MMA16>;
  MOAO_CUDA_TRY(set_smem_limit(kern, (int)TL::SMEM_BYTES, configured));
  KParams q = p;
  q.tiles_m = (int)((p.M + TL::BM - 1) / TL::BM);
  q.tiles_n = (int)((p.N + TL::BN - 1) / TL::BN);
  q.group_m = std::max(1, 4096 / TL::BM);  // bands of 4,096 rows
  long total = 0;
  for (int b0 = 0; b0 < q.tiles_m; b0 += q.group_m) {
    const int rows = std::min(q.group_m, q.tiles_m - b0);
    long cols = q.tiles_n;
    if (LOWERC) cols = std::min((long)q.tiles_n, ((long)(b0 + rows) * TL::BM - 1) / TL::BN + 1);
    total += rows * cols;
  }
  if (total <= 0) return MOAO_OK;
  if (total > 0x7fffffffL) return set_error(MOAO_ERR_BAD_ARG, "gemm: too many tiles");
  MOAO_CUDA_TRY(launch_chained(chained, kern, dim3((unsigned)total), dim3(TL::NTHREADS),
                               TL::SMEM_BYTES, s, q));
  return MOAO_OK;
}

// Products whose 128x128-tile count would fill fewer than two waves of the 148
// SMs take the 64x64 tiles (twice the CTAs of the 128x64 ones).
bool small_tiles(const KParams& p) {
  const long tiles = ((p.M + 127) / 128) * ((p.N + 127) / 128);
  return tiles < 2 * 148;
}

// Products of at most 74 tiles of 64 x 64 (half the SMs) take 32 x 32 ones: up to two
// per SM. The small products of an nmeas 640 reconstructor: 19.8 -> 11.9 us a launch
// on average, of an nmeas 12,032 one's diagonal blocks 18.3 -> 11.6 (B200, CUDA events
// around each launch).
bool tiny_tiles(const KParams& p, bool lower) {
  const long tiles = ((p.M + 63) / 64) * ((p.N + 63) / 64);
  return (lower ? (tiles + 1) / 2 : tiles) <= 74;
}

template <bool TRANSB, bool LOWERC, int VEC>
moao_status launch_gemm(const KParams& p, int cfg, bool ch, cudaStream_t s) {
  if (use_mma16() && tiny_tiles(p, LOWERC)) return launch_gemm_t<TileXS, TRANSB, LOWERC, VEC, true>(p, ch, s);
  if (small_tiles(p))
    return use_mma16() ? launch_gemm_t<TileS, TRANSB, LOWERC, VEC, true>(p, ch, s)
                       : launch_gemm_t<TileS, TRANSB, LOWERC, VEC, false>(p, ch, s);
  switch (cfg) {
    case 1: return launch_gemm_t<TileL32x2, TRANSB, LOWERC, VEC, true>(p, ch, s);
    case 2: return launch_gemm_t<TileL32x3, TRANSB, LOWERC, VEC, true>(p, ch, s);
    case 3: return launch_gemm_t<TileL16x6, TRANSB, LOWERC, VEC, true>(p, ch, s);
    default: break;
  }
  return use_mma16() ? launch_gemm_t<TileL, TRANSB, LOWERC, VEC, true>(p, ch, s)
                     : launch_gemm_t<TileL, TRANSB, LOWERC, VEC, false>(p, ch, s);
}

KParams params_of(const GemmArgs& g) {
  KParams p{g.M, g.N, g.K, g.alpha, g.beta, g.A, g.lda, g.B, g.ldb, g.C, g.ldc, (int)g.triB,
            g.tri_off};
  if (g.K == 0) p.alpha = 0.0;  // C = beta C
  return p;
}

template <bool TRANSB, bool LOWERC, int VEC>
moao_status launch_guard(const KParams& p, const TileWalk& w, long tile0, long tiles,
                         const int* flag_a, const int* flag_b, cudaStream_t s) {
  using TL = TileL32x2;
  static std::atomic<unsigned long long> configured{0};
  auto kern = gemm_f64_guard_kernel<TL, TRANSB, LOWERC, VEC>;
  MOAO_CUDA_TRY(set_smem_limit(kern, (int)TL::SMEM_BYTES, configured));
  kern<<<2 * 148, TL::NTHREADS, TL::SMEM_BYTES, s>>>(p, w, (int)tile0, (int)tiles, flag_a, flag_b);
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Leaf kernel of the blocked factorisation (leaf_factor_inverse, one CTA).
__global__ void __launch_bounds__(LEAF_THREADS, 1)
    potrf_inv_leaf_kernel(double* A, long lda, double* Linv, long ldi, int n, long col0,
                          int* info) {
  extern __shared__ __align__(16) double leaf_smem[];
  chain_wait();
  leaf_factor_inverse(A, lda, Linv, ldi, n, col0, info, leaf_smem);
}

// A whole diagonal block in one launch: the recursion of potrf_inv_block as a list of
// phases, a barrier over the (cooperative) grid between them. Its bound is the chain of
// phases: 16 leaves of 11 us for 1,024 columns and, per node of the recursion, three
// products of 1 to 9 us. As ~90 launches, chained, each phase cost 4 to 6 us more than its
// work; a barrier costs about 1.5. Products that no later leaf waits for (W2, the
// factor's block into place) run beside a leaf, and products with a triangle skip its
// zeros. A block of 1,024: 0.67 ms -> 0.52 on 96 CTAs, 0.56 on 64, 0.87 on 16, 1.28 on 8, where
// the FP64 units bound it (64 x 64 tiles once every CTA has one; 32 x 32 throughout: 1.85).
// nmeas 640 reconstructor 504 -> 421 us, the factorisation at nmeas 6,656 6.5 -> 6.1 ms, at
// 18,688 37.2 -> 35.3 ms, mixed 23.5 -> 21.9 ms.
// The operations on each element and their order are those of the launches.
enum DiagType { DIAG_LEAF = 0, DIAG_PANEL = 1, DIAG_TRAIL = 2, DIAG_JOIN = 3 };
struct DiagOp {
  int type, o, n1, n2;  // node: columns o.., n1 | n2; leaf: n1 columns
  unsigned w2;          // the node's W2 in the workspace
};
constexpr int kDiagOps = 128, kDiagMax = 2048;
struct DiagPlan {
  int n = 0;
  unsigned w1 = 0;  // doubles of the workspace for W1, the W2 of nodes above each other behind it
  DiagOp op[kDiagOps];
  void add(int type, int o, int n1, int n2, unsigned w2) { op[n++] = DiagOp{type, o, n1, n2, w2}; }
  void build(int o, int nb, unsigned w2) {
    if (nb <= LEAF) return add(DIAG_LEAF, o, nb, 0, 0);
    const int n1 = LEAF * ((nb + 2 * LEAF - 1) / (2 * LEAF)), n2 = nb - n1;
    w1 = std::max(w1, n1 * even(n2));
    build(o, n1, w2);
    add(DIAG_PANEL, o, n1, n2, w2);
    add(DIAG_TRAIL, o, n1, n2, w2);  // a leaf follows, with this node's products beside it
    build(o + n1, n2, w2 + (unsigned)n1 * even(n2));
    add(DIAG_JOIN, o, n1, n2, w2);
  }
  static unsigned even(int x) { return (unsigned)(x + 1) & ~1u; }
};
// 32 x 32 tiles by 8 warps of 16 x 8 (the leaf's 256 threads)
using TileD = Tile<32, 32, 16, 32, 4, 8>;
using TileD64 = Tile<64, 64, 32, 32, 4, 16>;
static_assert(TileD::NTHREADS == LEAF_THREADS && TileD64::NTHREADS == LEAF_THREADS, "one CTA shape for products and leaves");
constexpr size_t kDiagSmem =
    TileD64::SMEM_BYTES > LEAF_SMEM_BYTES ? TileD64::SMEM_BYTES : LEAF_SMEM_BYTES;
static_assert(TileD::SMEM_BYTES <= kDiagSmem, "one size for all");
constexpr unsigned kDiagPolls = 1u << 22;  // default of the barrier's wait: some seconds

// All CTAs of the grid have arrived, count of them since the launch; false when the
// wait ran out (then *err is raised and the kernel leaves).
__device__ __forceinline__ bool diag_barrier(unsigned* arrived, unsigned count, unsigned limit, int* err) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived, 1u);
    unsigned v, polls = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(arrived) : "memory");
    } while (v < count && ++polls < limit);
    ok = v >= count;
    if (!ok) atomicExch(err, 1);
    __threadfence();
  }
  return __syncthreads_and(ok || threadIdx.x != 0);
}

template <class TL, bool TRANSB, bool LOWERC, int VEC>
__device__ __forceinline__ void diag_tiles(const KParams& p, double* smem, int cta, int ctas) {
  const int tm = (int)((p.M + TL::BM - 1) / TL::BM), tiles = tm * (int)((p.N + TL::BN - 1) / TL::BN);
  if (LOWERC) {  // a square C: tiles m >= n only, by columns
    int n = 0, first = 0;  // column n starts at the first-th tile
    for (int v = cta; v < tm * (tm + 1) / 2; v += ctas) {
      while (v >= first + tm - n) first += tm - n++;
      const int m = n + v - first;
      gemm_tile<TL, TRANSB, LOWERC, VEC, true>(p, smem, (long)m * TL::BM, (long)n * TL::BN);
      __syncthreads();
    }
    return;
  }
  // a CTA's tiles spread over the rows: K grows along them with a triangular A
  for (int v = cta; v < tiles; v += ctas) {
    const int n = v / tm, m = (v + n) % tm;
    gemm_tile<TL, TRANSB, LOWERC, VEC, true>(p, smem, (long)m * TL::BM, (long)n * TL::BN);
    __syncthreads();
  }
}

template <bool TRANSB, bool LOWERC, int VEC>
__device__ __forceinline__ void diag_product(const KParams& p, double* smem, int cta, int ctas) {
  const long t64 = ((p.M + 63) / 64) * ((p.N + 63) / 64);
  if ((LOWERC ? (t64 + 1) / 2 : t64) >= ctas) diag_tiles<TileD64, TRANSB, LOWERC, VEC>(p, smem, cta, ctas);
  else diag_tiles<TileD, TRANSB, LOWERC, VEC>(p, smem, cta, ctas);
}

template <int VEC>
__global__ void __launch_bounds__(LEAF_THREADS, 1)
    diag_block_kernel(const __grid_constant__ DiagPlan plan, double* A, long lda, double* D, long ldd,
                      double* W, long col0, int* info, unsigned* arrived, unsigned limit) {
  extern __shared__ __align__(16) double diag_smem[];
  double* sm = diag_smem;
  const int ctas = gridDim.x;
  for (int k = 0; k < plan.n; ++k) {
    const DiagOp op = plan.op[k];
    if (op.type == DIAG_LEAF) {
      if (blockIdx.x == 0)
        leaf_factor_inverse(A + op.o * (lda + 1), lda, D + op.o * (ldd + 1), ldd, op.n1, col0 + op.o, info,
                            sm);
      __syncthreads();
      const int workers = ctas > 1 ? ctas - 1 : 1, me = ctas > 1 ? (int)blockIdx.x - 1 : 0;
      if (k > 0 && plan.op[k - 1].type == DIAG_TRAIL && me >= 0) {
        const DiagOp q = plan.op[k - 1];
        const long n1 = q.n1, n2 = q.n2, ldw = (n2 + 1) & ~1L;
        double* D11 = D + q.o * (ldd + 1);
        // W2 = L21 D11
        const KParams p{n2, n1, n1, 1.0, 0.0, W, ldw, D11, ldd, W + plan.w1 + q.w2, ldw, TRI_LOWER, 0};
        diag_product<false, false, VEC>(p, sm, me, workers);
        // L21 into place, zeros above the inverse's diagonal
        double *A21 = A + q.o * (lda + 1) + n1, *D12 = D11 + n1 * ldd;
        const int lane = threadIdx.x & 31, warps = workers * (LEAF_THREADS / 32);
        const int w0 = me * (LEAF_THREADS / 32) + (threadIdx.x >> 5);
        for (long c = w0; c < n1; c += warps)
#pragma unroll 4
          for (long r = lane; r < n2; r += 32) A21[c * lda + r] = W[c * ldw + r];
        for (long c = w0; c < n2; c += warps)
          for (long r = lane; r < n1; r += 32) D12[c * ldd + r] = 0.0;
      }
    } else {
      const long n1 = op.n1, n2 = op.n2, ldw = (n2 + 1) & ~1L;
      double *A11 = A + op.o * (lda + 1), *D11 = D + op.o * (ldd + 1);
      if (op.type == DIAG_PANEL) {  // W = L21 = A21 L11^-T
        const KParams p{n2, n1, n1, 1.0, 0.0, A11 + n1, lda, D11, ldd, W, ldw, TRI_LOWER, 0};
        diag_product<true, false, VEC>(p, sm, blockIdx.x, ctas);
      } else if (op.type == DIAG_TRAIL) {  // A22 -= L21 L21^T
        const KParams p{n2, n2, n1, -1.0, 1.0, W, ldw, W, ldw, A11 + n1 * (lda + 1), lda, 0, 0};
        diag_product<true, true, VEC>(p, sm, blockIdx.x, ctas);
      } else {  // D21 = -D22 W2
        KParams p{n2, n1, n2, -1.0, 0.0, D11 + n1 * (ldd + 1), ldd, W + plan.w1 + op.w2, ldw, D11 + n1, ldd,
                  0, 0};
        p.triA = 1;
        diag_product<false, false, VEC>(p, sm, blockIdx.x, ctas);
      }
    }
    if (k + 1 < plan.n && !diag_barrier(arrived, (unsigned)ctas * (k + 1), limit, info + 1)) return;
  }
}

// dst (m x n) = src: 1,024 rows of 4 columns a CTA, 16 loads in flight a thread. A panel
// of 17,664 x 1,024 takes 43 us (the driver's 2D copy 147).
__global__ void __launch_bounds__(256)
    copy_kernel(const double* __restrict__ src, long lds, double* __restrict__ dst, long ldd, long m,
                long n) {
  const long r0 = blockIdx.x * 1024L + threadIdx.x;
  for (long c0 = blockIdx.y * 4L; c0 < n; c0 += gridDim.y * 4L) {
    double v[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        v[c][u] = r0 + u * 256 < m && c0 + c < n ? src[(c0 + c) * lds + r0 + u * 256] : 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r0 + u * 256 < m && c0 + c < n) dst[(c0 + c) * ldd + r0 + u * 256] = v[c][u];
  }
}

// dst (m x n) = src, and the zn x zm block at z (null: none) = 0: the factor's block
// into place and the zeros above the diagonal of its inverse.
__global__ void copy_zero_kernel(const double* __restrict__ src, long lds, double* __restrict__ dst,
                                 long ldd, long m, long n, double* __restrict__ z, long ldz,
                                 long zm, long zn) {
  chain_wait();
  const long step = (long)gridDim.x * blockDim.x, e0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
  for (long e = e0; e < m * n; e += step) dst[(e / m) * ldd + e % m] = src[(e / m) * lds + e % m];
  for (long e = e0; e < zm * zn; e += step) z[(e / zm) * ldz + e % zm] = 0.0;
}

// Cee(i, j) = Cpp(max(i,j), min(i,j)); the diagonal goes through 2d * 0.5
// exactly like the reference's geadd + scal sequence.
__global__ void sym_from_lower_kernel(const double* __restrict__ P, long ldp,
                                      double* __restrict__ E, long lde, long n) {
  const long total = n * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const long i = e % n, j = e / n;
    double v;
    if (i > j) v = P[j * ldp + i];
    else if (i < j) v = P[i * ldp + j];
    else v = (P[j * ldp + i] + P[j * ldp + i]) * 0.5;
    E[j * lde + i] = v;
  }
}

unsigned grid_for(long total) {
  long b = (total + 255) / 256;
  return (unsigned)std::max(1L, std::min(b, 148L * 16));
}

}  // namespace

moao_status gemm_f64(const GemmArgs& g, cudaStream_t s, long long* launches) {
  if (g.M < 0 || g.N < 0 || g.K < 0) return set_error(MOAO_ERR_BAD_ARG, "gemm: negative size");
  if (g.M == 0 || g.N == 0) return MOAO_OK;
  if (g.lowerC && g.triB != TRI_FULL)
    return set_error(MOAO_ERR_UNSUPPORTED, "gemm: lowerC with a triangular B");
  if (g.lda < std::max(1L, g.M) || g.ldc < std::max(1L, g.M) ||
      g.ldb < std::max(1L, g.transB ? g.N : g.K))
    return set_error(MOAO_ERR_BAD_ARG, "gemm: leading dimension too small");
  KParams p = params_of(g);
  const bool v2 = aligned16(g.A) && aligned16(g.B) && (g.lda % 2 == 0) && (g.ldb % 2 == 0);
  moao_status st;
  const int c = g.cfg;
  if (v2) {
    if (g.transB) st = g.lowerC ? launch_gemm<true, true, 2>(p, c, g.chained, s) : launch_gemm<true, false, 2>(p, c, g.chained, s);
    else st = g.lowerC ? launch_gemm<false, true, 2>(p, c, g.chained, s) : launch_gemm<false, false, 2>(p, c, g.chained, s);
  } else {
    if (g.transB) st = g.lowerC ? launch_gemm<true, true, 1>(p, c, g.chained, s) : launch_gemm<true, false, 1>(p, c, g.chained, s);
    else st = g.lowerC ? launch_gemm<false, true, 1>(p, c, g.chained, s) : launch_gemm<false, false, 1>(p, c, g.chained, s);
  }
  if (st == MOAO_OK && launches) ++*launches;
  return st;
}

moao_status gemm_f64_guarded(const GemmArgs& g, long tile0, long tiles, const int* flag_a,
                             const int* flag_b, cudaStream_t s, long long* launches) {
  if (g.M <= 0 || g.N <= 0 || tiles <= 0) return MOAO_OK;
  TileWalk w{};
  fill_walk(&w, g.M, g.N, g.lowerC ? 1 : 0, 0, 128);
  const KParams p = params_of(g);
  const bool v2 = aligned16(g.A) && aligned16(g.B) && (g.lda % 2 == 0) && (g.ldb % 2 == 0);
  moao_status st;
  if (g.lowerC) {
    if (!g.transB) return set_error(MOAO_ERR_UNSUPPORTED, "guarded gemm: lower C without a transposed B");
    st = v2 ? launch_guard<true, true, 2>(p, w, tile0, tiles, flag_a, flag_b, s)
            : launch_guard<true, true, 1>(p, w, tile0, tiles, flag_a, flag_b, s);
  } else if (g.transB) {
    st = v2 ? launch_guard<true, false, 2>(p, w, tile0, tiles, flag_a, flag_b, s)
            : launch_guard<true, false, 1>(p, w, tile0, tiles, flag_a, flag_b, s);
  } else {
    st = v2 ? launch_guard<false, false, 2>(p, w, tile0, tiles, flag_a, flag_b, s)
            : launch_guard<false, false, 1>(p, w, tile0, tiles, flag_a, flag_b, s);
  }
  if (st == MOAO_OK && launches) ++*launches;
  return st;
}

moao_status potrf_inv_leaf(double* A, long lda, double* Linv, long ldi, int n, long col0,
                           int* d_info, bool chained, cudaStream_t s, long long* launches) {
  if (n <= 0) return MOAO_OK;
  if (n > LEAF) return set_error(MOAO_ERR_BAD_ARG, "potrf leaf: n > 64");
  static std::atomic<unsigned long long> configured{0};
  const int smem = LEAF_SMEM_BYTES;
  MOAO_CUDA_TRY(set_smem_limit(potrf_inv_leaf_kernel, smem, configured));
  MOAO_CUDA_TRY(launch_chained(chained, potrf_inv_leaf_kernel, dim3(1), dim3(LEAF_THREADS), (size_t)smem,
                               s, A, lda, Linv, ldi, n, col0, d_info));
  if (launches) ++*launches;
  return MOAO_OK;
}

bool diag_block_fits(long nb) { return nb > LEAF && nb <= kDiagMax; }

moao_status diag_block(double* A, long lda, double* D, long ldd, long nb, long col0, int* d_info,
                       double* W, unsigned* d_sync, int ctas, unsigned polls, cudaStream_t s,
                       long long* launches) {
  if (!diag_block_fits(nb)) return set_error(MOAO_ERR_BAD_ARG, "diag_block: size");
  DiagPlan plan;
  plan.build(0, (int)nb, 0);
  MOAO_CUDA_TRY(cudaMemsetAsync(d_sync, 0, sizeof(unsigned), s));
  const bool v2 = aligned16(A) && aligned16(D) && aligned16(W) && lda % 2 == 0 && ldd % 2 == 0;
  auto kern = v2 ? diag_block_kernel<2> : diag_block_kernel<1>;
  static std::atomic<unsigned long long> configured[2];
  MOAO_CUDA_TRY(set_smem_limit(kern, (int)kDiagSmem, configured[v2]));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(LEAF_THREADS);
  cfg.dynamicSmemBytes = kDiagSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MOAO_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, (const DiagPlan&)plan, A, lda, D, ldd, W, col0, d_info,
                                   d_sync, polls ? polls : kDiagPolls));
  if (launches) ++*launches;
  return MOAO_OK;
}

moao_status copy_matrix(const double* src, long lds, double* dst, long ldd, long m, long n,
                        cudaStream_t s, long long* launches) {
  if (m <= 0 || n <= 0) return MOAO_OK;
  const dim3 grid((unsigned)((m + 1023) / 1024), (unsigned)std::min((n + 3) / 4, 65535L));
  copy_kernel<<<grid, 256, 0, s>>>(src, lds, dst, ldd, m, n);
  if (launches) ++*launches;
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

moao_status copy_zero(const double* src, long lds, double* dst, long ldd, long m, long n, double* z,
                      long ldz, long zm, long zn, bool chained, cudaStream_t s,
                      long long* launches) {
  const long total = std::max(m * n, zm * zn);
  if (total <= 0) return MOAO_OK;
  MOAO_CUDA_TRY(launch_chained(chained, copy_zero_kernel, dim3(grid_for(total)), dim3(256), 0, s, src, lds,
                               dst, ldd, m, n, z, ldz, zm, zn));
  if (launches) ++*launches;
  return MOAO_OK;
}

moao_status sym_from_lower(const double* Cpp, long ldp, double* Cee, long lde, long n,
                           cudaStream_t s, long long* launches) {
  if (n <= 0) return MOAO_OK;
  sym_from_lower_kernel<<<grid_for(n * n), 256, 0, s>>>(Cpp, ldp, Cee, lde, n);
  if (launches) ++*launches;
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

}  // namespace moao
