// Intersample PSF: Cvv -> averaged covariance map -> phase structure function
// -> long-exposure PSF (common/tomo_struct/intersample.cpp:74-170).
//
// Device pipeline (N = 512 for every supported system) in seven launches. The
// reference's FFTW real-to-complex / complex-to-real steps are full complex
// transforms whose spectra are Hermitian from the half spectrum the real transforms
// keep, so the results are those of the half-spectrum pipeline. Every 2-D transform
// is row transforms of one index, written transposed, then of the other; the
// pointwise steps between transforms run inside the row kernels, and a column
// j > N/2 of a Hermitian spectrum is not transformed at all: its row transform is
// the conjugate of column N - j's.
//   map       Map cell c = sum of Cvv[i] over idx[i]-1 == c divided by its hit
//             count: partial maps in shared memory over the columns of Cvv where
//             the index table allows it, else a warp per cell
//   place     the map's rows on the N x N lattice with pitch dactupix, forward
//             transforms along j of those rows (the others are 0)
//   filter    per column j <= N/2: forward along i; re *= abs2fi[j*N+i] (transposed
//             index, as in the reference), im = 0; inverse along i
//   structure per row i: inverse along j; its real part is the phase covariance
//   otf       per column j <= N/2: exp(-0.5 (norm - dphi fact / fact2)) with the
//             reference's truncated pi in fact, read through the quadrant swap
//             (_eclat_double), times otf_tel[j*N+i]; inverse along i
//   psf       per row i: inverse along j, real part through the final quadrant swap
// The 64 x 64 system's PSF (3,000 actuators) takes 122 us: 517 with 17 launches and
// one thread per map cell, 171 with six launches and a warp per cell, whose gathers
// fetch a 32-byte sector for every 8-byte entry. The partial maps read Cvv and the
// index table once, in order (113 MB, 32 us); the rest is seven dependent launches
// of 10-18 us each on a cold cache.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "chain.cuh"
#include "context.h"
#include "fft.h"
#include "fft_row.cuh"

struct moao_isample {
  moao_ctx* ctx = nullptr;
  moao_isample_info info{};
  long nmap = 0, ncov = 0;
  // device
  double* abs2fi = nullptr;   // N*N
  double* otf = nullptr;      // N*N
  long nact = 0;              // > 0: partial maps by columns of Cvv (nidx = nact^2)
  int parts = 0;              // partial maps
  int* cell_of = nullptr;     // nidx: cell of every Cvv entry (partial maps)
  double* part = nullptr;     // parts x nmap
  int* cell_start = nullptr;  // nmap+1 (CSR over Cvv indices; a warp per cell)
  int* cell_idx = nullptr;    // nidx
  double* div = nullptr;      // nmap
  double* dphi = nullptr;     // N*N real: the phase covariance
  double* map = nullptr;      // nmap
  moao::Cplx* spec = nullptr;   // N*N: spectra
  moao::Cplx* rows = nullptr;   // N x ncov: transforms of the map's rows, by column
  double* in_host_cvv = nullptr;
  moao::Fft2d fft;
  double fact = 0, fact2 = 0;
  long idx_norm = 0;
};

namespace moao {
namespace {

constexpr int kGatherWarps = 8;

// A warp per map cell: lanes take its Cvv entries in turn. Consecutive cells (of one
// block) read neighbouring Cvv entries, so their sectors are shared in L1.
__global__ void __launch_bounds__(kGatherWarps * 32)
    gather_kernel(const double* __restrict__ cvv, const int* __restrict__ start,
                  const int* __restrict__ cidx, const double* __restrict__ div,
                  double* __restrict__ map, long nmap) {
  chain_wait();
  const long c = blockIdx.x * (long)kGatherWarps + (threadIdx.x >> 5);
  if (c >= nmap) return;
  const int lane = threadIdx.x & 31, k1 = start[c + 1];
  double s[4] = {};
  int k = start[c] + lane;
  for (; k + 96 < k1; k += 128) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] += cvv[cidx[k + 32 * q]];
  }
  for (; k < k1; k += 32) s[0] += cvv[cidx[k]];
  double v = (s[0] + s[1]) + (s[2] + s[3]);
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) map[c] = div[c] > 0 ? v / div[c] : v;
}

// Partial maps: CTA b adds its columns of Cvv (nact entries each, all in different
// cells: checked when the object is made) into a map in shared memory, one barrier
// per column, and writes it out. In units of 4 entries per thread, the next unit's
// loads in flight while the current one is added; the order is fixed, so are the
// sums.
constexpr int kMapThreads = 1024, kMapPer = 4;
__global__ void __launch_bounds__(kMapThreads)
    map_kernel(const double* __restrict__ cvv, const int* __restrict__ cell, int nact, int cols,
               int nmap, double* __restrict__ part) {
  extern __shared__ double m[];
  chain_wait();
  const int tid = threadIdx.x;
  for (int c = tid; c < nmap; c += kMapThreads) m[c] = 0.0;
  const int per_col = (nact + kMapThreads * kMapPer - 1) / (kMapThreads * kMapPer);
  const int j0 = blockIdx.x * cols, units = (min(nact, j0 + cols) - j0) * per_col;
  double v[kMapPer];
  int id[kMapPer];
  auto load = [&](int u) {
    const long base = (long)(j0 + u / per_col) * nact;
    const int i0 = (u % per_col) * kMapThreads * kMapPer + tid;
#pragma unroll
    for (int q = 0; q < kMapPer; ++q) {
      const int i = i0 + q * kMapThreads;
      id[q] = i < nact ? __ldcs(cell + base + i) : -1;
      v[q] = i < nact ? __ldcs(cvv + base + i) : 0.0;
    }
  };
  if (units > 0) load(0);
  for (int u = 0; u < units; ++u) {
    double w[kMapPer];
    int c[kMapPer];
#pragma unroll
    for (int q = 0; q < kMapPer; ++q) {
      w[q] = v[q];
      c[q] = id[q];
    }
    if (u + 1 < units) load(u + 1);
    __syncthreads();  // the previous unit's additions (or the zeros) are in place
#pragma unroll
    for (int q = 0; q < kMapPer; ++q)
      if (c[q] >= 0) m[c[q]] += w[q];
  }
  __syncthreads();
  for (int c = tid; c < nmap; c += kMapThreads) part[(long)blockIdx.x * nmap + c] = m[c];
}

// map = the sum of the partial maps over the hit counts: 32 cells a block, eight
// threads each.
__global__ void __launch_bounds__(256)
    map_sum_kernel(const double* __restrict__ part, int parts, const double* __restrict__ div,
                   double* __restrict__ map, int nmap) {
  __shared__ double sums[8][32];
  chain_wait();
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, c = blockIdx.x * 32 + x;
  double s[4] = {};
  if (c < nmap) {
    int b = y;
    for (; b + 24 < parts; b += 32) {
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += part[(long)(b + 8 * q) * nmap + c];
    }
    for (; b < parts; b += 8) s[0] += part[(long)b * nmap + c];
  }
  sums[y][x] = (s[0] + s[1]) + (s[2] + s[3]);
  __syncthreads();
  if (y > 0 || c >= nmap) return;
  double v = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) v += sums[q][x];
  map[c] = div[c] > 0 ? v / div[c] : v;
}

// Row ii of the map on the lattice (row a + ii pitch, columns a + jj pitch), forward
// along j: rows[j * ncov + ii].
__global__ void place_kernel(const double* __restrict__ map, Cplx* __restrict__ rows, int N, int logN,
                             const Cplx* __restrict__ tw, int ncov, int a, int pitch) {
  extern __shared__ Cplx row[];
  chain_wait();
  const int ii = blockIdx.x;
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    const int d = c - a, jj = d / pitch;
    const double v = (d >= 0 && d % pitch == 0 && jj < ncov) ? map[(long)ii * ncov + jj] : 0.0;
    row[fft_place(c, logN)] = {v, 0.0};
  }
  fft_row(row, logN, tw, -1);
  for (int c = threadIdx.x; c < N; c += blockDim.x) rows[(long)c * ncov + ii] = row[fft_at(c)];
}

// Column j of a Hermitian spectrum, transformed along i, into both its columns of
// the transposed array: out[i * N + j] and, for the mirrored column, its conjugate.
__device__ __forceinline__ void put_columns(const Cplx* row, Cplx* __restrict__ out, int N, int j) {
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    const Cplx v = row[fft_at(c)];
    out[(long)c * N + j] = v;
    if (j > 0 && j < N / 2) out[(long)c * N + N - j] = {v.x, -v.y};
  }
}

__global__ void filter_kernel(const Cplx* __restrict__ rows, const double* __restrict__ abs2fi,
                              Cplx* __restrict__ spec, int N, int logN, const Cplx* __restrict__ tw,
                              int ncov, int a, int pitch) {
  extern __shared__ Cplx row[];
  chain_wait();
  const int j = blockIdx.x;  // 0 .. N/2
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    const int d = c - a, ii = d / pitch;
    const bool on = d >= 0 && d % pitch == 0 && ii < ncov;
    row[fft_place(c, logN)] = on ? rows[(long)j * ncov + ii] : Cplx{0.0, 0.0};
  }
  fft_row(row, logN, tw, -1);
  double v[8];  // at most eight elements a thread
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = threadIdx.x + q * blockDim.x;
    v[q] = c < N ? row[fft_at(c)].x * abs2fi[(long)j * N + c] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = threadIdx.x + q * blockDim.x;
    if (c < N) row[fft_place(c, logN)] = {v[q], 0.0};
  }
  fft_row(row, logN, tw, +1);
  put_columns(row, spec, N, j);
}

// dphi[i * N + j] = re of the inverse along j of spec's row i
__global__ void structure_kernel(const Cplx* __restrict__ spec, double* __restrict__ dphi, int N,
                                 int logN, const Cplx* __restrict__ tw) {
  extern __shared__ Cplx row[];
  chain_wait();
  const long i = blockIdx.x;
  for (int c = threadIdx.x; c < N; c += blockDim.x) row[fft_place(c, logN)] = spec[i * N + c];
  fft_row(row, logN, tw, +1);
  for (int c = threadIdx.x; c < N; c += blockDim.x) dphi[i * N + c] = row[fft_at(c)].x;
}

__global__ void otf_kernel(const double* __restrict__ dphi, const double* __restrict__ otf,
                           Cplx* __restrict__ spec, int N, int logN, const Cplx* __restrict__ tw,
                           long idx_norm, double fact, double fact2) {
  extern __shared__ Cplx row[];
  chain_wait();
  const int j = blockIdx.x, h = N / 2;  // 0 .. N/2
  const double norm = dphi[idx_norm] / fact2 * fact;
  const double* src = dphi + (long)((j + h) % N) * N;
  for (int c = threadIdx.x; c < N; c += blockDim.x) {
    const double d = exp(-0.5 * (norm - src[(c + h) % N] / fact2 * fact));
    row[fft_place(c, logN)] = {otf[(long)j * N + c] * d, 0.0};
  }
  fft_row(row, logN, tw, +1);
  put_columns(row, spec, N, j);
}

__global__ void psf_kernel(const Cplx* __restrict__ spec, double* __restrict__ psf, int N, int logN,
                           const Cplx* __restrict__ tw) {
  extern __shared__ Cplx row[];
  chain_wait();
  const long i = blockIdx.x;
  const int h = N / 2;
  for (int c = threadIdx.x; c < N; c += blockDim.x) row[fft_place(c, logN)] = spec[i * N + c];
  fft_row(row, logN, tw, +1);
  double* dst = psf + ((i + h) % N) * N;
  for (int c = threadIdx.x; c < N; c += blockDim.x) dst[(c + h) % N] = row[fft_at(c)].x;
}

void free_isample(moao_isample* is) {
  if (!is) return;
  fft2d_free(&is->fft);
  void* ptrs[] = {is->abs2fi, is->otf, is->cell_start, is->cell_idx, is->div,
                  is->dphi, is->map, is->spec, is->rows, is->cell_of, is->part};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete is;
}

}  // namespace
}  // namespace moao

using namespace moao;

extern "C" {

moao_status moao_intersample_create(moao_ctx* ctx, long nidx, long np, double Dtel,
                                    const long* idx, const double* abs2fi, const double* otf_tel,
                                    moao_isample** out) {
  (void)Dtel;
  if (!ctx || !idx || !abs2fi || !otf_tel || !out || nidx <= 0 || np < 2)
    return set_error(MOAO_ERR_BAD_ARG, "intersample_create: bad arguments");
  if (nidx > 0x7fffffffL) return set_error(MOAO_ERR_UNSUPPORTED, "intersample: nidx too large");
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  moao_isample* is = new moao_isample;
  is->ctx = ctx;
  // intersample_prepare (intersample.cpp:176-207)
  const long N = std::max(512L, (long)(8 * std::pow(2, (long)(std::log((double)np) + 0.5))));
  is->info.N = N;
  is->info.np = np;
  is->info.nidx = nidx;
  is->info.lambda = 1.65e-06;
  is->info.dactupix = (double)(N / (3 * (np - 1)) + 1);
  is->ncov = 2 * np - 1;
  is->nmap = is->ncov * is->ncov;
  // Hit counts; indices are validated here instead of being written out of bounds.
  // Where Cvv is square with every column's entries in different cells and the map
  // fits in shared memory, each entry's cell; else the CSR gather lists.
  std::vector<int> count(is->nmap + 1, 0), cidx(nidx);
  const long na = std::lround(std::sqrt((double)nidx));
  bool columns = na * na == nidx && is->nmap * (long)sizeof(double) <= 200 * 1024;
  std::vector<long> seen(columns ? is->nmap : 0, -1);
  for (long i = 0, j = 0, r = 0; i < nidx; ++i) {
    const long c = idx[i] - 1;
    if (c < 0 || c >= is->nmap) {
      delete is;
      return set_error(MOAO_ERR_BAD_ARG, "intersample_create: idx[" + std::to_string(i) +
                                             "] outside the covariance map");
    }
    ++count[c + 1];
    cidx[i] = (int)c;
    if (columns) {
      if (seen[c] == j) columns = false;
      else seen[c] = j;
      if (++r == na) r = 0, ++j;
    }
  }
  std::vector<double> div(is->nmap);
  for (long c = 0; c < is->nmap; ++c) div[c] = (double)count[c + 1];
  if (columns) {
    is->nact = na;
    is->parts = (int)std::min(148L, (na + 3) / 4);
  } else {
    for (long c = 0; c < is->nmap; ++c) count[c + 1] += count[c];
    std::vector<int> fill(count.begin(), count.end() - 1);
    for (long i = 0; i < nidx; ++i) cidx[fill[idx[i] - 1]++] = (int)i;
  }

  const double dp = is->info.dactupix;
  is->fact = 2 * std::pow(2 * 3.14159 / is->info.lambda, 2);
  is->fact2 = N * N * dp * dp;
  const long ncmap = N / 2 + 1;
  is->idx_norm = N * (ncmap - 1) + ncmap - 1;

  const size_t NN = (size_t)N * N;
  moao_status st = MOAO_OK;
  auto alloc = [&](void** p, size_t bytes) {
    if (st == MOAO_OK && !device_alloc(ctx, p, bytes))
      st = set_error(MOAO_ERR_OOM, "intersample_create: device allocation");
  };
  alloc((void**)&is->abs2fi, NN * 8);
  alloc((void**)&is->otf, NN * 8);
  if (is->nact > 0) {
    alloc((void**)&is->cell_of, nidx * sizeof(int));
    alloc((void**)&is->part, (size_t)is->parts * is->nmap * 8);
  } else {
    alloc((void**)&is->cell_start, (is->nmap + 1) * sizeof(int));
    alloc((void**)&is->cell_idx, nidx * sizeof(int));
  }
  alloc((void**)&is->div, is->nmap * 8);
  alloc((void**)&is->dphi, NN * 8);
  alloc((void**)&is->spec, NN * sizeof(Cplx));
  alloc((void**)&is->map, is->nmap * 8);
  alloc((void**)&is->rows, (size_t)N * is->ncov * sizeof(Cplx));
  if (st == MOAO_OK) {
    cudaMemcpy(is->abs2fi, abs2fi, NN * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(is->otf, otf_tel, NN * 8, cudaMemcpyHostToDevice);
    if (is->nact == 0)
      cudaMemcpy(is->cell_start, count.data(), (is->nmap + 1) * sizeof(int), cudaMemcpyHostToDevice);
    cudaMemcpy(is->nact > 0 ? is->cell_of : is->cell_idx, cidx.data(), nidx * sizeof(int),
               cudaMemcpyHostToDevice);
    if (cudaMemcpy(is->div, div.data(), is->nmap * 8, cudaMemcpyHostToDevice) != cudaSuccess)
      st = set_error(MOAO_ERR_CUDA, "intersample_create: upload");
  }
  if (st == MOAO_OK) st = fft2d_plan(&is->fft, N);
  if (st != MOAO_OK) {
    free_isample(is);
    return st;
  }
  *out = is;
  return MOAO_OK;
}

moao_status moao_intersample_get_info(const moao_isample* is, moao_isample_info* out) {
  if (!is || !out) return set_error(MOAO_ERR_BAD_ARG, "intersample_get_info: null");
  *out = is->info;
  return MOAO_OK;
}

moao_status moao_intersample_process(moao_isample* is, const double* d_Cvv, double* d_psf) {
  if (!is || !d_Cvv || !d_psf) return set_error(MOAO_ERR_BAD_ARG, "intersample_process: null");
  moao_ctx* ctx = is->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  const long N = is->info.N;
  const long ncmap = N / 2 + 1, nelem = (is->ncov - 1) / 2;
  const long pitch = (long)is->info.dactupix;
  const long a = ncmap - nelem * pitch - 1;
  if (a < 0) return set_error(MOAO_ERR_BAD_ARG, "intersample: map does not fit the FFT support");
  const int n = (int)N, half = n / 2, nc = (int)is->ncov, lg = is->fft.logN;
  const size_t smem = fft_smem(n);
  const Cplx* tw = is->fft.tw;
  const bool ch = ctx->chained;
  const dim3 blk((unsigned)fft_threads(n)), cols((unsigned)half + 1), full((unsigned)n);
  // lattice rows inside the support (the last one may fall on its edge)
  const int on = (int)std::min<long>(is->ncov, (N - 1 - a) / pitch + 1);
  if (is->nact > 0) {
    static std::atomic<unsigned long long> configured{0};
    MOAO_CUDA_TRY(set_smem_limit(map_kernel, 200 * 1024, configured));
    const int cols = (int)((is->nact + is->parts - 1) / is->parts);
    MOAO_CUDA_TRY(launch_chained(ch, map_kernel, dim3((unsigned)is->parts), dim3(kMapThreads),
                                 sizeof(double) * is->nmap, s, d_Cvv, is->cell_of, (int)is->nact, cols,
                                 (int)is->nmap, is->part));
    MOAO_CUDA_TRY(launch_chained(ch, map_sum_kernel, dim3((unsigned)((is->nmap + 31) / 32)), dim3(256), 0, s,
                                 is->part, is->parts, is->div, is->map, (int)is->nmap));
    ++ctx->launches;
  } else {
    MOAO_CUDA_TRY(launch_chained(ch, gather_kernel,
                                 dim3((unsigned)((is->nmap + kGatherWarps - 1) / kGatherWarps)),
                                 dim3(kGatherWarps * 32), 0, s, d_Cvv, is->cell_start, is->cell_idx,
                                 is->div, is->map, is->nmap));
  }
  MOAO_CUDA_TRY(launch_chained(ch, place_kernel, dim3((unsigned)on), blk, smem, s,
                               is->map, is->rows, n, lg, tw, nc, (int)a, (int)pitch));
  MOAO_CUDA_TRY(launch_chained(ch, filter_kernel, cols, blk, smem, s, is->rows, is->abs2fi, is->spec, n,
                               lg, tw, nc, (int)a, (int)pitch));
  MOAO_CUDA_TRY(launch_chained(ch, structure_kernel, full, blk, smem, s, is->spec, is->dphi, n, lg, tw));
  MOAO_CUDA_TRY(launch_chained(ch, otf_kernel, cols, blk, smem, s, is->dphi, is->otf, is->spec, n, lg, tw,
                               is->idx_norm, is->fact, is->fact2));
  MOAO_CUDA_TRY(launch_chained(ch, psf_kernel, full, blk, smem, s, is->spec, d_psf, n, lg, tw));
  ctx->launches += 6;
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

moao_status moao_intersample_process_host(moao_isample* is, const double* Cvv, double* psf) {
  if (!is || !Cvv || !psf) return set_error(MOAO_ERR_BAD_ARG, "intersample_process_host: null");
  moao_ctx* ctx = is->ctx;
  MOAO_CUDA_TRY(cudaSetDevice(ctx->device));
  const long N = is->info.N;
  double *dc = nullptr, *dp = nullptr;
  if (!device_alloc(ctx, (void**)&dc, is->info.nidx * 8))
    return set_error(MOAO_ERR_OOM, "intersample_process_host: Cvv");
  if (!device_alloc(ctx, (void**)&dp, N * N * 8)) {
    cudaFree(dc);
    return set_error(MOAO_ERR_OOM, "intersample_process_host: psf");
  }
  moao_status st = MOAO_OK;
  if (cudaMemcpyAsync(dc, Cvv, is->info.nidx * 8, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess)
    st = set_error(MOAO_ERR_CUDA, "intersample_process_host: H2D");
  if (st == MOAO_OK) st = moao_intersample_process(is, dc, dp);
  if (st == MOAO_OK &&
      cudaMemcpyAsync(psf, dp, N * N * 8, cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess)
    st = set_error(MOAO_ERR_CUDA, "intersample_process_host: D2H");
  cudaStreamSynchronize(ctx->stream);
  cudaFree(dc);
  cudaFree(dp);
  return st;
}

void moao_intersample_destroy(moao_isample* is) {
  if (!is) return;
  cudaSetDevice(is->ctx->device);
  cudaStreamSynchronize(is->ctx->stream);
  free_isample(is);
}

}  // extern "C"
