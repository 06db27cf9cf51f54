// 2-D complex FFT (FP64) as row transforms, a transpose, row transforms and a
// transpose back. A row transform is one CTA (fft_row.cuh): the row is read into
// shared memory in bit-reversed order, then log2(N) radix-2 decimation-in-time stages
// run, three at a time in registers (Cooley-Tukey). Twiddles come from a table
// computed on the host in long double, so every factor is the correctly rounded
// double of exp(-2 pi i k / N). The transposes move 32 x 32 tiles through shared
// memory so that reads and writes are both coalesced.
#include "fft.h"
#include "fft_row.cuh"

#include <cmath>
#include <vector>

namespace moao {
namespace {

__global__ void fft_rows_kernel(Cplx* __restrict__ data, int N, int logN,
                                const Cplx* __restrict__ tw, int dir) {
  extern __shared__ Cplx row[];
  Cplx* g = data + (long)blockIdx.x * N;
  for (int c = threadIdx.x; c < N; c += blockDim.x) row[fft_place(c, logN)] = g[c];
  fft_row(row, logN, tw, dir);
  for (int c = threadIdx.x; c < N; c += blockDim.x) g[c] = row[fft_at(c)];
}

// dst[c * N + r] = src[r * N + c]
__global__ void transpose_kernel(const Cplx* __restrict__ src, Cplx* __restrict__ dst, int N) {
  __shared__ Cplx tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = by + k, c = bx + threadIdx.x;
    if (r < N && c < N) tile[k][threadIdx.x] = src[(long)r * N + c];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int c = bx + k, r = by + threadIdx.x;
    if (r < N && c < N) dst[(long)c * N + r] = tile[threadIdx.x][k];
  }
}

}  // namespace

moao_status fft2d_plan(Fft2d* f, long N) {
  int logN = 0;
  while ((1L << logN) < N) ++logN;
  if (N < 2 || N > 2048 || (1L << logN) != N)
    return set_error(MOAO_ERR_UNSUPPORTED, "fft2d: N must be a power of two in [2, 2048]");
  std::vector<Cplx> tw(N / 2);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (long k = 0; k < N / 2; ++k) {
    const long double a = -2.0L * pi * (long double)k / (long double)N;
    tw[k] = {(double)std::cos(a), (double)std::sin(a)};
  }
  f->N = N;
  f->logN = logN;
  if (cudaMalloc(&f->tw, sizeof(Cplx) * (N / 2)) != cudaSuccess ||
      cudaMalloc(&f->tmp, sizeof(Cplx) * N * N) != cudaSuccess) {
    fft2d_free(f);
    return set_error(MOAO_ERR_OOM, "fft2d: device buffers");
  }
  MOAO_CUDA_TRY(cudaMemcpy(f->tw, tw.data(), sizeof(Cplx) * (N / 2), cudaMemcpyHostToDevice));
  return MOAO_OK;
}

void fft2d_free(Fft2d* f) {
  if (f->tw) cudaFree(f->tw);
  if (f->tmp) cudaFree(f->tmp);
  f->tw = f->tmp = nullptr;
  f->N = 0;
}

moao_status fft2d(const Fft2d& f, Cplx* data, int dir, cudaStream_t s, long long* launches) {
  const int N = (int)f.N;
  if (N < 2 || !f.tw || !f.tmp) return set_error(MOAO_ERR_BAD_ARG, "fft2d: no plan");
  const size_t smem = fft_smem(N);
  const int threads = fft_threads(N);
  const dim3 tgrid((N + 31) / 32, (N + 31) / 32), tblock(32, 8);
  fft_rows_kernel<<<N, threads, smem, s>>>(data, N, f.logN, f.tw, dir);
  transpose_kernel<<<tgrid, tblock, 0, s>>>(data, f.tmp, N);
  fft_rows_kernel<<<N, threads, smem, s>>>(f.tmp, N, f.logN, f.tw, dir);
  transpose_kernel<<<tgrid, tblock, 0, s>>>(f.tmp, data, N);
  if (launches) *launches += 4;
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

}  // namespace moao
