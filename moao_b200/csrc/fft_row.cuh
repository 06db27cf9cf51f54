// One row transform in shared memory, by the fft_threads(N) threads of a CTA.
#ifndef MOAO_FFT_ROW_CUH
#define MOAO_FFT_ROW_CUH

#include "fft.h"

namespace moao {

// Eight elements per thread (at least a warp).
inline int fft_threads(int N) { return N / 8 > 32 ? N / 8 : 32; }
// Shared memory of a row: one element of padding per eight, so that threads eight
// elements apart (the first group of stages) hit different banks.
inline size_t fft_smem(int N) { return sizeof(Cplx) * (size_t)(N + N / 8 + 1); }
__device__ __forceinline__ int fft_at(int c) { return c + (c >> 3); }
// Where element c of a row of 2^logN goes before fft_row (bit-reversed order).
__device__ __forceinline__ int fft_place(int c, int logN) {
  return fft_at((int)(__brev((unsigned)c) >> (32 - logN)));
}

// G radix-2 stages s .. s + G - 1 on 2^G elements a thread, in registers.
template <int G>
__device__ __forceinline__ void fft_group(Cplx* row, int s, int logN, const Cplx* __restrict__ tw,
                                          int dir) {
  const int half = 1 << s;
  for (int t = threadIdx.x; t < (1 << (logN - G)); t += blockDim.x) {
    const int pos = t & (half - 1), base = ((t >> s) << (s + G)) + pos;
    Cplx e[1 << G];
#pragma unroll
    for (int k = 0; k < (1 << G); ++k) e[k] = row[fft_at(base + k * half)];
#pragma unroll
    for (int q = 0; q < G; ++q) {
#pragma unroll
      for (int k = 0; k < (1 << G); ++k) {
        if (k >> q & 1) continue;
        const int p = pos + (k & ((1 << q) - 1)) * half;
        Cplx w = tw[p << (logN - 1 - s - q)];
        if (dir > 0) w.y = -w.y;
        const Cplx u = e[k], v = e[k | (1 << q)];
        const Cplx vw = {v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x};
        e[k] = {u.x + vw.x, u.y + vw.y};
        e[k | (1 << q)] = {u.x - vw.x, u.y - vw.y};
      }
    }
#pragma unroll
    for (int k = 0; k < (1 << G); ++k) row[fft_at(base + k * half)] = e[k];
  }
  __syncthreads();
}

// In place: row holds its input in bit-reversed order (fft_place) and ends as the
// transform, element c at fft_at(c). log2(N) radix-2 decimation-in-time stages,
// three at a time in a thread's registers (eight elements), so a 512-point row takes
// three barriers instead of nine.
__device__ __forceinline__ void fft_row(Cplx* row, int logN, const Cplx* __restrict__ tw, int dir) {
  __syncthreads();
  int s = 0;
  for (; s + 3 <= logN; s += 3) fft_group<3>(row, s, logN, tw, dir);
  if (logN - s == 2) fft_group<2>(row, s, logN, tw, dir);
  else if (logN - s == 1) fft_group<1>(row, s, logN, tw, dir);
}

}  // namespace moao

#endif  // MOAO_FFT_ROW_CUH
