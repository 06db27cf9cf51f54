// Covariance generation on sm_100a: Cmm, Ctm, Ctt tiles from the von Karman
// phase structure function.
//
// Model (restated from the reference, common/kernels/matcov_kernels.cpp):
//   DPHI(r) = k1 L0^(5/3) f(2 pi r / L0)                          rodconan :92
//   f(x) = -x^(5/6) K_5/6(x) series (x <= Xlim)                   macdo_x56 :38
//   f(x) = k2 - k3 e^-x x^(1/3) (1 + a1/x + a2/x^2 + a3/x^3)      asymp_macdo :65
//   slope covariances are 4-point DPHI stencils                    cov_XX_gb.. :147-193
//   element = sum over layers of 0.5 cov kk cn2 (+ WFS noise)      compute_element_tiled_4 :206
//   Ctt uses the unprojected truth-sensor positions                compute_element_ts_tile :423
//
// Work decomposition (B200): one thread owns one subaperture pair (i, j) and
// produces the 2x2 slope block {x_i, y_i} x {x_j, y_j} of that pair, so the
// geometry decode, the per-layer loads and the separation are shared by the
// four covariances. When the two WFS have the same subaperture size on a layer
// (every NGS/NGS and equal-altitude LGS/LGS pair) the 16 stencil points of the
// block collapse to 9 distinct DPHI evaluations. Per-layer constants
// (2 pi / L0, k1 L0^(5/3), 0.5 kk cn2) are hoisted to shared memory. Pairs of equal
// projection gather from tables over grid offsets, edge-aligned ones share their
// points in matcov_edge_kernel, and f itself comes from a table of polynomials
// (dphi_v): its 40 to 55 FP64 operations bounded the direct form, reads of the
// table bound this one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "chain.cuh"
#include "moao_internal.h"

namespace moao {
namespace {

// Constants of the reference model (common/moao_defs.h:15-38).
struct Series {
  double c[11];
};
constexpr Series kGa = {{0, 12.067619015983075, 5.17183672113560444, 0.795667187867016068,
                         0.0628158306210802181, 0.00301515986981185091, 9.72632216068338833e-05,
                         2.25320204494595251e-06, 3.93000356676612095e-08, 5.34694362825451923e-10,
                         5.83302941264329804e-12}};
constexpr Series kGma = {{-3.74878707653729304, -2.04479295083852408, -0.360845814853857083,
                          -0.0313778969438136685, -0.001622994669507603, -5.56455315259749673e-05,
                          -1.35720808599938951e-06, -2.47515152461894642e-08, -3.50257291219662472e-10,
                          -3.95770950530691961e-12, -3.65327031259100284e-14}};
__constant__ Series c_Ga = kGa, c_Gma = kGma;
constexpr double kPi = 3.1415926535897932384626433;
constexpr double kK1 = 0.1716613621245709486;
constexpr double kK2 = 1.00563491799858928388289314170833;
constexpr double kK3 = 1.25331413731550012081;
constexpr double kA1 = 0.22222222222222222222;
constexpr double kA2 = -0.08641975308641974829;
constexpr double kA3 = 0.08001828989483310284;
constexpr double kXlim = 0.75 * 2 * kPi;
constexpr double kLambda2 = 0.00026942094446267851;  // (lambda/(2 pi) rasc)^2

// f(x) / (k1 L0^(5/3)) for x = 2 pi r / L0 >= 0 (so that DPHI = amp * f).
__device__ __forceinline__ double dphi_unit(double x) {
  if (x > kXlim) {
    const double xi = 1.0 / x;
    return kK2 - kK3 * exp(-x) * cbrt(x) * (1.0 + xi * (kA1 + xi * (kA2 + xi * kA3)));
  }
  const double c = cbrt(x);
  const double x2a = x * c * c;  // x^(5/3)
  const double z = 0.25 * x * x;  // (x/2)^2
  double pg = c_Gma.c[10];
#pragma unroll
  for (int n = 9; n >= 0; --n) pg = fma(pg, z, c_Gma.c[n]);
  double pa = c_Ga.c[10];
#pragma unroll
  for (int n = 9; n >= 1; --n) pa = fma(pa, z, c_Ga.c[n]);
  return -0.5 * (x2a * pg + z * pa);
}

// From here on f is taken of v = x^2 / Xlim^2, without square roots and cube roots. The
// two forms differ by 5e-7 of f where they meet, at separations of 0.75 L0, which a grid
// can hold exactly. So s = x^2 is summed as for the direct form, and scaled by the
// neighbour of 1 / Xlim^2 that puts s = Xlim^2 below 1 and the next double not.
constexpr double kXlim2 = kXlim * kXlim, kPerXlim2 = 0x1.70e6301e60654p-5;
static_assert(kXlim2 * kPerXlim2 < 1.0 && kXlim2 * (1.0 + 0x1p-52) * kPerXlim2 >= 1.0,
              "v >= 1 where s > Xlim^2");
// Rounded by itself (as are the sums that give s): no kernel's compilation may fuse it with
// what follows, so that they agree to the bit.
__device__ __forceinline__ double dphi_scaled(double s) { return __dmul_rn(s, kPerXlim2); }

// Values outside the other forms: 0, below kDphiTiny (whose float seeds would lose range),
// not finite.
__device__ __noinline__ double dphi_rare(double v) {
  const double s = v * kXlim2;
  return s > 0 ? dphi_unit(sqrt(s)) : 0.0;
}

// The series of small x, with the constants of z = (x/2)^2 = Xlim^2 v / 4 and x^(5/3)
// folded into the coefficients: f = v (y G(v) + A(v)), y = v^(-1/6), N terms of each. y
// comes from a seed 2^(-log2(v)/6) by the PTX approximations (flush-to-zero forms: v is a
// normal float here, and so is the seed; good to 2e-6) and one step of fourth order,
// r = 1 - v y^6, (1 - r)^(-1/6) = 1 + r/6 + 7 r^2/72 + 91 r^3/1296 + O(r^4). 9 + 2 N
// FP64 operations; within 3.7e-16 of f for v < 2^-12 with N = 5 and 6.4e-16 for v < 2^-6
// with N = 9 (sampled against 50 digits; all 11 terms with Newton's iteration, which it
// takes the place of, 6.7e-16 and 1.1e-15).
constexpr double kDphiTiny = 1e-31;
constexpr double kZ = 0.25 * kXlim2, kXlim53 = 13.245505975797633;  // kXlim^(5/3)
constexpr int kSeriesTerms = 9;
struct FoldedSeries {
  double G[kSeriesTerms], A[kSeriesTerms];
};
constexpr FoldedSeries folded_series() {
  FoldedSeries f{};
  double z = 1.0;
  for (int n = 0; n < kSeriesTerms; ++n, z *= kZ) {
    f.G[n] = -0.5 * kXlim53 * z * kGma.c[n];
    f.A[n] = -0.5 * z * kZ * kGa.c[n + 1];
  }
  return f;
}
template <int N>
__device__ __forceinline__ double dphi_series(double v) {
  constexpr FoldedSeries f = folded_series();
  float l2, seed;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l2) : "f"((float)v));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(seed) : "f"(l2 * (-1.0f / 6.0f)));
  const double y0 = (double)seed, y2 = y0 * y0;
  const double r = fma(-v, y2 * y2 * y2, 1.0);
  const double p = y0 * (r * fma(fma(91.0 / 1296, r, 7.0 / 72), r, 1.0 / 6));  // y = y0 + p
  double g = f.G[N - 1];
#pragma unroll
  for (int n = N - 2; n >= 0; --n) g = fma(g, v, f.G[n]);
  double a = f.A[N - 1];
#pragma unroll
  for (int n = N - 2; n >= 0; --n) a = fma(a, v, f.A[n]);
  return v * fma(y0, g, fma(p, g, a));
}
// Below the table, kDphiTiny < v < 2^kDphiLo.
__device__ __forceinline__ double dphi_low(double v) { return dphi_series<5>(v); }

// f from the table: kDphiSub intervals per octave
// from v's leading bits (the two forms of f meet at v = 1, an interval's edge), then
// a polynomial of degree 8 in the distance y from the interval's middle, against ~40
// FP64 operations of the series and ~55 of the asymptotic form with exp. The
// polynomials interpolate f, evaluated in 80-bit arithmetic, at Chebyshev nodes: an
// interval's half width is at most v / 32 and f's nearest singularity is v = 0, so the
// truncation is at most 3.1e-18 of f. The terms y^5 and up are at most 1.7e-9 of f (in
// an octave's first interval, relatively the widest), so their FP32 coefficients and
// evaluation cost at most 1.2e-16 of it; a whole evaluation is within 2.4e-16 of f
// (sampled against 50 digits). Below the table (separations under 0.0117 L0) the
// series; above it f is constant in 64 bits.
//
// What bounds it is shared-memory reads: 56 bytes a value. The table is held in
// copies, one per lane of a load's phase (8 lanes of 16 bytes, 16 of 8), each in banks
// of its own, so that lanes on different rows never conflict: 14 wavefronts a warp.
// One copy (degree 5, 64 intervals per octave, 48 bytes a value) took 21 in conflicts
// and 7.2 against 5.5 ms for the Ctm of nmeas 15,936; in L1 7.4 ms.
constexpr int kTab01 = 0, kTab23 = kTab01 + kDphiRows * 8 * 16, kTabF = kTab23 + kDphiRows * 8 * 16,
              kTab4 = kTabF + kDphiRows * 8 * 16, kTabBytes = kTab4 + kDphiRows * 16 * 8;

__device__ __forceinline__ void dphi_put(char* tab, const DphiRow& r, int q) {  // copy q % 16 of row q / 16
  const int k = q >> 4, p = q & 15;
  reinterpret_cast<double*>(tab + kTab4)[q] = r.c[4];
  if (p < 8) {
    reinterpret_cast<double2*>(tab + kTab01)[k * 8 + p] = make_double2(r.c[0], r.c[1]);
    reinterpret_cast<double2*>(tab + kTab23)[k * 8 + p] = make_double2(r.c[2], r.c[3]);
  } else {
    reinterpret_cast<float4*>(tab + kTabF)[k * 8 + p - 8] = make_float4(r.f[0], r.f[1], r.f[2], r.f[3]);
  }
}

template <int THREADS>
__device__ __forceinline__ void dphi_fill(char* tab, const DphiRow* __restrict__ rows) {
  constexpr int PER = kDphiRows * 16 / THREADS, REST = kDphiRows * 16 % THREADS;
  DphiRow r[PER];  // every row's loads in flight together
#pragma unroll
  for (int u = 0; u < PER; ++u) r[u] = rows[(threadIdx.x + u * THREADS) >> 4];
#pragma unroll
  for (int u = 0; u < PER; ++u) dphi_put(tab, r[u], threadIdx.x + u * THREADS);
  if (threadIdx.x < REST) {
    const int q = threadIdx.x + PER * THREADS;
    dphi_put(tab, rows[q >> 4], q);
  }
}

// Interval of v, counted from the table's first; intervals from the last row's on share
// it. Outside (unsigned) [0, kDphiInf): below the table, not finite, or negative.
constexpr int kDphiInf = 0x7ff0 - ((1023 + kDphiLo) << 4);
__device__ __forceinline__ int dphi_interval(double v) {
  return (__double2hiint(v) >> 16) - ((1023 + kDphiLo) << 4);
}
__device__ __forceinline__ double dphi_middle(double v) {
  return __hiloint2double((__double2hiint(v) & 0xffff0000) | 0x8000, 0);
}

// v in an interval from 0 on, from one copy of the rows.
__device__ __forceinline__ double dphi_one(const DphiRow* rows, double v) {
  const DphiRow& r = rows[min(dphi_interval(v), kDphiRows - 1)];
  const double y = v - dphi_middle(v);
  const float yf = (float)y;
  const float ph = fmaf(fmaf(fmaf(r.f[3], yf, r.f[2]), yf, r.f[1]), yf, r.f[0]);
  double p = fma((double)ph, y, r.c[4]);
  p = fma(p, y, r.c[3]);
  p = fma(p, y, r.c[2]);
  p = fma(p, y, r.c[1]);
  return fma(p, y, r.c[0]);
}

// The same from the copies.
__device__ __forceinline__ double dphi_v(const char* tab, double v) {
  const int lane = threadIdx.x & 31, k = min(dphi_interval(v), kDphiRows - 1);
  const double y = v - dphi_middle(v);
  const char* t = tab + (k * 8 + (lane & 7)) * 16;
  const float4 f = *reinterpret_cast<const float4*>(t + kTabF);
  const double2 c0 = *reinterpret_cast<const double2*>(t + kTab01);
  const double2 c2 = *reinterpret_cast<const double2*>(t + kTab23);
  const double c4 = *reinterpret_cast<const double*>(tab + kTab4 + (k * 16 + (lane & 15)) * 8);
  const float yf = (float)y;
  const float ph = fmaf(fmaf(fmaf(f.w, yf, f.z), yf, f.y), yf, f.x);
  double p = fma((double)ph, y, c4);
  p = fma(p, y, c2.y);
  p = fma(p, y, c2.x);
  p = fma(p, y, c0.y);
  return fma(p, y, c0.x);
}

// A value outside the table, in interval k.
__device__ __forceinline__ double dphi_outside(double v, int k) {
  return k < 0 && v > kDphiTiny ? dphi_low(v) : dphi_rare(v);
}
__device__ __noinline__ double dphi_outside_call(double v) { return dphi_outside(v, dphi_interval(v)); }

// Any v, with a branch for the lanes outside the table.
__device__ __forceinline__ double dphi_any(const char* tab, double v) {
  if ((unsigned)dphi_interval(v) >= (unsigned)kDphiInf) return dphi_outside_call(v);
  return dphi_v(tab, v);
}

// The same from the rows in global memory (the per-pair and table kernels; not
// inlined, so that their 9 or 16 points per layer share one body).
__device__ __noinline__ double dphi_row(const DphiRow* __restrict__ rows, double s) {
  const double v = dphi_scaled(s);
  const int k = dphi_interval(v);
  if ((unsigned)k >= (unsigned)kDphiInf) return dphi_outside(v, k);
  return dphi_one(rows, v);
}

constexpr double kDphiReach = 0.75 / 64;  // separation at the table's lower end, in outer scales
static_assert(kDphiLo == -12, "2^-6 of Xlim / 2 pi");
constexpr int kMaxJobs = 160;
constexpr long kMaxEdgeTiles = 1L << 27;  // tile pairs of a launch: the warps count eighths
constexpr int kTileI = 32;
constexpr int kTileJ = 8;

struct Job {
  int m, n;        // row WFS, column WFS
  int i0, ni;      // subaperture range of the row WFS
  int j0, nj;      // subaperture range of the column WFS
  int rb, cb;      // global row / column of the first slope of each WFS
  int tiles_i, tile_base;
};

struct LaunchDesc {
  int njobs, total_tiles, type;
  int r0, c0, nrows, ncols;
  long long ld;
  Job jobs[kMaxJobs];
};

// Element bits: 1 = (x_i, x_j), 2 = (x_i, y_j), 4 = (y_i, x_j), 8 = (y_i, y_j).
template <typename OutT>
__global__ void __launch_bounds__(kTileI* kTileJ)
    matcov_block_kernel(const __grid_constant__ LaunchDesc d, const DevGeometry g,
                        OutT* __restrict__ out) {
  __shared__ double s_tpl[kMaxLayers], s_amp[kMaxLayers], s_w[kMaxLayers];
  __shared__ double s_sm[kMaxLayers], s_sn[kMaxLayers];
  __shared__ int s_job;
  chain_wait();

  if (threadIdx.x == 0 && threadIdx.y == 0) {
    int k = 0;
    while (k + 1 < d.njobs && d.jobs[k + 1].tile_base <= (int)blockIdx.x) ++k;
    s_job = k;
  }
  __syncthreads();
  const Job& jb = d.jobs[s_job];
  const int nL = g.nLayer;
  const int m = jb.m, n = jb.n;
  const double sspm = g.diam / g.Nssp[m], sspn = g.diam / g.Nssp[n];
  const double kk = kLambda2 / (sspm * sspn);
  for (int l = threadIdx.y * kTileI + threadIdx.x; l < nL; l += kTileI * kTileJ) {
    s_tpl[l] = g.layer[l];
    s_amp[l] = g.layer[nL + l];
    s_w[l] = 0.5 * kk * g.layer[2 * nL + l];
    s_sm[l] = g.layer[3 * nL + m * nL + l];
    s_sn[l] = g.layer[3 * nL + n * nL + l];
  }
  __syncthreads();

  const int t = blockIdx.x - jb.tile_base;
  const int ti = t % jb.tiles_i, tj = t / jb.tiles_i;
  const int i = jb.i0 + ti * kTileI + threadIdx.x;
  const int j = jb.j0 + tj * kTileJ + threadIdx.y;
  if (i >= jb.i0 + jb.ni || j >= jb.j0 + jb.nj) return;

  const int Nm = g.Nsubap[m], Nn = g.Nsubap[n];
  const int rx = jb.rb + i, ry = jb.rb + Nm + i;
  const int cx = jb.cb + j, cy = jb.cb + Nn + j;
  const int r1 = d.r0 + d.nrows, c1 = d.c0 + d.ncols;
  const bool lower = (d.type == 1 || d.type == 5);
  auto want = [&](int r, int c) {
    return r >= d.r0 && r < r1 && c >= d.c0 && c < c1 && (!lower || r >= c);
  };
  unsigned mask = (want(rx, cx) ? 1u : 0u) | (want(rx, cy) ? 2u : 0u) |
                  (want(ry, cx) ? 4u : 0u) | (want(ry, cy) ? 8u : 0u);
  if (!mask) return;

  const int pi = g.off[m] + i, pj = g.off[n] + j;
  double cxx = 0, cxy = 0, cyx = 0, cyy = 0;
  const int tab = g.ttab ? g.tpair[m][n] : -1;
  if (tab >= 0) {
    const int N = g.nssp_grid, W = 2 * N - 1;
    const int2 a = reinterpret_cast<const int2*>(g.grid_cr)[i];
    const int2 b = reinterpret_cast<const int2*>(g.grid_cr)[j];
    const long off = ((long)tab * W * W + (long)(a.y - b.y + N - 1) * W + (a.x - b.x + N - 1)) * 4;
    const double4 t4 = *reinterpret_cast<const double4*>(g.ttab + off);
    cxx = t4.x;
    cxy = t4.y;
    cyx = t4.z;
    cyy = t4.w;
  }
  for (int l = 0; l < nL && tab < 0; ++l) {
    const double sml = s_sm[l], snl = s_sn[l];
    if (!(sml > 0 && snl > 0)) continue;
    const double* ul = g.u + (size_t)l * g.Nx;
    const double* vl = g.v + (size_t)l * g.Nx;
    const double du = __ldg(ul + pi) - __ldg(ul + pj);
    const double dv = __ldg(vl + pi) - __ldg(vl + pj);
    const double s1 = sml * 0.5, s2 = snl * 0.5;
    const double t2 = s_tpl[l] * s_tpl[l];
    const double w = s_w[l] * s_amp[l];
    auto D = [&](double x, double y) { return dphi_row(g.dphi, t2 * (x * x + y * y)); };
    if (s1 == s2) {
      // Equal subaperture sizes: ac = 0, ad = 2 s; XY and YX share 4 points.
      const double ad = s1 + s2;
      const double d0 = (mask & 9u) ? D(du, dv) : 0.0;
      if (mask & 1u) {
        const double xx = -d0 + D(du + ad, dv) + D(du - ad, dv) - d0;
        cxx += xx * w;
      }
      if (mask & 8u) {
        const double yy = -d0 + D(du, dv + ad) + D(du, dv - ad) - d0;
        cyy += yy * w;
      }
      if (mask & 6u) {
        const double pp = D(du + s1, dv + s2), pm = D(du + s1, dv - s2);
        const double mp = D(du - s1, dv + s2), mm = D(du - s1, dv - s2);
        cxy += (-pm + pp + mm - mp) * w;
        cyx += (-mp + pp + mm - pm) * w;
      }
    } else {
      const double ac = s1 - s2, ad = s1 + s2, bc = -ad, bd = -ac;
      if (mask & 1u)
        cxx += (-D(du + ac, dv) + D(du + ad, dv) + D(du + bc, dv) -
                D(du + bd, dv)) * w;
      if (mask & 8u)
        cyy += (-D(du, dv + ac) + D(du, dv + ad) + D(du, dv + bc) -
                D(du, dv + bd)) * w;
      if (mask & 2u)
        cxy += (-D(du + s1, dv - s2) + D(du + s1, dv + s2) +
                D(du - s1, dv - s2) - D(du - s1, dv + s2)) * w;
      if (mask & 4u)
        cyx += (-D(du - s2, dv + s1) + D(du + s2, dv + s1) +
                D(du - s2, dv - s1) - D(du + s2, dv - s1)) * w;
    }
  }

  // WFS noise on same-WFS blocks (compute_element_tiled_4 :310-330).
  if (m == n && d.type != 3) {
    if (m < g.nLgs) {
      if (i == j) {
        const int p = g.off[m] + i;
        cxx += g.noiseLGSxx[p];
        cyy += g.noiseLGSyy[p];
        cxy += g.noiseLGSxy[p];
        cyx += g.noiseLGSxy[p];
      }
      cxx += g.lgsCst;
      cyy += g.lgsCst;
    } else if (i == j) {
      cxx += g.noiseNGS[m - g.nLgs];
      cyy += g.noiseNGS[m - g.nLgs];
    }
  }

  const long long ld = d.ld;
  auto store = [&](int r, int c, double val) {
    out[(size_t)(c - d.c0) * ld + (r - d.r0)] = (OutT)val;
    if (d.type == 5 && r != c) out[(size_t)(r - d.c0) * ld + (c - d.r0)] = (OutT)val;
  };
  if (mask & 1u) store(rx, cx, cxx);
  if (mask & 2u) store(rx, cy, cxy);
  if (mask & 4u) store(ry, cx, cyx);
  if (mask & 8u) store(ry, cy, cyy);
}

// ---- Edge-aligned WFS pairs without an offset table (an LGS against an NGS or
// the truth sensor): shared stencil points.
//
// On every layer the projected subaperture of such a WFS spans [centre - s,
// centre + s] with 2 s the projected grid spacing, so its edges are the grid
// lines between neighbouring centres. The 4-point stencils then only ever
// evaluate DPHI at (edge or centre of i) - (edge or centre of j): XX at
// (x-edges, y-centres), YY at (x-centres, y-edges), XY at (x-edge of i minus
// x-centre of j, y-centre of i minus y-edge of j), YX the reverse. A block
// handles a 4x4-cell tile of WFS m against an 8x8-cell tile of WFS n: 4 x 1,440
// distinct points for its 1,024 pairs, 5.6 evaluations per pair instead of 16.
//
// A warp takes one covariance. A lane holds the two indices that are centres fixed
// (one of the i tile, one of the j tile) and walks the 9 x 5 edges of the other two,
// forming the stencil from the last two edges in registers, where the 32
// covariances of its (edge-walked) cells accumulate over the layers: no point
// passes through shared memory. With cells i = (a, b) and j = (c, e), columns and
// rows of the two tiles, and u the 5 i-edges, v the 9 j-edges:
//   XX  lane (b, e)  x = (u edge of a) - (v edge of c),   y = centres b - e
//   YY  lane (a, c)  y = (u edge of b) - (v edge of e),   x = centres a - c
//   XY  lane (b, c)  x = (u edge of a) - centre c,        y = centre b - (v edge of e)
//   YX  lane (a, e)  y = (u edge of b) - centre e,        x = centre a - (v edge of c)
// so s = S(u, v) + const for XX and YY (S: 45 values a layer, shared by the lanes)
// and s = U(u) + V(v) for XY and YX.
constexpr int kEA = 4, kEB = 8;                              // cells per tile side
constexpr int kEWarps = 16;                                  // per CTA, one CTA per SM
constexpr int kEU = kEA + 1, kEV = kEB + 1;                  // edges per tile side
constexpr int kECoord = 2 * (kEU + kEV);                     // centres: xm ym xn yn
constexpr int kEPairs = kEA * kEA * kEB * kEB;               // 1,024
static_assert(kEA * kEB == 32 && kECoord <= 32, "a lane per pair of fixed indices and per centre");
// Shared memory: the structure-function table, then per warp half of the staged
// output, the layer's centres, S, and the valid indices of the two tiles' cells.
constexpr int kEWarpDoubles = kEPairs / 2 + kECoord + kEU * kEV + (kEA * kEA + kEB * kEB) / 2 + 1;
constexpr size_t kESmem = (size_t)kTabBytes + kEWarps * kEWarpDoubles * sizeof(double);
static_assert(kESmem <= 232448, "shared memory per CTA");
// XX and YY: the lanes' (i, j) fixed indices in order of j - i, so that the eight lanes
// of a 16-byte shared load's phase hold close separations and read few table rows.
__constant__ unsigned char c_edge_lane[32] = {
    3, 2, 7, 1, 6, 11, 0, 5, 10, 15, 4, 9, 14, 19, 8, 13, 18, 23, 12, 17, 22, 27,
    16, 21, 26, 31, 20, 25, 30, 24, 29, 28};  // i + 4 j

struct EdgeJob {
  int m, n;        // row WFS, column WFS
  int rb, cb;      // global row / column of the first slope of each WFS
  int ta0, nta;    // the 4 x 4 tiles of the row WFS, the 8 x 8 tiles of the column WFS that
  int tb0, ntb;    // hold subapertures of the window
  int tile_base;
};

struct EdgeLaunch {
  int njobs, total_tiles, type;
  int r0, c0, nrows, ncols;
  long long ld;
  EdgeJob jobs[kMaxJobs];
};

// Projected centre of grid column (or row) c of WFS w on a layer:
// ((bornemin + pitch (c + 1/2)) + pup) (1 - h gsAlt) + alpha h, the same
// expression as the host projection (tomo.cpp projectedSubap) with no rotation
// and unit magnification.
__device__ __forceinline__ double grid_centre(const DevGeometry& g, int c, double pup,
                                              double rr, double shift) {
  // fused here, not by choice of a kernel's compilation: its variants agree to the bit
  const double x = fma(g.pitch / 2., 2. * c + 1., g.bornemin);
  return fma(x + pup, rr, shift);
}

// The values of one step of the walk below in a system where many lie below the table:
// all five in flight, by the form that covers every lane of the warp. Called by whole
// warps. (One call a value by the lanes below the table took 1.46 times as long at
// L0 = 10 km as at 25 m, 29 x 29; the direct form in FP64 that was there before the
// table, 0.79 times.)
struct EdgeRow {
  double v[kEU];
};
__device__ __noinline__ EdgeRow edge_low(const char* tab, EdgeRow r) {
  int least = dphi_interval(r.v[0]), most = least;
#pragma unroll
  for (int u = 1; u < kEU; ++u) {
    least = min(least, dphi_interval(r.v[u]));
    most = max(most, dphi_interval(r.v[u]));
  }
  EdgeRow o;
  if (!__any_sync(0xffffffffu, least < 0 || most >= kDphiInf)) {
#pragma unroll
    for (int u = 0; u < kEU; ++u) o.v[u] = dphi_v(tab, r.v[u]);
    return o;
  }
  if (!__any_sync(0xffffffffu, most >= 0)) {
#pragma unroll
    for (int u = 0; u < kEU; ++u) o.v[u] = dphi_low(r.v[u]);
  } else if (!__any_sync(0xffffffffu, most >= (-6 - kDphiLo) * kDphiSub)) {  // v < 2^-6
#pragma unroll
    for (int u = 0; u < kEU; ++u) o.v[u] = dphi_series<9>(r.v[u]);
  } else {
#pragma unroll
    for (int u = 0; u < kEU; ++u) {
      const bool low = dphi_interval(r.v[u]) < 0;
      const double p = dphi_low(r.v[u]), q = dphi_v(tab, low ? 1.0 : r.v[u]);
      o.v[u] = low ? p : q;
    }
  }
#pragma unroll
  for (int u = 0; u < kEU; ++u)
    if (!(r.v[u] > kDphiTiny) || dphi_interval(r.v[u]) >= kDphiInf) o.v[u] = dphi_rare(r.v[u]);
  return o;
}

// Accumulates the 8 x 4 covariances of a lane over one layer. S: kEV x kEU shared
// values (UNIFORM), or u_sep[5] of the lane and its v coordinate against the edges
// ve[v] - en (v_sep = t2 (vc - (ve[v] - en))^2). LOW: many values lie below the table.
template <bool UNIFORM, bool LOW, int NV>
__device__ __forceinline__ void edge_layer(const char* tab, const double* S, double c0,
                                           const double (&u_sep)[kEU], double vc, const double* ve, double en,
                                           double t2, double w, double (&acc)[NV][kEA]) {
  double prev[kEU];
#pragma unroll
  for (int v = 0; v <= NV; ++v) {
    double cur[kEU];
    double b = c0;
    if (!UNIFORM) {
      const double d = vc - (ve[v] - en);
      b = t2 * (d * d);
    }
    EdgeRow r;
#pragma unroll
    for (int u = 0; u < kEU; ++u) r.v[u] = dphi_scaled(__dadd_rn(UNIFORM ? S[v * kEU + u] : u_sep[u], b));
    if (LOW) r = edge_low(tab, r);
#pragma unroll
    for (int u = 0; u < kEU; ++u) cur[u] = LOW ? r.v[u] : dphi_any(tab, r.v[u]);
    // the reference's stencil (cov_XX/YY/XY/YX, matcov_kernels.cpp:147-193): right and
    // top edges are index + 1, left and bottom edges index + 0
    if (v > 0) {
#pragma unroll
      for (int u = 0; u < kEA; ++u)
        acc[v - 1][u] = fma(((-cur[u + 1] + prev[u + 1]) + cur[u]) - prev[u], w, acc[v - 1][u]);
    }
#pragma unroll
    for (int u = 0; u < kEU; ++u) prev[u] = cur[u];
  }
}

// Item v: tile pair v / 4 and covariance v % 4, by one warp; wsm is the warp's shared
// memory.
template <typename OutT, bool LOW, int PARTS>
__device__ __forceinline__ void edge_item(const EdgeLaunch& d, const DevGeometry& g,
                                          OutT* __restrict__ out, const char* tab, double* wsm,
                                          int v_item) {
  constexpr int NV = kEB / PARTS;
  const int lane = threadIdx.x & 31, kind = v_item & 3, tile = (v_item >> 2) / PARTS;
  const int v0 = (v_item >> 2) % PARTS * NV;  // the edges v0 .. v0 + NV
  double* o = wsm;                       // [32 j cells][i cell]
  double* co = o + kEPairs / 2;              // centres of the current layer
  double* S = co + kECoord;
  int* s_vi = reinterpret_cast<int*>(S + kEU * kEV + 1);
  int* s_vj = s_vi + kEA * kEA;
  int job = 0;
  while (job + 1 < d.njobs && d.jobs[job + 1].tile_base <= tile) ++job;
  const EdgeJob& jb = d.jobs[job];
  const int t = tile - jb.tile_base;
  const int ta = jb.ta0 + t % jb.nta, tb = jb.tb0 + t / jb.nta;
  const int ci0 = g.tiles_a[2 * ta], ri0 = g.tiles_a[2 * ta + 1];
  const int cj0 = g.tiles_b[2 * tb], rj0 = g.tiles_b[2 * tb + 1];
  const int N = g.nssp_grid, m = jb.m, n = jb.n;
  const int Nm = g.Nsubap[m], Nn = g.Nsubap[n];
  __syncwarp();
  for (int q = lane; q < kEA * kEA + kEB * kEB; q += 32) {
    const bool of_i = q < kEA * kEA;
    const int k = of_i ? q : q - kEA * kEA, side = of_i ? kEA : kEB;
    const int c = (of_i ? ci0 : cj0) + k % side, r = (of_i ? ri0 : rj0) + k / side;
    s_vi[q] = (c < N && r < N) ? g.cell_idx[r * N + c] : -1;  // s_vj follows s_vi
  }
  __syncwarp();
  // rows and columns of pair (i, j) in this covariance (slope bit 1: y of i, bit 0: of j)
  const int slope = kind == 0 ? 0 : (kind == 1 ? 3 : kind - 1);  // XX YY XY YX
  const int r1 = d.r0 + d.nrows, c1 = d.c0 + d.ncols;
  const bool lower = (d.type == 1 || d.type == 5);
  const int rbase = jb.rb + (slope & 2 ? Nm : 0), cbase = jb.cb + (slope & 1 ? Nn : 0);
  auto wanted = [&](int i, int j) {
    if (s_vi[i] < 0 || s_vj[j] < 0) return false;
    const int r = rbase + s_vi[i], c = cbase + s_vj[j];
    return r >= d.r0 && r < r1 && c >= d.c0 && c < c1 && (!lower || r >= c);
  };
  bool any = false;
  for (int q = lane; q < kEPairs; q += 32) any |= wanted(q & 15, q >> 4);
  if (!__any_sync(0xffffffffu, any)) return;  // nothing of this covariance is written

  double acc[NV][kEA];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int u = 0; u < kEA; ++u) acc[v][u] = 0.0;
  // the lane's fixed i and j indices
  const int fix = kind < 2 ? c_edge_lane[lane] : lane, fi = fix & 3, fj = fix >> 2;
  // centres in co: xm [0, 5), ym [5, 10), xn [10, 19), yn [19, 28)
  const double *xm = co, *ym = co + kEU, *xn = co + 2 * kEU, *yn = xn + kEV;
  const int nL = g.nLayer;
  const double sspm = g.diam / g.Nssp[m], sspn = g.diam / g.Nssp[n];
  const double kk = kLambda2 / (sspm * sspn);
  for (int l = 0; l < nL; ++l) {
    const double sml = g.layer[3 * nL + m * nL + l], snl = g.layer[3 * nL + n * nL + l];
    if (!(sml > 0 && snl > 0)) continue;
    const double h = g.layer[3 * nL + g.nW * nL + l];
    const double tpl = g.layer[l];
    const double t2 = tpl * tpl;
    const double w = 0.5 * kk * g.layer[2 * nL + l] * g.layer[nL + l];
    __syncwarp();
    if (lane < kECoord) {
      const bool of_m = lane < 2 * kEU;
      const int k = of_m ? lane : lane - 2 * kEU, ne = of_m ? kEU : kEV;
      const bool yax = k >= ne;
      const int wf = of_m ? m : n;
      const int c = (yax ? k - ne : k) + (of_m ? (yax ? ri0 : ci0) : (yax ? rj0 : cj0));
      co[lane] = grid_centre(g, c, yax ? g.YPup[wf] : g.XPup[wf], fma(-h, g.gsAlt[wf], 1.),
                             __dmul_rn(yax ? g.alphaY[wf] : g.alphaX[wf], h));
    }
    __syncwarp();
    // edge k of a WFS's tile is half a projected subaperture below centre k
    const double em = sml * 0.5, en = snl * 0.5;
    double u_sep[kEU];
    if (kind < 2) {
      const double *am = kind == 0 ? xm : ym, *an = kind == 0 ? xn : yn;
      const double *bm = kind == 0 ? ym : xm, *bn = kind == 0 ? yn : xn;
      for (int q = lane; q < kEU * kEV; q += 32) {
        const double dv = (am[q % kEU] - em) - (an[q / kEU] - en);
        S[q] = t2 * (dv * dv);
      }
      const double dc = bm[fi] - bn[fj];
      __syncwarp();
      edge_layer<true, LOW, NV>(tab, S + v0 * kEU, t2 * (dc * dc), u_sep, 0.0, nullptr, 0.0, t2, w, acc);
    } else {
      const double *am = kind == 2 ? xm : ym, *an = kind == 2 ? xn : yn;  // u edges - centre
      const double *bm = kind == 2 ? ym : xm, *bn = kind == 2 ? yn : xn;  // centre - v edges
#pragma unroll
      for (int u = 0; u < kEU; ++u) {
        const double dv = (am[u] - em) - an[fj];
        u_sep[u] = t2 * (dv * dv);
      }
      edge_layer<false, LOW, NV>(tab, nullptr, 0.0, u_sep, bm[fi], bn + v0, en, t2, w, acc);
    }
  }
  // through shared memory in two halves (v < 4, v >= 4), so that neighbouring lanes
  // store neighbouring rows
  const long long ld = d.ld;
  const bool fixed_j = kind == 0 || kind == 3;  // j = 8 fj + v, else 8 v + fj
#pragma unroll
  for (int h = 0; h < 2 / PARTS; ++h) {
    const int half = PARTS == 2 ? v0 / NV : h;
    __syncwarp();
#pragma unroll
    for (int v = 0; v < kEB / 2; ++v)
#pragma unroll
      for (int u = 0; u < kEA; ++u) {
        const int i = (kind == 0 || kind == 2) ? fi * kEA + u : u * kEA + fi;  // b * 4 + a
        const int j = fixed_j ? fj * 4 + v : v * kEB + fj;
        o[j * kEA * kEA + i] = acc[h * 4 + v][u];
      }
    __syncwarp();
    for (int q = lane; q < kEPairs / 2; q += 32) {
      const int i = q & 15, jj = q >> 4;
      const int j = fixed_j ? (jj >> 2) * kEB + half * 4 + (jj & 3) : half * 32 + jj;  // e * 8 + c
      if (!wanted(i, j)) continue;
      const int r = rbase + s_vi[i], c = cbase + s_vj[j];
      out[(size_t)(c - d.c0) * ld + (r - d.r0)] = (OutT)o[q];
      if (d.type == 5 && r != c) out[(size_t)(r - d.c0) * ld + (c - d.r0)] = (OutT)o[q];
    }
  }
}

// Persistent: one CTA per SM holds the table in shared memory; item v of the launch
// goes to warp v / gridDim.x of CTA v % gridDim.x, so that a short launch spreads
// over the SMs.
template <typename OutT, bool LOW, int PARTS>
__global__ void __launch_bounds__(kEWarps * 32, 1)
    matcov_edge_kernel(const __grid_constant__ EdgeLaunch d, const DevGeometry g,
                       OutT* __restrict__ out) {
  extern __shared__ __align__(16) char esm[];
  dphi_fill<kEWarps * 32>(esm, g.dphi);  // written once, long before: no need to wait for it
  chain_wait();
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  double* wsm = reinterpret_cast<double*>(esm + kTabBytes) + warp * kEWarpDoubles;
  for (int v = blockIdx.x + warp * gridDim.x; v < 4 * PARTS * d.total_tiles; v += kEWarps * gridDim.x)
    edge_item<OutT, LOW, PARTS>(d, g, out, esm, wsm, v);
}

// Ctt (type 4): truth-sensor auto-covariance from the unprojected positions,
// compute_element_ts_tile (common/kernels/matcov_kernels.cpp:423-483). The
// reference indexes the truth sensor at Nsubap_ts * (nW - 1), which assumes
// every WFS has the same number of valid subapertures; kept as is. Where they are on
// the common grid, the pair's offset table holds every value (toeplitz_table_kernel):
// 13.4 -> 0.1 ms for nmeasts 5,944.
template <typename OutT>
__global__ void __launch_bounds__(kTileI* kTileJ)
    matcov_ts_kernel(const DevGeometry g, int r0, int c0, int nrows, int ncols,
                     long long ld, OutT* __restrict__ out) {
  __shared__ double s_tpl[kMaxLayers], s_w[kMaxLayers];
  chain_wait();
  const int nL = g.nLayer;
  const int ts = g.nW - 1;
  const int Nt = g.Nsubap[ts];
  const double ssp = g.diam / g.Nssp[ts];
  const double kk = kLambda2 / (ssp * ssp);
  for (int l = threadIdx.y * kTileI + threadIdx.x; l < nL; l += kTileI * kTileJ) {
    s_tpl[l] = g.layer[l];
    s_w[l] = 0.5 * kk * g.layer[2 * nL + l] * g.layer[nL + l];
  }
  __syncthreads();
  // Pair grid covers the subaperture bounding range of the window.
  const int i = blockIdx.x * kTileI + threadIdx.x;
  const int j = blockIdx.y * kTileJ + threadIdx.y;
  if (i >= Nt || j >= Nt) return;
  const int r1 = r0 + nrows, c1 = c0 + ncols;
  auto want = [&](int r, int c) { return r >= r0 && r < r1 && c >= c0 && c < c1; };
  const unsigned mask = (want(i, j) ? 1u : 0u) | (want(i, Nt + j) ? 2u : 0u) |
                        (want(Nt + i, j) ? 4u : 0u) | (want(Nt + i, Nt + j) ? 8u : 0u);
  if (!mask) return;
  const int tab = g.ttab ? g.tpair[ts][ts] : -1;
  double cxx = 0, cxy = 0, cyx = 0, cyy = 0;
  if (tab >= 0) {
    const int N = g.nssp_grid, W = 2 * N - 1;
    const int2 a = reinterpret_cast<const int2*>(g.grid_cr)[i];
    const int2 b = reinterpret_cast<const int2*>(g.grid_cr)[j];
    const long off = ((long)tab * W * W + (long)(a.y - b.y + N - 1) * W + (a.x - b.x + N - 1)) * 4;
    const double4 t4 = *reinterpret_cast<const double4*>(g.ttab + off);
    cxx = t4.x;
    cxy = t4.y;
    cyx = t4.z;
    cyy = t4.w;
  }
  const int base = Nt * (g.nW - 1);
  const double du = g.X[base + i] - g.X[base + j];
  const double dv = g.Y[base + i] - g.Y[base + j];
  const double s = ssp * 0.5, ad = 2.0 * s;
  for (int l = 0; l < nL && tab < 0; ++l) {
    const double t2 = s_tpl[l] * s_tpl[l], w = s_w[l];
    auto D = [&](double x, double y) { return dphi_row(g.dphi, t2 * (x * x + y * y)); };
    const double d0 = (mask & 9u) ? D(du, dv) : 0.0;
    if (mask & 1u) cxx += (-d0 + D(du + ad, dv) + D(du - ad, dv) - d0) * w;
    if (mask & 8u) cyy += (-d0 + D(du, dv + ad) + D(du, dv - ad) - d0) * w;
    if (mask & 6u) {
      const double pp = D(du + s, dv + s), pm = D(du + s, dv - s);
      const double mp = D(du - s, dv + s), mm = D(du - s, dv - s);
      cxy += (-pm + pp + mm - mp) * w;
      cyx += (-mp + pp + mm - pm) * w;
    }
  }
  auto store = [&](int r, int c, double val) {
    out[(size_t)(c - c0) * ld + (r - r0)] = (OutT)val;
  };
  if (mask & 1u) store(i, j, cxx);
  if (mask & 2u) store(i, Nt + j, cxy);
  if (mask & 4u) store(Nt + i, j, cyx);
  if (mask & 8u) store(Nt + i, Nt + j, cyy);
}

// Offset tables of the equal-projection WFS pairs. Two WFS with the same guide
// star altitude, grid, magnification and rotation see every layer through the
// same affine map up to a constant shift, so the separation of subapertures i
// and j depends only on their grid offset (dc, dr):
//   du = G rr (dx cos - dy sin) + rr (XPup_m - XPup_n) + (alphaX_m - alphaX_n) h
//   dv = G rr (dx sin + dy cos) + rr (YPup_m - YPup_n) + (alphaY_m - alphaY_n) h
// with dx = dc pitch, dy = dr pitch and rr = 1 - h gsAlt. One thread per
// (pair, offset) evaluates the 2x2 slope block over all layers; the matrix
// kernel then gathers from the table. The separation is formed from the grid
// offset instead of from two projected positions, which changes it by rounding
// only (a few ulp of a position).
__global__ void toeplitz_table_kernel(const DevGeometry g, const int2* __restrict__ pairs,
                                      int npairs, double* __restrict__ out) {
  const int N = g.nssp_grid, W = 2 * N - 1;
  const long total = (long)npairs * W * W;
  const int nL = g.nLayer;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const int pidx = (int)(e / ((long)W * W));
    const int off = (int)(e % ((long)W * W));
    const int dr = off / W - (N - 1), dc = off % W - (N - 1);
    const int m = pairs[pidx].x, n = pairs[pidx].y;
    const double dx = dc * g.pitch, dy = dr * g.pitch;
    const double sspm = g.diam / g.Nssp[m], sspn = g.diam / g.Nssp[n];
    const double kk = kLambda2 / (sspm * sspn);
    const bool ctt = m == n && m == g.nW - 1;  // unprojected positions and sizes
    const double bx = ctt ? dx : g.G[m] * (dx * g.cth[m] - dy * g.sth[m]);
    const double by = ctt ? dy : g.G[m] * (dx * g.sth[m] + dy * g.cth[m]);
    double cxx = 0, cxy = 0, cyx = 0, cyy = 0;
    for (int l = 0; l < nL; ++l) {
      const double sml = ctt ? sspm : g.layer[3 * nL + m * nL + l];
      if (!(sml > 0)) continue;
      const double h = ctt ? 0.0 : g.layer[3 * nL + g.nW * nL + l];
      const double rr = 1. - h * g.gsAlt[m];
      const double du = (bx + (g.XPup[m] - g.XPup[n])) * rr + (g.alphaX[m] - g.alphaX[n]) * h;
      const double dv = (by + (g.YPup[m] - g.YPup[n])) * rr + (g.alphaY[m] - g.alphaY[n]) * h;
      const double s = sml * 0.5, ad = s + s;
      const double t2 = g.layer[l] * g.layer[l];
      auto D = [&](double x, double y) { return dphi_row(g.dphi, t2 * (x * x + y * y)); };
      const double w = 0.5 * kk * g.layer[2 * nL + l] * g.layer[nL + l];
      const double d0 = D(du, dv);
      cxx += (-d0 + D(du + ad, dv) + D(du - ad, dv) - d0) * w;
      cyy += (-d0 + D(du, dv + ad) + D(du, dv - ad) - d0) * w;
      const double pp = D(du + s, dv + s), pm = D(du + s, dv - s);
      const double mp = D(du - s, dv + s), mm = D(du - s, dv - s);
      cxy += (-pm + pp + mm - mp) * w;
      cyx += (-mp + pp + mm - pm) * w;
    }
    double* o = out + 4 * e;
    o[0] = cxx;
    o[1] = cxy;
    o[2] = cyx;
    o[3] = cyy;
  }
}

// Bounding subaperture range [lo, hi) of a WFS whose x slopes start at global
// index base and y slopes at base + N, intersected with the window [w0, w1).
void subap_range(int base, int N, int w0, int w1, int* lo, int* hi) {
  int a = std::max(w0 - base, 0), b = std::min(w1 - base, N);          // x part
  int c = std::max(w0 - base - N, 0), e = std::min(w1 - base - N, N);  // y part
  int l = N, h = 0;
  if (a < b) { l = std::min(l, a); h = std::max(h, b); }
  if (c < e) { l = std::min(l, c); h = std::max(h, e); }
  *lo = l;
  *hi = h;
}

// The tiles (of T x T cells, `first` of each row of them) that hold the valid
// subapertures [i0, i0 + n): whole rows of tiles.
void tiles_of(const GridRows& g, const std::vector<int>& first, int T, int i0, int n, int* t0, int* nt) {
  *t0 = 0;
  *nt = first.back();
  if (n == (int)g.row.size()) return;
  const auto r = std::minmax_element(g.row.begin() + i0, g.row.begin() + i0 + n);
  *t0 = first[*r.first / T];
  *nt = first[*r.second / T + 1] - *t0;
}

template <typename OutT>
moao_status launch_impl(const DevGeometry& g, OutT* data, int nrows, int ncols, int xoffset,
                        int yoffset, int lda, int type_mat, cudaStream_t s,
                        long long* launches, bool chained) {
  if (nrows < 0 || ncols < 0 || xoffset < 0 || yoffset < 0)
    return set_error(MOAO_ERR_BAD_ARG, "matcov: negative size or offset");
  if (nrows == 0 || ncols == 0) return MOAO_OK;
  if (lda < nrows) return set_error(MOAO_ERR_BAD_ARG, "matcov: lda < nrows");
  if (!data) return set_error(MOAO_ERR_BAD_ARG, "matcov: null data");
  if (g.nLayer > kMaxLayers || g.nW > kMaxWfs)
    return set_error(MOAO_ERR_UNSUPPORTED, "matcov: too many layers or WFS");
  const int ts = g.nW - 1;
  long nmeas = 0;
  for (int w = 0; w < ts; ++w) nmeas += 2L * g.Nsubap[w];
  const long nts = 2L * g.Nsubap[ts];

  if (type_mat == 4) {
    if (xoffset + (long)nrows > nts || yoffset + (long)ncols > nts)
      return set_error(MOAO_ERR_BAD_ARG, "matcov: Ctt tile outside nmeasts x nmeasts");
    const int Nt = g.Nsubap[ts];
    if ((long)Nt * g.nW > g.Nx)  // the reference's uniform-Nsubap indexing would overrun X, Y
      return set_error(MOAO_ERR_UNSUPPORTED, "matcov: Ctt needs equal subaperture counts per WFS");
    dim3 grid((Nt + kTileI - 1) / kTileI, (Nt + kTileJ - 1) / kTileJ);
    MOAO_CUDA_TRY(launch_chained(chained, matcov_ts_kernel<OutT>, grid, dim3(kTileI, kTileJ), 0, s, g,
                                 xoffset, yoffset, nrows, ncols, (long long)lda, data));
    if (launches) ++*launches;
    return MOAO_OK;
  }
  if (type_mat != 1 && type_mat != 2 && type_mat != 3 && type_mat != 5)
    return set_error(MOAO_ERR_BAD_ARG, "matcov: unrecognized type_mat " + std::to_string(type_mat));
  const long rows_total = (type_mat == 3) ? nts : nmeas;
  const long cols_total = (type_mat == 2) ? nts : nmeas;
  if (xoffset + (long)nrows > rows_total || yoffset + (long)ncols > cols_total)
    return set_error(MOAO_ERR_BAD_ARG, "matcov: tile outside the matrix");
  if (type_mat == 5 && (xoffset != yoffset || nrows != ncols))
    return set_error(MOAO_ERR_BAD_ARG, "matcov: type 5 needs a square diagonal tile");

  // Row / column WFS lists and their slope bases.
  std::vector<int> rw, cw, rbase, cbase;
  if (type_mat == 3) { rw.push_back(ts); rbase.push_back(0); }
  else { int b = 0; for (int w = 0; w < ts; ++w) { rw.push_back(w); rbase.push_back(b); b += 2 * g.Nsubap[w]; } }
  if (type_mat == 2) { cw.push_back(ts); cbase.push_back(0); }
  else { int b = 0; for (int w = 0; w < ts; ++w) { cw.push_back(w); cbase.push_back(b); b += 2 * g.Nsubap[w]; } }

  const bool lower = (type_mat == 1 || type_mat == 5);
  std::vector<Job> jobs;
  for (size_t a = 0; a < rw.size(); ++a) {
    for (size_t b = 0; b < cw.size(); ++b) {
      const int m = rw[a], n = cw[b];
      if (lower && m < n) continue;  // entirely above the diagonal
      Job jb{};
      jb.m = m; jb.n = n; jb.rb = rbase[a]; jb.cb = cbase[b];
      int ilo, ihi, jlo, jhi;
      subap_range(jb.rb, g.Nsubap[m], xoffset, xoffset + nrows, &ilo, &ihi);
      subap_range(jb.cb, g.Nsubap[n], yoffset, yoffset + ncols, &jlo, &jhi);
      if (ilo >= ihi || jlo >= jhi) continue;
      jb.i0 = ilo; jb.ni = ihi - ilo; jb.j0 = jlo; jb.nj = jhi - jlo;
      jb.tiles_i = (jb.ni + kTileI - 1) / kTileI;
      jobs.push_back(jb);
    }
  }
  // Edge-aligned pairs without an offset table go to the shared-point kernel.
  std::vector<Job> plain;
  std::vector<EdgeJob> edge;
  for (const Job& jb : jobs) {
    const bool tab = g.ttab && g.tpair[jb.m][jb.n] >= 0;
    if (!tab && jb.m != jb.n && g.aligned[jb.m] && g.aligned[jb.n] && g.cell_idx &&
        g.ntiles_a > 0 && g.ntiles_b > 0) {
      EdgeJob e{};
      e.m = jb.m; e.n = jb.n; e.rb = jb.rb; e.cb = jb.cb;
      tiles_of(*g.rows, g.rows->first_a, kEA, jb.i0, jb.ni, &e.ta0, &e.nta);
      tiles_of(*g.rows, g.rows->first_b, kEB, jb.j0, jb.nj, &e.tb0, &e.ntb);
      edge.push_back(e);
    } else {
      plain.push_back(jb);
    }
  }
  jobs.swap(plain);
  for (size_t base = 0; base < edge.size();) {
    EdgeLaunch d{};
    d.type = type_mat;
    d.r0 = xoffset; d.c0 = yoffset; d.nrows = nrows; d.ncols = ncols; d.ld = lda;
    long tiles = 0;
    for (; base < edge.size() && d.njobs < kMaxJobs; ++base) {
      EdgeJob e = edge[base];
      const long more = (long)e.nta * e.ntb;
      if (more > kMaxEdgeTiles) return set_error(MOAO_ERR_UNSUPPORTED, "matcov: window too large");
      if (tiles + more > kMaxEdgeTiles) break;
      e.tile_base = (int)tiles;
      tiles += more;
      d.jobs[d.njobs++] = e;
    }
    d.total_tiles = (int)tiles;
    if (tiles == 0) continue;
    static std::atomic<unsigned long long> configured[4];
    // edge_low where an outer scale puts separations of a subaperture and a 32nd of the pupil
    // below the table (Cmm, ms, a branch at each value and edge_low: 39 m, 29 x 29,
    // 10 layers, L0 = 25 m 1.62 and 1.79, 100 m 1.79 and 1.83, 300 m 1.97 and 1.79; the
    // direct form before the table 3.03, 2.30 and 2.30). By the geometry alone, so that an
    // element has the same bits in every window.
    const bool low = kDphiReach * g.outer > std::max(g.pitch, g.diam / 32);
    // Half tiles (25 values a lane for 45, and 8 % more a value) where the warps then go
    // through fewer: a small launch is as long as its longest chain. Cmm and Ctm, us, whole
    // and half: 8 m, 10 x 10, 3 layers 49 + 48 and 40 + 39; 39 m, 10 layers, 10 x 10
    // 87 + 82 and 66 + 61, 20 x 20 264 + 167 and 270 + 158.
    const long warps = 148 * kEWarps;
    const bool half = (8 * tiles + warps - 1) / warps * 27 < (4 * tiles + warps - 1) / warps * 45;
    const auto kern = half ? (low ? matcov_edge_kernel<OutT, true, 2> : matcov_edge_kernel<OutT, false, 2>)
                           : (low ? matcov_edge_kernel<OutT, true, 1> : matcov_edge_kernel<OutT, false, 1>);
    MOAO_CUDA_TRY(set_smem_limit(kern, (int)kESmem, configured[2 * half + low]));
    const int ctas = (int)std::min(148L, (half ? 8 : 4) * tiles);
    MOAO_CUDA_TRY(launch_chained(chained, kern, dim3((unsigned)ctas),
                                 dim3(kEWarps * 32), kESmem, s, d, g, data));
    if (launches) ++*launches;
  }
  // Launch in chunks of kMaxJobs jobs.
  for (size_t base = 0; base < jobs.size(); base += kMaxJobs) {
    LaunchDesc d{};
    d.type = type_mat;
    d.r0 = xoffset; d.c0 = yoffset; d.nrows = nrows; d.ncols = ncols; d.ld = lda;
    int tiles = 0;
    for (size_t k = base; k < jobs.size() && k < base + kMaxJobs; ++k) {
      Job jb = jobs[k];
      jb.tile_base = tiles;
      tiles += jb.tiles_i * ((jb.nj + kTileJ - 1) / kTileJ);
      d.jobs[d.njobs++] = jb;
    }
    d.total_tiles = tiles;
    if (tiles == 0) continue;
    MOAO_CUDA_TRY(launch_chained(chained, matcov_block_kernel<OutT>, dim3((unsigned)tiles),
                                 dim3(kTileI, kTileJ), 0, s, d, g, data));
    if (launches) ++*launches;
  }
  return MOAO_OK;
}

// Ordered WFS pairs that get an offset table: Cmm pairs (m >= n) and the truth
// sensor against each WFS, in both orders, when their projections match.
void table_pairs(const DevGeometry& g, int2* pairs, int* npairs) {
  *npairs = 0;
  const int ts = g.nW - 1;
  auto same = [&](int m, int n) {
    return g.gsAlt[m] == g.gsAlt[n] && g.G[m] == g.G[n] && g.cth[m] == g.cth[n] &&
           g.sth[m] == g.sth[n] && g.Nssp[m] == g.nssp_grid && g.Nssp[n] == g.nssp_grid &&
           g.Nsubap[m] == g.Nsubap[0] && g.Nsubap[n] == g.Nsubap[0];
  };
  for (int m = 0; m < g.nW; ++m)
    for (int n = 0; n < g.nW; ++n) {
      const bool needed = (m < ts && n < ts && m >= n) || (m == ts && n < ts) || (n == ts && m < ts);
      // Ctt by the truth sensor with itself, where every WFS is on the common grid (its
      // positions are then the grid's)
      bool ctt = m == ts && n == ts;
      for (int q = 0; q < g.nW && ctt; ++q)
        ctt = g.Nsubap[q] == g.Nsubap[0] && g.Nssp[q] == g.nssp_grid;
      if ((needed && same(m, n)) || ctt) pairs[(*npairs)++] = make_int2(m, n);
    }
}

}  // namespace

const DphiRow* dphi_table() {
  static const std::vector<DphiRow> table = [] {
    auto f = [](long double v, bool asym) {
      const long double x = std::sqrt(v) * (long double)kXlim;
      if (asym) {
        const long double xi = 1.0L / x;
        return (long double)kK2 - (long double)kK3 * std::exp(-x) * std::cbrt(x) *
                                      (1.0L + xi * (kA1 + xi * (kA2 + xi * (long double)kA3)));
      }
      const long double c = std::cbrt(x), z = 0.25L * x * x;
      long double pg = kGma.c[10], pa = kGa.c[10];
      for (int n = 9; n >= 0; --n) pg = pg * z + kGma.c[n];
      for (int n = 9; n >= 1; --n) pa = pa * z + kGa.c[n];
      return -0.5L * (x * c * c * pg + z * pa);
    };
    constexpr int D = 8;  // degree
    std::vector<DphiRow> t(kDphiRows);
    for (int k = 0; k + 1 < kDphiRows; ++k) {
      const int e = kDphiLo + k / kDphiSub;
      const long double w = std::ldexp(1.0L, e) / kDphiSub;  // interval width
      const long double mid = std::ldexp(1.0L, e) + w * (k % kDphiSub) + w / 2;
      // Newton's divided differences at Chebyshev nodes in tau = (v - mid) / (w / 2),
      // expanded to powers of tau
      long double node[D + 1], d[D + 1], mono[D + 1] = {}, basis[D + 2] = {1.0L};
      for (int i = 0; i <= D; ++i) {
        node[i] = std::cos(3.141592653589793238462643L * (2 * i + 1) / (2 * (D + 1)));
        d[i] = f(mid + node[i] * w / 2, e >= 0);
      }
      for (int o = 1; o <= D; ++o)
        for (int i = D; i >= o; --i) d[i] = (d[i] - d[i - 1]) / (node[i] - node[i - o]);
      for (int o = 0; o <= D; ++o) {
        for (int i = 0; i <= o; ++i) mono[i] += d[o] * basis[i];
        for (int i = o + 1; i >= 1; --i) basis[i] = basis[i - 1] - node[o] * basis[i];
        basis[0] *= -node[o];
      }
      long double scale = 1.0L;
      for (int i = 0; i <= D; ++i, scale *= 2.0L / w) {
        if (i < 5) t[k].c[i] = (double)(mono[i] * scale);
        else t[k].f[i - 5] = (float)(mono[i] * scale);
      }
    }
    t[kDphiRows - 1] = DphiRow{{kK2, 0, 0, 0, 0}, {0, 0, 0, 0}};
    return t;
  }();
  return table.data();
}

long toeplitz_table_doubles(const DevGeometry& g, int* npairs) {
  int2 pairs[kMaxWfs * kMaxWfs];
  table_pairs(g, pairs, npairs);
  const long W = 2L * g.nssp_grid - 1;
  return (long)*npairs * W * W * 4;
}

moao_status build_toeplitz_tables(DevGeometry& g, cudaStream_t s, long long* launches) {
  int2 pairs[kMaxWfs * kMaxWfs];
  int np = 0;
  table_pairs(g, pairs, &np);
  for (int m = 0; m < kMaxWfs; ++m)
    for (int n = 0; n < kMaxWfs; ++n) g.tpair[m][n] = -1;
  if (np == 0 || !g.ttab) {
    g.ttab = nullptr;
    return MOAO_OK;
  }
  for (int k = 0; k < np; ++k) g.tpair[pairs[k].x][pairs[k].y] = k;
  // the pair list travels in the table's tail (4 doubles per offset before it)
  const long W = 2L * g.nssp_grid - 1;
  int2* d_pairs = reinterpret_cast<int2*>(g.ttab + (long)np * W * W * 4);
  MOAO_CUDA_TRY(cudaMemcpyAsync(d_pairs, pairs, np * sizeof(int2), cudaMemcpyHostToDevice, s));
  const long total = (long)np * W * W;
  const unsigned blocks = (unsigned)std::min<long>((total + 127) / 128, 148L * 64);
  toeplitz_table_kernel<<<blocks, 128, 0, s>>>(g, d_pairs, np, g.ttab);
  if (launches) ++*launches;
  MOAO_CUDA_TRY(cudaGetLastError());
  return MOAO_OK;
}

moao_status launch_matcov(const DevGeometry& g, double* data, int nrows, int ncols,
                          int xoffset, int yoffset, int lda, int type_mat, cudaStream_t s,
                          long long* launches, bool chained) {
  return launch_impl<double>(g, data, nrows, ncols, xoffset, yoffset, lda, type_mat, s,
                             launches, chained);
}

moao_status launch_matcov_f32(const DevGeometry& g, float* data, int nrows, int ncols,
                              int xoffset, int yoffset, int lda, int type_mat, cudaStream_t s,
                              long long* launches) {
  return launch_impl<float>(g, data, nrows, ncols, xoffset, yoffset, lda, type_mat, s,
                            launches, false);
}

}  // namespace moao
