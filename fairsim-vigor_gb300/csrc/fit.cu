// The parameter fit on line pairs: SimAlgorithm.estimateParameters (S/SimAlgorithm.java:37-159)
// and the live refit (LM/ReconstructionRunner.java:642-746) for all directions at once.
//
// The fit always correlates two bands of one direction, so the two bands are the two lines of a
// pair (fft_pair.cuh): a plane holds {re0, re1, im0, im1} per pixel, and every transform,
// attenuation and common region of the search works on both. Transforms run columns first, then
// rows, so that a row pass ends with whole rows of both bands in registers and forms what follows:
//   spectra  raw rows x border fade, FFT along x; FFT along y; separation           -> S (band pairs)
//   coarse   columns: S x attenuation, inverse along y; rows: inverse along x, band1 conj(band0),
//            FFT along x; columns of that: FFT along y and the largest magnitude beyond kMin
//   search   three times: columns: common region of S, inverse along y; rows: inverse along x, the
//            row's ten ramp sums of band1 conj(band0) and its share of norm2(band0); one block per
//            grid point: the sum over rows, the last block to finish scans the grid in the
//            reference's order and sets up the next step
//   getPeak  region, two-pass inverse transforms and row sums as Correlation.getPeak's vector form
// The search's transforms run on pairs, so its own phase and magnitude (reported with the peaks) carry
// other roundings of the same size as the form that ran one vector operation at a time; ramps, products
// and sums hold what they held there. The spectra and getPeak, whose phase and modulation the fit
// stores, keep that form's roundings (transforms line by line, sums in its order). It took 2.87 ms at
// 1024^2 (3 x 3, f32): 13 launches per search step and direction, each pass over memory.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "corr_grid.cuh"
#include "estimate.cuh"
#include "fft_pair.cuh"
#include "filters.cuh"
#include "otf.cuh"
#include "runtime.cuh"
#include "sim_host.h"
#include "vec_ops.cuh"

namespace fsim {
namespace {

constexpr int NG = 10;       // grid side of a search step (Correlation.fitPeak)
constexpr int NV = 2 * NG;   // sums per row: NG complex ramp sums (norm2 has its own)
constexpr int NR = 2 * NG;   // ramps per direction: the grid's columns, then its rows

// One direction's state: the search of the current step (position, width, shifts, common region)
// and the best correlation so far.
struct FitDir {
  double kx, ky, search, phase, mag;
  double kxs[NG], kys[NG];
  CrParams cp;
  double2 corr[NG * NG];
  int done;  // grid points finished in this step
  int pad;
};
struct FitArgs {  // what the passes need besides planes and state
  const OtfTable* otf;
  const float* att;      // attenuation of the coarse correlation, N*N (symmetric)
  const float* weight;   // 1 / OTF inside the weight limit, 0 beyond, N*N (symmetric)
  float wlf;             // weight limit: the smallest float >= it
  float d2_keep, d2_drop;  // squared distance (px^2) surely inside / beyond the weight limit; d2_drop < 0: unknown
  // Per direction NR ramps of N entries. Search: x ramps j and j + NG/2 together, {re, re, im, im} per
  // entry, then the y ramps one by one. getPeak: its x ramp first, its y ramp at NG * N.
  float2* ramps;
  double2* Q;            // per direction: NG x N row sums
  double* n2;            // per direction: N row norms
  float* pmag;           // per direction and peak block
  int* pidx;
  FitDir* dir;
  double* results;       // per direction: kx, ky, phase, magnitude, getPeak of the low and the high band
};

template <int N>
struct FCfg {
  static constexpr int E = (N % 3 == 0) ? 12 : 8;
  static constexpr int T = N / E;
  static constexpr int G = T >= 64 ? 1 : 64 / T;  // rows per block, row passes
  static constexpr int C = T >= 256 ? 2 : 4;      // columns per block, column passes
  static constexpr int R = E <= 8 ? (C * T >= 512 ? 64 : 80) : 128;
  static constexpr int XS = pair_elems(N, 1), XC = pair_elems(N, C);
  static constexpr int blocks(int threads, int regs) {
    const int n = threads < 32 ? 32 : threads, b = 65536 / (n * regs);
    return b < 1 ? 1 : (b > 32 ? 32 : b);
  }
  static constexpr int PT = T > 32 ? 32 : T;  // partial sums per value and row, added in FP64
};

struct MixCoef {  // separation coefficients of both bands of a plane
  float2 c[FSIM_MAX_DIRS][2][FSIM_MAX_PHASES];
};

// ---- band spectra -----------------------------------------------------------------------------
// separateBands of both bands of a plane from the frame spectra
struct SpecIn {
  const float2* in[FSIM_MAX_DIRS * FSIM_MAX_PHASES];
};
__global__ void k_fit_separate(const __grid_constant__ SpecIn si, const __grid_constant__ MixCoef mc, int nP, size_t n,
                               ulonglong2* __restrict__ S) {
  const int a = blockIdx.y;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    // the products and sums of k_separate, rounded one by one: the same bits
    float re[2] = {0.f, 0.f}, im[2] = {0.f, 0.f};
    for (int p = 0; p < nP; p++) {
      const float2 v = __ldg(si.in[a * nP + p] + i);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float2 c = mc.c[a][h][p];
        re[h] = __fadd_rn(re[h], __fsub_rn(__fmul_rn(c.x, v.x), __fmul_rn(c.y, v.y)));
        im[h] = __fadd_rn(im[h], __fadd_rn(__fmul_rn(c.y, v.x), __fmul_rn(c.x, v.y)));
      }
    }
    S[a * n + i] = make_ulonglong2(p_pack(re[0], re[1]), p_pack(im[0], im[1]));
  }
}

// ---- column passes ----------------------------------------------------------------------------
// Is |OTF(r -+ k)| below the weight limit? Decided by the squared distance where it is clear (the
// estimated OTF falls with the radius), else by the lookup.
__device__ __forceinline__ bool otf_inside(const FitArgs& A, int xh, int yh, FShift k, double kx, double ky) {
  const float dx = __fsub_rn(__fsub_rn((float)xh, k.xh), k.xl), dy = __fsub_rn(__fsub_rn((float)yh, k.yh), k.yl);
  const float d2 = dx * dx + dy * dy;
  if (A.d2_drop >= 0.f) {
    if (d2 < A.d2_keep) return true;
    if (d2 > A.d2_drop) return false;
  }
  float2 c;
  const float v = otf_at_fast(*A.otf, 0, xh, yh, k, kx, ky, false, &c) ? c.x : 0.f;
  return !(fabsf(v) < A.wlf);
}
// Factors of both bands at (x, y): Correlation.commonRegion (java:227-288) with division by the OTF.
struct Region {  // CrParams with what a pixel needs of it in 32 bits
  double kx, ky, dist;
  FShift kf, kn;
  int r2_lo, r2_hi, ikx, iky, mx_zero;
};
template <int N>
__device__ __forceinline__ Region region_of(const CrParams& cp, double dist) {
  Region r;
  r.kx = cp.kx;
  r.ky = cp.ky;
  r.dist = dist;
  r.kf = cp.kf;
  r.kn = fshift_neg(cp.kf);
  r.r2_lo = (int)cp.r2_lo;
  r.r2_hi = (int)cp.r2_hi;
  r.ikx = ((int)cp.kx % N + N) % N;
  r.iky = ((int)cp.ky % N + N) % N;
  r.mx_zero = cp.mx_zero;
  return r;
}
template <int N>
__device__ __forceinline__ f32x2 common_factor(const FitArgs& A, const Region& R, int x, int y) {
  const float w = __ldg(A.weight + (size_t)x * N + y);
  if (w == 0.f) return 0ull;
  const int xh = freq_x(x, N), yh = freq_y(y, N);
  auto cut = [&](int xx, int yy) {
    const int a = freq_x(xx, N), b = freq_x(yy, N), r2 = a * a + b * b;
    if (R.mx_zero) {  // ratio = sqrt(r^2) / 0: the reference's expression (NaN at the origin)
      const double ratio = sqrt((double)r2) / 0.0;
      return (ratio < R.dist) || (ratio > (1 - R.dist));
    }
    return r2 < R.r2_lo || r2 > R.r2_hi;
  };
  const float f0 = !cut(x, y) && otf_inside(A, xh, yh, R.kf, R.kx, R.ky) ? w : 0.f;
  // band1 is zeroed at ((x-(int)kx+w)%w, (y+(int)ky+h)%h) for every cut (x,y)
  int xs = x + R.ikx, ys = y - R.iky;
  xs = xs >= N ? xs - N : xs;
  ys = ys < 0 ? ys + N : ys;
  const float f1 = !cut(xs, ys) && otf_inside(A, xh, yh, R.kn, -R.kx, -R.ky) ? w : 0.f;
  return p_pack(f0, f1);
}
__device__ __forceinline__ float2 ramp_at(double k, int x, int N) {  // exp(2 pi i k x / N), reduced in double
  double f = k * (double)x / (double)N;
  f -= floor(f);
  double s, c;
  sincospi(2.0 * f, &s, &c);
  return make_float2((float)c, (float)s);
}
// One ramp of the search by a block, in FP64 and rounded once, as ramp_at: exp(2 pi i k (32 m + l) / N) is
// the product of two factors out of N/32 + 32. (GB300 runs two FP64 operations per clock and SM: with a
// sine and cosine for every entry the ramps of a step took longer than its column pass.)
__device__ __forceinline__ double2 turn(double f) {
  f -= floor(f);
  double s, c;
  sincospi(2.0 * f, &s, &c);
  return make_double2(c, s);
}
template <class F>
__device__ __forceinline__ void ramp_search(double k, int N, double2* f, F put) {
  const int nh = N / 32;
  for (int i = threadIdx.x; i < nh + 32; i += blockDim.x) f[i] = turn(k * (double)(i < nh ? 32 * i : i - nh) / (double)N);
  __syncthreads();
  for (int x = threadIdx.x; x < N; x += blockDim.x) {
    const double2 h = f[x >> 5], l = f[nh + (x & 31)];
    put(x, make_float2((float)(h.x * l.x - h.y * l.y), (float)(h.x * l.y + h.y * l.x)));
  }
}
// SEARCH false: times the attenuation, inverse. true: common region, inverse; the first NR blocks of a
// direction compute the step's ramps instead.
template <int N, bool SEARCH>
__global__ void __launch_bounds__(FCfg<N>::C* FCfg<N>::T, FCfg<N>::blocks(FCfg<N>::C* FCfg<N>::T, FCfg<N>::R))
    k_fit_cols(const ulonglong2* __restrict__ in, ulonglong2* __restrict__ out, const __grid_constant__ FitArgs A,
               double dist) {
  using P = FCfg<N>;
  constexpr int T = P::T, C = P::C, E = P::E;
  extern __shared__ ulonglong2 smp[];
  static_assert((N / 32 + 32) * sizeof(double2) <= P::XC * sizeof(ulonglong2), "a ramp's factors fit the exchange buffer");
  const int lt = threadIdx.x, lane = lt % C, t = lt / C, a = blockIdx.y;
  if constexpr (SEARCH) {
    if (blockIdx.x < NR) {  // fourierShift(kx, -ky) of every grid column and row
      const FitDir& d = A.dir[a];
      float2* r = A.ramps + (size_t)a * NR * N;
      const int j = blockIdx.x;
      double2* f = reinterpret_cast<double2*>(smp);
      if (j < NG) {
        float* q = reinterpret_cast<float*>(r + (size_t)(j % (NG / 2)) * 2 * N) + j / (NG / 2);
        ramp_search(d.kxs[j], N, f, [&](int x, float2 v) {
          q[4 * x] = v.x;
          q[4 * x + 2] = v.y;
        });
      } else {
        ramp_search(-d.kys[j - NG], N, f, [&](int y, float2 v) { r[(size_t)j * N + y] = v; });
      }
      return;
    }
  }
  const int x = (blockIdx.x - (SEARCH ? NR : 0)) * C + lane;
  const ulonglong2* ip = in + (size_t)a * N * N + x;
  cpair v[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const ulonglong2 u = __ldg(ip + (size_t)(t + i * T) * N);
    v[i] = cpair{u.x, u.y};
  }
  if constexpr (SEARCH) {
    const Region R = region_of<N>(A.dir[a].cp, dist);
#pragma unroll
    for (int i = 0; i < E; i++) {
      const float2 f = p_unpack(common_factor<N>(A, R, x, t + i * T)), re = p_unpack(v[i].re), im = p_unpack(v[i].im);
      // (a bin that is cut is 0, whatever it held)
      v[i] = cpair{p_pack(f.x == 0.f ? 0.f : re.x * f.x, f.y == 0.f ? 0.f : re.y * f.y),
                   p_pack(f.x == 0.f ? 0.f : im.x * f.x, f.y == 0.f ? 0.f : im.y * f.y)};
    }
  } else {
#pragma unroll
    for (int i = 0; i < E; i++) {
      const f32x2 f = p_dup(__ldg(A.att + (size_t)x * N + t + i * T));
      v[i] = cpair{p_mul(v[i].re, f), p_mul(v[i].im, f)};
    }
  }
  line_fft_pair<N, T, C, true>(v, smp, lane, t, g_stw + stw_offset(N, E));
  ulonglong2* op = out + (size_t)a * N * N + x;
#pragma unroll
  for (int i = 0; i < E; i++) op[(size_t)(t + i * T) * N] = make_ulonglong2(v[i].re, v[i].im);
}

// ---- row passes -------------------------------------------------------------------------------
// Coarse correlation: inverse along x of both bands, band1 conj(band0) scaled as two scaled inverse
// transforms, forward along x. The product row is stored as float2.
template <int N>
__global__ void __launch_bounds__(FCfg<N>::G* FCfg<N>::T, FCfg<N>::blocks(FCfg<N>::G* FCfg<N>::T, FCfg<N>::R))
    k_fit_rows_product(const ulonglong2* __restrict__ W, float2* __restrict__ V) {
  using P = FCfg<N>;
  constexpr int T = P::T, E = P::E;
  const int g = threadIdx.x / T, t = threadIdx.x % T, y = blockIdx.x * P::G + g, a = blockIdx.y;
  extern __shared__ ulonglong2 smp[];
  ulonglong2* s = smp + g * P::XS;
  const float2* tw = g_stw + stw_offset(N, E);
  const size_t row = ((size_t)a * N + y) * N + t;
  cpair x[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const ulonglong2 u = W[row + i * T];
    x[i] = cpair{u.x, u.y};
  }
  line_fft_pair<N, T, 1, true>(x, s, 0, t, tw);
  const float sc = 1.f / ((float)N * (float)N);
  float2 p[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    float2 b0, b1;
    cp_split(x[i], b0, b1);
    p[i] = cmulc(cscale(b1, sc), cscale(b0, sc));
  }
  line_fft_reg<N, T, 1, false>(p, reinterpret_cast<float2*>(s), 0, t, tw);
#pragma unroll
  for (int i = 0; i < E; i++) V[row + i * T] = p[i];
}
// Grid row sums: Q[j] = sum_x b1 conj(b0) exp(2 pi i kxs[j] x / N), two ramps at a time in packed
// arithmetic, and sum_x |b0|^2. A thread's pixels and the threads of equal lane are added in float, as the
// 32 partial sums of a warp-per-row evaluation, then those in FP64; the norm's float squares are added
// exactly to 2^-45 (a sum of two floats), then in FP64. The transforms' 1/N^2 cancels against the norm. 35 us at
// 1024^2, 3 directions (29 with eight of the ramps as float products of two others and a float norm).
template <int N>
__global__ void __launch_bounds__(FCfg<N>::G* FCfg<N>::T, FCfg<N>::blocks(FCfg<N>::G* FCfg<N>::T, FCfg<N>::E <= 8 ? 96 : 128))
    k_fit_rows(const ulonglong2* __restrict__ W, const __grid_constant__ FitArgs A) {
  using P = FCfg<N>;
  constexpr int T = P::T, E = P::E;
  const int g = threadIdx.x / T, t = threadIdx.x % T, y = blockIdx.x * P::G + g, a = blockIdx.y;
  extern __shared__ ulonglong2 smp[];
  ulonglong2* s = smp + g * P::XS;
  const size_t row = ((size_t)a * N + y) * N + t;
  cpair x[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const ulonglong2 u = __ldg(W + row + i * T);
    x[i] = cpair{u.x, u.y};
  }
  line_fft_pair<N, T, 1, true>(x, s, 0, t, g_stw + stw_offset(N, E));
  const ulonglong2* r = reinterpret_cast<const ulonglong2*>(A.ramps + (size_t)a * NR * N) + t;
  cpair q[NG / 2];  // ramps j and j + NG/2
#pragma unroll
  for (int j = 0; j < NG / 2; j++) q[j] = cp_zero();
  float ns = 0.f, ne = 0.f;
  auto add_norm = [&](float v) {
    float s, z;
    ff_two_sum(ns, v, s, z);
    ns = s;
    ne = __fadd_rn(ne, z);
  };
#pragma unroll
  for (int i = 0; i < E; i++) {
    float2 b0, b1;
    cp_split(x[i], b0, b1);
    add_norm(__fmul_rn(b0.x, b0.x));
    add_norm(__fmul_rn(b0.y, b0.y));
    const wpair p = w_dup(cmulc(b1, b0));
#pragma unroll
    for (int j = 0; j < NG / 2; j++) {
      const ulonglong2 w = __ldg(r + (size_t)j * N + i * T);
      q[j] = cadd(q[j], cmul(cpair{w.x, w.y}, p));
    }
  }
  float* part = reinterpret_cast<float*>(smp + P::G * P::XS) + (size_t)g * NV * (T + 1);  // [value][T + 1]
#pragma unroll
  for (int j = 0; j < NG / 2; j++) {
    float2 u, v;
    cp_split(q[j], u, v);
    part[(2 * j) * (T + 1) + t] = u.x;
    part[(2 * j + 1) * (T + 1) + t] = u.y;
    part[(2 * j + NG) * (T + 1) + t] = v.x;
    part[(2 * j + NG + 1) * (T + 1) + t] = v.y;
  }
  constexpr int NWP = (T + 31) / 32;  // warps per row
  __shared__ double norm[P::G][NWP];
#pragma unroll
  for (int o = P::PT / 2; o > 0; o >>= 1) {  // PT lanes: the warp, or the row's share of it
    const float s = __shfl_xor_sync(0xffffffffu, ns, o), z = __shfl_xor_sync(0xffffffffu, ne, o);
    add_norm(s);
    ne = __fadd_rn(ne, z);
  }
  if (t % P::PT == 0) norm[g][t / P::PT] = (double)ns + (double)ne;
  __syncthreads();
  if (t == 0) {
    double d = norm[g][0];
    for (int k = 1; k < NWP; k++) d += norm[g][k];
    A.n2[(size_t)a * N + y] = d;
  }
  // four threads per value (neighbours in a warp), an eighth of the PT partial sums at a time
  for (int k = t; k < 4 * NV; k += T) {
    const int v = k / 4, h = k % 4;
    const float* pv = part + v * (T + 1);
    double d = 0;
#pragma unroll
    for (int l = 0; l < P::PT; l += 4) {
      float f = pv[l + h];
#pragma unroll
      for (int w = P::PT; w < T; w += P::PT) f += pv[w + l + h];
      d += f;
    }
    const unsigned four = 0xfu << (threadIdx.x & 28);  // enter together: T and 4 * NV are multiples of 4
    d += __shfl_xor_sync(four, d, 1);
    d += __shfl_xor_sync(four, d, 2);
    if (h == 0) reinterpret_cast<double*>(A.Q + ((size_t)a * NG + v / 2) * N + y)[v & 1] = d;
  }
}

// ---- search -----------------------------------------------------------------------------------
// The next step at (kx, ky): shifts k + ((i - 4.5) / 4.5) search and the common region, by the threads
// of a block of at least 128 (each chain of FP64 operations on a warp of its own).
__device__ void fit_setup(FitDir& d, double kx, double ky, double search, double dist, int n) {
  const int i = threadIdx.x;
  const double mx = __dsqrt_rn(__dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky)));
  const long long r2max = 2 * (long long)(n / 2) * (n / 2);
  if (i < NG) {
    const double o = __dmul_rn(__ddiv_rn((double)i - 4.5, 4.5), search);
    d.kxs[i] = __dadd_rn(kx, o);
    d.kys[i] = __dadd_rn(ky, o);
  } else if (i == 32) {
    d.cp.r2_lo = mx > 0 ? cr_threshold_lo(mx, dist, r2max) : 0;
  } else if (i == 64) {
    d.cp.r2_hi = mx > 0 ? cr_threshold_hi(mx, dist, r2max) : 0;
  } else if (i == 96) {
    d.kx = kx;
    d.ky = ky;
    d.search = search;
    d.cp.kx = kx;
    d.cp.ky = ky;
    d.cp.kf = fshift_host(kx, ky);
    d.cp.mx_zero = mx > 0 ? 0 : 1;
    d.done = 0;
  }
}
// Column transforms of the coarse correlation (two adjacent columns per pair) and the largest
// magnitude of the block's columns beyond kMin (r^2 > r2_lim), the first in y-major order among
// equals: Correlation.locatePeak (java:144-167). Cplx.Float.abs() is evaluated in double only where
// a float estimate (within 4e-7 of it) can reach the running maximum.
template <int N>
__global__ void __launch_bounds__(FCfg<N>::C* FCfg<N>::T, FCfg<N>::blocks(FCfg<N>::C* FCfg<N>::T, FCfg<N>::R))
    k_fit_peak(const float2* __restrict__ V, long long r2_lim, const __grid_constant__ FitArgs A) {
  using P = FCfg<N>;
  constexpr int T = P::T, C = P::C, E = P::E, NT = C * T;
  const int lt = threadIdx.x, lane = lt % C, t = lt / C, a = blockIdx.y, x = 2 * (blockIdx.x * C + lane);
  extern __shared__ ulonglong2 smp[];
  const float4* ip = reinterpret_cast<const float4*>(V + (size_t)a * N * N + x);
  cpair v[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const float4 u = ip[(size_t)(t + i * T) * (N / 2)];
    v[i] = cpair{p_pack(u.x, u.z), p_pack(u.y, u.w)};
  }
  line_fft_pair<N, T, C, false>(v, smp, lane, t, g_stw + stw_offset(N, E));
  auto inside = [&](int i, int h) {
    const long long xx = freq_x(x + h, N), yy = freq_y(t + i * T, N);
    return xx * xx + yy * yy > r2_lim;
  };
  float est[E][2], top = -1.f;  // float estimates, and the largest of the warp
#pragma unroll
  for (int i = 0; i < E; i++) {
    float2 z[2];
    cp_split(v[i], z[0], z[1]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      est[i][h] = inside(i, h) ? sqrtf(z[h].x * z[h].x + z[h].y * z[h].y) : -1.f;
      top = fmaxf(top, est[i][h]);
    }
  }
  if constexpr (NT % 32 == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  }
  float best = -1.f;
  int bi = 0x7fffffff;
#pragma unroll
  for (int i = 0; i < E; i++) {
    float2 z[2];
    cp_split(v[i], z[0], z[1]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      // NaN estimates fail every comparison, as the reference's
      if (est[i][h] >= 0.f && est[i][h] >= top * (1.f - 1e-6f)) {
        const float m = (float)sqrt((double)z[h].x * z[h].x + (double)z[h].y * z[h].y);
        const int id = (t + i * T) * N + x + h;
        if (m > best || (m == best && id < bi)) {
          best = m;
          bi = id;
        }
      }
    }
  }
  float* sm = reinterpret_cast<float*>(smp);  // the transform is done with the buffer
  int* si = reinterpret_cast<int*>(sm + NT);
  sm[lt] = best;
  si[lt] = bi;
  __syncthreads();
  for (int n = NT; n > 1;) {  // any thread count
    const int h = (n + 1) / 2;
    if (lt + h < n && (sm[lt + h] > sm[lt] || (sm[lt + h] == sm[lt] && si[lt + h] < si[lt]))) {
      sm[lt] = sm[lt + h];
      si[lt] = si[lt + h];
    }
    __syncthreads();
    n = h;
  }
  if (lt == 0) {
    A.pmag[(size_t)a * gridDim.x + blockIdx.x] = sm[0];
    A.pidx[(size_t)a * gridDim.x + blockIdx.x] = si[0];
  }
}
// locatePeak's result as fitPeak's start (-x, -y), search width 2.5
__global__ void __launch_bounds__(256) k_fit_start(const __grid_constant__ FitArgs A, int nb, int n, double dist) {
  __shared__ float sm[256];
  __shared__ int si[256];
  const int i = threadIdx.x, a = blockIdx.x;
  float best = -1.f;
  int bi = 0x7fffffff;
  for (int k = i; k < nb; k += 256) {
    const float m = A.pmag[(size_t)a * nb + k];
    const int id = A.pidx[(size_t)a * nb + k];
    if (m > best || (m == best && id < bi)) {
      best = m;
      bi = id;
    }
  }
  sm[i] = best;
  si[i] = bi;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (i < o && (sm[i + o] > sm[i] || (sm[i + o] == sm[i] && si[i + o] < si[i]))) {
      sm[i] = sm[i + o];
      si[i] = si[i + o];
    }
    __syncthreads();
  }
  double xPos = -0., yPos = -1;
  if (si[0] != 0x7fffffff && sm[0] >= 0) {
    xPos = si[0] % n;
    yPos = si[0] / n;
  }
  if (xPos > n / 2) xPos = xPos - n;
  if (yPos > n / 2) yPos = n - yPos;
  else yPos *= -1;
  if (i == 0) {
    A.dir[a].phase = 0;
    A.dir[a].mag = 0;
  }
  fit_setup(A.dir[a], -xPos, -yPos, 2.5, dist, n);
}
// One block per grid point and direction: sum_y Q[jx][y] ty[jy][y] in FP64 in a fixed order. The last
// block of a direction sums norm2, scans the normalised grid in the reference's order (yi outer,
// xi inner, strict >: the largest value, the first of equals; Correlation.java:104-132) and sets up
// the next step; after the last one it stores the fit and sets up getPeak at `scale` times it.
__global__ void __launch_bounds__(128) k_fit_grid(const __grid_constant__ FitArgs A, int n, int step, double dist,
                                                  double scale) {
  constexpr int NT = 128;
  const int g = blockIdx.x, a = blockIdx.y, i = threadIdx.x, lane = i % 32, wp = i / 32;
  const int jx = g % NG, jy = g / NG;
  FitDir& d = A.dir[a];
  const double2* Q = A.Q + ((size_t)a * NG + jx) * n;
  const float2* ty = A.ramps + ((size_t)a * NR + NG + jy) * n;
  double re = 0, im = 0;
  for (int y = i; y < n; y += NT) {
    const double2 q = Q[y];
    const float2 r = ty[y];
    re += q.x * r.x - q.y * r.y;
    im += q.x * r.y + q.y * r.x;
  }
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  __shared__ double part[NT / 32][2];
  __shared__ int last;
  if (lane == 0) {
    part[wp][0] = re;
    part[wp][1] = im;
  }
  __syncthreads();
  if (i == 0) {
    d.corr[g] = make_double2((part[0][0] + part[1][0]) + (part[2][0] + part[3][0]),
                             (part[0][1] + part[1][1]) + (part[2][1] + part[3][1]));
    __threadfence();
    last = atomicAdd(&d.done, 1) == NG * NG - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double hv[NT];
  __shared__ int hi[NT];
  double nn = 0;
  for (int y = i; y < n; y += NT) nn += A.n2[(size_t)a * n + y];
  for (int o = 16; o > 0; o >>= 1) nn += __shfl_down_sync(0xffffffffu, nn, o);
  if (lane == 0) part[wp][0] = nn;
  __syncthreads();
  const double sc = 1. / ((part[0][0] + part[1][0]) + (part[2][0] + part[3][0]));
  const volatile double2* cv = d.corr;
  hv[i] = -1.;
  if (i < NG * NG) hv[i] = hypot(cv[i].x * sc, cv[i].y * sc);
  if (!(hv[i] > 0)) hv[i] = -1.;  // the reference starts at 0 with a strict >; NaN never wins
  hi[i] = i;
  __syncthreads();
  for (int o = NT / 2; o > 0; o >>= 1) {
    if (i < o && (hv[i + o] > hv[i] || (hv[i + o] == hv[i] && hi[i + o] < hi[i]))) {
      hv[i] = hv[i + o];
      hi[i] = hi[i + o];
    }
    __syncthreads();
  }
  const int best = hv[0] > 0 ? hi[0] : -1;
  const double kx = best >= 0 ? d.kxs[best % NG] : 0., ky = best >= 0 ? d.kys[best / NG] : 0., search = d.search / 5;
  __syncthreads();  // every thread has the shifts before they are replaced
  if (i == 0) {
    if (best >= 0) {
      d.phase = atan2(cv[best].y, cv[best].x);
      d.mag = hv[0];
    }
    if (step == 2) {
      double* res = A.results + 8 * a;
      res[0] = kx;
      res[1] = ky;
      res[2] = d.phase;
      res[3] = d.mag;
    }
  }
  // getPeak's one shift is the fit times a power of two
  if (step == 2) fit_setup(d, kx * scale, ky * scale, 0., dist, n);
  else fit_setup(d, kx, ky, search, dist, n);
}

// ---- getPeak (Correlation.java:183-209) ---------------------------------------------------------
// Common region of both bands into single planes, and the two ramps of the shift.
template <int N>
__global__ void __launch_bounds__(128) k_fit_region(const ulonglong2* __restrict__ S, float2* __restrict__ b,
                                                    const __grid_constant__ FitArgs A, double dist) {
  const int x = blockIdx.x * 128 + threadIdx.x, y = blockIdx.y, a = blockIdx.z;
  if (x >= N) return;
  const FitDir& d = A.dir[a];
  if (y < 2) A.ramps[((size_t)a * NR + NG * y) * N + x] = ramp_at(y == 0 ? d.kxs[0] : -d.kys[0], x, N);
  const size_t n = (size_t)N * N, i = (size_t)y * N + x;
  const Region R = region_of<N>(d.cp, dist);
  const float2 f = p_unpack(common_factor<N>(A, R, x, y));
  const ulonglong2 u = __ldg(S + a * n + i);
  const float2 re = p_unpack(u.x), im = p_unpack(u.y);
  // (a bin that is cut is +0, whatever its sign was)
  b[(2 * a) * n + i] = f.x == 0.f ? make_float2(0.f, 0.f) : make_float2(__fmul_rn(re.x, f.x), __fmul_rn(im.x, f.x));
  b[(2 * a + 1) * n + i] = f.y == 0.f ? make_float2(0.f, 0.f) : make_float2(__fmul_rn(re.y, f.y), __fmul_rn(im.y, f.y));
}
// Row norms of b0: the float squares added as a sum of two floats (exact to 2^-45), then in FP64. The
// row sums of b1 conj(b0) are k_corr_rows' (corr_grid.cuh).
__global__ void __launch_bounds__(256) k_fit_norm(const float2* __restrict__ b, int n, const __grid_constant__ FitArgs A) {
  const int lane = threadIdx.x % 32, y = blockIdx.x * 8 + threadIdx.x / 32, a = blockIdx.y;
  if (y >= n) return;  // uniform per warp
  const float2* b0 = b + ((size_t)(2 * a) * n + y) * n;
  float s = 0.f, e = 0.f;
  for (int x = lane; x < n; x += 32) {
    const float2 v = b0[x];
    float t, z;
    ff_two_sum(s, __fmul_rn(v.x, v.x), t, z);
    e = __fadd_rn(e, z);
    ff_two_sum(t, __fmul_rn(v.y, v.y), s, z);
    e = __fadd_rn(e, z);
  }
  double nn = (double)s + (double)e;
  for (int o = 16; o > 0; o >>= 1) nn += __shfl_down_sync(0xffffffffu, nn, o);
  if (lane == 0) A.n2[(size_t)a * n + y] = nn;
}
// The sum over rows, normalised, to results[out], [out + 1]; then the next band's getPeak (scale != 0).
__global__ void __launch_bounds__(128) k_fit_peak_sum(const __grid_constant__ FitArgs A, int n, int out, double dist,
                                                      double scale) {
  constexpr int NT = 128;
  const int a = blockIdx.x, i = threadIdx.x, lane = i % 32, wp = i / 32;
  FitDir& d = A.dir[a];
  double* res = A.results + 8 * a;
  const double2* Q = A.Q + (size_t)a * NG * n;
  const float2* ty = A.ramps + ((size_t)a * NR + NG) * n;
  double v[3] = {0, 0, 0};
  for (int y = i; y < n; y += NT) {
    const double2 q = Q[y];
    const float2 r = ty[y];
    v[0] += q.x * r.x - q.y * r.y;
    v[1] += q.x * r.y + q.y * r.x;
    v[2] += A.n2[(size_t)a * n + y];
  }
  __shared__ double part[3][NT / 32];
  for (int k = 0; k < 3; k++) {
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0) part[k][wp] = v[k];
  }
  __syncthreads();
  if (i == 0) {
    for (int k = 0; k < 3; k++) v[k] = (part[k][0] + part[k][1]) + (part[k][2] + part[k][3]);
    const double sc = 1. / v[2];
    res[out] = v[0] * sc;
    res[out + 1] = v[1] * sc;
  }
  if (scale != 0) fit_setup(d, res[0] * scale, res[1] * scale, 0., dist, n);
}
// 1 / OTF inside the weight limit, 0 beyond (Cplx.Float.reciproc's real part)
__global__ void k_fit_weight(float* __restrict__ w, int n, const OtfTable* __restrict__ otf, float wlf) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= n) return;
  float2 c;
  const float v = otf_at_fast(*otf, 0, freq_x(x, n), freq_y(y, n), FShift{0.f, 0.f, 0.f, 0.f}, 0, 0, false, &c) ? c.x : 0.f;
  w[(size_t)y * n + x] = fabsf(v) < wlf ? 0.f : __fdiv_rn(v, __fmul_rn(v, v));
}

struct FitBuf {  // planes and tables of one call, one allocation
  ulonglong2 *S = nullptr, *L = nullptr, *W = nullptr;
  float2* V = nullptr;  // the coarse product, then getPeak's two bands per direction
  FitArgs A{};
  double* fx = nullptr;
  float* fy = nullptr;
  void* base = nullptr;
};

struct PeakTask {  // getPeak of (band 0, a band) at the fit's shift times scale, results to out, out + 1
  const ulonglong2* S;
  double scale;
  int out;
};

template <int N>
int fit_run(const SpecIn& spec, const MixCoef& fitted, const MixCoef* other, int nA, int nP, const FitBuf& B,
            long long r2_lim, const PeakTask* task, int ntask, cudaStream_t st) {
  using P = FCfg<N>;
  constexpr size_t E16 = sizeof(ulonglong2);
  constexpr int PB = N / (2 * P::C);  // peak blocks
  constexpr size_t sm_row = E16 * P::G * P::XS, sm_col = E16 * P::XC;
  constexpr size_t sm_q = sm_row + sizeof(float) * P::G * NV * (P::T + 1);
  constexpr size_t sm_peak = std::max(sm_col, (size_t)P::C * P::T * 8);
  static bool attr = false;
  if (!attr) {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    FSIM_CUDA(cudaFuncSetAttribute(k_fit_cols<N, false>, a, (int)sm_col));
    FSIM_CUDA(cudaFuncSetAttribute(k_fit_cols<N, true>, a, (int)sm_col));
    FSIM_CUDA(cudaFuncSetAttribute(k_fit_rows_product<N>, a, (int)sm_row));
    FSIM_CUDA(cudaFuncSetAttribute(k_fit_rows<N>, a, (int)sm_q));
    FSIM_CUDA(cudaFuncSetAttribute(k_fit_peak<N>, a, (int)sm_peak));
    attr = true;
  }
  const dim3 gr(N / P::G, nA), gc(N / P::C, nA);
  const int nr = P::G * P::T, nc = P::C * P::T;
  const double dist = 0.15;
  const dim3 gsep(std::max(1, 8 * ctx().num_sms / nA), nA);
  k_fit_separate<<<gsep, 256, 0, st>>>(spec, fitted, nP, (size_t)N * N, B.S);
  if (other) k_fit_separate<<<gsep, 256, 0, st>>>(spec, *other, nP, (size_t)N * N, B.L);
  k_fit_cols<N, false><<<gc, nc, sm_col, st>>>(B.S, B.W, B.A, dist);
  k_fit_rows_product<N><<<gr, nr, sm_row, st>>>(B.W, B.V);
  k_fit_peak<N><<<dim3(PB, nA), nc, sm_peak, st>>>(B.V, r2_lim, B.A);
  k_fit_start<<<nA, 256, 0, st>>>(B.A, PB, N, dist);
  for (int step = 0; step < 3; step++) {
    k_fit_cols<N, true><<<dim3(NR + N / P::C, nA), nc, sm_col, st>>>(B.S, B.W, B.A, dist);
    k_fit_rows<N><<<gr, nr, sm_q, st>>>(B.W, B.A);
    k_fit_grid<<<dim3(NG * NG, nA), 128, 0, st>>>(B.A, N, step, dist, task[0].scale);
  }
  for (int k = 0; k < ntask; k++) {
    k_fit_region<N><<<dim3(div_up(N, 128), N, nA), 128, 0, st>>>(task[k].S, B.V, B.A, dist);
    FSIM_CHECK_LAUNCH();
    int rc = fft2d_lines_device(B.V, N, st, 2 * nA, nullptr);
    if (rc) return rc;
    k_fit_norm<<<dim3(N / 8, nA), 256, 0, st>>>(B.V, N, B.A);
    for (int a = 0; a < nA; a++)
      k_corr_rows<1><<<N / CORR_ROWS_PER_BLOCK, 32 * CORR_ROWS_PER_BLOCK, 0, st>>>(
          B.V + (size_t)(2 * a) * N * N, B.V + (size_t)(2 * a + 1) * N * N, B.A.ramps + (size_t)a * NR * N, N, 1,
          B.A.Q + (size_t)a * NG * N);
    k_fit_peak_sum<<<nA, 128, 0, st>>>(B.A, N, task[k].out, dist, k + 1 < ntask ? task[k + 1].scale : 0.);
  }
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

#define FSIM_FIT_SIZES(X) X(128) X(256) X(384) X(512) X(768) X(1024) X(2048)

}  // namespace

bool fit_pairs_supported(const fsim_sim_param* p, int fade_px) {
  if (otf_measured(p) || fade_px < 0 || 2 * fade_px > p->w) return false;
  switch (p->w) {
#define CASE(v) case v:
    FSIM_FIT_SIZES(CASE)
#undef CASE
    return true;
    default:
      return false;
  }
}

// Fits every direction; res receives 8 doubles per direction: kx, ky, phase, magnitude of fitPeak,
// getPeak of the low band (4, 5) and of the high one (6, 7). Synchronises st.
int fit_pairs(const fsim_sim_param* p, const FitSource& src, int fit_band, double fit_exclude, bool live, double* res,
              cudaStream_t st) {
  const int N = p->w, nA = p->nr_dirs, nP = p->nr_phases, nB = p->nr_bands;
  const size_t n = (size_t)N * N;
  const int lb = 1, hb = (nB == 3) ? 3 : 1;
  const int fb = live ? hb : (fit_band == 1 ? lb : hb);
  // planes: S (band 0, fitted band) and, where getPeak takes another band, L (band 0, that band)
  const int other = !live && lb != hb ? (fb == lb ? hb : lb) : (fb != lb ? lb : -1);
  auto coef = [&](int comp) {
    MixCoef m{};
    for (int a = 0; a < nA; a++) {
      const auto c = separation_coeffs(p, a, true);  // phaOff 0, fac null
      for (int q = 0; q < nP; q++) {
        m.c[a][0][q] = make_float2(c[q].real(), c[q].imag());
        m.c[a][1][q] = make_float2(c[comp * nP + q].real(), c[comp * nP + q].imag());
      }
    }
    return m;
  };
  const MixCoef cf = coef(fb), co = other >= 0 ? coef(other) : MixCoef{};
  // the estimated OTF falls with the radius: its sample first below the weight limit gives the
  // squared distance of the limit; unknown unless every other sample clears the limit by 1e-6
  OtfTable ht;
  build_otf_table(p, &ht);
  const double wl = 0.05;
  const float wlf = (double)(float)wl < wl ? std::nextafter((float)wl, INFINITY) : (float)wl;
  int lthr = 0;
  while (lthr < OTF_SAMPLES && ht.vals[lthr] >= wlf) lthr++;
  bool sure = true;
  for (int l = 0; l < OTF_SAMPLES; l++)
    sure = sure && (l < lthr ? ht.vals[l] > wl * (1 + 1e-6) : ht.vals[l] < wl * (1 - 1e-6));
  if (lthr + 1 >= OTF_SAMPLES) sure = false;
  const double dl = lthr * ht.cycles_per_sample / ht.vec_cpm;
  // the last r^2 with sqrt((double)r^2) <= kMin (locatePeak's radius test)
  const double kmin = fit_exclude * ht.cutoff / ht.vec_cpm;
  long long lo = -1, hi = 2 * (long long)(N / 2) * (N / 2);
  while (lo < hi) {
    const long long m = hi - (hi - lo) / 2;
    if (std::sqrt((double)m) > kmin) hi = m - 1;
    else lo = m;
  }
  // one allocation; OTF table and border fade together (one upload)
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t plane = al(sizeof(ulonglong2) * n * nA);
  // the frames' spectra are separated before the work planes W and V are written: they share memory
  const size_t spectra = src.raw ? al(sizeof(float2) * n * nA * nP) : 0, work = plane + al(sizeof(float2) * n * 2 * nA);
  // an estimated OTF's table ends before the measured bands
  const size_t o_fx = al(offsetof(OtfTable, mvals)), o_fy = o_fx + sizeof(double) * N, consts = al(o_fy + sizeof(float) * N);
  const size_t sizes[] = {plane, other >= 0 ? plane : 0, plane, std::max(spectra, work) - plane, al(sizeof(float) * n),
                          al(sizeof(float) * n), al(sizeof(float2) * NR * N * nA), al(sizeof(double2) * NG * N * nA),
                          al(sizeof(double) * N * nA), al(sizeof(float) * N * nA), al(sizeof(int) * N * nA),
                          al(sizeof(FitDir) * nA), al(sizeof(double) * 8 * nA), consts};
  size_t total = 0;
  for (size_t s : sizes) total += s;
  FitBuf B;
  cudaError_t e = fsim::dev_alloc_async(&B.base, total, st);
  if (e != cudaSuccess) {
    set_error("parameter fit scratch (%zu bytes): %s", total, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? FSIM_EOOM : FSIM_ECUDA;
  }
  char* q = (char*)B.base;
  void* ptr[14];
  for (int i = 0; i < 14; i++) {
    ptr[i] = q;
    q += sizes[i];
  }
  B.S = (ulonglong2*)ptr[0];
  B.L = (ulonglong2*)ptr[1];
  B.W = (ulonglong2*)ptr[2];
  B.V = (float2*)ptr[3];
  float *d_att = (float*)ptr[4], *d_weight = (float*)ptr[5];
  B.A.att = d_att;
  B.A.weight = d_weight;
  B.A.ramps = (float2*)ptr[6];
  B.A.Q = (double2*)ptr[7];
  B.A.n2 = (double*)ptr[8];
  B.A.pmag = (float*)ptr[9];
  B.A.pidx = (int*)ptr[10];
  B.A.dir = (FitDir*)ptr[11];
  B.A.results = (double*)ptr[12];
  OtfTable* d_otf = (OtfTable*)ptr[13];
  B.A.otf = d_otf;
  B.A.wlf = wlf;
  B.A.d2_keep = (float)(dl * dl * (1 - 4e-6));
  B.A.d2_drop = sure ? (float)(dl * dl * (1 + 4e-6)) : -1.f;
  auto run = [&]() -> int {
    std::vector<char> host(consts);
    std::memcpy(host.data(), &ht, offsetof(OtfTable, mvals));
    if (src.raw && src.fade_px > 0) {  // fadeBorderCos as a float row factor and a double column factor
      double* fx = reinterpret_cast<double*>(host.data() + o_fx);
      float* fy = reinterpret_cast<float*>(host.data() + o_fy);
      std::fill(fx, fx + N, 1.0);
      std::fill(fy, fy + N, 1.f);
      const double fac = 1. / src.fade_px * M_PI / 2.;
      for (int i = 0; i < src.fade_px; i++) {
        const double c = std::pow(std::sin(i * fac), 2);
        fx[i] = fx[N - 1 - i] = c;
        fy[i] = fy[N - 1 - i] = (float)c;
      }
    }
    FSIM_CUDA(cudaMemcpyAsync(d_otf, host.data(), consts, cudaMemcpyHostToDevice, st));
    B.fx = reinterpret_cast<double*>((char*)d_otf + o_fx);
    B.fy = reinterpret_cast<float*>((char*)d_otf + o_fy);
    SpecIn spec{};
    if (src.raw) {
      RawFade rf;
      rf.raw = src.raw;
      rf.u16 = src.u16;
      rf.fade = src.fade_px;
      rf.fx = B.fx;
      rf.fy = B.fy;
      float2* sp = reinterpret_cast<float2*>(B.W);
      int rc = fft2d_lines_device(sp, N, st, nA * nP, &rf);
      if (rc) return rc;
      for (int i = 0; i < nA * nP; i++) spec.in[i] = sp + i * n;
    } else {
      for (int i = 0; i < nA * nP; i++) spec.in[i] = src.spec[i];
    }
    // otfAtt = writeAttenuationVector(.99, 0.15*cutoff, 0, 0) (SimAlgorithm.java:65-66)
    int rc = att_device(d_att, N, N, ht.vec_cpm, .99, 0.15 * ht.cutoff, 0, 0, st);
    if (rc) return rc;
    k_fit_weight<<<dim3(div_up(N, 128), N), 128, 0, st>>>(d_weight, N, d_otf, wlf);
    FSIM_CHECK_LAUNCH();
    // getPeak of the low band and, in a three-band fit, of the high one, each at the fit scaled to
    // the band's shift
    PeakTask task[2];
    int ntask = 0;
    auto peak = [&](int comp, double scale, int out) { task[ntask++] = PeakTask{comp == fb ? B.S : B.L, scale, out}; };
    if (live) {
      peak(lb, 1.0 / (nB - 1), 4);
    } else if (lb != hb) {
      const double f2 = fit_band == 1 ? 2.0 : 1.0;  // the host doubles a band-1 fit
      peak(lb, f2 / 2, 4);
      peak(hb, f2, 6);
    } else {
      peak(lb, 1.0, 4);
    }
    switch (N) {
#define CASE(v)                                                                                              \
  case v:                                                                                                    \
    rc = fit_run<v>(spec, cf, other >= 0 ? &co : nullptr, nA, nP, B, lo, task, ntask, st);                    \
    break;
      FSIM_FIT_SIZES(CASE)
#undef CASE
    }
    if (rc) return rc;
    FSIM_CUDA(cudaMemcpyAsync(res, B.A.results, sizeof(double) * 8 * nA, cudaMemcpyDeviceToHost, st));
    FSIM_CUDA(cudaStreamSynchronize(st));
    return FSIM_OK;
  };
  int rc = run();
  cudaFreeAsync(B.base, st);
  return rc;
}

}  // namespace fsim
