// Fused live reconstruction: the per-stack work of ReconstructionThread.run
// (LM/ReconstructionRunner.java:434-542) with the filters of setupFilters (:773-813):
// u16 frames x border damping, FFT_N, band separation, times conj(OTF) (band 0,
// attenuated), the *fast* shift of SimUtils.pasteAndFourierShift (S/SimUtils.java:65-91:
// fractional shift on the N grid, then pasteFreq at the integer offset), sum, times
// Wiener denominator and apodization (bend 1, cutoff 2), iFFT_W, real part; plus the
// widefield mean of the damped frames.
//
// The fractional shift FFT_N(ramp * iFFT_N(.)) is separable, but the OTF product sits
// between the forward transforms and the shift, so four passes are used:
//   LA rows    (per dataset x raw row pair):  damp, widefield, band mix, FFT_N along x
//   LB columns (per dataset x 4 columns):     FFT_N along y, x conj(OTF), y half of the shift
//   LC rows    (per dataset x output row pair): x half of the shift, paste at the integer
//                                             offsets, sum, x Wiener*apo, iFFT_W along x
//   LD columns (per dataset x columns):       complex-to-real inverse along y, 1/W^2
// Three symmetries leave 4 of the 9 components of a 3 x 3 stack, and half of the output grid:
//  * band 0 of every angle has the same OTF and no shift: the angles are summed before LA's
//    transform;
//  * the neg component of a band pair is the conjugate of the pos one in real space, and the
//    fast shift's two ramps are conjugates up to a whole bin: with V the shifted pos spectrum,
//    fx = kx - floor(kx), dx = (fx != 0) and likewise along y,
//      V_neg[m, n] = conj V[dx - m, dy - n]   (indices modulo N),
//    pasted at -floor(kx) - dx. So V sits at X = floor(kx) + p, p in [-N/2, N/2 - 1], and its
//    conjugate mirror image at X = -(floor(kx) + p), p in [dx - N/2 + 1, dx + N/2];
//  * the image is real: only H(X, Y) = (F(X, Y) + conj F(-X, -Y)) / 2 matters, to which V[p]
//    contributes at +-(floor(k) + p) with weight 1, or 1/2 for the bins on the edge of the two
//    ranges, and only the rows Y = 0..N of H are formed (LD completes each column by symmetry).
// The OTF also zeroes every column beyond its support: only a window of columns leaves LA.
// Rows (LA, LC) and columns (LB, LD) are transformed two at a time (fft_pair.cuh). Bound by the
// shared-memory pipe and instruction issue of 11.6k transforms of length N per 512^2 3x3 stack (26k
// with every component and the full grid): 64 stacks in 1069 us on GB300, 2382 us before; one
// stack 62.6 us, 109 before.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "fft_pair.cuh"
#include "filters.cuh"
#include "otf.cuh"
#include "recon.cuh"
#include "runtime.cuh"
#include "sim_host.h"

namespace fsim {

std::vector<float> fade_vector(int w, int h, int px);
int plan_window(const fsim_sim_param* p, double R, int* nwin);

template <int N>
struct LCfg {
  static constexpr int W = 2 * N;
  static constexpr int E = (N % 3 == 0) ? 12 : 8;
  static constexpr int T = N / E;                   // threads per line pair
  static constexpr int G = T >= 64 ? 1 : 64 / T;    // row pairs per block, passes LA and LC
  static constexpr int CP = 2;                      // column pairs per block, pass LB
  static constexpr int CD = N >= 2048 ? 2 : 4;      // column pairs per block, pass LD
  // Registers per thread at 8 elements: 64 in passes LB and LD (against 80, 64 x 512^2: 217 -> 212 and
  // 129 -> 125 us; 16 x 1024^2: 305 -> 301 and 186 -> 152), 96 in pass LA, which keeps two frames' pixels in
  // flight while it mixes (64 x 512^2: 361 -> 318 us; three frames 342), and 128 in pass LC, which
  // loads the next contribution during a transform (474 -> 436 us; 531 at 80, where it spills).
  static constexpr int RA = 96, RC = 128, F = 2;
  static constexpr int blocks(int threads, int regs8 = 64) {
    const int n = threads < 32 ? 32 : threads, b = 65536 / (n * (E <= 8 ? regs8 : 128));
    return b < 1 ? 1 : (b > 32 ? 32 : b);
  }
  static constexpr int XS = pair_elems(N, 1);       // exchange buffer of one pair
};
// window column of spectrum column m (nWin columns from Xs, modulo N), or beyond nWin
template <int N>
__device__ __forceinline__ int live_col(int m, int Xs) {
  const int x = m - Xs;
  return x < 0 ? x + N : x;
}

// ---- LA -----------------------------------------------------------------------------------
// blockIdx.y < nA: the pos components of that angle; blockIdx.y == nA: band 0 of all angles, and
// the widefield.
template <int N>
__global__ void __launch_bounds__(LCfg<N>::G* LCfg<N>::T, LCfg<N>::blocks(LCfg<N>::G* LCfg<N>::T, LCfg<N>::RA))
    k_live_a(const JobDesc* __restrict__ jobs) {
  using P = LCfg<N>;
  constexpr int T = P::T, G = P::G, E = P::E;
  const JobDesc& J = jobs[blockIdx.z];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int y = 2 * (blockIdx.x * G + g), a = blockIdx.y;
  extern __shared__ ulonglong2 smp[];
  ulonglong2* s = smp + g * P::XS;
  const float2* tw = g_stw + stw_offset(N, E);  // stage twiddles through L1
  const size_t frame = (size_t)N * N, row = (size_t)y * N;
  const int nA = J.nA, nP = J.nP, nC = J.nC, nPair = (nC - 1) / 2, nWin = J.nWin, Xs = J.win[0];
  if (a > nA) return;  // uniform per block
  // setFrom16bitPixels + times(dampBorder) of both rows of frame f at this thread's elements
  // t + i*T; frames outer and elements inner, so that the rows' loads are in flight at once
  auto px_rows = [&](int f, f32x2 (&v)[E]) {
    const size_t at = (size_t)f * frame + row + t;
    if (J.input_u16) {
      const uint16_t* r = (const uint16_t*)J.raw + at;
#pragma unroll
      for (int i = 0; i < E; i++) v[i] = p_pack((float)__ldg(r + i * T), (float)__ldg(r + N + i * T));
    } else {
      const float* r = (const float*)J.raw + at;
#pragma unroll
      for (int i = 0; i < E; i++) v[i] = p_pack(__ldg(r + i * T), __ldg(r + N + i * T));
    }
    if (J.damp) {
      const float* d = J.damp + row + t;
#pragma unroll
      for (int i = 0; i < E; i++) v[i] = p_mul(v[i], p_pack(__ldg(d + i * T), __ldg(d + N + i * T)));
    }
  };
  // frames f0 .. f0 + nf - 1, several frames' loads in flight at once
  auto mix = [&](int f0, int nf, auto add) {
    constexpr int F = P::F;
    int f = f0;
#pragma unroll 1
    for (; f + F <= f0 + nf; f += F) {
      f32x2 v[F][E];
#pragma unroll
      for (int k = 0; k < F; k++) px_rows(f + k, v[k]);
#pragma unroll
      for (int k = 0; k < F; k++) add(v[k], f + k);
    }
#pragma unroll 1
    for (; f < f0 + nf; f++) {
      f32x2 v[E];
      px_rows(f, v);
      add(v, f);
    }
  };
  // both rows' value of the window columns, to the quad layout [xl/4][y][xl%4]
  cpair x[E];  // element t + i*T of both rows, in registers through the transform
  auto put = [&](int slot) {
    float2* I = J.I + (size_t)slot * nWin * N;
#pragma unroll
    for (int i = 0; i < E; i++) {
      const int xl = live_col<N>(t + i * T, Xs);
      if (xl < nWin) {
        float2 r0, r1;
        cp_split(x[i], r0, r1);
        float2* o = I + ((size_t)(xl >> 2) * N + y) * 4 + (xl & 3);
        o[0] = r0;
        o[4] = r1;
      }
    }
  };
  if (a == nA) {
    f32x2 wf[E];
#pragma unroll
    for (int i = 0; i < E; i++) {
      x[i] = cp_zero();
      wf[i] = 0ull;
    }
    auto add = [&](const f32x2 (&v)[E], int f) {
      const wpair m = w_dup(__ldg(J.coef + (f / nP) * nC * nP + f % nP));
#pragma unroll
      for (int i = 0; i < E; i++) {
        wf[i] = p_add(wf[i], v[i]);
        x[i] = cpair{p_fma(m.x, v[i], x[i].re), p_fma(m.y, v[i], x[i].im)};
      }
    };
    mix(0, nA * nP, add);
    if (J.widefield) {
      const f32x2 sc = p_dup(1.f / (float)(nA * nP));
#pragma unroll
      for (int i = 0; i < E; i++) {
        const float2 w = p_unpack(p_mul(wf[i], sc));
        J.widefield[row + t + i * T] = w.x;
        J.widefield[row + N + t + i * T] = w.y;
      }
    }
    line_fft_pair<N, T, 1, false>(x, s, 0, t, tw);
    put(0);
    return;
  }
  for (int b = 1; b <= nPair; b++) {
    const float2* coef = J.coef + (a * nC + 2 * b) * nP;
#pragma unroll
    for (int i = 0; i < E; i++) x[i] = cp_zero();
    mix(a * nP, nP, [&](const f32x2 (&v)[E], int f) {
      const wpair m = w_dup(__ldg(coef + (f - a * nP)));
#pragma unroll
      for (int i = 0; i < E; i++) x[i] = cpair{p_fma(m.x, v[i], x[i].re), p_fma(m.y, v[i], x[i].im)};
    });
    line_fft_pair<N, T, 1, false>(x, s, 0, t, tw);
    put(1 + a * nPair + (b - 1));
  }
}

// ---- LB -----------------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(LCfg<N>::CP* LCfg<N>::T, LCfg<N>::blocks(LCfg<N>::CP* LCfg<N>::T))
    k_live_b(const JobDesc* __restrict__ jobs) {
  using P = LCfg<N>;
  constexpr int T = P::T, C = P::CP, E = P::E;
  const JobDesc& J = jobs[blockIdx.z];
  const int lt = threadIdx.x, lane = lt % C, t = lt / C;
  const int nPair = (J.nC - 1) / 2, nWin = J.nWin, slot = blockIdx.y;
  if (slot > J.nA * nPair || (int)blockIdx.x * 2 * C >= nWin) return;  // uniform per block
  const int xl = blockIdx.x * 2 * C + 2 * lane;  // and xl + 1: nWin is a multiple of 4
  extern __shared__ ulonglong2 smp[];
  const float2* tw = g_stw + stw_offset(N, E);
  // rows two float4 apart; the columns are this block's alone and are transformed in place
  float4* I = reinterpret_cast<float4*>(J.I + (size_t)slot * nWin * N + ((size_t)(xl >> 2) * N) * 4 + (xl & 3));
  cpair x[E];  // element t + i*T of both columns, in registers through the transforms
#pragma unroll
  for (int i = 0; i < E; i++) {
    const float4 v = I[(size_t)(t + i * T) * 2];
    x[i] = cpair{p_pack(v.x, v.z), p_pack(v.y, v.w)};
  }
  line_fft_pair<N, T, C, false>(x, smp, lane, t, tw);
  // times conj(OTF): the OTF vector is real (estimate); band 0 carries its weight 1/2
  const float* o = J.masks + (size_t)xl * N + t;
  const float h = slot == 0 ? 0.5f : 1.f;
#pragma unroll
  for (int i = 0; i < E; i++) {
    const f32x2 f = p_pack(h * __ldg(o + i * T), h * __ldg(o + N + i * T));
    x[i] = cpair{p_mul(x[i].re, f), p_mul(x[i].im, f)};
  }
  if (slot > 0) {
    line_fft_pair<N, T, C, true>(x, smp, lane, t, tw);
    const float2* ry = J.ramps + (size_t)(slot - 1) * 2 * N + N;
#pragma unroll
    for (int i = 0; i < E; i++) x[i] = cmul(x[i], w_dup(__ldg(ry + t + i * T)));
    line_fft_pair<N, T, C, false>(x, smp, lane, t, tw);
  }
#pragma unroll
  for (int i = 0; i < E; i++) {
    float2 r0, r1;
    cp_split(x[i], r0, r1);
    I[(size_t)(t + i * T) * 2] = make_float4(r0.x, r0.y, r1.x, r1.y);
  }
}

// ---- LC -----------------------------------------------------------------------------------
// One row pair (Y, Y + 1) of H per group of T threads, Y even, Y <= N. The rows of a slot that
// land on them directly (row Y - floor(ky)) or mirrored (row -Y - floor(ky)) are transformed as
// a pair and added to the rows' sums in shared memory; then x Wiener*apo, and iFFT_W along x as
// two N-point inverse transforms (even and odd samples).
template <int N>
struct LCPass {
  using P = LCfg<N>;
  static constexpr int NT = P::G * P::T;
  static constexpr int GS = P::XS + 2 * N;  // exchange buffer and the sums of a row pair
  static constexpr size_t SMEM = sizeof(ulonglong2) * (size_t)P::G * GS;
};
template <int N>
__global__ void __launch_bounds__(LCPass<N>::NT, LCfg<N>::blocks(LCPass<N>::NT, LCfg<N>::RC))
    k_live_c(const JobDesc* __restrict__ jobs) {
  using P = LCfg<N>;
  constexpr int W = P::W, T = P::T, E = P::E, G = P::G;
  const JobDesc& J = jobs[blockIdx.y];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int Y0 = 2 * (blockIdx.x * G + g);  // rows Y0 and Y0 + 1; stored up to row N
  extern __shared__ ulonglong2 smp[];
  ulonglong2* s = smp + g * LCPass<N>::GS;
  ulonglong2* acc = s + P::XS;  // (re, im) of both rows, W columns
  const float2* tw = g_stw + stw_offset(N, E);
  const float2* twW = g_tw + tw_offset(W);
  const int nPair = (J.nC - 1) / 2, nWin = J.nWin, Xs = J.win[0], nS = 1 + J.nA * nPair;
  const float* wa = J.wa;
  auto wrap = [](int v) { return v < 0 ? v + W : (v >= W ? v - W : v); };
#pragma unroll
  for (int i = 0; i < 2 * E; i++) acc[t + i * T] = make_ulonglong2(0ull, 0ull);
  // Contribution k: slot k / 2, direct (even k) or mirrored (odd), from the slot's rows q[0], q[1]
  // relative to its origin. Rows are in the pos range [-N/2, N/2 - 1], in the neg range
  // [dy - N/2 + 1, dy + N/2] (band 0: the pos range only, its mirror image included); wp, wn: weights
  // of an element inside the pos / the neg x range.
  struct Part {
    int sl, mir, xi, dx, q[2];
    float wp[2], wn[2];
    bool any;
  };
  auto part = [&](int k) {
    Part c;
    c.sl = k >> 1;
    c.mir = k & 1;
    const int* w = J.win + 4 * c.sl;  // slot 0: (Xs, 0, -, -); pairs: floor(kx), floor(-ky), dx, dy
    const int yi = c.sl ? w[1] : 0, dy = c.sl ? w[3] : 0;
    c.xi = c.sl ? w[0] : 0;
    c.dx = c.sl ? w[2] : 0;
    c.any = false;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      int q = (c.mir ? -(Y0 + h) : Y0 + h) - yi;
      if (q < -N) q += W;  // floor(k) shifts reach beyond the grid's half
      else if (q >= N) q -= W;
      const bool in_p = q >= -N / 2 && q <= N / 2 - 1, in_n = c.sl && q >= dy - N / 2 + 1 && q <= dy + N / 2;
      c.q[h] = q;
      c.wp[h] = in_p ? (c.sl ? 0.5f : 1.f) : 0.f;
      c.wn[h] = in_n ? 0.5f : 0.f;
      c.any = c.any || in_p || in_n;
    }
    return c;
  };
  // the next contribution at or after k that some row pair of the block takes part in
  auto next = [&](int k) {
    for (; k < 2 * nS; k++) {
      const bool any = part(k).any;
      if (P::G == 1 ? any : (bool)__syncthreads_or(any)) break;
    }
    return k;
  };
  auto load = [&](int k, cpair (&v)[E]) {
    const Part c = part(k);
    const float2* I = J.I + (size_t)c.sl * nWin * N;
    const bool on0 = c.wp[0] + c.wn[0] > 0.f, on1 = c.wp[1] + c.wn[1] > 0.f;
    const int y0 = c.q[0] < 0 ? c.q[0] + N : c.q[0], y1 = c.q[1] < 0 ? c.q[1] + N : c.q[1];
#pragma unroll
    for (int i = 0; i < E; i++) {
      const int xl = live_col<N>(t + i * T, Xs);
      const size_t col = (size_t)(xl >> 2) * N * 4 + (xl & 3);
      const float2 z = make_float2(0.f, 0.f);
      v[i] = cp_make(on0 && xl < nWin ? __ldg(I + col + (size_t)y0 * 4) : z,
                     on1 && xl < nWin ? __ldg(I + col + (size_t)y1 * 4) : z);
    }
  };
  cpair x[E], xn[E];
  int k = next(0);
  if (k < 2 * nS) load(k, xn);
  while (k < 2 * nS) {
    const Part c = part(k);
    const int sl = c.sl, mir = c.mir, xi = c.xi, dx = c.dx;
#pragma unroll
    for (int i = 0; i < E; i++) x[i] = xn[i];
    k = next(k + 1);
    if (k < 2 * nS) load(k, xn);  // in flight during this contribution's transforms
    __syncthreads();              // the previous contribution's sums are complete
    if (sl) {
      line_fft_pair<N, T, 1, true>(x, s, 0, t, tw);
      const float2* rx = J.ramps + (size_t)(sl - 1) * 2 * N;
#pragma unroll
      for (int i = 0; i < E; i++) x[i] = cmul(x[i], w_dup(__ldg(rx + t + i * T)));
      line_fft_pair<N, T, 1, false>(x, s, 0, t, tw);
    }
    // v at p = px; sp, sn: inside the pos / the neg range along x
    auto add = [&](int px, bool sp, bool sn, cpair v) {
      int X = xi + px;
      if (mir) X = -X;
      X = wrap(wrap(X));
      float u[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float fp = 1.f, fn = 1.f;
        if (X == N || Y0 == N) {
          // The Nyquist column and row are their own mirror images, but Wiener and apodization
          // differ between the coordinates -N and +N: each part is weighted here, at its own
          // position (the pos range's at floor(k) + p, the neg range's at the mirrored one).
          const float f0 = __ldg(wa + (size_t)(Y0 + h) * W + X);
          const float f1 = __ldg(wa + (size_t)wrap(-(Y0 + h)) * W + wrap(-X));
          fp = mir ? f1 : f0;
          fn = mir ? f0 : f1;
        }
        u[h] = (sp ? c.wp[h] * fp : 0.f) + (sn ? c.wn[h] * fn : 0.f);
      }
      const f32x2 f = p_pack(u[0], u[1]);
      ulonglong2 o = acc[X];
      o.x = p_fma(v.re, f, o.x);
      o.y = p_fma(v.im, mir ? p_neg(f) : f, o.y);
      acc[X] = o;
    };
    // element m at p = m~ (signed), and, for the bins on the edge, at m~ + N in the neg range
    // (no two elements of a contribution meet)
#pragma unroll
    for (int i = 0; i < E; i++) {
      const int m = t + i * T, px = m < N / 2 ? m : m - N;
      const bool in_n = px >= dx - N / 2 + 1;
      add(px, true, in_n, x[i]);
      if (sl && !in_n) add(px + N, false, true, x[i]);
    }
  }
  __syncthreads();
  // x Wiener*apo, then iFFT_W: out[2n] = iFFT_N(A[k] + A[k+N]), out[2n+1] = iFFT_N((A[k] - A[k+N]) e^(i pi k/N))
  cpair z[E];
  const int Y1 = Y0 + 1 < W ? Y0 + 1 : 0;
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int k = t + i * T;
    const ulonglong2 a = acc[k], b = acc[k + N];
    f32x2 f0 = p_dup(1.f), f1 = p_dup(1.f);
    if (Y0 != N) {
      f0 = p_pack(__ldg(wa + (size_t)Y0 * W + k), __ldg(wa + (size_t)Y1 * W + k));
      if (k != 0) f1 = p_pack(__ldg(wa + (size_t)Y0 * W + k + N), __ldg(wa + (size_t)Y1 * W + k + N));
    }
    const cpair u0 = cpair{p_mul(a.x, f0), p_mul(a.y, f0)}, u1 = cpair{p_mul(b.x, f1), p_mul(b.y, f1)};
    x[i] = cadd(u0, u1);
    z[i] = cmulj(csub(u0, u1), w_dup(__ldg(twW + k)));
  }
  // the odd samples wait in the sums' place (each thread its own entries)
#pragma unroll
  for (int i = 0; i < E; i++) acc[t + i * T] = make_ulonglong2(z[i].re, z[i].im);
  line_fft_pair<N, T, 1, true>(x, s, 0, t, tw);
#pragma unroll
  for (int i = 0; i < E; i++) {
    const ulonglong2 u = acc[t + i * T];
    z[i] = cpair{u.x, u.y};
    acc[t + i * T] = make_ulonglong2(x[i].re, x[i].im);
  }
  line_fft_pair<N, T, 1, true>(z, s, 0, t, tw);
  // both samples of a column pair together: 16 bytes per thread and row
#pragma unroll
  for (int i = 0; i < E; i++) {
    const ulonglong2 u = acc[t + i * T];
    float2 e0, e1, o0, o1;
    cp_split(cpair{u.x, u.y}, e0, e1);
    cp_split(z[i], o0, o1);
    float4* O = reinterpret_cast<float4*>(J.O + (size_t)Y0 * W) + t + i * T;
    if (Y0 <= N) O[0] = make_float4(e0.x, e0.y, o0.x, o0.y);
    if (Y0 < N) O[W / 2] = make_float4(e1.x, e1.y, o1.x, o1.y);
  }
}

// ---- LD -----------------------------------------------------------------------------------
// Column x of the image is out[y] = sum_Y h[Y] exp(+2 pi i y Y/W) / W^2 with h[W-Y] = conj h[Y]:
// Z[k] = (h[k] + conj h[N-k]) + i exp(+2 pi i k/W) (h[k] - conj h[N-k]) gives
// iFFT_N(Z)[n] = out[2n] + i out[2n+1].
template <int N>
__global__ void __launch_bounds__(LCfg<N>::CD* LCfg<N>::T, LCfg<N>::blocks(LCfg<N>::CD* LCfg<N>::T))
    k_live_d(const JobDesc* __restrict__ jobs) {
  using P = LCfg<N>;
  constexpr int W = P::W, T = P::T, E = P::E, C = P::CD;
  const JobDesc& J = jobs[blockIdx.y];
  const int lt = threadIdx.x, lane = lt % C, t = lt / C;
  const int X = 2 * (blockIdx.x * C + lane);
  extern __shared__ ulonglong2 smp[];
  const float2* tw = g_stw + stw_offset(N, E);
  const float2* twW = g_tw + tw_offset(W);
  const float4* O = reinterpret_cast<const float4*>(J.O) + X / 2;  // rows W/2 float4 apart
  cpair v[E];  // element t + i*T of Z, in registers through the transform
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int k = t + i * T;
    const float4 a = O[(size_t)k * (W / 2)], b = O[(size_t)(N - k) * (W / 2)];
    const cpair h = cpair{p_pack(a.x, a.z), p_pack(a.y, a.w)}, m = cpair{p_pack(b.x, b.z), p_pack(-b.y, -b.w)};
    const cpair e = cadd(h, m), d = cmulj(csub(h, m), w_dup(__ldg(twW + k)));
    v[i] = cpair{p_sub(e.re, d.im), p_add(e.im, d.re)};  // e + i d
  }
  line_fft_pair<N, T, C, true>(v, smp, lane, t, tw);
  const f32x2 scale = p_dup(1.f / ((float)W * (float)W));
#pragma unroll
  for (int i = 0; i < E; i++) {
    const size_t y = 2 * (size_t)(t + i * T);
    *reinterpret_cast<float2*>(J.out + y * W + X) = p_unpack(p_mul(v[i].re, scale));
    *reinterpret_cast<float2*>(J.out + (y + 1) * W + X) = p_unpack(p_mul(v[i].im, scale));
  }
}

// ---- plan tables ----------------------------------------------------------------------------
// conj(OTF) over the window columns, column by column [xl][y]
__global__ void k_live_otf(float* __restrict__ v, int N, int Xs, const OtfTable* __restrict__ t, int att) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x, xl = blockIdx.y, x = (Xs + xl) % N;
  if (y >= N) return;
  float2 o = make_float2(0.f, 0.f);
  if (!otf_at_fast(*t, 0, freq_x(x, N), freq_y(y, N), FShift{0.f, 0.f, 0.f, 0.f}, 0, 0, att != 0, &o)) o.x = 0.f;
  v[(size_t)xl * N + y] = o.x;
}
// getDenominator x writeApoVector (the apodization from its octant table, W/2 + 1 per row)
__global__ void k_live_wa(float* __restrict__ wa, int W, const OtfTable* __restrict__ t, ShiftSet shifts, FShiftSet fsh,
                          int use_att, float wp, const float* __restrict__ apo) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
  if (X >= W) return;
  const int xh = freq_x(X, W), yh = freq_y(Y, W);
  float acc = 0.f;
  for (int d = 0; d < shifts.n_dirs; d++)
    for (int b = 0; b < shifts.n_bands; b++) {
      const double kx = shifts.px[d] * b, ky = shifts.py[d] * b;
      const FShift k = fsh.k[d][b];
      const float v1 = wiener_term(*t, 0, xh, yh, k, kx, ky, use_att != 0);
      const float v2 = wiener_term(*t, 0, xh, yh, fshift_neg(k), -kx, -ky, use_att != 0);
      acc = __fadd_rn(__fadd_rn(acc, v1), v2);
    }
  const float den = __fdiv_rn(1.f, __fadd_rn(acc, wp));
  const int ax = abs(xh), ay = abs(yh);
  wa[(size_t)Y * W + X] = __fmul_rn(den, __ldg(apo + (size_t)max(ax, ay) * (W / 2 + 1) + min(ax, ay)));
}

int Plan::build_live(cudaStream_t st) {
  const int N = prm.w, W = 2 * N, nA = prm.nr_dirs, nP = prm.nr_phases, nC = 2 * prm.nr_bands - 1;
  OtfTable ht;
  build_otf_table(&prm, &ht);
  const int old_nwin = nwin;
  // window of spectrum columns inside the OTF support (all columns when it is wider), from Xs
  plan_window(&prm, ht.cutoff / ht.vec_cpm, &nwin);
  if (nwin > N) nwin = N;
  const int Xs = nwin == N ? 0 : N - nwin / 2;
  std::vector<float2> coef((size_t)nA * nC * nP);
  for (int a = 0; a < nA; a++) {
    auto m = separation_coeffs(&prm, a, false);
    for (int c = 0; c < nC; c++)
      for (int q = 0; q < nP; q++) coef[(a * nC + c) * nP + q] = make_float2(m[c * nP + q].real(), m[c * nP + q].imag());
  }
  // per pos component: fractional shift ramps {x[N], y[N]} (1/N folded in), and the paste
  // offsets and edge flags of its slot {floor(kx), floor(-ky), dx, dy}; slot 0 holds Xs
  const int nPair = prm.nr_bands - 1;
  std::vector<float2> ramps((size_t)nA * nPair * 2 * N);
  std::vector<int> off((size_t)(1 + nA * nPair) * 4, 0);
  off[0] = Xs;
  for (int a = 0; a < nA; a++)
    for (int b = 1; b <= nPair; b++) {
      const int ab = a * nPair + (b - 1);
      const double kx = band_px(&prm, a, b), ky = band_py(&prm, a, b);
      // SimUtils.pasteAndFourierShift, fast mode (S/SimUtils.java:77-86)
      const double xFrac = kx - std::floor(kx), yFrac = -ky - std::floor(-ky);
      int* o = &off[4 * (1 + ab)];
      // pasteFreq takes its offsets modulo the output size: into [-N, N)
      auto mod = [&](double f) {
        const int m = (int)std::fmod(f, (double)W);
        return m >= N ? m - W : (m < -N ? m + W : m);
      };
      o[0] = mod(std::floor(kx));
      o[1] = mod(std::floor(-ky));
      o[2] = xFrac != 0;
      o[3] = yFrac != 0;
      float2* rx = &ramps[(size_t)ab * 2 * N];
      float2* ry = rx + N;
      for (int n = 0; n < N; n++) {
        double fx = xFrac * n / N, fy = yFrac * n / N;
        fx -= std::floor(fx);
        fy -= std::floor(fy);
        rx[n] = make_float2((float)(std::cos(2 * M_PI * fx) / N), (float)(std::sin(2 * M_PI * fx) / N));
        ry[n] = make_float2((float)(std::cos(2 * M_PI * fy) / N), (float)(std::sin(2 * M_PI * fy) / N));
      }
    }
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  size_t o_coef = 0, o_ramp = o_coef + al(coef.size() * sizeof(float2));
  size_t o_off = o_ramp + al(ramps.size() * sizeof(float2));
  size_t o_otf = o_off + al(off.size() * sizeof(int));
  size_t o_damp = o_otf + al(sizeof(OtfTable));
  size_t o_mask = o_damp + al((size_t)N * N * sizeof(float));
  size_t o_wa = o_mask + al((size_t)N * N * sizeof(float));
  size_t o_apo = o_wa + al((size_t)W * W * sizeof(float));
  size_t total = o_apo + al((size_t)(N + 1) * (N + 1) * sizeof(float));
  const void* old_dev = dev;
  if (total > dev_bytes) {
    if (dev) cudaFree(dev);
    dev = nullptr;
    dev_bytes = 0;
    FSIM_CUDA(fsim::dev_alloc(&dev, total));
    dev_bytes = total;
  }
  if (old_dev != dev || old_nwin != nwin) layout->fetch_add(1);
  char* b = (char*)dev;
  d_coef = (float2*)(b + o_coef);
  d_ramps = (float2*)(b + o_ramp);
  d_win = (int*)(b + o_off);
  d_otf = (OtfTable*)(b + o_otf);
  d_damp = fade_px > 0 ? (float*)(b + o_damp) : nullptr;
  d_masks = (float*)(b + o_mask);
  d_wa = (float*)(b + o_wa);
  FSIM_CUDA(cudaMemcpyAsync(d_coef, coef.data(), coef.size() * sizeof(float2), cudaMemcpyHostToDevice, st));
  FSIM_CUDA(cudaMemcpyAsync(d_ramps, ramps.data(), ramps.size() * sizeof(float2), cudaMemcpyHostToDevice, st));
  FSIM_CUDA(cudaMemcpyAsync(d_win, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice, st));
  FSIM_CUDA(cudaMemcpyAsync(d_otf, &ht, sizeof(OtfTable), cudaMemcpyHostToDevice, st));
  std::vector<float> dv;
  if (d_damp) {
    dv = fade_vector(N, N, fade_px);
    FSIM_CUDA(cudaMemcpyAsync(d_damp, dv.data(), dv.size() * sizeof(float), cudaMemcpyHostToDevice, st));
  }
  FSIM_CUDA(cudaStreamSynchronize(st));
  k_live_otf<<<dim3(div_up(N, 128), nwin), 128, 0, st>>>(d_masks, N, Xs, d_otf, prm.use_attenuation);
  // setupFilters: getDenominator(wienParam) and writeApoVector(apo, 1, 2)
  {
    float* d_apo = (float*)(b + o_apo);
    int rc = apo_octant_device(d_apo, N, ht.vec_cpm, ht.cutoff * 2.0, 1.0, st);
    if (rc) return rc;
    const ShiftSet sh = shift_set(&prm);
    k_live_wa<<<dim3(div_up(W, 128), W), 128, 0, st>>>(d_wa, W, d_otf, sh, fshift_set(sh), prm.use_attenuation,
                                                       (float)(prm.wiener * prm.wiener), d_apo);
  }
  FSIM_CHECK_LAUNCH();
  FSIM_CUDA(cudaStreamSynchronize(st));
  filter_bytes = total;
  return FSIM_OK;
}

// I: column windows of band 0 and of every pos component; O: rows 0..N of the half spectrum
static size_t live_i_bytes(const fsim_sim_param& p, int nwin) {
  const size_t b = (size_t)(1 + p.nr_dirs * (p.nr_bands - 1)) * nwin * p.w * sizeof(float2);
  return (b + 255) & ~(size_t)255;
}
size_t Plan::workspace_bytes_live() const {
  const size_t O = (size_t)(prm.w + 1) * 2 * prm.w * sizeof(float2);
  return live_i_bytes(prm, nwin) + ((O + 255) & ~(size_t)255);
}

void Plan::fill_job_live(JobDesc& j, const void* raw, float* out, float* wf, char* ws) const {
  const int nC = 2 * prm.nr_bands - 1;
  j.raw = raw;
  j.out = out;
  j.widefield = wf;
  j.input_u16 = input_type == FSIM_INPUT_U16;
  j.nA = prm.nr_dirs;
  j.nP = prm.nr_phases;
  j.nC = nC;
  j.nWin = nwin;
  j.bgr = 0.f;
  j.damp = d_damp;
  j.coef = d_coef;
  j.ramps = d_ramps;
  j.win = d_win;
  j.masks = d_masks;
  j.wa = d_wa;
  j.nyq = nullptr;
  j.D = nullptr;
  j.G = nullptr;
  j.Tw = nullptr;
  j.On = nullptr;
  j.clip_max = nullptr;
  j.clip = 0;
  j.cmask = 0;
  j.edge = nullptr;
  j.fwf = nullptr;
  j.wff = nullptr;
  j.Wf = nullptr;
  j.I = (float2*)ws;
  j.O = (float2*)(ws + live_i_bytes(prm, nwin));
}

template <int N>
static int launch_live(const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, cudaStream_t st) {
  using P = LCfg<N>;
  constexpr size_t E16 = sizeof(ulonglong2);
  const size_t sm_a = E16 * P::G * P::XS, sm_b = E16 * pair_elems(N, P::CP), sm_c = LCPass<N>::SMEM,
               sm_d = E16 * pair_elems(N, P::CD);
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(k_live_a<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_a));
    FSIM_CUDA(cudaFuncSetAttribute(k_live_b<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_b));
    FSIM_CUDA(cudaFuncSetAttribute(k_live_c<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_c));
    FSIM_CUDA(cudaFuncSetAttribute(k_live_d<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_d));
    attr = true;
  }
  cudaEvent_t* ev = profile_events();
  if (ev) cudaEventRecord(ev[0], st);
  k_live_a<N><<<dim3(N / (2 * P::G), maxA + 1, njobs), P::G * P::T, sm_a, st>>>(d_jobs);
  if (ev) cudaEventRecord(ev[1], st);
  k_live_b<N><<<dim3((maxWin + 2 * P::CP - 1) / (2 * P::CP), 1 + maxA * maxPair, njobs), P::CP * P::T, sm_b, st>>>(
      d_jobs);
  if (ev) cudaEventRecord(ev[2], st);
  // rows 0..N in pairs, whole groups
  k_live_c<N><<<dim3((N / 2 + 1 + P::G - 1) / P::G, njobs), LCPass<N>::NT, sm_c, st>>>(d_jobs);
  if (ev) cudaEventRecord(ev[3], st);
  k_live_d<N><<<dim3(N / P::CD, njobs), P::CD * P::T, sm_d, st>>>(d_jobs);
  if (ev) {
    cudaEventRecord(ev[4], st);
    profile_mark(4);
  }
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

#define FSIM_LIVE_SIZES(X) X(64) X(128) X(256) X(384) X(512) X(768) X(1024) X(2048)

bool live_size_supported(int n) {
  switch (n) {
#define CASE(v) case v:
    FSIM_LIVE_SIZES(CASE)
#undef CASE
    return true;
    default:
      return false;
  }
}

int launch_live_size(int n, const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, cudaStream_t st) {
  switch (n) {
#define CASE(v) \
  case v:       \
    return launch_live<v>(d_jobs, njobs, maxA, maxPair, maxWin, st);
    FSIM_LIVE_SIZES(CASE)
#undef CASE
  }
  set_error("live reconstruction: unsupported image size %d", n);
  return FSIM_EINVAL;
}

}  // namespace fsim
