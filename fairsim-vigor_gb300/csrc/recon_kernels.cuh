// Kernels of the fused offline reconstruction (templates instantiated per size in
// recon_inst_*.cu). See recon.cu for the algorithm and the pass structure.
//
// Every 1D operation here is done with N-length line FFTs. The reference's shift of a
// pasted N-point spectrum Z on the W = 2N grid, FFT_W(r * iFFT_W(paste(Z))), is evaluated
// through its exact even/odd split: with u = iFFT_W(paste(Z)),
//   u[2n]   = z[n] / 2                       (z = iFFT_N(Z), the line in real space)
//   u[2n+1] = iFFT_N(Z * s)[n] / W,  s(m) = exp(+i pi m~/N), m~ the pasted signed frequency
// so that, with E = FFT_N(r[2n] u[2n]) and O = FFT_N(r[2n+1] u[2n+1]),
//   FFT_W(r * u)[X] = E[X mod N] + exp(-2 pi i X/W) O[X mod N].
// The per-component ramps r (even and odd samples, 1/2 and 1/W folded in) are resident
// tables; s and exp(-2 pi i X/W) come from the W-point twiddle table. The final inverse
// FFT_W along y is folded the same way into two N-point inverse FFTs (even/odd rows).
#pragma once

#include "common.cuh"
#include "fft_line.cuh"
#include "fft_pair.cuh"
#include "filters.cuh"
#include "otf.cuh"
#include "recon.cuh"
#include "runtime.cuh"

namespace fsim {

// ---- launch configuration (variants picked per size by the autotuner) --------------------
// ENV: elements per thread of the N-length lines (radix plan and threads per line follow);
// CBV: interleaved columns per block in pass B.
template <int N, int ENV = 0, int CBV = 0>
struct Cfg {
  static constexpr int W = 2 * N;
  static constexpr int EN = ENV ? ENV : ((N % 3 == 0) ? 12 : 8);
  static constexpr int T = N / EN;  // threads per line
  static constexpr int CB = CBV ? CBV : 4;  // passes B1, B2: interleaved columns per block
  static constexpr int GC = (T >= 128) ? 1 : (128 / T);  // pass C: rows per block
};

// Copies a job descriptor into shared memory once per block (the passes read its fields
// after global stores, which would otherwise force reloads).
__device__ __forceinline__ void load_job(JobDesc* dst, const JobDesc* src, int tid, int nthreads) {
  const int* s = reinterpret_cast<const int*>(src);
  int* d = reinterpret_cast<int*>(dst);
  for (int i = tid; i < (int)(sizeof(JobDesc) / sizeof(int)); i += nthreads) d[i] = s[i];
}

// exp(+i pi m~ / N) for the pasted signed frequency m~ of index m (m < N/2: m, else m - N)
template <int N>
__device__ __forceinline__ float2 half_shift(const float2* twW, int m) {
  const int ms = m < N / 2 ? m : m - N;
  return cconjf(twW[ms < 0 ? ms + 2 * N : ms]);
}
// source index in an N-point spectrum of output index X of pasteFreq onto 2N (or -1)
template <int N>
__device__ __forceinline__ int paste_src(int X) {
  return X < N / 2 ? X : (X >= 3 * N / 2 ? X - N : -1);
}

// ---- pass A: rows ----------------------------------------------------------------------------
// Blocks per SM for regs8 registers per thread at 8 elements, 128 at 12 or 16, 255 beyond (a line pair
// holds 4 registers per element; a partial warp takes a whole one's registers).
__host__ __device__ constexpr int pair_min_blocks(int threads, int EN, int regs8) {
  const int r = EN <= 8 ? regs8 : (EN <= 16 ? 128 : 255), n = threads < 32 ? 32 : threads;
  return 65536 / (n * r) > 0 ? (65536 / (n * r) < 32 ? 65536 / (n * r) : 32) : 1;
}
// Raw pixels of the rows at `row` and the row below (frame offset fo) with the background clip:
// all loads of the two rows are issued before any is used.
template <int N, int EN, int T>
__device__ __forceinline__ void raw_rows(const JobDesc& J, size_t fo, size_t row, int t, float (&v)[2][EN]) {
  if (J.input_u16) {
    const uint16_t* r = (const uint16_t*)J.raw + fo + row + t;
#pragma unroll
    for (int i = 0; i < EN; i++) {
      v[0][i] = (float)__ldg(r + i * T);
      v[1][i] = (float)__ldg(r + N + i * T);
    }
  } else {
    const float* r = (const float*)J.raw + fo + row + t;
#pragma unroll
    for (int i = 0; i < EN; i++) {
      v[0][i] = __ldg(r + i * T);
      v[1][i] = __ldg(r + N + i * T);
    }
  }
  if (J.bgr != 0.f) {
#pragma unroll
    for (int i = 0; i < EN; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        v[h][i] = v[h][i] - J.bgr;
        if (v[h][i] < 0) v[h][i] = 0;
      }
  }
}
// The border damping of mixed rows: the mix of damped rows is the damped mix (the damping
// is one real factor per pixel), so the factors are read once per row, not once per frame.
template <int N, int EN, int T>
__device__ __forceinline__ void damp_rows(const JobDesc& J, size_t row, int t, cpair (&z)[EN]) {
  if (J.damp) {
    const float* d = J.damp + row + t;
#pragma unroll
    for (int i = 0; i < EN; i++) {
      const f32x2 f = p_pack(__ldg(d + i * T), __ldg(d + N + i * T));
      z[i].re = p_mul(z[i].re, f);
      z[i].im = p_mul(z[i].im, f);
    }
  }
}

// A group of T threads transforms two adjacent rows as one line pair; groups are joined to
// blocks of at least 64 threads. Dynamic shared memory: the exchange buffer of each group's pair.
template <int N, int ENV>
struct PassA {
  static constexpr int T = Cfg<N, ENV>::T, EN = Cfg<N, ENV>::EN;
  static constexpr int G = T >= 64 ? 1 : 64 / T;  // row pairs per block
  static constexpr int NT = G * T;
  static constexpr int RB = 2 * G;  // rows per block
  static constexpr int XS = pair_elems(N, 1);
  static constexpr size_t SMEM = sizeof(ulonglong2) * (size_t)G * XS;
  // Frames whose pixels are in flight at once while a thread mixes them, and the registers that
  // takes: with 64 threads 3 (96 registers) against 1 (80) is 447 us against 451 for 64 x 512^2, with
  // 128 threads 531 against 565 for 16 x 1024^2; at 256 threads 96 registers leave two blocks per
  // SM instead of three (a 2048^2 3x5 stack: 238 us, 201 with one frame, 195 with two). 12
  // elements per thread leave no room for more than one.
  static constexpr int F = EN > 8 ? 1 : (NT <= 128 ? 3 : 2);
  static constexpr int MINB = pair_min_blocks(NT, EN, F == 3 ? 96 : 80);
  static_assert(N % RB == 0, "whole blocks of rows");
};

// blockIdx.y < nA: the band pairs of that angle; blockIdx.y == nA: band 0 of all angles (in one
// launch, so that both read a dataset's frames while they are in L2: as two launches the
// frames of 16 datasets of 512^2 came from DRAM twice, 105 + 37 us against 111 us).
template <int N, int ENV>
__global__ void __launch_bounds__(PassA<N, ENV>::NT, PassA<N, ENV>::MINB) k_pass_a(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV>;
  using PA = PassA<N, ENV>;
  constexpr int W = P::W, T = P::T, EN = P::EN, NT = PA::NT;
  const int tid = threadIdx.x, g = tid / T, t = tid % T;
  const int y = blockIdx.x * PA::RB + 2 * g, a = blockIdx.y;
  __shared__ JobDesc J;
  __shared__ float2 coef[FSIM_MAX_DIRS * FSIM_MAX_PHASES];
  extern __shared__ ulonglong2 smp[];
  ulonglong2* s = smp + g * PA::XS;
  const float2* twN = g_stw + stw_offset(N, EN);  // stage table, read through L1
  const float2* twW = g_tw + tw_offset(W);
  const JobDesc* jg = jobs + blockIdx.z;
  load_job(&J, jg, tid, NT);
  // the counts and the separation coefficients straight from the descriptor in global
  // memory, so that one barrier covers both shared-memory copies
  const int nA = jg->nA, nP = jg->nP, nC = jg->nC, nPair = (nC - 1) / 2;
  if (a > nA) return;  // uniform per block
  if (a == nA) {
    for (int i = tid; i < nA * nP; i += NT) coef[i] = jg->coef[((i / nP) * nC) * nP + i % nP];
  } else {
    for (int i = tid; i < nC * nP; i += NT) coef[i] = jg->coef[a * nC * nP + i];
  }
  __syncthreads();
  const size_t frame = (size_t)N * N, row = (size_t)y * N;
  const int nWin = J.nWin;
  // Both rows' value of window column xl, written to the quad layout [xl/4][y][xl%4]: the
  // threads of a warp write whole 32-byte sectors.
  auto put = [&](float2* I, int xl, cpair v) {
    float2 r0, r1;
    cp_split(v, r0, r1);
    float2* o = I + ((size_t)(xl >> 2) * N + y) * 4 + (xl & 3);
    o[0] = r0;
    o[4] = r1;
  };
  // Band separation in real space of frames f0 .. f0 + nf - 1 with coefficients c: the frames
  // outer, so that every element's load of a frame's rows is in flight at once.
  cpair x[EN];  // element t + i*T of both rows, in registers from one transform to the next
  auto mix = [&](int f0, int nf, const float2* c) {
#pragma unroll
    for (int i = 0; i < EN; i++) x[i] = cp_zero();
    auto add = [&](float (&v)[2][EN], float2 k) {
      const wpair m = w_dup(k);
#pragma unroll
      for (int i = 0; i < EN; i++) {
        const f32x2 r = p_pack(v[0][i], v[1][i]);
        x[i].re = p_fma(m.x, r, x[i].re);
        x[i].im = p_fma(m.y, r, x[i].im);
      }
    };
    constexpr int F = PA::F;
    int p = 0;
#pragma unroll 1
    for (; p + F <= nf; p += F) {
      float v[F][2][EN];
#pragma unroll
      for (int f = 0; f < F; f++) raw_rows<N, EN, T>(J, (size_t)(f0 + p + f) * frame, row, t, v[f]);
#pragma unroll
      for (int f = 0; f < F; f++) add(v[f], c[p + f]);
    }
#pragma unroll 1
    for (; p < nf; p++) {
      float v[2][EN];
      raw_rows<N, EN, T>(J, (size_t)(f0 + p) * frame, row, t, v);
      add(v, c[p]);
    }
    damp_rows<N, EN, T>(J, row, t, x);
  };
  if (a == nA) {
    // Band 0 is summed over the angles before the column pass, and its band separation
    // and row FFT are linear: one row group mixes the band-0 rows of every angle and
    // transforms the sum once into slot 0 (band 0 has no shift: one window for all angles).
    mix(0, nA * nP, coef);
    line_fft_pair<N, T, 1, false>(x, s, 0, t, twN);
    const int Xs = J.win[0];
#pragma unroll
    for (int i = 0; i < EN; i++) {
      const int m = t + i * T;
      int xl = (m < N / 2 ? m : m + N) - Xs;  // pasted column
      if (xl < 0) xl += W;
      if (xl < nWin) put(J.I, xl, x[i]);
    }
    for (int xl = t; xl < nWin; xl += T) {  // window columns that pasteFreq leaves empty
      int X = Xs + xl;
      if (X >= W) X -= W;
      if (paste_src<N>(X) < 0) put(J.I, xl, cp_zero());
    }
    if (y == 0 && t == 0) *J.clip_max = 0.f;  // CLIPSCALE.BOTH: pass C takes the maximum from 0
    return;
  }
  // Components: band 0, then per band b the pair neg = 2b-1, pos = 2b. The separation
  // coefficients of a pair are complex conjugates, so z_pos = conj(z_neg).
  // Pair (neg, pos): only the neg component is transformed and stored. The image is real, so
  // the two components enter it as m_neg (V_neg + V+) / 2 and its mirror image, V+(X, Y) =
  // conj V_pos(-X, -Y). With z_pos = conj(z_neg) and opposite shifts, V_neg and V+ are the same
  // transform of z_neg except for the half-sample phase of the pasted Nyquist bin, s(N/2) = -i
  // in V_neg and +i in V+: with T the shift whose s(N/2) is 0 and Q the Nyquist bin's rank-one
  // part, along x and y, V_neg = (Ty - iQy)(Tx - iQx) z, V+ = (Ty + iQy)(Tx + iQx) z, and
  //   (V_neg + V+) / 2 = Ty Tx z - Qy Qx z.
  // So this pass drops the Nyquist bin (s(N/2) = 0) and keeps its value per row (D); the column
  // pass puts -Qy Qx z back as the column's own Nyquist value.
  // z holds the mixed rows, then E: in shared memory (8 or 12 more 16-byte elements per thread each
  // way, twice) the shared-memory pipe, which bounds this pass, took 474 us per 64 x 512^2 in place of
  // 447, and 374 us per 16 x 768^2 in place of 333.
  cpair z[EN];
  for (int b = 1; b <= nPair; b++) {
    const int cn = 2 * b - 1;
    mix(a * nP, nP, coef + cn * nP);
#pragma unroll
    for (int i = 0; i < EN; i++) z[i] = x[i];
    const float2* re = J.ramps + (size_t)(a * nC + cn) * 2 * W;
    const float2* ro = re + N;
    // even samples times the even-sample ramp, FFT: E (changes places with the mixed rows)
#pragma unroll
    for (int i = 0; i < EN; i++) x[i] = cmul(x[i], w_dup(__ldg(re + t + i * T)));
    line_fft_pair<N, T, 1, false>(x, s, 0, t, twN);
#pragma unroll
    for (int i = 0; i < EN; i++) {
      const cpair e = x[i];
      x[i] = z[i];
      z[i] = e;
    }
    line_fft_pair<N, T, 1, false>(x, s, 0, t, twN);  // Z = FFT_N(z)
    if (t == (N / 2) % T) {
      float2 r0, r1;
      cp_split(x[(N / 2) / T], r0, r1);
      float2* D = J.D + (size_t)(a * nPair + (b - 1)) * N + y;
      D[0] = r0;
      D[1] = r1;
      x[(N / 2) / T] = cp_zero();
    }
    // odd samples of the upsampled line, iFFT_N(Z * s), times the odd-sample ramp, FFT: O
#pragma unroll
    for (int i = 0; i < EN; i++) x[i] = cmul(x[i], w_dup(half_shift<N>(twW, t + i * T)));
    line_fft_pair<N, T, 1, true>(x, s, 0, t, twN);
#pragma unroll
    for (int i = 0; i < EN; i++) x[i] = cmul(x[i], w_dup(__ldg(ro + t + i * T)));
    line_fft_pair<N, T, 1, false>(x, s, 0, t, twN);
    // neg window of the shifted spectrum: E[X mod N] + exp(-2 pi i X/W) O[X mod N]. Element m
    // is column X = m or m + N; a window wider than N holds both of some.
    const int Xs = J.win[2 * (a * nC + cn)];
    float2* I = J.I + (size_t)(1 + a * nPair + (b - 1)) * nWin * N;  // slot of (a, b)
#pragma unroll
    for (int i = 0; i < EN; i++) {
      int xl = t + i * T - Xs;
      if (xl < 0) xl += W;
      if (xl >= N) xl -= N;
      if (xl < nWin) {
        int X = Xs + xl;
        if (X >= W) X -= W;
        const cpair o = cmul(x[i], w_dup(__ldg(twW + X)));
        put(I, xl, cadd(z[i], o));
        if (xl + N < nWin) put(I, xl + N, csub(z[i], o));
      }
    }
  }
  // At its end, as pass B's: blocks that start early are placed on SMs that still run this pass and
  // wait there (4 x 128^2 30.7 us, 39.5 with this at the start; one 192^2 stack 41.0, 47.4).
  pdl_trigger();
}

// ---- pass G: the Nyquist column of the row transforms (complex masks, edge weights) ---------------------
// A complex mask m (measured OTFs) weighs V_neg with m and V+ with conj(m), so a pair enters the
// image as Re(m) (V_neg + V+)/2 + i Im(m) (V_neg - V+)/2 and its mirror image, and
//   i (V_neg - V+) / 2 = Ty Qx z + Qy Tx z   (pass A's notation).
// The same term enters the output's Nyquist column and row (pass B1) where a support reaches them.
// Qx z is D(y) times a plan table along x: this pass transforms D along y once per angle and pair.
template <int N, int ENV>
__global__ void __launch_bounds__(Cfg<N, ENV>::T) k_pass_g(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV>;
  constexpr int W = P::W, T = P::T, EN = P::EN;
  const int t = threadIdx.x, ab = blockIdx.x;
  __shared__ JobDesc J;
  __shared__ float2 bz[smem_line_elems(N, 1)], bh[smem_line_elems(N, 1)];
  const float2* twN = g_stw + stw_offset(N, EN);
  const float2* twW = g_tw + tw_offset(W);
  load_job(&J, jobs + blockIdx.y, t, T);
  pdl_trigger();
  pdl_wait();
  __syncthreads();
  const int nC = J.nC, nPair = (nC - 1) / 2;
  if (!(J.cmask || J.edge) || ab >= J.nA * nPair) return;  // uniform per block
  const int a = ab / nPair, cn = 2 * (ab % nPair) + 1;
  const float2* d = J.D + (size_t)ab * N;
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int k = t + i * T;
    const float2 v = d[k];
    bz[sidx(k)] = v;
    bh[sidx(k)] = v;
  }
  __syncthreads();
  line_fft_st<N, T, 1, false>(bh, t, twN);
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int m = t + i * T;
    bh[sidx(m)] = m == N / 2 ? make_float2(0.f, 0.f) : cmul(bh[sidx(m)], half_shift<N>(twW, m));
  }
  __syncthreads();
  line_fft_st<N, T, 1, true>(bh, t, twN);
  const float2* re = J.ramps + (size_t)(a * nC + cn) * 2 * W + W;  // y ramps
  const float2* ro = re + N;
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int m = t + i * T;
    bz[sidx(m)] = cmul(bz[sidx(m)], __ldg(re + m));
    bh[sidx(m)] = cmul(bh[sidx(m)], __ldg(ro + m));
  }
  __syncthreads();
  line_fft_st<N, T, 1, false>(bz, t, twN);
  line_fft_st<N, T, 1, false>(bh, t, twN);
  const int Ys = J.win[2 * (a * nC + cn) + 1];
  for (int yl = t; yl < J.nWin; yl += T) {
    int Y = Ys + yl;
    if (Y >= W) Y -= W;
    const int m = Y < N ? Y : Y - N;
    J.G[(size_t)ab * J.nWin + yl] = cadd(bz[sidx(m)], cmul(twW[Y], bh[sidx(m)]));
  }
}

// ---- pass B1: column transforms of band 0 and of the neg components, masked ---------------------
// One block per CB window columns of one component: band 0 (the windows of all angles summed: they
// share one unshifted mask) is transformed along y and pasted; each pair's neg component gets the
// full y shift (even/odd split, the Nyquist bin as pass A's comment says).
// The result over the component's row window, times its OTF mask, is the component's
// contribution P to the image's spectrum S, stored column by column ([column][row]):
//   H(X, Y) = S(X, Y) + conj S(-X, -Y),  S = sum of P over band 0 (mask/2) and the pairs,
// because mask_pos(X, Y) = mask_neg(-X, -Y). That fails on the output's Nyquist column X = N and row
// Y = N: they are their own mirror images, but masks and Wiener x apodization (wa) are evaluated at
// one coordinate of the two (-N along x, +N along y). With M = (-X, -Y), a pair's share of the image is
//   2 H(X, Y) = f(X, Y) + conj f(M),  f(X, Y) = wa(X, Y) (m_neg(X, Y) V_neg(X, Y) + m_pos(X, Y) conj V+(M)),
// and with V_neg = P - i G, V+ = P + i G, where P = (V_neg + V+)/2 and G is pass G's term,
//   H(X, Y) = S(X, Y) + conj S(M),  S = alpha P + gamma G,
//   alpha = (wa m_neg + wa(M) conj m_pos(M)) / 2,  gamma = -i (wa m_neg - wa(M) conj m_pos(M)) / 2.
// A plan whose supports and apodization reach these lines holds alpha and gamma along them (edge): its
// jobs run pass G, this pass weights the two lines with them and pass B2 leaves wa out there. (Band 0's
// paste is 0 on both lines.)
// With the masks and the Nyquist terms applied here, where the column is in registers, pass B2 only
// adds windows (it took 0.358 ms per 64 datasets of 512^2 3x3 while it read neg and pos masks and
// formed the Nyquist terms per pixel).
// Adjacent columns form a line pair: CB/2 pairs of T threads per block. Each thread keeps the
// column and then E in registers, as pass A does (in shared memory 395 us per 64 x 512^2 in place
// of 367); the transforms' operands beside them fit 80 registers without spills worth their time
// (72: 396 us, 96: 382).
template <int N, int ENV, int CBV>
struct PassB1 {
  using P = Cfg<N, ENV, CBV>;
  static constexpr int CP = P::CB / 2, NT = CP * P::T;
  static constexpr int XS = pair_elems(N, CP);
  static constexpr size_t SMEM = sizeof(ulonglong2) * (size_t)XS;
  static constexpr int MINB = pair_min_blocks(NT, P::EN, 80);
  static constexpr bool BYJOB = P::EN > 8 && NT >= 128;  // grid order of k_pass_b01
};
// Row yl of window columns xl and xl + 1 of a component (col: the position of its first row in
// the component-by-component window layout), times their masks, to Tw.
template <bool CM>
__device__ __forceinline__ void b1_put(const JobDesc& J, size_t col, int nWin, int yl, cpair v) {
  float2* out = J.Tw + col + yl;
  float2 r0, r1;
  if constexpr (CM) {
    const float2* mk = reinterpret_cast<const float2*>(J.masks) + col + yl;
    cp_split(v, r0, r1);
    out[0] = cmul(r0, __ldg(mk));
    out[nWin] = cmul(r1, __ldg(mk + nWin));
  } else {
    const float* mk = J.masks + col + yl;
    const f32x2 f = p_pack(__ldg(mk), __ldg(mk + nWin));
    cp_split(cpair{p_mul(v.re, f), p_mul(v.im, f)}, r0, r1);
    out[0] = r0;
    out[nWin] = r1;
  }
}
// The output's Nyquist row and column among window columns xl and xl + 1 of pair ab, each weighted at its
// own coordinates in place of the masks: rewrites what this thread has stored there. x, z: O and E of
// this thread's rows; nyquist(yl, h): the term G.
template <int N, int T, int EN, class F>
__device__ __forceinline__ void b1_edges(const JobDesc& J, int ab, int xl, int t, const cpair (&x)[EN], const cpair (&z)[EN],
                                         F nyquist) {
  constexpr int W = 2 * N;
  const int nWin = J.nWin, nPair = (J.nC - 1) / 2, c = (ab / nPair) * J.nC + 2 * (ab % nPair) + 1;
  const int Xs = J.win[2 * c], Ys = J.win[2 * c + 1];
  const int xN = Xs <= N ? N - Xs : N - Xs + W, yN = Ys <= N ? N - Ys : N - Ys + W;  // beyond nWin: not in the window
  const float4* e = J.edge + (size_t)2 * ab * nWin;
  float2* out = J.Tw + ((size_t)(1 + ab) * nWin + xl) * nWin;
  auto put = [&](int yl, int h, cpair v, float4 w) {
    float2 r[2];
    cp_split(v, r[0], r[1]);
    out[(size_t)h * nWin + yl] =
        cadd(cmul(h ? r[1] : r[0], make_float2(w.x, w.y)), cmul(nyquist(yl, h), make_float2(w.z, w.w)));
  };
  if (t == 0 && yN < nWin)  // row N is element 0's: E - O
    for (int h = 0; h < 2; h++) put(yN, h, csub(z[0], x[0]), __ldg(e + nWin + xl + h));
  if ((xN & ~1) != xl || xN >= nWin) return;
  const float2* twW = g_tw + tw_offset(W);
#pragma unroll
  for (int i = 0; i < EN; i++)
    for (int yl = t + i * T - Ys + (t + i * T < Ys ? W : 0), k = 0; k < 2; k++, yl += yl < N ? N : -N) {
      if (yl >= nWin) continue;
      const int Y = Ys + yl < W ? Ys + yl : Ys + yl - W;
      put(yl, xN & 1, cadd(z[i], cmul(x[i], w_dup(__ldg(twW + Y)))), __ldg(e + yl));
    }
}
// elements t + i*T of window columns xl and xl + 1 from pass A's slot
template <int N, int T, int EN>
__device__ __forceinline__ void b1_load(const JobDesc& J, int slot, int nWin, int xl, int t, cpair (&x)[EN]) {
  const float4* I = reinterpret_cast<const float4*>(J.I + (size_t)slot * nWin * N + ((size_t)(xl >> 2) * N) * 4 +
                                                    (xl & 3));  // rows 2 float4 apart
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const float4 v = I[(size_t)(t + i * T) * 2];
    x[i] = cpair{p_pack(v.x, v.z), p_pack(v.y, v.w)};
  }
}
// Band 0: summed over the angles and row-transformed in pass A (slot 0); one transform per column.
template <int N, int ENV, int CBV, bool CM>
__device__ __forceinline__ void b1_band0(const JobDesc& J, int xl, int lane, int t, ulonglong2* s) {
  using P = Cfg<N, ENV, CBV>;
  constexpr int W = P::W, T = P::T, EN = P::EN, CP = PassB1<N, ENV, CBV>::CP;
  const int nWin = J.nWin;
  const size_t col = (size_t)xl * nWin;
  cpair x[EN];
  b1_load<N, T, EN>(J, 0, nWin, xl, t, x);
  line_fft_pair<N, T, CP, false>(x, s, lane, t, g_stw + stw_offset(N, EN));
  const int Ys = J.win[1];
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int m = t + i * T;
    int yl = (m < N / 2 ? m : m + N) - Ys;  // pasted row
    if (yl < 0) yl += W;
    if (yl < nWin) b1_put<CM>(J, col, nWin, yl, x[i]);
  }
  for (int yl = t; yl < nWin; yl += T) {  // window rows that pasteFreq leaves empty
    int Y = Ys + yl;
    if (Y >= W) Y -= W;
    if (paste_src<N>(Y) < 0) J.Tw[col + yl] = J.Tw[col + nWin + yl] = make_float2(0.f, 0.f);
  }
}
template <int N, int ENV, int CBV, bool CM>
__device__ __noinline__ void b1_band0_call(const JobDesc& J, int xl, int lane, int t, ulonglong2* s) {
  b1_band0<N, ENV, CBV, CM>(J, xl, lane, t, s);
}
// The neg component comp = 1 + a*nPair + (b-1) of (a, b), window columns xl and xl + 1.
template <int N, int ENV, int CBV, bool CM, bool EDGE>
__device__ __forceinline__ void b1_pair(const JobDesc& J, int comp, int xl, int lt, ulonglong2* s) {
  using P = Cfg<N, ENV, CBV>;
  using PB = PassB1<N, ENV, CBV>;
  constexpr int W = P::W, T = P::T, CB = P::CB, EN = P::EN, CP = PB::CP, NT = PB::NT, WS = NT < 32 ? NT : 32;
  const int lane = lt % CP, t = lt / CP, nC = J.nC, nWin = J.nWin, nPair = (nC - 1) / 2;
  __shared__ float2 part[(NT + 31) / 32];
  cpair z[EN];
  const float2* twN = g_stw + stw_offset(N, EN);
  const float2* twW = g_tw + tw_offset(W);
  const size_t col = ((size_t)comp * nWin + xl) * nWin;
  cpair x[EN];  // element t + i*T of this lane's columns, in registers through the transforms
  b1_load<N, T, EN>(J, comp, nWin, xl, t, x);
  const int ab = comp - 1, a = ab / nPair, cn = 2 * (ab % nPair) + 1;
  const float2* re = J.ramps + (size_t)(a * nC + cn) * 2 * W + W;  // y ramps
  const float2* ro = re + N;
  {  // sum over rows of (-1)^y D(y): the 2D Nyquist corner of the component
    float2 z = make_float2(0.f, 0.f);
    for (int y = lt; y < N; y += NT) z = cadd(z, J.D[(size_t)ab * N + y]);  // NT is even: one parity per thread
    if (lt & 1) z = make_float2(-z.x, -z.y);
#pragma unroll
    for (int o = WS / 2; o > 0; o >>= 1) {
      z.x += __shfl_down_sync(0xffffffffu >> (32 - WS), z.x, o);
      z.y += __shfl_down_sync(0xffffffffu >> (32 - WS), z.y, o);
    }
    if (lt % 32 == 0) part[lt / 32] = z;  // read after the transforms' barriers
  }
  // even samples times the even-sample ramp, FFT: E (changes places with the column)
#pragma unroll
  for (int i = 0; i < EN; i++) {
    z[i] = x[i];
    x[i] = cmul(x[i], w_dup(__ldg(re + t + i * T)));
  }
  line_fft_pair<N, T, CP, false>(x, s, lane, t, twN);
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const cpair e = x[i];
    x[i] = z[i];
    z[i] = e;
  }
  line_fft_pair<N, T, CP, false>(x, s, lane, t, twN);  // Z along y
  const float2* nx = J.nyq + (size_t)ab * 2 * nWin;  // Qx over the window columns, Qy over its rows
  __shared__ float2 szc[CM || EDGE ? CB : 1];
  cpair zq = cp_zero();
  if (t == (N / 2) % T) {
    float2 z = part[0];
    for (int k = 1; k < (NT + 31) / 32; k++) z = cadd(z, part[k]);
    if constexpr (CM || EDGE) cp_split(x[(N / 2) / T], szc[2 * lane], szc[2 * lane + 1]);  // read after barriers
    z = make_float2(-z.x, -z.y);
    zq = cp_make(cmul(z, __ldg(nx + xl)), cmul(z, __ldg(nx + xl + 1)));
  }
  // odd samples, iFFT_N(Z * s), times the odd-sample ramp, FFT: O
#pragma unroll
  for (int i = 0; i < EN; i++) x[i] = cmul(x[i], w_dup(half_shift<N>(twW, t + i * T)));
  if (t == (N / 2) % T) x[(N / 2) / T] = zq;
  line_fft_pair<N, T, CP, true>(x, s, lane, t, twN);
#pragma unroll
  for (int i = 0; i < EN; i++) x[i] = cmul(x[i], w_dup(__ldg(ro + t + i * T)));
  line_fft_pair<N, T, CP, false>(x, s, lane, t, twN);
  // shifted column E[Y mod N] + exp(-2 pi i Y/W) O[Y mod N] over the row window (as pass A's)
  const int Ys = J.win[2 * (a * nC + cn) + 1];
  auto finish = [&](int yl, cpair v) {
    if constexpr (CM) {  // Re(m) v + Im(m) (Ty Qx z + Qy Tx z)
      const float2 gy = J.G[(size_t)ab * nWin + yl], qy = __ldg(nx + nWin + yl);
      const float2* mk = reinterpret_cast<const float2*>(J.masks) + col + yl;
      float2 r[2];
      cp_split(v, r[0], r[1]);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float2 m = __ldg(mk + h * nWin), q = cadd(cmul(__ldg(nx + xl + h), gy), cmul(qy, szc[2 * lane + h]));
        J.Tw[col + (size_t)h * nWin + yl] = make_float2(m.x * r[h].x + m.y * q.x, m.x * r[h].y + m.y * q.y);
      }
    } else {
      b1_put<CM>(J, col, nWin, yl, v);
    }
  };
#pragma unroll
  for (int i = 0; i < EN; i++) {
    int yl = t + i * T - Ys;
    if (yl < 0) yl += W;
    if (yl >= N) yl -= N;
    if (yl < nWin) {
      int Y = Ys + yl;
      if (Y >= W) Y -= W;
      const cpair o = cmul(x[i], w_dup(__ldg(twW + Y)));
      finish(yl, cadd(z[i], o));
      if (yl + N < nWin) finish(yl + N, csub(z[i], o));
    }
  }
  if constexpr (EDGE) {
    b1_edges<N, T>(J, ab, xl, t, x, z, [&](int yl, int h) {
      return cadd(cmul(__ldg(nx + xl + h), J.G[(size_t)ab * nWin + yl]), cmul(__ldg(nx + nWin + yl), szc[2 * lane + h]));
    });
  }
}

template <int N, int ENV, int CBV, bool CM>
__global__ void __launch_bounds__(PassB1<N, ENV, CBV>::NT, PassB1<N, ENV, CBV>::MINB)
    k_pass_b0(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV, CBV>;
  using PB = PassB1<N, ENV, CBV>;
  const int lt = threadIdx.x, x0 = blockIdx.x * P::CB;
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  load_job(&J, jobs + blockIdx.y, lt, PB::NT);
  __syncthreads();
  if ((J.cmask != 0) != CM || J.edge || x0 >= J.nWin) return;  // another launch's job (uniform per block)
  // the thread's columns xl and xl + 1: nWin is a multiple of 4, both are inside
  b1_band0<N, ENV, CBV, CM>(J, x0 + 2 * (lt % PB::CP), lt % PB::CP, lt / PB::CP, smp);
}
template <int N, int ENV, int CBV, bool CM>
__global__ void __launch_bounds__(PassB1<N, ENV, CBV>::NT, PassB1<N, ENV, CBV>::MINB)
    k_pass_b1(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV, CBV>;
  using PB = PassB1<N, ENV, CBV>;
  const int lt = threadIdx.x, x0 = blockIdx.x * P::CB, comp = 1 + blockIdx.y;
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  load_job(&J, jobs + blockIdx.z, lt, PB::NT);
  __syncthreads();
  if ((J.cmask != 0) != CM || J.edge || comp > J.nA * (J.nC - 1) / 2 || x0 >= J.nWin) return;  // uniform per block
  b1_pair<N, ENV, CBV, CM, false>(J, comp, x0 + 2 * (lt % PB::CP), lt, smp);
}
// Band 0 and the pairs in one launch: the form of dependent launches, whose blocks all wait for pass A
// (and G) before they read what it wrote, and of the jobs with edge weights (EDGE). Band 0, the shorter
// work, comes last of all jobs (4 x 1024^2 358 us, 366 with it last of each job; 7 x 384^2 three-band 197, 202), but
// job by job where 12 elements per thread make blocks of 128 threads (4 x 768^2 231 us, 240 the other way): four
// of those fill an SM. As ordinary launches the two kernels are faster: band 0 by itself needs fewer
// registers (16 x 512^2 306 us, 309 in one).
template <int N, int ENV, int CBV, bool CM, bool EDGE>
__global__ void __launch_bounds__(PassB1<N, ENV, CBV>::NT, PassB1<N, ENV, CBV>::MINB)
    k_pass_b01(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV, CBV>;
  using PB = PassB1<N, ENV, CBV>;
  constexpr bool BYJOB = PB::BYJOB;
  const int lt = threadIdx.x, x0 = blockIdx.x * P::CB;
  const int c = BYJOB ? blockIdx.y : blockIdx.z, comp = c + 1 < (int)(BYJOB ? gridDim.y : gridDim.z) ? c + 1 : 0;
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  load_job(&J, jobs + (BYJOB ? blockIdx.z : blockIdx.y), lt, PB::NT);  // written before pass A
  pdl_wait();
  __syncthreads();
  if ((J.cmask != 0) != CM || (J.edge != nullptr) != EDGE || comp > J.nA * (J.nC - 1) / 2 || x0 >= J.nWin)
    return;  // uniform per block
  const int lane = lt % PB::CP, xl = x0 + 2 * lane;
  if (comp == 0) b1_band0_call<N, ENV, CBV, CM>(J, xl, lane, lt / PB::CP, smp);
  else b1_pair<N, ENV, CBV, CM, EDGE>(J, comp, xl, lt, smp);
  pdl_trigger();
}

// ---- pass B2: Hermitian sum over components, Wiener x apodization, inverse along y -------------
// The image is real: out = Re iFFT2(F) = iFFT2(H) with the Hermitian part
// H(X, Y) = S(X, Y) + conj S(-X, -Y) of pass B1's masked windows, so only the columns
// X = 0..N of H are formed and stored (pass C completes each row by symmetry).
// CB output columns per block, T threads per column: each thread keeps the rows k = t + i*T
// and k + N of its column in registers. Each window column is contiguous, at X for
// the direct term and at -X, read backwards, for the mirrored one, so a warp's loads are
// whole sectors at any window origin; all loads of a window column are issued before they
// are added.
// iFFT_W along y as two N-point inverse FFTs of one line pair:
//   out[2n] = iFFT_N(A[k] + A[k+N]),  out[2n+1] = iFFT_N((A[k] - A[k+N]) exp(i pi k/N)).
template <int N, int ENV, int CBV>
struct PassB2 {
  using P = Cfg<N, ENV, CBV>;
  static constexpr int NT = P::CB * P::T;
  static constexpr size_t SMEM = sizeof(ulonglong2) * (size_t)pair_elems(N, P::CB);
  // 80 registers hold the sums without spills (64 x 512^2: 207 us, 240 at 64); at 512 threads they leave
  // one block per SM, and 64 leave two (a 2048^2 3x5 stack: 94 -> 86 us)
  static constexpr int MINB = pair_min_blocks(NT, P::EN, NT >= 512 ? 64 : 80);
};
template <int N, int ENV, int CBV, bool EDGE>
__global__ void __launch_bounds__(PassB2<N, ENV, CBV>::NT, PassB2<N, ENV, CBV>::MINB)
    k_pass_b2(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N, ENV, CBV>;
  constexpr int W = P::W, T = P::T, CB = P::CB, EN = P::EN, NT = CB * T;
  const int lt = threadIdx.x, lane = lt % CB, t = lt / CB;
  const int X = blockIdx.x * CB + lane;  // X <= N + CB - 1 < W; only X <= N is stored
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  const float2* twN = g_stw + stw_offset(N, EN);
  const float2* twW = g_tw + tw_offset(W);
  load_job(&J, jobs + blockIdx.y, lt, NT);
  pdl_trigger();
  pdl_wait();
  __syncthreads();
  if ((J.edge != nullptr) != EDGE) return;  // another launch's job (uniform per block)
  const int nC = J.nC, nWin = J.nWin, nPair = (nC - 1) / 2, nS = 1 + J.nA * nPair;
  auto wrap = [](int v) { return v < 0 ? v + W : (v >= W ? v - W : v); };
  const int Xm = wrap(-X);
  float2 acc[2][EN];  // rows t + i*T, and N beyond
#pragma unroll
  for (int i = 0; i < EN; i++) acc[0][i] = acc[1][i] = make_float2(0.f, 0.f);
  for (int s = 0; s < nS; s++) {
    const int c = s == 0 ? 0 : ((s - 1) / nPair) * nC + 2 * ((s - 1) % nPair) + 1;
    const int Xs = J.win[2 * c], Ys = J.win[2 * c + 1];
    const int xd = wrap(X - Xs), xm = wrap(Xm - Xs);
    const float2* w = J.Tw + (size_t)s * nWin * nWin;
    if (xd < nWin) {
      const float2* col = w + (size_t)xd * nWin;
      float2 u[2][EN];
#pragma unroll
      for (int i = 0; i < EN; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int yl = wrap(t + i * T + h * N - Ys);
          u[h][i] = yl < nWin ? __ldg(col + yl) : make_float2(0.f, 0.f);
        }
#pragma unroll
      for (int i = 0; i < EN; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) acc[h][i] = cadd(acc[h][i], u[h][i]);
    }
    if (xm < nWin) {
      const float2* col = w + (size_t)xm * nWin;
      float2 u[2][EN];
#pragma unroll
      for (int i = 0; i < EN; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int yl = wrap(wrap(-(t + i * T + h * N)) - Ys);
          u[h][i] = yl < nWin ? __ldg(col + yl) : make_float2(0.f, 0.f);
        }
#pragma unroll
      for (int i = 0; i < EN; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) acc[h][i] = make_float2(acc[h][i].x + u[h][i].x, acc[h][i].y - u[h][i].y);
    }
  }
  const float* wa = J.wa + (size_t)(X >> 2) * W * 4 + (X & 3);
  cpair x[EN];  // even rows' sequence, odd rows' sequence
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int k = t + i * T;
    float f0 = __ldg(wa + (size_t)k * 4), f1 = __ldg(wa + (size_t)(k + N) * 4);
    if constexpr (EDGE) {  // pass B1 has weighted the Nyquist column and row
      if (X == N) f0 = f1 = 1.f;
      if (k == 0) f1 = 1.f;
    }
    const float2 u0 = cscale(acc[0][i], f0), u1 = cscale(acc[1][i], f1);
    x[i] = cp_make(cadd(u0, u1), cmul(csub(u0, u1), cconjf(__ldg(twW + k))));
  }
  line_fft_pair<N, T, CB, true>(x, smp, lane, t, twN);
  float2* o = X < N ? J.O + X : J.On;
  const size_t st = X < N ? N : 1;
  if (X <= N) {
#pragma unroll
    for (int i = 0; i < EN; i++) {
      const size_t r = 2 * (size_t)(t + i * T);
      float2 r0, r1;
      cp_split(x[i], r0, r1);
      o[r * st] = r0;
      o[(r + 1) * st] = r1;
    }
  }
}

// ---- pass C: rows of the output (complex-to-real) ------------------------------------------------
// Row y of the image is out[x] = sum_X H[X] exp(+2 pi i x X/W) / W^2 with H[W-X] = conj H[X],
// H[0..N-1] = O[y][.] and H[N] = On[y]. Both halves of the output come from one N-point
// inverse FFT: Z[k] = (H[k] + conj H[N-k]) + i exp(+2 pi i k/W) (H[k] - conj H[N-k]) gives
// iFFT_N(Z)[n] = out[2n] + i out[2n+1] (the two sub-sequences' transforms are real).
// clip != 0 clips negative values (CLIPSCALE.CLIP); clip == 2 also records the image's
// maximum (CLIPSCALE.BOTH: k_scale_clip scales afterwards, before clipping).
template <int N>
__global__ void __launch_bounds__(Cfg<N>::GC* Cfg<N>::T) k_pass_c(const JobDesc* __restrict__ jobs) {
  using P = Cfg<N>;
  constexpr int W = P::W, T = P::T, G = P::GC, EN = P::EN;
  const JobDesc& J = jobs[blockIdx.y];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int y = blockIdx.x * G + g;
  __shared__ float2 sm[G * smem_line_elems(N, 1)];
  // stage twiddles through L1 (a per-block shared copy of the 511-entry table cost a 4 KB
  // copy and a barrier per pair of rows)
  const float2* tw = g_stw + stw_offset(N, EN);
  float2* s = sm + g * smem_line_elems(N, 1);
  const float2* twW = g_tw + tw_offset(W);
  pdl_wait();
  const float2* row = J.O + (size_t)y * N;
  const float2 hn = J.On[y];
  float2 x[EN];  // element t + i*T of Z, in registers through the transform
#pragma unroll
  for (int i = 0; i < EN; i++) {
    const int k = t + i * T;
    const float2 h = row[k];
    const float2 hm = cconjf(k == 0 ? hn : row[N - k]);
    const float2 e = cadd(h, hm), d = cmul(csub(h, hm), cconjf(twW[k]));
    x[i] = make_float2(e.x - d.y, e.y + d.x);  // e + i d
  }
  line_fft_reg<N, T, 1, true>(x, s, 0, t, tw);
  const float scale = 1.f / ((float)W * (float)W);
  const int clip = J.clip;
  float2* out = reinterpret_cast<float2*>(J.out + (size_t)y * W);
  float mx = 0.f;
#pragma unroll
  for (int i = 0; i < EN; i++) {
    float2 v = make_float2(x[i].x * scale, x[i].y * scale);
    if (clip == 2) mx = fmaxf(mx, fmaxf(v.x, v.y));
    if (clip == 1) {
      if (v.x < 0) v.x = 0.f;
      if (v.y < 0) v.y = 0.f;
    }
    out[t + i * T] = v;
  }
  if (clip == 2) {  // non-negative floats order as their bit patterns
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx > 0.f) atomicMax(reinterpret_cast<unsigned int*>(J.clip_max), __float_as_uint(mx));
  }
}

// CLIPSCALE.BOTH (SimUtils.clipAndScale(vec, true, true), S/SimUtils.java:244-264): every pixel
// times 255/max (max over the image, starting at 0), then negative values set to 0.
static __global__ void k_scale_clip(const JobDesc* __restrict__ jobs, int W) {
  const JobDesc& J = jobs[blockIdx.y];
  if (J.clip != 2) return;
  const float f = __fdiv_rn(255.f, *J.clip_max);
  float* out = J.out;
  const size_t n = (size_t)W * W;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v = __fmul_rn(out[i], f);
    if (v < 0) v = 0.f;
    out[i] = v;
  }
}

// ---- launch ----------------------------------------------------------------------------------------
// Each pass has its own launch-shape variants (autotuner: tuning.json); a batch launches
// A, (G,) B1, B2, C in order on one stream; G only where some job needs it.
// Dynamic shared memory of a kernel instantiation, granted once per process.
template <class K>
static int grant_smem(K kern, size_t bytes, bool& done) {
  if (!done) {
    FSIM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done = true;
  }
  return FSIM_OK;
}
template <int N, int ENA>
static int launch_a(const JobDesc* d_jobs, int njobs, int maxA, cudaStream_t st) {
  using PA = PassA<N, ENA>;
  static bool attr = false;
  int rc = grant_smem(k_pass_a<N, ENA>, PA::SMEM, attr);
  if (rc) return rc;
  // blockIdx.x: RB rows; blockIdx.y: the angles' band pairs, then (y == nA) the band-0 rows
  k_pass_a<N, ENA><<<dim3(N / PA::RB, maxA + 1, njobs), PA::NT, PA::SMEM, st>>>(d_jobs);
  return FSIM_OK;
}

template <int N, int ENA>
static int launch_g(bool dep, const JobDesc* d_jobs, int njobs, int maxA, int maxPair, cudaStream_t st) {
  FSIM_CUDA(launch_pass(dep, k_pass_g<N, ENA>, dim3(maxA * maxPair, njobs), Cfg<N, ENA>::T, 0, st, d_jobs));
  return FSIM_OK;
}
// Band 0 and the pairs of one kind of jobs: two launches, or one (k_pass_b01).
template <int N, int ENB, int CBB, bool CM>
static int launch_b_two(const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, cudaStream_t st) {
  using PB = PassB1<N, ENB, CBB>;
  constexpr int CB = 2 * PB::CP;
  static bool attr0 = false, attr = false;
  int rc = grant_smem(k_pass_b0<N, ENB, CBB, CM>, PB::SMEM, attr0);
  if (!rc) rc = grant_smem(k_pass_b1<N, ENB, CBB, CM>, PB::SMEM, attr);
  if (rc) return rc;
  const int gx = (maxWin + CB - 1) / CB;
  k_pass_b0<N, ENB, CBB, CM><<<dim3(gx, njobs), PB::NT, PB::SMEM, st>>>(d_jobs);
  k_pass_b1<N, ENB, CBB, CM><<<dim3(gx, maxA * maxPair, njobs), PB::NT, PB::SMEM, st>>>(d_jobs);
  return FSIM_OK;
}
template <int N, int ENB, int CBB, bool CM, bool EDGE>
static int launch_b_one(bool dep, const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, cudaStream_t st) {
  using PB = PassB1<N, ENB, CBB>;
  constexpr int CB = 2 * PB::CP;
  static bool attr = false;
  int rc = grant_smem(k_pass_b01<N, ENB, CBB, CM, EDGE>, PB::SMEM, attr);
  if (rc) return rc;
  const int gx = (maxWin + CB - 1) / CB, comps = 1 + maxA * maxPair;
  FSIM_CUDA(launch_pass(dep, k_pass_b01<N, ENB, CBB, CM, EDGE>, PB::BYJOB ? dim3(gx, comps, njobs) : dim3(gx, njobs, comps),
                        PB::NT, PB::SMEM, st, d_jobs));
  return FSIM_OK;
}
// jobs without edge weights, in long batches
template <int N, int ENB, int CBB>
static int launch_b1(const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, int kinds, cudaStream_t st) {
  int rc = FSIM_OK;
  if (kinds & JOB_REAL) rc = launch_b_two<N, ENB, CBB, false>(d_jobs, njobs, maxA, maxPair, maxWin, st);
  if (!rc && (kinds & JOB_COMPLEX)) rc = launch_b_two<N, ENB, CBB, true>(d_jobs, njobs, maxA, maxPair, maxWin, st);
  return rc;
}
// the same in one launch, and the jobs with edge weights: one variant
template <int N, int ENB, int CBB>
static int launch_b01(bool dep, const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, int kinds, cudaStream_t st) {
  int rc = FSIM_OK;
  if (kinds & JOB_REAL) rc = launch_b_one<N, ENB, CBB, false, false>(dep, d_jobs, njobs, maxA, maxPair, maxWin, st);
  if (!rc && (kinds & JOB_COMPLEX)) rc = launch_b_one<N, ENB, CBB, true, false>(dep, d_jobs, njobs, maxA, maxPair, maxWin, st);
  if (!rc && (kinds & JOB_REAL_EDGE)) rc = launch_b_one<N, ENB, CBB, false, true>(dep, d_jobs, njobs, maxA, maxPair, maxWin, st);
  if (!rc && (kinds & JOB_COMPLEX_EDGE)) rc = launch_b_one<N, ENB, CBB, true, true>(dep, d_jobs, njobs, maxA, maxPair, maxWin, st);
  return rc;
}
template <int N, int ENB, int CBB, bool EDGE>
static int launch_b2(bool dep, const JobDesc* d_jobs, int njobs, cudaStream_t st) {
  using PB = PassB2<N, ENB, CBB>;
  constexpr int CB = Cfg<N, ENB, CBB>::CB;
  static bool attr = false;
  int rc = grant_smem(k_pass_b2<N, ENB, CBB, EDGE>, PB::SMEM, attr);
  if (rc) return rc;
  FSIM_CUDA(launch_pass(dep, k_pass_b2<N, ENB, CBB, EDGE>, dim3(N / CB + 1, njobs), PB::NT, PB::SMEM, st, d_jobs));  // 0..N
  return FSIM_OK;
}

// tuned variants per size: index into the variant lists of launch_offline
extern int g_var_a[16], g_var_b[16], g_var_b2[16];
__host__ inline int size_slot(int n) {
  switch (n) {
    case 64: return 0;
    case 128: return 1;
    case 192: return 2;
    case 256: return 3;
    case 384: return 4;
    case 512: return 5;
    case 768: return 6;
    case 1024: return 7;
    case 2048: return 8;
  }
  return -1;
}

// variant lists: pass A (and G) elements/thread {E0, E1}; passes B1 (long batches: the form of dependent
// launches has one variant) and B2, each on its own, (elements, columns per block) {(E0,4), (E0,2),
// (E1,4), (E1,2)} with E0 = 8, E1 = 16 (3*2^k sizes: 12, 24). The extremes (N <= 128, N >= 2048) have
// one variant.
template <int N>
int launch_offline(const JobDesc* d_jobs, int njobs, int maxA, int maxPair, int maxWin, bool scale_clip, int kinds,
                   bool alone, cudaStream_t st) {
  constexpr bool p3 = (N % 3 == 0);
  constexpr int E0 = p3 ? 12 : 8, E1 = p3 ? 24 : 16;
  constexpr bool single = (N <= 128 || N >= 2048);
  constexpr int CBX = N >= 2048 ? 2 : 4;
  const int k = size_slot(N);
  const int va = single ? 0 : g_var_a[k], vb1 = single ? 0 : g_var_b[k], vb2 = single ? 0 : g_var_b2[k];
  // Passes as dependent launches while a batch is short (as graphs, without and with: one 256^2 stack 36.9
  // and 30.7 us, 4 x 512^2 101 and 93, 8 x 512^2 167 and 160), but not in a batch of several size classes,
  // whose waiting blocks take the room of another class's passes (3% longer). The line was drawn while
  // pass B was two dependent launches, when 64 x 512^2 took 1183 us without and 1195 with; as one launch,
  // longer batches gain too (16 x 512^2 307 and 297, 64 x 512^2 1100 and 1092).
  const bool dep = alone && (long long)(N / PassA<N, E0>::RB) * (maxA + 1) * njobs <= 64LL * ctx().num_sms;
  cudaEvent_t* ev = profile_events();
  if (ev) cudaEventRecord(ev[0], st);
  int rc = FSIM_OK;
  if (va == 0) rc = launch_a<N, E0>(d_jobs, njobs, maxA, st);
  else if constexpr (!single) rc = launch_a<N, E1>(d_jobs, njobs, maxA, st);
  if (rc) return rc;
  if (ev) cudaEventRecord(ev[1], st);
  if (kinds & ~JOB_REAL) {
    if (va == 0) rc = launch_g<N, E0>(dep, d_jobs, njobs, maxA, maxPair, st);
    else if constexpr (!single) rc = launch_g<N, E1>(dep, d_jobs, njobs, maxA, maxPair, st);
    if (rc) return rc;
  }
  const bool edge = kinds & (JOB_REAL_EDGE | JOB_COMPLEX_EDGE), plain = kinds & (JOB_REAL | JOB_COMPLEX);
  if (!dep) {
    if constexpr (single) {
      rc = launch_b1<N, E0, CBX>(d_jobs, njobs, maxA, maxPair, maxWin, kinds, st);
    } else {
      switch (vb1) {
        case 0: rc = launch_b1<N, E0, 4>(d_jobs, njobs, maxA, maxPair, maxWin, kinds, st); break;
        case 1: rc = launch_b1<N, E0, 2>(d_jobs, njobs, maxA, maxPair, maxWin, kinds, st); break;
        case 2: rc = launch_b1<N, E1, 4>(d_jobs, njobs, maxA, maxPair, maxWin, kinds, st); break;
        default: rc = launch_b1<N, E1, 2>(d_jobs, njobs, maxA, maxPair, maxWin, kinds, st); break;
      }
    }
  }
  const int one = dep ? kinds : kinds & (JOB_REAL_EDGE | JOB_COMPLEX_EDGE);
  if (!rc && one) rc = launch_b01<N, E0, CBX>(dep, d_jobs, njobs, maxA, maxPair, maxWin, one, st);
  if (rc) return rc;
  if (ev) cudaEventRecord(ev[2], st);
  if (plain) {
    if constexpr (single) {
      rc = launch_b2<N, E0, CBX, false>(dep, d_jobs, njobs, st);
    } else {
      switch (vb2) {
        case 0: rc = launch_b2<N, E0, 4, false>(dep, d_jobs, njobs, st); break;
        case 1: rc = launch_b2<N, E0, 2, false>(dep, d_jobs, njobs, st); break;
        case 2: rc = launch_b2<N, E1, 4, false>(dep, d_jobs, njobs, st); break;
        default: rc = launch_b2<N, E1, 2, false>(dep, d_jobs, njobs, st); break;
      }
    }
  }
  if (!rc && edge) rc = launch_b2<N, E0, CBX, true>(dep, d_jobs, njobs, st);
  if (rc) return rc;
  if (ev) cudaEventRecord(ev[3], st);
  using PC = Cfg<N>;
  FSIM_CUDA(launch_pass(dep, k_pass_c<N>, dim3(PC::W / PC::GC, njobs), PC::GC * PC::T, 0, st, d_jobs));
  if (scale_clip) k_scale_clip<<<dim3(2 * N, njobs), 256, 0, st>>>(d_jobs, 2 * N);
  if (ev) {
    cudaEventRecord(ev[4], st);
    profile_mark(4);
  }
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

}  // namespace fsim
