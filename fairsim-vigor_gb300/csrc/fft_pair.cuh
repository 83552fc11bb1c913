// Stockham line FFT of two lines at a time, in the packed single-precision form of sm_103a.
//
// A thread holds the same elements of two lines: `re` packs the two real parts, `im` the two
// imaginary parts, and add/mul/fma.rn.f32x2 work on both lines in one instruction with the
// rounding of the scalar ones. The transforms of fft_line.cuh are bound by instruction issue
// and by the shared-memory pipe together; measured on GB300 (152 SMs, one million iterations in
// registers), a complex butterfly runs at 100 flop per SM and clock packed against 77 scalar,
// a complex product at 124 against 95, in half the issue slots, and everything a line pair
// shares (twiddle loads and powers, table products, addresses) is issued once instead of twice.
// The exchanges move 16-byte elements (both lines' value), which a quarter-warp of eight lanes
// accesses in one wavefront when the eight addresses differ modulo 8.
//
// Same plan as line_fft_reg: x[i] = element t + i*T on entry and exit, T = L / E threads per
// pair, C pairs interleaved in the exchange buffer (element k of pair c at layout(k*C + c)).
#pragma once

#include "fft_line.cuh"

namespace fsim {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 p_pack(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 p_unpack(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 p_dup(float a) { return p_pack(a, a); }
__device__ __forceinline__ f32x2 p_add(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 p_sub(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 p_mul(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 p_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 p_neg(f32x2 v) {  // folds into the consumer's operand
  const float2 r = p_unpack(v);
  return p_pack(-r.x, -r.y);
}

struct cpair {  // one element of two lines
  f32x2 re, im;
};
struct wpair {  // one factor, for both lines
  f32x2 x, y;
};
__device__ __forceinline__ wpair w_dup(float2 w) { return wpair{p_dup(w.x), p_dup(w.y)}; }
__device__ __forceinline__ cpair cp_zero() { return cpair{0ull, 0ull}; }
__device__ __forceinline__ cpair cp_make(float2 a, float2 b) { return cpair{p_pack(a.x, b.x), p_pack(a.y, b.y)}; }
// the element of line 0 / 1
__device__ __forceinline__ void cp_split(cpair v, float2& a, float2& b) {
  const float2 r = p_unpack(v.re), i = p_unpack(v.im);
  a = make_float2(r.x, i.x);
  b = make_float2(r.y, i.y);
}
__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return cpair{p_add(a.re, b.re), p_add(a.im, b.im)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b) { return cpair{p_sub(a.re, b.re), p_sub(a.im, b.im)}; }
__device__ __forceinline__ cpair cmul(cpair v, wpair w) {
  return cpair{p_fma(v.re, w.x, p_neg(p_mul(v.im, w.y))), p_fma(v.im, w.x, p_mul(v.re, w.y))};
}
__device__ __forceinline__ cpair cmulj(cpair v, wpair w) {  // v * conj(w)
  return cpair{p_fma(v.re, w.x, p_mul(v.im, w.y)), p_fma(v.im, w.x, p_neg(p_mul(v.re, w.y)))};
}
__device__ __forceinline__ wpair wmul(wpair a, wpair b) {
  return wpair{p_fma(a.x, b.x, p_neg(p_mul(a.y, b.y))), p_fma(a.x, b.y, p_mul(a.y, b.x))};
}
// a + q w b, a - q w b for w = exp(-+ i pi/4) (K = 1) or exp(-+ 3 i pi/4) (K = 3), q = sqrt(1/2) in
// qq: both products are one addition and one subtraction of b's parts, scaled in the sums' FMAs
template <bool INV, int K>
__device__ __forceinline__ void bfly_w8(cpair a, cpair b, f32x2 qq, cpair& s, cpair& d) {
  const f32x2 u = p_add(b.re, b.im), v = p_sub(b.im, b.re), n = p_neg(qq);
  if constexpr (!INV && K == 1) {  // (u, v)
    s = cpair{p_fma(u, qq, a.re), p_fma(v, qq, a.im)};
    d = cpair{p_fma(u, n, a.re), p_fma(v, n, a.im)};
  } else if constexpr (!INV) {  // (v, -u)
    s = cpair{p_fma(v, qq, a.re), p_fma(u, n, a.im)};
    d = cpair{p_fma(v, n, a.re), p_fma(u, qq, a.im)};
  } else if constexpr (K == 1) {  // (-v, u)
    s = cpair{p_fma(v, n, a.re), p_fma(u, qq, a.im)};
    d = cpair{p_fma(v, qq, a.re), p_fma(u, n, a.im)};
  } else {  // (-u, -v)
    s = cpair{p_fma(u, n, a.re), p_fma(v, n, a.im)};
    d = cpair{p_fma(u, qq, a.re), p_fma(v, qq, a.im)};
  }
}
// a + r b, a - r b for r = -i (forward) / +i (inverse)
template <bool INV>
__device__ __forceinline__ void bfly_rot(cpair a, cpair b, cpair& s, cpair& d) {
  const cpair p = cpair{p_add(a.re, b.im), p_sub(a.im, b.re)}, m = cpair{p_sub(a.re, b.im), p_add(a.im, b.re)};
  s = INV ? m : p;
  d = INV ? p : m;
}

template <bool INV>
__device__ __forceinline__ void dft4(cpair& v0, cpair& v1, cpair& v2, cpair& v3) {
  const cpair t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3), t3 = csub(v1, v3);
  v0 = cadd(t0, t2);
  v2 = csub(t0, t2);
  bfly_rot<INV>(t1, t3, v1, v3);
}
template <bool INV>
__device__ __forceinline__ void dft3(cpair& a, cpair& b, cpair& c) {
  const f32x2 h = p_dup(0.86602540378443864676f), mh = p_dup(-0.5f);
  const cpair s = cadd(b, c), d = csub(b, c);
  const cpair m = cpair{p_fma(s.re, mh, a.re), p_fma(s.im, mh, a.im)};
  a = cadd(a, s);
  const f32x2 n = p_neg(h);  // m +- h r d, r = -i / +i
  const cpair p = cpair{p_fma(d.im, h, m.re), p_fma(d.re, n, m.im)}, q = cpair{p_fma(d.im, n, m.re), p_fma(d.re, h, m.im)};
  b = INV ? q : p;
  c = INV ? p : q;
}
template <bool INV>
__device__ __forceinline__ void dft8(cpair* v) {
  const f32x2 qq = p_dup(0.70710678118654752440f);
  cpair e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  cpair o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<INV>(e0, e1, e2, e3);
  dft4<INV>(o0, o1, o2, o3);
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  bfly_w8<INV, 1>(e1, o1, qq, v[1], v[5]);
  bfly_rot<INV>(e2, o2, v[2], v[6]);
  bfly_w8<INV, 3>(e3, o3, qq, v[3], v[7]);
}
template <bool INV>
__device__ __forceinline__ void dft12(cpair* v) {
  // 3 x 4 without twiddles: with n = 4 n1 + 3 n2 and k = k1 mod 3 = k2 mod 4 (both modulo 12),
  // W12^{nk} = W3^{n1 k1} W4^{n2 k2}
  cpair x[4][3];
#pragma unroll
  for (int n2 = 0; n2 < 4; n2++) {
#pragma unroll
    for (int n1 = 0; n1 < 3; n1++) x[n2][n1] = v[(4 * n1 + 3 * n2) % 12];
    dft3<INV>(x[n2][0], x[n2][1], x[n2][2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < 3; k1++) {
    dft4<INV>(x[0][k1], x[1][k1], x[2][k1], x[3][k1]);
#pragma unroll
    for (int k2 = 0; k2 < 4; k2++) v[(4 * k1 + 9 * k2) % 12] = x[k2][k1];
  }
}
template <bool INV>
__device__ __forceinline__ void dft16(cpair* v) {
  // 4 x 4: sub-DFTs over m for v[q + 4m], twiddle W16^{q*k1}, then DFT4 over q.
  cpair x[4][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    x[q][0] = v[q];
    x[q][1] = v[q + 4];
    x[q][2] = v[q + 8];
    x[q][3] = v[q + 12];
    dft4<INV>(x[q][0], x[q][1], x[q][2], x[q][3]);
  }
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, q = 0.70710678118654752440f;
  const wpair W1 = w_dup(make_float2(c1, s1)), W2 = w_dup(make_float2(q, q)), W3 = w_dup(make_float2(s1, c1));
  auto mulw = [](cpair a, wpair w) { return INV ? cmul(a, w) : cmulj(a, w); };
  x[1][1] = mulw(x[1][1], W1);
  x[1][2] = mulw(x[1][2], W2);
  x[1][3] = mulw(x[1][3], W3);
  x[2][1] = mulw(x[2][1], W2);
  // x[2][2] turns by -+ i inside the last butterfly of k1 = 2
  x[2][3] = mulw(x[2][3], wpair{p_neg(W2.x), W2.y});
  x[3][1] = mulw(x[3][1], W3);
  x[3][2] = mulw(x[3][2], wpair{p_neg(W2.x), W2.y});
  x[3][3] = mulw(x[3][3], wpair{p_neg(W1.x), p_neg(W1.y)});
#pragma unroll
  for (int k1 = 0; k1 < 4; k1++) {
    const cpair a = x[0][k1], b = x[1][k1], c = x[2][k1], d = x[3][k1];
    cpair t0, t1;
    if (k1 == 2) bfly_rot<INV>(a, c, t0, t1);
    else {
      t0 = cadd(a, c);
      t1 = csub(a, c);
    }
    const cpair t2 = cadd(b, d), t3 = csub(b, d);
    v[k1] = cadd(t0, t2);
    v[k1 + 8] = csub(t0, t2);
    bfly_rot<INV>(t1, t3, v[k1 + 4], v[k1 + 12]);
  }
}
template <int R, bool INV>
__device__ __forceinline__ void dft(cpair* v) {
  if constexpr (R == 2) {
    const cpair t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  } else if constexpr (R == 3) dft3<INV>(v[0], v[1], v[2]);
  else if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  else if constexpr (R == 8) dft8<INV>(v);
  else if constexpr (R == 12) dft12<INV>(v);
  else if constexpr (R == 16) dft16<INV>(v);
}

// Exchange layouts: one element of padding per 8, or per 16 where a radix-16 stage writes with
// stride 16; a stage's writes at stride R and its contiguous reads are then free of conflicts
// at power-of-two strides, and the position of element base + offset is layout(base) +
// layout(offset) where no carry reaches the padding, so that a thread's R accesses share one
// address register.
__host__ __device__ constexpr int pair_pad(int R) { return R == 16 ? 4 : 3; }
template <int S>
__host__ __device__ constexpr int pair_lay(int a) { return a + (a >> S); }
__host__ __device__ constexpr int pair_elems(int L, int C) { return L * C + (L * C) / 8 + 1; }

template <int L, int T, int C, int R, int NS, bool INV, bool FIRST, bool LAST, int SIN>
__device__ __forceinline__ void fft_stage_pair(cpair (&x)[L / T], ulonglong2* s, int c, int t, const float2* tw) {
  constexpr int E = L / T, NB = E / R, LR = L / R, SOUT = pair_pad(R);
  constexpr bool ADD_IN = is_pow2(L) || (LR * C) % (1 << SIN) == 0, ADD_OUT = is_pow2(NS * R);
  // stage table [r-1][k]: W^k, and W^2k, W^4k, W^8k where the radix has them; the other powers
  // by products (one rounding beyond the table's)
  constexpr int NT = NS > 1 ? (R > 8 ? 4 : (R >= 8 ? 3 : (R == 2 ? 1 : 2))) : 1;
  float2 tl[NB][NT];
  if constexpr (NS > 1) {
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const int k = (t + b * T) % NS;
      tl[b][0] = tw[k];
      if constexpr (R >= 3) tl[b][1] = tw[NS + k];
      if constexpr (R >= 8) tl[b][2] = tw[3 * NS + k];
      if constexpr (R > 8) tl[b][3] = tw[7 * NS + k];
    }
  }
  cpair v[NB][R];
#pragma unroll
  for (int b = 0; b < NB; b++) {
    const int rb = (t + b * T) * C + c, lb = pair_lay<SIN>(rb);
#pragma unroll
    for (int r = 0; r < R; r++) {
      if constexpr (FIRST) v[b][r] = x[b + NB * r];
      else {
        const ulonglong2 u = s[ADD_IN ? lb + pair_lay<SIN>(r * LR * C) : pair_lay<SIN>(rb + r * LR * C)];
        v[b][r] = cpair{u.x, u.y};
      }
    }
  }
  if constexpr (!FIRST) __syncthreads();
#pragma unroll
  for (int b = 0; b < NB; b++) {
    const int j = t + b * T;
    const int k = j % NS;
    if constexpr (NS > 1) {
      wpair w[R];
      w[1] = w_dup(tl[b][0]);
      if constexpr (R >= 3) w[2] = w_dup(tl[b][1]);
      if constexpr (R >= 4) w[3] = wmul(w[2], w[1]);
      if constexpr (R >= 8) {
        w[4] = w_dup(tl[b][2]);
#pragma unroll
        for (int r = 5; r < 8; r++) w[r] = wmul(w[4], w[r - 4]);
      }
      if constexpr (R > 8) {
        w[8] = w_dup(tl[b][3]);
#pragma unroll
        for (int r = 9; r < R; r++) w[r] = wmul(w[8], w[r - 8]);
      }
#pragma unroll
      for (int r = 1; r < R; r++) v[b][r] = INV ? cmulj(v[b][r], w[r]) : cmul(v[b][r], w[r]);
    }
    dft<R, INV>(v[b]);
    if constexpr (LAST) {
#pragma unroll
      for (int r = 0; r < R; r++) x[b + NB * r] = v[b][r];
    } else {
      const int wb = ((j / NS) * NS * R + k) * C + c, lb = pair_lay<SOUT>(wb);
#pragma unroll
      for (int r = 0; r < R; r++)
        s[ADD_OUT ? lb + pair_lay<SOUT>(r * NS * C) : pair_lay<SOUT>(wb + r * NS * C)] =
            make_ulonglong2(v[b][r].re, v[b][r].im);
    }
  }
  if constexpr (!LAST) __syncthreads();
}
template <int L, int T, int C, bool INV, int NS, int SIN>
__device__ __forceinline__ void fft_stages_pair(cpair (&x)[L / T], ulonglong2* s, int c, int t, const float2* tw) {
  constexpr int R = pick_radix_pair(L / NS, L / T);
  static_assert((L / NS) % R == 0 && (L / T) % R == 0, "bad radix plan");
  fft_stage_pair<L, T, C, R, NS, INV, NS == 1, NS * R == L, SIN>(x, s, c, t, tw);
  if constexpr (NS * R < L) fft_stages_pair<L, T, C, INV, NS * R, pair_pad(R)>(x, s, c, t, tw + (R - 1) * NS);
}
// Transform pair c of C interleaved line pairs held in registers (x[i] = element t + i*T), with
// `s` (pair_elems(L, C) elements) as scratch; stage tables (g_stw layout). Called by all threads
// of the block (it contains __syncthreads); `s` must not be in use on entry and is free on return.
template <int L, int T, int C, bool INV>
__device__ __forceinline__ void line_fft_pair(cpair (&x)[L / T], ulonglong2* s, int c, int t, const float2* stw) {
  static_assert(supported_len(L) && plan_ok(L, T) && stw_ok(L, L / T), "no stage table for this plan");
  fft_stages_pair<L, T, C, INV, 1, 3>(x, s, c, t, stw + (pair_own_plan(L, L / T) ? stw_plan_len(L, L / T, false) : 0));
}

}  // namespace fsim
