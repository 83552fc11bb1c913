// Widefield side outputs of the offline reconstruction (SimAlgorithm.runReconstruction's
// Wiener path, S/SimAlgorithm.java:533-576):
//   "Widefield"          = spatial(sum over directions a of placeFreq(band0_a))
//   "filtered Widefield" = spatial(placeFreq(sum_a band0_a) * conj(OTF_0) * 1/(2 |OTF_0|^2 + w^2)
//                          inside the OTF support)   (WienerFilter.getWidefieldDenominator,
//                          S/WienerFilter.java:129-139; OtfProvider.maskOtf at (0, 0));
//                          the product of the three factors is a resident per-plan table
// Band separation is linear, so sum_a band0_a = FFT_N(sum_{a,p} M^-1_a[0][p] * prep(raw_{a,p})):
// one N x N transform per dataset. The 2N x 2N inverse of the pasted spectrum splits into
// N-point inverse FFTs of the even and odd output samples (as in the main passes):
//   out[2m]   = iFFT_N(S)[m],   out[2m+1] = iFFT_N(S * s)[m],   s(k) = exp(+i pi k~/N)
// along each axis (k~ the pasted signed frequency), scaled by 1/W^2 once at the end. The
// filter of the pasted grid equals the filter of the N grid at the source index (both use
// the same signed coordinates and cycles per micron), so it is applied before pasting.
// Three passes per dataset, run after pass C in the job's own (then free) workspace, each on line
// pairs (two adjacent rows or columns per thread group, fft_pair.cuh), as the main passes:
//   WA rows:    band-0 mix over all frames, FFT_N along x            -> Wf [N][N]
//   WB columns: FFT_N along y, (filter), even/odd inverse along y    -> V_o [W][N], o = 0, 1
//   WC rows:    even/odd inverse along x (one transform: the two real parts
//               from the Hermitian halves), 1/W^2                     -> widefield / fwf [W][W]
// On single lines the passes took 44 + 70 + 62 us per 16 x 512^2 (cold), on pairs 32 + 53 + 58: the
// batch with both images 513 -> 490 us. WC waits on memory: at 56 registers (18 blocks of 64 threads
// per SM) the batch is 3 us faster than at 64, at 48 it spills; WB keeps the spectrum beside a
// transform: 96 registers.
// Algorithmic bytes per dataset (f32 raw): nA nP 4N^2 + 8N^2 | 8N^2 + 4N^2 + 2 x 16N^2 |
// 2 x (16N^2 + 16N^2).
#include "recon_kernels.cuh"

namespace fsim {

template <int N>
struct WfCfg {
  static constexpr int W = 2 * N;
  static constexpr int E = (N % 3 == 0) ? 12 : 8;   // elements per thread of an N-length line
  static constexpr int T = N / E;                   // threads per line pair
  static constexpr int G = T >= 64 ? 1 : 64 / T;    // row pairs per block, WA and WC
  static constexpr int CP = T >= 128 ? 2 : 4;       // column pairs per block, WB
  static constexpr int XR = pair_elems(N, 1);       // exchange buffers
  static constexpr size_t SMEM_R = sizeof(ulonglong2) * (size_t)G * XR;
  static constexpr size_t SMEM_C = sizeof(ulonglong2) * (size_t)pair_elems(N, CP);
};

size_t widefield_ws_bytes(int n) {
  // Wf (N*N) then V_0 and V_1 (W*N each), complex
  return (size_t)n * n * sizeof(float2) * 5;
}

// WA: G row pairs per block; rows y, y + 1 of sum_{a,p} c0[a][p] * prep(raw[a][p]), FFT_N along x.
template <int N>
__global__ void __launch_bounds__(WfCfg<N>::G* WfCfg<N>::T, pair_min_blocks(WfCfg<N>::G* WfCfg<N>::T, WfCfg<N>::E, 80))
    k_wf_rows(const JobDesc* __restrict__ jobs) {
  using P = WfCfg<N>;
  constexpr int E = P::E, T = P::T, G = P::G;
  __shared__ JobDesc J;
  __shared__ float2 c0[FSIM_MAX_DIRS * FSIM_MAX_PHASES];
  extern __shared__ ulonglong2 smp[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  load_job(&J, jobs + blockIdx.y, threadIdx.x, G * T);
  __syncthreads();
  if (!J.widefield && !J.fwf) return;  // uniform per block
  const int nA = J.nA, nP = J.nP, nC = J.nC, nF = nA * nP;
  for (int i = threadIdx.x; i < nF; i += G * T) c0[i] = J.coef[((i / nP) * nC) * nP + i % nP];
  __syncthreads();
  const int y = 2 * (blockIdx.x * G + g);  // N is a multiple of 2 G
  const size_t frame = (size_t)N * N, row = (size_t)y * N;
  cpair x[E];
#pragma unroll
  for (int i = 0; i < E; i++) x[i] = cp_zero();
#pragma unroll 1
  for (int f = 0; f < nF; f++) {
    float v[2][E];
    raw_rows<N, E, T>(J, f * frame, row, t, v);
    const wpair m = w_dup(c0[f]);
#pragma unroll
    for (int i = 0; i < E; i++) {
      const f32x2 r = p_pack(v[0][i], v[1][i]);
      x[i].re = p_fma(m.x, r, x[i].re);
      x[i].im = p_fma(m.y, r, x[i].im);
    }
  }
  damp_rows<N, E, T>(J, row, t, x);
  line_fft_pair<N, T, 1, false>(x, smp + g * P::XR, 0, t, g_stw + stw_offset(N, E));
  float2* o = J.Wf + row + t;
#pragma unroll
  for (int i = 0; i < E; i++) cp_split(x[i], o[i * T], o[N + i * T]);
}

// WB: CP column pairs per block. Columns x, x + 1: FFT_N along y gives the band-0 sum S(x, k); for
// each requested output, the even and odd rows of the 2N-point inverse along y go to V_o.
template <int N>
__global__ void __launch_bounds__(WfCfg<N>::CP* WfCfg<N>::T, pair_min_blocks(WfCfg<N>::CP* WfCfg<N>::T, WfCfg<N>::E, 96))
    k_wf_cols(const JobDesc* __restrict__ jobs) {
  using P = WfCfg<N>;
  constexpr int E = P::E, T = P::T, CP = P::CP, W = P::W;
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  const int lane = threadIdx.x % CP, t = threadIdx.x / CP;
  load_job(&J, jobs + blockIdx.y, threadIdx.x, CP * T);
  __syncthreads();
  if (!J.widefield && !J.fwf) return;  // uniform per block
  const int x = 2 * (blockIdx.x * CP + lane);  // N is a multiple of 2 CP
  const float2* twN = g_stw + stw_offset(N, E);
  const float2* twW = g_tw + tw_offset(W);
  cpair S[E], y[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const float4 v = *reinterpret_cast<const float4*>(J.Wf + (size_t)(t + i * T) * N + x);
    S[i] = cpair{p_pack(v.x, v.z), p_pack(v.y, v.w)};
  }
  line_fft_pair<N, T, CP, false>(S, smp, lane, t, twN);
  for (int o = 0; o < 2; o++) {
    if (!(o == 0 ? J.widefield : J.fwf)) continue;  // uniform per block
    if (o == 1) {  // the plan's resident filter (k_build_wff)
#pragma unroll
      for (int i = 0; i < E; i++) {
        const float2 w = __ldg(reinterpret_cast<const float2*>(J.wff + (size_t)(t + i * T) * N + x));
        const f32x2 f = p_pack(w.x, w.y);
        S[i] = cpair{p_mul(S[i].re, f), p_mul(S[i].im, f)};
      }
    }
    float2* V = J.Wf + (size_t)N * N + (size_t)o * W * N + x;
    auto put = [&](int odd) {
#pragma unroll
      for (int i = 0; i < E; i++) {
        float2 a, b;
        cp_split(y[i], a, b);
        *reinterpret_cast<float4*>(V + (size_t)(2 * (t + i * T) + odd) * N) = make_float4(a.x, a.y, b.x, b.y);
      }
    };
#pragma unroll
    for (int i = 0; i < E; i++) y[i] = S[i];
    line_fft_pair<N, T, CP, true>(y, smp, lane, t, twN);
    put(0);
#pragma unroll
    for (int i = 0; i < E; i++) y[i] = cmul(S[i], w_dup(half_shift<N>(twW, t + i * T)));
    line_fft_pair<N, T, CP, true>(y, smp, lane, t, twN);
    put(1);
  }
}

// WC: G row pairs per block of output o = blockIdx.y. Rows Y, Y + 1 of V_o: even and odd columns of
// the 2N-point inverse along x, real part, scaled by 1/W^2 (JTransforms complexInverse, scale).
template <int N>
__global__ void __launch_bounds__(WfCfg<N>::G* WfCfg<N>::T, pair_min_blocks(WfCfg<N>::G* WfCfg<N>::T, WfCfg<N>::E, 56))
    k_wf_out(const JobDesc* __restrict__ jobs) {
  using P = WfCfg<N>;
  constexpr int E = P::E, T = P::T, G = P::G, W = P::W;
  __shared__ JobDesc J;
  extern __shared__ ulonglong2 smp[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  load_job(&J, jobs + blockIdx.z, threadIdx.x, G * T);
  __syncthreads();
  const int o = blockIdx.y;
  float* out = o == 0 ? J.widefield : J.fwf;
  if (!out) return;  // uniform per block
  const int Y = 2 * (blockIdx.x * G + g);  // W is a multiple of 2 G
  const float2* twN = g_stw + stw_offset(N, E);
  const float2* twW = g_tw + tw_offset(W);
  const float2* V = J.Wf + (size_t)N * N + (size_t)o * W * N + (size_t)Y * N;
  ulonglong2* s = smp + g * P::XR;
  // Only the real parts of iFFT_N(a) (even columns, a = v) and iFFT_N(b) (odd columns,
  // b = v * s) are kept. Re(iFFT(a)) = iFFT(Ha), Ha[k] = (a[k] + conj(a[-k]))/2 is real, so
  // one transform of Ha + i Hb gives both: even columns in its real part, odd in its imaginary.
  cpair y[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int k = t + i * T;
    y[i] = cp_make(V[k], V[N + k]);
    s[pair_lay<3>(k)] = make_ulonglong2(y[i].re, y[i].im);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int k = t + i * T, km = k == 0 ? 0 : N - k;
    const ulonglong2 u = s[pair_lay<3>(km)];
    const cpair a = y[i], am = cpair{u.x, u.y};
    const float2 w = half_shift<N>(twW, k);  // s(-k) = conj s(k), but the pasted Nyquist bin is its own
    const cpair b = cmul(a, w_dup(w)), bm = cmul(am, w_dup(make_float2(w.x, k == N / 2 ? w.y : -w.y)));
    // 2 (Ha + i Hb)
    y[i] = cpair{p_sub(p_add(a.re, am.re), p_sub(b.im, bm.im)), p_add(p_sub(a.im, am.im), p_add(b.re, bm.re))};
  }
  __syncthreads();  // the mirrored reads are done before the transform writes the scratch
  line_fft_pair<N, T, 1, true>(y, s, 0, t, twN);
  const f32x2 sc = p_dup(0.5f * (float)(1.0 / ((double)W * (double)W)));
  float2* orow = reinterpret_cast<float2*>(out + (size_t)Y * W) + t;
#pragma unroll
  for (int i = 0; i < E; i++) cp_split(cpair{p_mul(y[i].re, sc), p_mul(y[i].im, sc)}, orow[i * T], orow[N + i * T]);
}

// The filtered widefield's filter on the N grid, built once per plan: conj(OTF_0) (the OTF
// table is real), times 1/(|OTF_0|^2 + |OTF_0|^2 + (float)(wiener^2)), zero where the
// frequency lies beyond the cutoff: OtfProvider.otfToVector (S/OtfProvider.java:331-373, no
// attenuation), WienerFilter.getWidefieldDenominator (S/WienerFilter.java:129-139, from
// addWienerDenominator at band 0, java:46-79) and OtfProvider.maskOtf(0, 0) (java:538-559).
// Table positions as otf_pos_ff (the reference's double-precision radius, MTool.fhypot, at
// the boundaries of its tests); coordinates x~ = x < N/2 ? x : x - N, y~ = y < N/2 ? -y : N - y.
__global__ void k_build_wff(float* __restrict__ f, int N, const OtfTable* __restrict__ otf, float wp) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= N) return;
  float2 o;
  float v = 0.f;
  if (otf_at_fast(*otf, 0, freq_x(x, N), freq_y(y, N), FShift{0.f, 0.f, 0.f, 0.f}, 0, 0, false, &o)) {
    const float a2 = __fmul_rn(o.x, o.x);
    v = __fmul_rn(o.x, __frcp_rn(__fadd_rn(__fadd_rn(a2, a2), wp)));
  }
  f[(size_t)y * N + x] = v;
}

int build_widefield_filter(float* d_wff, int n, const OtfTable* d_otf, float wp, cudaStream_t st) {
  k_build_wff<<<dim3(div_up(n, 128), n), 128, 0, st>>>(d_wff, n, d_otf, wp);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

template <int N>
static int launch_wf(const JobDesc* d_jobs, int njobs, cudaStream_t st) {
  using P = WfCfg<N>;
  static bool attr_r = false, attr_c = false, attr_o = false;
  int rc = grant_smem(k_wf_rows<N>, P::SMEM_R, attr_r);
  if (!rc) rc = grant_smem(k_wf_cols<N>, P::SMEM_C, attr_c);
  if (!rc) rc = grant_smem(k_wf_out<N>, P::SMEM_R, attr_o);
  if (rc) return rc;
  k_wf_rows<N><<<dim3(N / (2 * P::G), njobs), P::G * P::T, P::SMEM_R, st>>>(d_jobs);
  k_wf_cols<N><<<dim3(N / (2 * P::CP), njobs), P::CP * P::T, P::SMEM_C, st>>>(d_jobs);
  k_wf_out<N><<<dim3(P::W / (2 * P::G), 2, njobs), P::G * P::T, P::SMEM_R, st>>>(d_jobs);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

int launch_widefield_size(int n, const JobDesc* d_jobs, int njobs, cudaStream_t st) {
  switch (n) {
#define CASE(v) \
  case v:       \
    return launch_wf<v>(d_jobs, njobs, st);
    CASE(64) CASE(128) CASE(192) CASE(256) CASE(384) CASE(512) CASE(768) CASE(1024) CASE(2048)
#undef CASE
  }
  set_error("widefield: unsupported image size %d", n);
  return FSIM_EINVAL;
}

}  // namespace fsim
