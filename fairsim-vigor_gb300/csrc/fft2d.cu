// 2D complex FFT (the replacement of the reference's cufftExecC2C path,
// accel/cuda_cplx.cu:475-514) built from the line-pair FFT of fft_pair.cuh:
//   pass 1: rows    - two adjacent rows per thread group, coalesced row loads;
//   pass 2: columns - pairs of adjacent columns, CP pairs interleaved in shared memory so that
//           every global access of a row moves CP * 16 contiguous bytes.
// Small power-of-two arrays run line by line instead (lines_faster, below).
// Each pass reads and writes the array once (16 bytes per complex element per pass): 16 planes of
// 1024^2 in 112 us on GB300, 134 one line at a time (79 at the rate of a plain copy); the column
// pass, with 64-byte pieces of each row, is the slower one.
// Twiddles come from the per-stage tables, read through L1; lines enter and leave the transform
// in registers.
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "fft_pair.cuh"
#include "runtime.cuh"
#include "vec_ops.cuh"

namespace fsim {

// 8 elements of both lines per thread (12 for 3*2^k lengths, 4 for the shortest).
template <int L>
struct LinePlan {
  static constexpr int E = (L % 3 == 0) ? 12 : (L >= 64 ? 8 : 4);
  static constexpr int T = L / E;
  static constexpr int G = T >= 128 ? 1 : 128 / T;                     // row pairs per block
  // column pairs per block; two at the longest lines although one block then fills an SM: one pair reads 16
  // bytes of every row, half a sector (4096^2: 176 us, 141 with two)
  static constexpr int CP = T >= 256 ? 2 : (T >= 32 ? 4 : 8);
  static constexpr int R = E <= 8 ? 64 : 128;                          // registers per thread
  static constexpr int blocks(int threads) { return 65536 / (threads * R) > 0 ? 65536 / (threads * R) : 1; }
};

template <int L, bool INV>
__global__ void __launch_bounds__(LinePlan<L>::G* LinePlan<L>::T, LinePlan<L>::blocks(LinePlan<L>::G* LinePlan<L>::T))
    k_fft_rows(float2* __restrict__ data, int nrows, size_t item_stride, float scale) {
  using P = LinePlan<L>;
  constexpr int T = P::T, E = P::E;
  extern __shared__ ulonglong2 smp[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int row = 2 * (blockIdx.x * P::G + g);  // nrows is even
  const bool in = row < nrows;
  float2* base = data + blockIdx.y * item_stride + (size_t)row * L + t;
  cpair x[E];  // element t + i*T of both rows: in and out of the transform in registers
#pragma unroll
  for (int i = 0; i < E; i++) x[i] = in ? cp_make(base[i * T], base[L + i * T]) : cp_zero();
  line_fft_pair<L, T, 1, INV>(x, smp + g * pair_elems(L, 1), 0, t, g_stw + stw_offset(L, E));
  if (in) {
    const f32x2 sc = p_dup(scale);
#pragma unroll
    for (int i = 0; i < E; i++) {
      float2 a, b;
      cp_split(cpair{p_mul(x[i].re, sc), p_mul(x[i].im, sc)}, a, b);
      base[i * T] = a;
      base[L + i * T] = b;
    }
  }
}

// A16: the columns' pairs are 16-byte aligned (the base address and the row length allow it)
template <int L, bool INV, bool A16>
__global__ void __launch_bounds__(LinePlan<L>::CP* LinePlan<L>::T, LinePlan<L>::blocks(LinePlan<L>::CP* LinePlan<L>::T))
    k_fft_cols(float2* __restrict__ data, int ncols, size_t item_stride, float scale) {
  using P = LinePlan<L>;
  constexpr int T = P::T, E = P::E, CP = P::CP;
  extern __shared__ ulonglong2 smp[];
  const int lane = threadIdx.x % CP, t = threadIdx.x / CP;
  const int x = 2 * (blockIdx.x * CP + lane);  // ncols is even
  const bool in = x < ncols;
  float2* base = data + blockIdx.y * item_stride + x;
  cpair v[E];  // element t + i*T of both columns: in and out of the transform in registers
#pragma unroll
  for (int i = 0; i < E; i++) {
    const float2* p = base + (size_t)(t + i * T) * ncols;
    if (!in) v[i] = cp_zero();
    else if constexpr (A16) {
      const float4 u = *reinterpret_cast<const float4*>(p);
      v[i] = cpair{p_pack(u.x, u.z), p_pack(u.y, u.w)};
    } else {
      v[i] = cp_make(p[0], p[1]);
    }
  }
  line_fft_pair<L, T, CP, INV>(v, smp, lane, t, g_stw + stw_offset(L, E));
  if (in) {
    const f32x2 sc = p_dup(scale);
#pragma unroll
    for (int i = 0; i < E; i++) {
      float2 a, b;
      cp_split(cpair{p_mul(v[i].re, sc), p_mul(v[i].im, sc)}, a, b);
      float2* p = base + (size_t)(t + i * T) * ncols;
      if constexpr (A16) {
        *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
      } else {
        p[0] = a;
        p[1] = b;
      }
    }
  }
}

template <int L, bool INV>
static int launch_rows(float2* d, int nrows, int batch, size_t stride, float scale, cudaStream_t st) {
  using P = LinePlan<L>;
  const size_t smem = sizeof(ulonglong2) * (size_t)P::G * pair_elems(L, 1);
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(k_fft_rows<L, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = true;
  }
  k_fft_rows<L, INV><<<dim3(div_up(nrows, 2 * P::G), batch), P::G * P::T, smem, st>>>(d, nrows, stride, scale);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}

template <int L, bool INV, bool A16>
static int launch_cols_kind(float2* d, int ncols, int batch, size_t stride, float scale, cudaStream_t st) {
  using P = LinePlan<L>;
  const size_t smem = sizeof(ulonglong2) * (size_t)pair_elems(L, P::CP);
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(k_fft_cols<L, INV, A16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = true;
  }
  k_fft_cols<L, INV, A16><<<dim3(div_up(ncols, 2 * P::CP), batch), P::CP * P::T, smem, st>>>(d, ncols, stride, scale);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}
template <int L, bool INV>
static int launch_cols(float2* d, int ncols, int batch, size_t stride, float scale, cudaStream_t st) {
  // rows are an even number of 8-byte elements long, so every pair is aligned if the base is
  return ((uintptr_t)d % 16) == 0 && stride % 2 == 0 ? launch_cols_kind<L, INV, true>(d, ncols, batch, stride, scale, st)
                                                     : launch_cols_kind<L, INV, false>(d, ncols, batch, stride, scale, st);
}

#define FSIM_FFT_LENGTHS(X) \
  X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768) X(1024) X(1536) X(2048) X(3072) X(4096)

static bool len_ok(int L) {
  switch (L) {
#define CASE(n) case n:
    FSIM_FFT_LENGTHS(CASE)
#undef CASE
    return true;
    default:
      return false;
  }
}

bool fft2d_supported(int w, int h) { return len_ok(w) && len_ok(h); }

// ---- the same transform one line at a time ----------------------------------------------------
// For small arrays (lines_faster), and in the fit: the parameter fit's spectra and getPeak's inverse transforms keep this plan (16 elements per
// thread at 1024 and beyond): the fitted modulations are reported in double, and another order
// of the same roundings moves them by 5e-9 relative, so callers that compare fits would see it.
template <int L>
struct LineOne {
  static constexpr int E = (L % 3 == 0) ? 12 : (L <= 512 ? 8 : 16);
  static constexpr int T = L / E;
  static constexpr int G = T >= 256 ? 1 : 256 / T;  // rows per block in the row pass
  static constexpr int C = (E <= 8) ? (T >= 128 ? 4 : 8) : (L <= 1024 ? 8 : (L <= 3072 ? 4 : 2));
  static constexpr int MINB_R = (E <= 8) ? 4 : 1;
  static constexpr int MINB_C = (E <= 8) ? 65536 / (C * T * 64) : 1;
};
// RAW: the rows come from raw frames (f32 or u16) times the border fade, the imaginary part 0
template <int L, bool INV, bool RAW>
__global__ void __launch_bounds__(LineOne<L>::G* LineOne<L>::T, LineOne<L>::MINB_R)
    k_fft1_rows(float2* __restrict__ data, int nrows, size_t item_stride, const RawFade rf) {
  using P = LineOne<L>;
  constexpr int T = P::T, E = P::E, G = P::G, SL = smem_line_elems(L, 1);
  extern __shared__ float2 sm1[];
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int row = blockIdx.x * G + g;
  float2* base = data + blockIdx.y * item_stride + (size_t)row * L;
  float2 x[E];
  if constexpr (RAW) {
    // a zero the compiler does not see: with a constant one it would order the first stage's
    // roundings differently from the transform of a stored complex row
    float zero;
    asm("mov.f32 %0, 0f00000000;" : "=f"(zero));
    const size_t at = blockIdx.y * item_stride + (size_t)row * L + t;
    float v[E];  // all loads before their first use
#pragma unroll
    for (int i = 0; i < E; i++) v[i] = 0.f;
    if (row < nrows) {
      if (rf.u16) {
#pragma unroll
        for (int i = 0; i < E; i++) v[i] = (float)__ldg((const uint16_t*)rf.raw + at + i * T);
      } else {
#pragma unroll
        for (int i = 0; i < E; i++) v[i] = __ldg((const float*)rf.raw + at + i * T);
      }
      if (rf.fade) {  // fadeBorderCos: the float row factor, then the column's in double
        const float r = __ldg(rf.fy + row);
#pragma unroll
        for (int i = 0; i < E; i++) {
          const int c = t + i * T;
          float f = r;
          if (c < rf.fade || c >= L - rf.fade) f = (float)((double)r * __ldg(rf.fx + c));
          v[i] = __fmul_rn(v[i], f);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < E; i++) x[i] = make_float2(v[i], zero);
  } else {
#pragma unroll
    for (int i = 0; i < E; i++) x[i] = row < nrows ? base[t + i * T] : make_float2(0.f, 0.f);
  }
  line_fft_reg<L, T, 1, INV>(x, sm1 + g * SL, 0, t, g_stw + stw_offset(L, E));
  if (row < nrows) {
#pragma unroll
    for (int i = 0; i < E; i++) base[t + i * T] = x[i];
  }
}
template <int L, bool INV>
__device__ __forceinline__ void fft1_cols_body(float2* __restrict__ data, int ncols, size_t item_stride, float scale) {
  using P = LineOne<L>;
  constexpr int T = P::T, E = P::E, C = P::C;
  extern __shared__ float2 sm1[];
  const int c = threadIdx.x % C, t = threadIdx.x / C;
  const int x = blockIdx.x * C + c;
  float2* base = data + blockIdx.y * item_stride;
  float2 v[E];
#pragma unroll
  for (int i = 0; i < E; i++) v[i] = (x < ncols) ? base[(size_t)(t + i * T) * ncols + x] : make_float2(0.f, 0.f);
  line_fft_reg<L, T, C, INV>(v, sm1, c, t, g_stw + stw_offset(L, E));
  if (x < ncols) {
#pragma unroll
    for (int i = 0; i < E; i++) base[(size_t)(t + i * T) * ncols + x] = cscale(v[i], scale);
  }
}
template <int L, bool INV>
__global__ void __launch_bounds__(LineOne<L>::C* LineOne<L>::T, LineOne<L>::MINB_C)
    k_fft1_cols(float2* __restrict__ data, int ncols, size_t item_stride, float scale) {
  fft1_cols_body<L, INV>(data, ncols, item_stride, scale);
}
// longer plans: the compiler's own register choice (a bound of 512 threads raised it from
// 96 to 121 registers at 1024)
template <int L, bool INV>
__global__ void k_fft1_cols_wide(float2* __restrict__ data, int ncols, size_t item_stride, float scale) {
  fft1_cols_body<L, INV>(data, ncols, item_stride, scale);
}
template <int L, bool INV>
constexpr auto cols1_kernel() {
  if constexpr (LineOne<L>::E <= 8) return k_fft1_cols<L, INV>;
  else return k_fft1_cols_wide<L, INV>;
}
// In small arrays the pairs' half as many threads and, at 1024 and beyond, one exchange more show as
// latency: 64^2 3.6 us, 3.3 by lines, 256^2 5.4 and 5.2, 1024^2 11.0 and 10.1, 256 x 1024 8.5 and 7.7, 512 x 2048 11.2
// and 10.3; 4 x 512^2 take 9.0 either way, 2 x 1024^2 16.0 and 17.4. Lengths 3*2^k are faster in pairs at
// every size (768^2 9.5, 11.4 by lines).
static bool lines_faster(int w, int h, int batch) {
  auto ok = [](int L) { return (L & (L - 1)) == 0 && L >= 64; };
  return ok(w) && ok(h) && (size_t)w * h * batch <= (size_t)(std::max(w, h) >= 1024 ? 1 << 20 : 1 << 19);
}
template <int L, bool INV>
static int line_rows(float2* d, int nrows, int batch, size_t stride, cudaStream_t st) {
  using P = LineOne<L>;
  const size_t smem = sizeof(float2) * (size_t)P::G * smem_line_elems(L, 1);
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(k_fft1_rows<L, INV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = true;
  }
  k_fft1_rows<L, INV, false><<<dim3(div_up(nrows, P::G), batch), P::G * P::T, smem, st>>>(d, nrows, stride, RawFade{});
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}
template <int L, bool INV>
static int line_cols(float2* d, int ncols, int batch, size_t stride, float scale, cudaStream_t st) {
  using P = LineOne<L>;
  const size_t smem = sizeof(float2) * smem_line_elems(L, P::C);
  auto cols = cols1_kernel<L, INV>();
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = true;
  }
  cols<<<dim3(div_up(ncols, P::C), batch), P::C * P::T, smem, st>>>(d, ncols, stride, scale);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}
static int lines_2d(float2* d, int w, int h, bool inv, cudaStream_t st, int batch) {
  const size_t stride = (size_t)w * h;
  const float scale = inv ? (float)(1.0 / ((double)w * (double)h)) : 1.f;
  int rc = FSIM_EINVAL;
#define FSIM_LINE_LENGTHS(X) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096)
  switch (w) {
#define CASE(n) \
  case n: rc = inv ? line_rows<n, true>(d, h, batch, stride, st) : line_rows<n, false>(d, h, batch, stride, st); break;
    FSIM_LINE_LENGTHS(CASE)
#undef CASE
  }
  if (rc) return rc;
  switch (h) {
#define CASE(n) \
  case n:       \
    return inv ? line_cols<n, true>(d, w, batch, stride, scale, st) : line_cols<n, false>(d, w, batch, stride, scale, st);
    FSIM_LINE_LENGTHS(CASE)
#undef CASE
  }
  return FSIM_EINVAL;
}
template <int L>
static int raw_rows_launch(float2* d, int batch, const RawFade& rf, cudaStream_t st) {
  using P = LineOne<L>;
  const size_t smem = sizeof(float2) * (size_t)P::G * smem_line_elems(L, 1);
  static bool attr = false;
  if (!attr) {
    FSIM_CUDA(cudaFuncSetAttribute(k_fft1_rows<L, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr = true;
  }
  k_fft1_rows<L, false, true><<<dim3(div_up(L, P::G), batch), P::G * P::T, smem, st>>>(d, L, (size_t)L * L, rf);
  FSIM_CHECK_LAUNCH();
  return FSIM_OK;
}
template <int L>
static int fit_lines(float2* d, int batch, const RawFade* raw, cudaStream_t st) {
  const size_t stride = (size_t)L * L;
  int rc = raw ? raw_rows_launch<L>(d, batch, *raw, st) : line_rows<L, true>(d, L, batch, stride, st);
  if (rc) return rc;
  return raw ? line_cols<L, false>(d, L, batch, stride, 1.f, st)
             : line_cols<L, true>(d, L, batch, stride, (float)(1.0 / ((double)L * (double)L)), st);
}
#define FSIM_LINE_SIZES(X) X(128) X(256) X(384) X(512) X(768) X(1024) X(2048)
int fft2d_lines_device(float2* data, int n, cudaStream_t st, int batch, const RawFade* raw) {
  switch (n) {
#define CASE(v) \
  case v:       \
    return fit_lines<v>(data, batch, raw, st);
    FSIM_LINE_SIZES(CASE)
#undef CASE
  }
  set_error("line-by-line FFT: unsupported size %d", n);
  return FSIM_EINVAL;
}

static int rows_dispatch(int L, bool inv, float2* d, int nrows, int batch, size_t stride, float scale, cudaStream_t st) {
  switch (L) {
#define CASE(n)                                                                          \
  case n:                                                                                \
    return inv ? launch_rows<n, true>(d, nrows, batch, stride, scale, st)               \
               : launch_rows<n, false>(d, nrows, batch, stride, scale, st);
    FSIM_FFT_LENGTHS(CASE)
#undef CASE
  }
  set_error("unsupported FFT length %d", L);
  return FSIM_EINVAL;
}
static int cols_dispatch(int L, bool inv, float2* d, int ncols, int batch, size_t stride, float scale, cudaStream_t st) {
  switch (L) {
#define CASE(n)                                                                          \
  case n:                                                                                \
    return inv ? launch_cols<n, true>(d, ncols, batch, stride, scale, st)               \
               : launch_cols<n, false>(d, ncols, batch, stride, scale, st);
    FSIM_FFT_LENGTHS(CASE)
#undef CASE
  }
  set_error("unsupported FFT length %d", L);
  return FSIM_EINVAL;
}

int fft2d_device(float2* data, int w, int h, bool inverse, cudaStream_t stream, int batch) {
  FSIM_REQUIRE(fft2d_supported(w, h), FSIM_EINVAL,
               "fft2d: unsupported size %d x %d (lengths 2^k in 32..4096 and 3*2^k in 48..3072)", w, h);
  if (lines_faster(w, h, batch)) return lines_2d(data, w, h, inverse, stream, batch);
  size_t stride = (size_t)w * h;
  int rc = rows_dispatch(w, inverse, data, h, batch, stride, 1.f, stream);
  if (rc) return rc;
  float scale = inverse ? (float)(1.0 / ((double)w * (double)h)) : 1.f;
  return cols_dispatch(h, inverse, data, w, batch, stride, scale, stream);
}

}  // namespace fsim

extern "C" int fsim_vec_fft2d(fsim_vec* v, int inverse) {
  int rc = fsim::ensure_init();
  if (rc) return rc;
  FSIM_REQUIRE(v && v->d && v->cplx, FSIM_EINVAL, "fft2d: complex vector required");
  return fsim::fft2d_device(reinterpret_cast<float2*>(v->d), v->w, v->h, inverse != 0, fsim::ctx().stream, 1);
}

extern "C" int fsim_fft2d_batch(void* data, int w, int h, int batch, int inverse, void* stream) {
  FSIM_REQUIRE(data && batch > 0, FSIM_EINVAL, "fft2d_batch: bad arguments");
  FSIM_REQUIRE(fsim::fft2d_supported(w, h), FSIM_EINVAL, "fft2d_batch: unsupported size %d x %d", w, h);
  int rc = fsim::ensure_init();
  if (rc) return rc;
  cudaStream_t st = stream ? (cudaStream_t)stream : fsim::ctx().stream;
  return fsim::fft2d_device(static_cast<float2*>(data), w, h, inverse != 0, st, batch);
}
