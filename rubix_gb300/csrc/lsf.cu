// Kernel (d): 1-D convolution of every spectrum of a datacube along wavelength,
// the full convolution cropped to [crop, n + crop) (rubix/telescope/lsf/lsf.py:29-105).
//
// A block stages one spectrum in shared memory with K-1 zeros of halo.  Up to 28 taps a
// thread produces 12 consecutive outputs (4 for short rows and in the fused dot) from float4
// loads of its window; longer kernels take one output at a time.
#include "common.cuh"
#include "dot_reduce.cuh"

namespace rubix {
namespace {

constexpr int kLsfThreads = 256;
constexpr int kLsfMaxTaps = 255;

struct LsfArgs {
  const float* in;
  float* out;
  long long rows;
  int n;
  long long sin, sout;
  int K, crop;
  float taps[kLsfMaxTaps + 1];
  const float* taps_dev;  // when set, the taps are read from device memory instead
};

// out[t] = sum_q w[q] * s[t + q] with s[i] = in[i - (K-1-crop)] and w[q] = taps[K-1-q].
// kDot: instead of storing out, sum wt[row][t] * out[t] over the cube (wt with the
// output's layout, row stride sout) into *dot_out, deterministically.
template <int KC, bool kDot = false>
__global__ void __launch_bounds__(kLsfThreads)
    lsf_vec_kernel(LsfArgs a, const float* __restrict__ wt = nullptr,
                   FusedDotScratch* dot_ws = nullptr, double* dot_out = nullptr) {
  extern __shared__ __align__(16) float s_row[];
  __shared__ float s_w[KC * 4];
  float dot = 0.f;
  const int tid = threadIdx.x;
  const float* tp = a.taps_dev ? a.taps_dev : a.taps;
  for (int q = tid; q < KC * 4; q += kLsfThreads) s_w[q] = (q < a.K) ? tp[a.K - 1 - q] : 0.f;
  const int lead = a.K - 1 - a.crop;           // zeros before in[0]
  const int n4 = (a.n + 3) / 4;                 // output groups of 4
  const int span = n4 * 4 + KC * 4;             // staged length (multiple of 4)
  for (long long row = blockIdx.x; row < a.rows; row += gridDim.x) {
    __syncthreads();
    const float* src = a.in + row * a.sin;
    for (int i = tid; i < span; i += kLsfThreads) {
      const int g = i - lead;
      s_row[i] = (g >= 0 && g < a.n) ? src[g] : 0.f;
    }
    __syncthreads();
    float* dst = a.out + row * a.sout;
    for (int u = tid; u < n4; u += kLsfThreads) {
      // dot mode: the four weights first, so the window loads and FMAs hide them
      float wq[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (kDot) {
        const float* wr = wt + row * a.sout;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (4 * u + c < a.n) wq[c] = wr[4 * u + c];
      }
      float win[KC * 4 + 4];
      const float4* p = reinterpret_cast<const float4*>(s_row + 4 * u);
#pragma unroll
      for (int c = 0; c <= KC; ++c) {
        float4 v = p[c];
        win[4 * c] = v.x;
        win[4 * c + 1] = v.y;
        win[4 * c + 2] = v.z;
        win[4 * c + 3] = v.w;
      }
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int q = 0; q < KC * 4; ++q) {
        const float w = s_w[q];
        o0 = fmaf(w, win[q], o0);
        o1 = fmaf(w, win[q + 1], o1);
        o2 = fmaf(w, win[q + 2], o2);
        o3 = fmaf(w, win[q + 3], o3);
      }
      const int t = 4 * u;
      if constexpr (kDot) {
        // wq is 0 past the row's end
        dot = fmaf(wq[3], o3, fmaf(wq[2], o2, fmaf(wq[1], o1, fmaf(wq[0], o0, dot))));
      } else {
        if (t < a.n) dst[t] = o0;
        if (t + 1 < a.n) dst[t + 1] = o1;
        if (t + 2 < a.n) dst[t + 2] = o2;
        if (t + 3 < a.n) dst[t + 3] = o3;
      }
    }
  }
  if constexpr (kDot) {
    __shared__ double s_red[kLsfThreads / 32];
    __shared__ int s_last;
    fused_dot_finish(dot, dot_ws, dot_out, s_red, &s_last);
  }
}

// The same products in the same order (bit-identical outputs) with the traffic of the
// store path and of the weights spread over more outputs.  One group of 12 outputs per
// thread: the window costs (12 + 4 KC) / 4 vector loads, 40 wavefronts per 384 outputs where
// 4 outputs a thread need 96, the weights one broadcast load per 12 outputs, and a lane
// stride of 48 bytes keeps the 16-byte loads free of bank conflicts.  The outputs return to
// shared memory and leave as whole 128-byte lines; the next row waits in registers
// behind the arithmetic (178 us; as 4-byte asynchronous copies into a second buffer, 187).  Bound by FMA issue and shared memory together, then HBM: 84 M outputs
// (150 x 150 x 3721, 25 taps) take 178 us, where the 4-output kernel took 246 us, bound
// by shared-memory wavefronts; one read and one write at the copy rate are 98 us.
constexpr int kLsfOut = 12;
constexpr int kLsfRowThreads = 320;  // 320 * 12 = 3840 outputs at a time
constexpr int kLsfPre = 13;           // rows of up to 13 * 320 staged floats

// Floats of one staged row: the last group's window ends 4 KC past a multiple of 12.
__host__ __device__ constexpr int lsf_row_floats(int n, int KC) {
  return (n + kLsfOut - 1) / kLsfOut * kLsfOut + 4 * KC;
}

template <int KC>
__global__ void __launch_bounds__(kLsfRowThreads) lsf_row_kernel(LsfArgs a) {
  extern __shared__ __align__(16) float s_buf[];
  __shared__ __align__(16) float s_w[KC * 4];
  const int tid = threadIdx.x;
  const int span = lsf_row_floats(a.n, KC);
  const int groups = (a.n + kLsfOut - 1) / kLsfOut;
  const int lead = a.K - 1 - a.crop;  // zeros before in[0]
  const float* tp = a.taps_dev ? a.taps_dev : a.taps;
  for (int q = tid; q < KC * 4; q += kLsfRowThreads) s_w[q] = (q < a.K) ? tp[a.K - 1 - q] : 0.f;
  float pre[kLsfPre];  // the next row's values at places tid, tid + 320, ...
  auto fetch = [&](long long row) {
    const float* src = a.in + row * a.sin + tid - lead;
#pragma unroll
    for (int k = 0; k < kLsfPre; ++k) {
      const int g = tid - lead + k * kLsfRowThreads;
      pre[k] = (unsigned)g < (unsigned)a.n ? __ldcs(src + k * kLsfRowThreads) : 0.f;
    }
  };
  if (blockIdx.x < a.rows) fetch(blockIdx.x);
  for (long long row = blockIdx.x; row < a.rows; row += gridDim.x) {
    float* cur = s_buf;
    __syncthreads();  // the row before is stored
#pragma unroll
    for (int k = 0; k < kLsfPre; ++k)
      if (tid + k * kLsfRowThreads < span) cur[tid + k * kLsfRowThreads] = pre[k];
    __syncthreads();
    if (row + gridDim.x < a.rows) fetch(row + gridDim.x);
    float* dst = a.out + row * a.sout;
    for (int u0 = 0; u0 < groups; u0 += kLsfRowThreads) {
      const int u = u0 + tid;
      float2 o[kLsfOut / 2];
      if (u < groups) {
        // the window in pairs from even and from odd places: one packed FMA per tap and
        // two outputs
        constexpr int NP = (kLsfOut + KC * 4) / 2;
        float2 even[NP];
        const float4* p = reinterpret_cast<const float4*>(cur + kLsfOut * u);
#pragma unroll
        for (int c = 0; c < NP / 2; ++c) {
          const float4 v = p[c];
          even[2 * c] = make_float2(v.x, v.y);
          even[2 * c + 1] = make_float2(v.z, v.w);
        }
#pragma unroll
        for (int r = 0; r < kLsfOut / 2; ++r) o[r] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          const float4 w4 = *reinterpret_cast<const float4*>(s_w + 4 * c);
          const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 wq = make_float2(w[q], w[q]);
#pragma unroll
            for (int r = 0; r < kLsfOut / 2; ++r) {
              const int m = 2 * c + q / 2 + r;  // pair of window places 4c + q + 2r, + 1
              o[r] = __ffma2_rn(
                  wq, (q & 1) ? make_float2(even[m].y, even[m + 1 < NP ? m + 1 : m].x) : even[m],
                  o[r]);
            }
          }
        }
      }
      // a window reaches 4 KC past its outputs, into the next groups': store only when
      // every window of this round has been read, and the next round's first are safe
      // because its outputs start after them
      __syncthreads();
      if (u < groups) {
        float4* p = reinterpret_cast<float4*>(cur + kLsfOut * u);
#pragma unroll
        for (int c = 0; c < kLsfOut / 4; ++c)
          p[c] = make_float4(o[2 * c].x, o[2 * c].y, o[2 * c + 1].x, o[2 * c + 1].y);
      }
      __syncthreads();
      const int t1 = min(a.n, (u0 + kLsfRowThreads) * kLsfOut);
#pragma unroll 4
      for (int t = u0 * kLsfOut + tid; t < t1; t += kLsfRowThreads) dst[t] = cur[t];
    }
  }
}

// Generic path for long kernels: one output per thread iteration.
__global__ void __launch_bounds__(kLsfThreads) lsf_scalar_kernel(LsfArgs a) {
  extern __shared__ __align__(16) float s_row[];
  __shared__ float s_w[kLsfMaxTaps + 1];
  const int tid = threadIdx.x;
  const float* tp = a.taps_dev ? a.taps_dev : a.taps;
  for (int q = tid; q < a.K; q += kLsfThreads) s_w[q] = tp[a.K - 1 - q];
  const int lead = a.K - 1 - a.crop;
  const int span = a.n + a.K - 1;
  for (long long row = blockIdx.x; row < a.rows; row += gridDim.x) {
    __syncthreads();
    const float* src = a.in + row * a.sin;
    for (int i = tid; i < span; i += kLsfThreads) {
      const int g = i - lead;
      s_row[i] = (g >= 0 && g < a.n) ? src[g] : 0.f;
    }
    __syncthreads();
    float* dst = a.out + row * a.sout;
    for (int t = tid; t < a.n; t += kLsfThreads) {
      float o = 0.f;
      for (int q = 0; q < a.K; ++q) o = fmaf(s_w[q], s_row[t + q], o);
      dst[t] = o;
    }
  }
}

// Whether lsf_row_kernel is the faster one: a row of n occupies n / 12 of its 320 threads, and of
// the 4-output kernel's 256 n / 4, which short rows and few taps prefer.  22 500 rows, us of the
// 4-output kernel / of this: 25 taps 37 / 77 at 300, 66 / 78 at 550, 81 / 79 at 600, 105 / 89 at
// 960, 72 / 91 at 1000 and 81 / 91 at 1025 (one round of the other is full), 89 / 90 at 1060, 120 /
// 94 at 1450; 13 taps 59 / 62 at 550, 73 / 64 at 600, 94 / 70 at 800; 9 taps 54 / 66 at 1000, 69 /
// 70 at 1401, 74 / 72 at 1500.  A cube that stays in L2 (9000 rows): 25 taps at most 34 / 39 at
// 1150, both the launch's time at 1350.
bool lsf_row_pays(long long rows, int n, int KC) {
  if (KC <= 3) return n > 1400;
  if (KC > 4 && n <= 1300 && rows * n < 16'000'000) return false;
  return n >= 600 && (n <= 980 || n > 1048);
}

template <int KC>
int launch_row(const LsfArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(float) * (size_t)lsf_row_floats(a.n, KC);
  if (!lsf_row_pays(a.rows, a.n, KC) || lsf_row_floats(a.n, KC) > kLsfPre * kLsfRowThreads) {
    const size_t one = sizeof(float) * ((size_t)(a.n + 3) / 4 * 4 + KC * 4 + 4);
    cudaError_t e = cudaFuncSetAttribute(lsf_vec_kernel<KC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one);
    if (e != cudaSuccess)
      return set_error(RUBIX_E_CUDA, "cudaFuncSetAttribute(lsf_vec_kernel): %s",
                       cudaGetErrorString(e));
    const long long grid = std::min<long long>(a.rows, (long long)sm_count() * 8);
    lsf_vec_kernel<KC><<<(int)grid, kLsfThreads, one, st>>>(a);
    RUBIX_LAUNCH_CHECK("lsf_vec_kernel");
    return RUBIX_OK;
  }
  cudaError_t e = cudaFuncSetAttribute(lsf_row_kernel<KC>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess)
    return set_error(RUBIX_E_CUDA, "cudaFuncSetAttribute(lsf_row_kernel): %s",
                     cudaGetErrorString(e));
  const int per_sm =
      blocks_per_sm(reinterpret_cast<const void*>(lsf_row_kernel<KC>), kLsfRowThreads, smem);
  const long long grid = std::min<long long>(a.rows, (long long)sm_count() * std::max(per_sm, 1));
  lsf_row_kernel<KC><<<(int)grid, kLsfRowThreads, smem, st>>>(a);
  RUBIX_LAUNCH_CHECK("lsf_row_kernel");
  return RUBIX_OK;
}

template <int KC>
int launch_vec_dot(const LsfArgs& a, const float* wt, FusedDotScratch* ws, double* out,
                   cudaStream_t st) {
  const int n4 = (a.n + 3) / 4;
  const size_t smem = sizeof(float) * ((size_t)n4 * 4 + KC * 4 + 4);
  cudaError_t e = cudaFuncSetAttribute(lsf_vec_kernel<KC, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess)
    return set_error(RUBIX_E_CUDA, "cudaFuncSetAttribute(lsf_vec_kernel): %s", cudaGetErrorString(e));
  const long long grid = std::min<long long>(
      std::min<long long>(a.rows, (long long)sm_count() * 8), kFusedDotMaxBlocks);
  lsf_vec_kernel<KC, true><<<(int)grid, kLsfThreads, smem, st>>>(a, wt, ws, out);
  RUBIX_LAUNCH_CHECK("lsf_vec_kernel");
  return RUBIX_OK;
}

}  // namespace
}  // namespace rubix

using namespace rubix;

namespace rubix {
namespace {

int lsf_fwd_impl(const float* in, float* out, int64_t n_rows, int32_t n_wave_t,
                 int64_t row_stride_in, int64_t row_stride_out, const float* taps,
                 int32_t n_taps, int32_t crop, bool device_taps, void* stream) {
  RUBIX_REQUIRE(n_rows >= 0 && n_wave_t >= 0, RUBIX_E_SHAPE, "rubix_lsf_fwd: negative size");
  RUBIX_REQUIRE(n_taps >= 1 && n_taps <= kLsfMaxTaps, RUBIX_E_SHAPE,
                "rubix_lsf_fwd: n_taps must be in [1, %d]", kLsfMaxTaps);
  RUBIX_REQUIRE(crop >= 0 && crop <= n_taps - 1, RUBIX_E_SHAPE,
                "rubix_lsf_fwd: crop must be in [0, n_taps-1]");
  RUBIX_REQUIRE(row_stride_in >= n_wave_t && row_stride_out >= n_wave_t, RUBIX_E_SHAPE,
                "rubix_lsf_fwd: row stride smaller than n_wave_t");
  RUBIX_REQUIRE((long long)n_wave_t + n_taps + 8 <= 48 * 1024, RUBIX_E_SHAPE,
                "rubix_lsf_fwd: spectrum too long for one shared-memory row");
  if (n_rows == 0 || n_wave_t == 0) return RUBIX_OK;
  RUBIX_REQUIRE(in && out && taps, RUBIX_E_INVALID, "rubix_lsf_fwd: null pointer");
  RUBIX_REQUIRE(in != out, RUBIX_E_INVALID, "rubix_lsf_fwd: in and out must differ");
  LsfArgs a;
  a.in = in;
  a.out = out;
  a.rows = n_rows;
  a.n = n_wave_t;
  a.sin = row_stride_in;
  a.sout = row_stride_out;
  a.K = n_taps;
  a.crop = crop;
  a.taps_dev = device_taps ? taps : nullptr;
  for (int i = 0; i <= kLsfMaxTaps; ++i) a.taps[i] = (!device_taps && i < n_taps) ? taps[i] : 0.f;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // KC = ceil(K/4) weight chunks; each thread's window is KC+1 float4 loads.
  switch ((n_taps + 3) / 4) {
    case 0:
    case 1: return launch_row<1>(a, st);
    case 2: return launch_row<2>(a, st);
    case 3: return launch_row<3>(a, st);
    case 4: return launch_row<4>(a, st);
    case 5: return launch_row<5>(a, st);
    case 6: return launch_row<6>(a, st);
    case 7: return launch_row<7>(a, st);
    default: break;
  }
  const size_t smem = sizeof(float) * ((size_t)n_wave_t + n_taps + 4);
  RUBIX_CUDA_TRY(cudaFuncSetAttribute(lsf_scalar_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  long long grid = std::min<long long>(n_rows, (long long)sm_count() * 8);
  lsf_scalar_kernel<<<(int)grid, kLsfThreads, smem, st>>>(a);
  RUBIX_LAUNCH_CHECK("lsf_scalar_kernel");
  return RUBIX_OK;
}

}  // namespace
}  // namespace rubix

extern "C" int rubix_lsf_fwd(const float* in, float* out, int64_t n_rows, int32_t n_wave_t,
                             int64_t row_stride_in, int64_t row_stride_out, const float* taps,
                             int32_t n_taps, int32_t crop, void* stream) {
  return lsf_fwd_impl(in, out, n_rows, n_wave_t, row_stride_in, row_stride_out, taps, n_taps,
                      crop, false, stream);
}

extern "C" int rubix_lsf_dot_dtaps(const float* in, int64_t n_rows, int32_t n_wave_t,
                                   int64_t row_stride_in, const float* w, int64_t row_stride_w,
                                   const float* taps, int32_t n_taps, int32_t crop, double* out,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  RUBIX_REQUIRE(n_rows >= 0 && n_wave_t >= 0, RUBIX_E_SHAPE, "rubix_lsf_dot_dtaps: negative size");
  RUBIX_REQUIRE(n_taps >= 1 && n_taps <= 28, RUBIX_E_UNSUPPORTED,
                "rubix_lsf_dot_dtaps: n_taps must be in [1, 28], got %d", n_taps);
  RUBIX_REQUIRE(crop >= 0 && crop <= n_taps - 1, RUBIX_E_SHAPE,
                "rubix_lsf_dot_dtaps: crop must be in [0, n_taps-1]");
  RUBIX_REQUIRE(row_stride_in >= n_wave_t && row_stride_w >= n_wave_t, RUBIX_E_SHAPE,
                "rubix_lsf_dot_dtaps: row stride smaller than n_wave_t");
  RUBIX_REQUIRE((long long)n_wave_t + n_taps + 8 <= 48 * 1024, RUBIX_E_SHAPE,
                "rubix_lsf_dot_dtaps: spectrum too long for one shared-memory row");
  RUBIX_REQUIRE(out != nullptr, RUBIX_E_INVALID, "rubix_lsf_dot_dtaps: null output");
  RUBIX_REQUIRE(workspace != nullptr && workspace_bytes >= sizeof(FusedDotScratch) &&
                    (reinterpret_cast<uintptr_t>(workspace) & 7) == 0,
                RUBIX_E_WORKSPACE,
                "rubix_lsf_dot_dtaps: workspace of %zu bytes (8-byte aligned) needed",
                sizeof(FusedDotScratch));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n_rows == 0 || n_wave_t == 0) {
    RUBIX_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(double), st));
    return RUBIX_OK;
  }
  RUBIX_REQUIRE(in && w && taps, RUBIX_E_INVALID, "rubix_lsf_dot_dtaps: null pointer");
  LsfArgs a;
  a.in = in;
  a.out = nullptr;
  a.rows = n_rows;
  a.n = n_wave_t;
  a.sin = row_stride_in;
  a.sout = row_stride_w;
  a.K = n_taps;
  a.crop = crop;
  a.taps_dev = taps;
  for (int i = 0; i <= kLsfMaxTaps; ++i) a.taps[i] = 0.f;
  auto* ws = static_cast<FusedDotScratch*>(workspace);
  RUBIX_CUDA_TRY(cudaMemsetAsync(&ws->counter, 0, sizeof(unsigned), st));
  switch ((n_taps + 3) / 4) {
    case 1: return launch_vec_dot<1>(a, w, ws, out, st);
    case 2: return launch_vec_dot<2>(a, w, ws, out, st);
    case 3: return launch_vec_dot<3>(a, w, ws, out, st);
    case 4: return launch_vec_dot<4>(a, w, ws, out, st);
    case 5: return launch_vec_dot<5>(a, w, ws, out, st);
    case 6: return launch_vec_dot<6>(a, w, ws, out, st);
    default: return launch_vec_dot<7>(a, w, ws, out, st);
  }
}

extern "C" int rubix_lsf_fwd_dtaps(const float* in, float* out, int64_t n_rows,
                                   int32_t n_wave_t, int64_t row_stride_in,
                                   int64_t row_stride_out, const float* taps, int32_t n_taps,
                                   int32_t crop, void* stream) {
  return lsf_fwd_impl(in, out, n_rows, n_wave_t, row_stride_in, row_stride_out, taps, n_taps,
                      crop, true, stream);
}
