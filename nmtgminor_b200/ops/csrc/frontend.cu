// Front end of the raw-audio encoders without gradients: convolution over the waveform, LayerNorm over the channels and GELU.
//
//   conv_norm_gelu  first layer (one input channel) -> LayerNorm -> GELU -> bf16 frames, channels last
//   norm_gelu       LayerNorm -> GELU of the frames that the later layers' products leave
//
// In tensor operations the first layer of six utterances of 20 s (384000 frames x 512 channels) went through memory in 32 bits six times
// (convolution, transposition, LayerNorm, GELU, rounding, the copy into the next layer's padded rows); the bytes that must move are the
// 0.39 GB written once (0.06 ms).  The frames are written where the next convolution's overlapping rows are read.  The whole front end of
// those utterances took 6.37 ms and takes 1.16, 0.47 of them the products; one utterance of 1 s 0.73 and 0.27.
// What bounds these kernels is the instructions of GELU and LayerNorm (about 60 for two channels): 0.33 ms for the first layer's frames and
// 0.15 for the 192000 of the second (0.34 and 0.16 with the affine parameters in registers, at half the warps).
#include "gemm_common.cuh"
#include "seq_api.h"

namespace b200 {

int num_sms();

namespace {

__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) { return fma2(a, Pair(1.f), b); }

// LayerNorm and GELU of one row, kPairs channel pairs to a lane, in place; pair j is at channel j / kRun * 64 kRun + j % kRun * 2 of the
// lane's affine parameters
template <int kPairs, int kRun>
__device__ __forceinline__ void norm_gelu(Pair (&x)[kPairs], const float* gamma, const float* beta, int channels, float eps) {
  Pair s(0.f);
#pragma unroll
  for (int j = 0; j < kPairs; ++j) s = add2(x[j], s);
  const float mu = lane_sum(s.split().x + s.split().y) / channels;
  Pair sq(0.f);
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    x[j] = add2(x[j], Pair(-mu));
    sq = fma2(x[j], x[j], sq);
  }
  const Pair rs(rsqrtf(lane_sum(sq.split().x + sq.split().y) / channels + eps));
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int c = j / kRun * 64 * kRun + j % kRun * 2;
    const float2 g = *reinterpret_cast<const float2*>(gamma + c), b = *reinterpret_cast<const float2*>(beta + c);
    const Pair y = fma2(mul2(x[j], rs), Pair(g.x, g.y), Pair(b.x, b.y));
    Pair bell;
    x[j] = mul2(y, normal_cdf2(y, bell));
  }
}

__device__ __forceinline__ uint32_t round2(Pair x) {
  const float2 f = x.split();
  const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

constexpr int kFrontWarps = 8, kFrames = 4, kTaps = 16, kStride = 64;      // taps and stride: at most

// A warp takes four neighbouring frames of an utterance, a lane the channel pairs 2 lane + 64 j: the weights of a tap are read from shared
// memory once for the four.
template <int kPairs>
__global__ void __launch_bounds__(32 * kFrontWarps, 2)
conv_norm_gelu_kernel(const float* __restrict__ wav, long wav_stride, const float* __restrict__ w, const float* __restrict__ bias,
                      const float* __restrict__ gamma, const float* __restrict__ beta, float eps, __nv_bfloat16* __restrict__ out, int B,
                      int samples, int T, int out_rows, int taps, int stride) {
  constexpr int C = 64 * kPairs;
  extern __shared__ __align__(16) float shared[];
  float* ws = shared;                                    // [taps][C]
  float* affine = ws + taps * C;                         // gamma, beta, bias
  float* seg = affine + 3 * C + (threadIdx.x >> 5) * ((kFrames - 1) * stride + taps);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < taps * C; i += blockDim.x) ws[(i % taps) * C + i / taps] = w[i];
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    affine[i] = gamma[i];
    affine[C + i] = beta[i];
    affine[2 * C + i] = bias ? bias[i] : 0.f;
  }
  __syncthreads();
  const int groups = (T + kFrames - 1) / kFrames, window = (kFrames - 1) * stride + taps;
  const long tasks = static_cast<long>(B) * groups;
  for (long task = static_cast<long>(blockIdx.x) * kFrontWarps + warp; task < tasks; task += static_cast<long>(gridDim.x) * kFrontWarps) {
    const int b = static_cast<int>(task / groups), t0 = static_cast<int>(task % groups) * kFrames;
    const long first = static_cast<long>(t0) * stride;
    __syncwarp();
    for (int i = lane; i < window; i += 32) seg[i] = first + i < samples ? wav[b * wav_stride + first + i] : 0.f;
    __syncwarp();
    Pair x[kFrames][kPairs];
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const float2 f = *reinterpret_cast<const float2*>(affine + 2 * C + 2 * lane + 64 * j);
#pragma unroll
      for (int i = 0; i < kFrames; ++i) x[i][j] = Pair(f.x, f.y);
    }
#pragma unroll 1
    for (int k = 0; k < taps; ++k) {
      Pair at[kFrames];
#pragma unroll
      for (int i = 0; i < kFrames; ++i) at[i] = Pair(seg[i * stride + k]);
#pragma unroll
      for (int j = 0; j < kPairs; ++j) {
        const float2 f = *reinterpret_cast<const float2*>(ws + k * C + 2 * lane + 64 * j);
        const Pair v(f.x, f.y);
#pragma unroll
        for (int i = 0; i < kFrames; ++i) x[i][j] = fma2(at[i], v, x[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < kFrames; ++i) {
      if (t0 + i >= T) break;
      norm_gelu<kPairs, 1>(x[i], affine + 2 * lane, affine + C + 2 * lane, C, eps);
      __nv_bfloat16* row = out + (static_cast<long>(b) * out_rows + t0 + i) * C + 2 * lane;
#pragma unroll
      for (int j = 0; j < kPairs; ++j) *reinterpret_cast<uint32_t*>(row + 64 * j) = round2(x[i][j]);
    }
  }
}

// A warp to a row, eight channels of a lane side by side.
template <int kVec>
__global__ void __launch_bounds__(32 * kFrontWarps, 4)
norm_gelu_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, float eps,
                 __nv_bfloat16* __restrict__ out, int B, int T, int in_rows, int out_rows) {
  constexpr int C = 256 * kVec;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ __align__(16) float affine[2 * C];
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    affine[i] = gamma[i];
    affine[C + i] = beta[i];
  }
  __syncthreads();
  const long rows = static_cast<long>(B) * T;
  for (long r = static_cast<long>(blockIdx.x) * kFrontWarps + warp; r < rows; r += static_cast<long>(gridDim.x) * kFrontWarps) {
    const long b = r / T, t = r % T;
    const uint4* from = reinterpret_cast<const uint4*>(x + (b * in_rows + t) * C) + lane;
    uint4* to = reinterpret_cast<uint4*>(out + (b * out_rows + t) * C) + lane;
    Pair v[4 * kVec];
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const uint4 u = from[32 * i];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        v[4 * i + j] = Pair(f.x, f.y);
      }
    }
    norm_gelu<4 * kVec, 4>(v, affine + 8 * lane, affine + C + 8 * lane, C, eps);
#pragma unroll
    for (int i = 0; i < kVec; ++i) to[32 * i] = make_uint4(round2(v[4 * i]), round2(v[4 * i + 1]), round2(v[4 * i + 2]), round2(v[4 * i + 3]));
  }
}

int front_grid(long warps_of_work) {
  const long ctas = (warps_of_work + kFrontWarps - 1) / kFrontWarps, most = 4L * num_sms();
  return static_cast<int>(ctas < most ? ctas : most);
}

template <int kPairs>
const char* launch_conv(const float* wav, long wav_stride, const float* w, const float* bias, const float* gamma, const float* beta, float eps,
                        __nv_bfloat16* out, int B, int samples, int T, int out_rows, int taps, int stride, cudaStream_t stream) {
  static_assert(sizeof(float) * ((kTaps + 3) * 64 * kPairs + kFrontWarps * ((kFrames - 1) * kStride + kTaps)) <= 48 * 1024, "shared memory");
  const size_t smem = sizeof(float) * ((taps + 3) * 64 * kPairs + kFrontWarps * ((kFrames - 1) * stride + taps));
  conv_norm_gelu_kernel<kPairs><<<front_grid(static_cast<long>(B) * ((T + kFrames - 1) / kFrames)), 32 * kFrontWarps, smem, stream>>>(
      wav, wav_stride, w, bias, gamma, beta, eps, out, B, samples, T, out_rows, taps, stride);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

const char* nmtg_conv_norm_gelu(const float* wav, long wav_stride, const float* w, const float* bias, const float* gamma, const float* beta,
                                float eps, void* out, int B, int samples, int T, int out_rows, int channels, int taps, int stride,
                                cudaStream_t stream) {
  if (B <= 0 || T <= 0) return nullptr;
  if (taps < 1 || taps > kTaps || stride < 1 || stride > kStride || out_rows < T || static_cast<long>(T - 1) * stride + taps > samples)
    return "conv_norm_gelu: sizes out of range";
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  switch (channels) {
    case 256: return launch_conv<4>(wav, wav_stride, w, bias, gamma, beta, eps, o, B, samples, T, out_rows, taps, stride, stream);
    case 512: return launch_conv<8>(wav, wav_stride, w, bias, gamma, beta, eps, o, B, samples, T, out_rows, taps, stride, stream);
    default: return "conv_norm_gelu: 256 or 512 channels";
  }
}

const char* nmtg_norm_gelu(const void* x, const float* gamma, const float* beta, float eps, void* out, int B, int T, int in_rows, int out_rows,
                           int channels, cudaStream_t stream) {
  if (B <= 0 || T <= 0) return nullptr;
  if (in_rows < T || out_rows < T) return "norm_gelu: fewer rows than frames";
  const __nv_bfloat16* i = static_cast<const __nv_bfloat16*>(x);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  const int grid = front_grid(static_cast<long>(B) * T);
  if (channels == 256) norm_gelu_kernel<1><<<grid, 32 * kFrontWarps, 0, stream>>>(i, gamma, beta, eps, o, B, T, in_rows, out_rows);
  else if (channels == 512) norm_gelu_kernel<2><<<grid, 32 * kFrontWarps, 0, stream>>>(i, gamma, beta, eps, o, B, T, in_rows, out_rows);
  else return "norm_gelu: 256 or 512 channels";
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // extern "C"
