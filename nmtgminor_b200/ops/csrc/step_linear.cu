// Linear layers of a decoding step with up to 32 rows: out[M, N] = epilogue([LayerNorm](X) W^T), bf16.
//
// A step is a chain of such products, one waiting for the other, and each costs latency, not bandwidth: the wait for the kernel before,
// one round trip for the rows, the arithmetic, the way back.  So
//   * everything that does not depend on the kernel before happens while that one runs (programmatic launch): a CTA owns 8 to 32 features
//     over the whole of K and holds their weights in registers, K cut over its warps;
//   * a CTA sees whole rows, so with up to 8 of them (one to a warp) the LayerNorm in front of the product is computed here, by every CTA
//     for itself (the same bf16 values that the LayerNorm kernel writes): one kernel less in the chain, 3.7 us each, for 0.6 to 1.5 more
//     in this one.  Each further row to a warp costs 1.4: with 16 rows both ways take the same;
//   * no tensor memory, descriptors, barriers or clusters to set up and take down: m16n8k16 products (rows of X are the 16 rows, weights the
//     8 columns) and one sum over the warps through shared memory.  tcgen05 with K cut over a cluster (gemm_skinny_tcgen05.cu) takes over
//     from 33 rows, where every CTA reading all of X costs more than the set-up.
// us a product, back to back with programmatic launch, few-row tcgen05 kernel / this one (with its LayerNorm: two kernels / one), weights
// from six matrices in turn: 1024 x 1024, 4 rows 3.6 / 1.7 (5.7 / 2.8), 32 rows 4.3 / 3.3; 4096 x 1024, 4 rows 4.6 / 2.4 (6.2 / 3.3);
// 1024 x 4096, 4 rows 5.2 / 2.5; 3840 x 1280, 32 rows 5.8 / 4.8.  A search for one sentence 19.1 / 12.9 ms.
// As the contraction's order is free, a lane takes eight consecutive values of K (one 16-byte load) where the instruction wants four
// scattered pairs, of X and W alike.
#include "gemm_common.cuh"

namespace b200 {

bool step_overlap();
int num_sms();

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct StepArgs {
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  const __nv_bfloat16* gamma;      // null: no LayerNorm
  const __nv_bfloat16* beta;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  __nv_bfloat16* out;
  int ldx, ldw, ld_res, ld_out;
  int M, N, K, act;
  float eps;
};

constexpr int kMaxVec = 5;          // 16-byte vectors of a row to a lane (staged rows: K up to 1280)

// Row of X in shared memory: whole 128 bytes plus 64, so that the eight lanes of a load phase (two rows, four pieces) meet 32 banks.
__host__ __device__ constexpr int staged_ld(int K) { return (K + 63) / 64 * 64 + 32; }

// The arithmetic of ln_fwd_kernel (layernorm.cu), value for value, over a row in shared memory.
__device__ __forceinline__ void normalise(__nv_bfloat16* row, const __nv_bfloat16* gamma, const __nv_bfloat16* beta, int K, float eps, int lane) {
  const int nvec = K >> 3;
  uint4 u[kMaxVec];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i) u[i] = lane + i * 32 < nvec ? reinterpret_cast<const uint4*>(row)[lane + i * 32] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[i]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      s += f.x + f.y;
    }
  }
  const float mu = row_sum(s) / K;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i)
    if (lane + i * 32 < nvec) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        const float dx = f.x - mu, dy = f.y - mu;
        sq += dx * dx;
        sq += dy * dy;
      }
    }
  const float rs = rsqrtf(row_sum(sq) / K + eps);
#pragma unroll
  for (int i = 0; i < kMaxVec; ++i) {
    const int vi = lane + i * 32;
    if (vi >= nvec) break;
    const uint4 g = reinterpret_cast<const uint4*>(gamma)[vi], b = reinterpret_cast<const uint4*>(beta)[vi];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[i]);
    const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&g);
    const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
    uint4 o;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]), gf = __bfloat1622float2(g2[j]), bf = __bfloat1622float2(b2[j]);
      o2[j] = __floats2bfloat162_rn((f.x - mu) * rs * gf.x + bf.x, (f.y - mu) * rs * gf.y + bf.y);
    }
    reinterpret_cast<uint4*>(row)[vi] = o;
  }
}

__device__ __forceinline__ float step_act(float v, int act) {
  if (act == kActRelu) return fmaxf(v, 0.f);
  if (act == kActGelu) return gelu_f(v);
  if (act == kActSilu) return v * sigmoid_f(v);
  return v;
}

// kWarps warps, each with kChunks pieces of 32 of K (piece i of warp w is w + kWarps i); kTiles tiles of 8 features; kRows8 x 8 rows.
// kDirect: the rows come straight from global memory, each value once per CTA (no LayerNorm, one group of 8 rows).
template <int kWarps, int kChunks, int kTiles, int kRows8, bool kDirect>
__global__ void __launch_bounds__(32 * kWarps, kWarps == 8 ? 2 : 1)
step_linear_kernel(const StepArgs p) {
  constexpr int kF = 8 * kTiles, kPairs = (kRows8 + 1) / 2;
  constexpr int kEach = (kRows8 * 8 * kF / 2 + 32 * kWarps - 1) / (32 * kWarps);      // pairs of outputs to a thread
  extern __shared__ __align__(16) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kF;
  const int ld = staged_ld(p.K);
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem);                          // [8 kRows8][ld], staged rows
  __nv_bfloat16* affine = xs + (kDirect ? 0 : kRows8 * 8 * ld);                          // [2][ld] gamma, beta
  float* red = reinterpret_cast<float*>(smem);                                           // [kWarps][8 kRows8][kF], over the rows
  let_next_start();
  uint4 w[kChunks][kTiles];
#pragma unroll
  for (int i = 0; i < kChunks; ++i)
#pragma unroll
    for (int f = 0; f < kTiles; ++f) {
      const int col = (warp + kWarps * i) * 32 + 8 * t, row = n0 + 8 * f + g;
      w[i][f] = col < p.K && row < p.N ? __ldg(reinterpret_cast<const uint4*>(p.w + static_cast<size_t>(row) * p.ldw + col)) : make_uint4(0u, 0u, 0u, 0u);
    }
  float2 bias[kEach];
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int col = n0 + 2 * ((threadIdx.x + e * 32 * kWarps) % (kF / 2));
    bias[e] = make_float2(0.f, 0.f);
    if (p.bias && col < p.N) bias[e] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p.bias + col));
  }
  if constexpr (!kDirect) {
    if (kRows8 == 1 && p.gamma)
      for (int i = threadIdx.x; i < p.K / 8; i += 32 * kWarps) {
        reinterpret_cast<uint4*>(affine)[i] = __ldg(reinterpret_cast<const uint4*>(p.gamma) + i);
        reinterpret_cast<uint4*>(affine + ld)[i] = __ldg(reinterpret_cast<const uint4*>(p.beta) + i);
      }
    __syncthreads();
  }
  wait_for_previous();
  // ---- from here on: what the kernel before wrote
  uint4 xd[kDirect ? kChunks : 1];
  if constexpr (kDirect) {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int col = (warp + kWarps * i) * 32 + 8 * t;
      xd[i] = col < p.K && g < p.M ? *reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(g) * p.ldx + col) : make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    for (int r = warp; r < p.M; r += kWarps)
      for (int i = lane; i < p.K / 8; i += 32) cp_async16(xs + r * ld + 8 * i, p.x + static_cast<size_t>(r) * p.ldx + 8 * i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __nv_bfloat162 res[kEach];
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int o = threadIdx.x + e * 32 * kWarps, row = o / (kF / 2), col = n0 + 2 * (o % (kF / 2));
    res[e] = __floats2bfloat162_rn(0.f, 0.f);
    if (p.residual && row < p.M && col < p.N) res[e] = *reinterpret_cast<const __nv_bfloat162*>(p.residual + static_cast<size_t>(row) * p.ld_res + col);
  }
  if constexpr (!kDirect) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    if (kRows8 == 1 && p.gamma)
      if (warp < p.M) normalise(xs + warp * ld, affine, affine + ld, p.K, p.eps, lane);
    __syncthreads();
  }
  float acc[kPairs][kTiles][4];
#pragma unroll
  for (int m = 0; m < kPairs; ++m)
#pragma unroll
    for (int f = 0; f < kTiles; ++f) acc[m][f][0] = acc[m][f][1] = acc[m][f][2] = acc[m][f][3] = 0.f;
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int col = (warp + kWarps * i) * 32 + 8 * t;
#pragma unroll
    for (int m = 0; m < kPairs; ++m) {
      uint4 lo, hi = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (kDirect) lo = xd[i];
      else {
        lo = hi;
        if (col < p.K) {
          lo = *reinterpret_cast<const uint4*>(xs + (16 * m + g) * ld + col);
          if (kRows8 > 1) hi = *reinterpret_cast<const uint4*>(xs + (16 * m + 8 + g) * ld + col);
        }
      }
#pragma unroll
      for (int f = 0; f < kTiles; ++f) {
        mma_bf16(acc[m][f], lo.x, hi.x, lo.y, hi.y, w[i][f].x, w[i][f].y);
        mma_bf16(acc[m][f], lo.z, hi.z, lo.w, hi.w, w[i][f].z, w[i][f].w);
      }
    }
  }
  if (!kDirect) __syncthreads();
#pragma unroll
  for (int m = 0; m < kPairs; ++m)
#pragma unroll
    for (int f = 0; f < kTiles; ++f) {
      float* at = red + (warp * kRows8 * 8 + 16 * m + g) * kF + 8 * f + 2 * t;
      *reinterpret_cast<float2*>(at) = make_float2(acc[m][f][0], acc[m][f][1]);
      if (kRows8 > 1) *reinterpret_cast<float2*>(at + 8 * kF) = make_float2(acc[m][f][2], acc[m][f][3]);
    }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int o = threadIdx.x + e * 32 * kWarps, row = o / (kF / 2), c = 2 * (o % (kF / 2));
    if (row >= p.M || n0 + c >= p.N) continue;
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
      const float2 part = *reinterpret_cast<const float2*>(red + (i * kRows8 * 8 + row) * kF + c);
      s.x += part.x;
      s.y += part.y;
    }
    const float2 r = __bfloat1622float2(res[e]);
    *reinterpret_cast<__nv_bfloat162*>(p.out + static_cast<size_t>(row) * p.ld_out + n0 + c) =
        __floats2bfloat162_rn(step_act(s.x + bias[e].x, p.act) + r.x, step_act(s.y + bias[e].y, p.act) + r.y);
  }
}

template <int kWarps, int kChunks, int kTiles, int kRows8, bool kDirect>
const char* launch_step(const StepArgs& a, cudaStream_t stream) {
  auto kern = step_linear_kernel<kWarps, kChunks, kTiles, kRows8, kDirect>;
  const size_t sums = static_cast<size_t>(kWarps) * kRows8 * 8 * kTiles * 8 * 4;
  const size_t rows = kDirect ? 0 : static_cast<size_t>(kRows8 * 8 + (kRows8 == 1 ? 2 : 0)) * staged_ld(a.K) * 2;
  const size_t smem = sums > rows ? sums : rows;
  static bool configured = false;
  if (!configured && smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024);
    if (e != cudaSuccess) return cudaGetErrorString(e);
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.N + 8 * kTiles - 1) / (8 * kTiles));
  cfg.blockDim = dim3(32 * kWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = step_overlap() ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

template <int kChunks, int kRows8>
const char* staged(const StepArgs& a, int tiles, cudaStream_t stream) {
  // weights of kChunks x tiles loads stay in registers beside the sums: 15 of them with 32 rows, 20 with fewer
  constexpr int kMost = (kRows8 == 4 ? 15 : 20) / kChunks < 4 ? (kRows8 == 4 ? 15 : 20) / kChunks : 4;
  if (tiles >= 4 && kMost >= 4) return launch_step<8, kChunks, kMost < 4 ? 1 : 4, kRows8, false>(a, stream);
  if (tiles >= 3 && kMost >= 3) return launch_step<8, kChunks, kMost < 3 ? 1 : 3, kRows8, false>(a, stream);
  if (tiles >= 2) return launch_step<8, kChunks, 2, kRows8, false>(a, stream);
  return launch_step<8, kChunks, 1, kRows8, false>(a, stream);
}

template <int kRows8>
const char* staged_by_length(const StepArgs& a, int tiles, cudaStream_t stream) {
  switch ((a.K + 255) / 256) {
    case 1: return staged<1, kRows8>(a, tiles, stream);
    case 2: return staged<2, kRows8>(a, tiles, stream);
    case 3: return staged<3, kRows8>(a, tiles, stream);
    case 4: return staged<4, kRows8>(a, tiles, stream);
    default: return staged<5, kRows8>(a, tiles, stream);
  }
}

template <int kWarps, int kChunks>
const char* direct(const StepArgs& a, int tiles, cudaStream_t stream) {
  return tiles >= 2 ? launch_step<kWarps, kChunks, 2, 1, true>(a, stream) : launch_step<kWarps, kChunks, 1, 1, true>(a, stream);
}

}  // namespace

constexpr int kStagedK = 256 * kMaxVec, kDirectK = 5120, kNormRows = 8;

bool step_linear_takes(int M, int N, int K, bool norm, int sms) {
  if (M < 1 || M > (norm ? kNormRows : 32) || K % 8 || N % 2 || K < 8) return false;
  if (K > kStagedK) return !norm && M <= 8 && K <= kDirectK && (N + 15) / 16 <= sms;
  return (N + 31) / 32 <= 2 * sms;
}

const char* launch_step_linear(const StepArgs& a, int sms, cudaStream_t stream) {
  // as few tiles to a CTA as give every SM one
  const int tiles = ((a.N + 7) / 8 + sms - 1) / sms;
  if (!a.gamma && a.M <= 8 && tiles <= 2) {
    const int chunks = (a.K + 31) / 32;
    if (chunks <= 8) return direct<8, 1>(a, tiles, stream);
    if (chunks <= 16) return direct<8, 2>(a, tiles, stream);
    if (chunks <= 24) return direct<8, 3>(a, tiles, stream);
    if (chunks <= 32) return direct<8, 4>(a, tiles, stream);
    if (chunks <= 40) return direct<8, 5>(a, tiles, stream);
    if (chunks <= 64) return direct<16, 4>(a, tiles, stream);
    if (chunks <= 96) return direct<16, 6>(a, tiles, stream);
    if (chunks <= 128) return direct<16, 8>(a, tiles, stream);
    return direct<16, 10>(a, tiles, stream);
  }
  if (a.M <= 8) return staged_by_length<1>(a, tiles, stream);
  if (a.M <= 16) return staged_by_length<2>(a, tiles, stream);
  return staged_by_length<4>(a, tiles, stream);
}

}  // namespace b200

using namespace b200;

int nmtg_step_linear_takes(int M, int N, int K, int norm) { return step_linear_takes(M, N, K, norm != 0, num_sms()) ? 1 : 0; }

const char* nmtg_step_linear(const void* x, int ldx, const void* gamma, const void* beta, float eps, const void* w, int ldw, const void* bias,
                             const void* residual, int ld_res, void* out, int ld_out, int M, int N, int K, int act, cudaStream_t stream) {
  const int sms = num_sms();
  if (!step_linear_takes(M, N, K, gamma != nullptr, sms)) return "step_linear: sizes out of range";
  if (act < 0 || act > kActSilu) return "step_linear: unknown activation";
  if (ldx % 8 || ldw % 8 || ld_out % 2 || (residual && ld_res % 2)) return "step_linear: rows must start on a 16-byte boundary";
  const uintptr_t wide = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta);
  const uintptr_t pairs = reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(out);
  if ((wide & 15) || (pairs & 3)) return "step_linear: unaligned operand";
  StepArgs a;
  a.x = static_cast<const __nv_bfloat16*>(x); a.ldx = ldx;
  a.w = static_cast<const __nv_bfloat16*>(w); a.ldw = ldw;
  a.gamma = static_cast<const __nv_bfloat16*>(gamma); a.beta = static_cast<const __nv_bfloat16*>(beta); a.eps = eps;
  a.bias = static_cast<const __nv_bfloat16*>(bias);
  a.residual = static_cast<const __nv_bfloat16*>(residual); a.ld_res = ld_res;
  a.out = static_cast<__nv_bfloat16*>(out); a.ld_out = ld_out;
  a.M = M; a.N = N; a.K = K; a.act = act;
  return launch_step_linear(a, sms, stream);
}
