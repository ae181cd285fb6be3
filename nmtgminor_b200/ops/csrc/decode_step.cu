// Kernels of a replayed beam-search step: everything between two embedding look-ups that is not a GEMM or a LayerNorm.
//
//   decode_self   append this position's keys / values to the caches and attend over them.  Hypotheses are never copied when
//                 the search re-ranks them: `anc[r][j]` names the cache row that holds position j of hypothesis r, and only that
//                 table is permuted (copying the caches cost 12 launches of 14.7 us a step, 64 sentences x 4 hypotheses).
//   decode_cross  attention over the encoder states of a sentence, all its hypotheses in one CTA, so the keys and values are read
//                 once per sentence; long sources are cut over a cluster (1500 frames x 20 heads x 8 sentences: 31 MB of keys and
//                 as much of values per layer).
//   beam_part     log-sum-exp and best 2K of every 4096-column piece of the logits, one pass, the piece in registers.
//   beam_advance  per sentence: merge the pieces, finish hypotheses that end, choose the next K, update the tables.
//   beam_trace    the finished hypotheses' words, walked backwards through the step records.
//
// All are launched with programmatic overlap inside a step (nmtg_set_step_overlap) and touch an earlier kernel's data only
// after griddepcontrol.wait.
//
// Counterpart of the reference's BeamSearch.step / _translate_batch bookkeeping (onmt/inference/search.py:62-106,
// onmt/inference/fast_translator.py:428-1010).
#include "b200_ptx.cuh"
#include "seq_api.h"
#include "ops_api.h"

namespace b200 {

bool step_overlap();

namespace {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... A, typename... P>
const char* launch(void (*kernel)(A...), dim3 grid, dim3 block, size_t smem, int cluster_z, cudaStream_t stream, P... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (step_overlap()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster_z > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = cluster_z;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, A(args)...);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(h[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
// exp(a - b) with exp(-inf - -inf) = 0: an empty part has no weight
__device__ __forceinline__ float exp_diff(float a, float b) { return a == -INFINITY ? 0.f : __expf(a - b); }

// Both attention kernels serve all hypotheses of a sentence (KB at a time) from one CTA, in blocks of 4 KU keys.  A load
// instruction of a warp covers four 128-byte rows (eight lanes a row, 16 bytes a lane), so a lane (sub = lane / 8, eighth = lane
// % 8) holds dimensions 8 eighth .. + 7 of the keys 4 u + sub, u < KU; a row is loaded and unpacked once and used for KB queries.
// KU is 8, or 4 where the queries' sums need the registers.  A CTA has 2 to 8 warps, each with blocks of its own: a lone
// sentence wants its few blocks side by side, 64 sentences want many small CTAs on an SM instead.

// Partial dot products of the lane's KU keys -> the score of key 4 slot + sub, slot = eighth (KU = 8) or eighth / 2 (KU = 4): the
// eight lanes of a row halve their lists while they add.
template <int KU>
__device__ __forceinline__ float fold_scores(const float (&d)[KU], int eighth) {
  static_assert(KU == 8 || KU == 4, "");
  float a[KU / 2], b[KU / 4];
  const bool hi4 = eighth & 4, hi2 = eighth & 2, hi1 = eighth & 1;
#pragma unroll
  for (int i = 0; i < KU / 2; ++i) {
    const float keep = hi4 ? d[i + KU / 2] : d[i], give = hi4 ? d[i] : d[i + KU / 2];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
  }
#pragma unroll
  for (int i = 0; i < KU / 4; ++i) {
    const float keep = hi2 ? a[i + KU / 4] : a[i], give = hi2 ? a[i] : a[i + KU / 4];
    b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
  }
  if constexpr (KU == 4) return b[0] + __shfl_xor_sync(0xffffffffu, b[0], 1);
  else {
    const float keep = hi1 ? b[1] : b[0], give = hi1 ? b[0] : b[1];
    return keep + __shfl_xor_sync(0xffffffffu, give, 1);
  }
}
template <int KU> __device__ __forceinline__ int slot_of(int eighth) { return KU == 8 ? eighth : eighth >> 1; }
template <int KU> __device__ __forceinline__ int owner_of(int lane, int u) { return (lane & 24) | (KU == 8 ? u : u << 1); }

__device__ __forceinline__ float dot8(const float (&f)[8], const float* q) {
  float s = 0.f;
#pragma unroll
  for (int d = 0; d < 8; ++d) s = fmaf(f[d], q[d], s);
  return s;
}

// running softmax of one query over blocks of keys: maximum, this lane's share of the sum, dimensions 8 eighth .. + 7 of the keys
// with this `sub`
struct Running {
  float m, l, acc[8];
  __device__ __forceinline__ void clear() {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int d = 0; d < 8; ++d) acc[d] = 0.f;
  }
  // s: score of this lane's key (-inf where there is none) -> its weight relative to the new maximum; `once`: of the lanes that hold
  // the same key, the one that counts it
  __device__ __forceinline__ float weigh(float s, bool once) {
    const float mn = fmaxf(m, warp_max(s)), corr = exp_diff(m, mn), p = exp_diff(s, mn);
    m = mn;
    l = l * corr + (once ? p : 0.f);
#pragma unroll
    for (int d = 0; d < 8; ++d) acc[d] *= corr;
    return p;
  }
  __device__ __forceinline__ void add(float p, const float (&f)[8]) {
#pragma unroll
    for (int d = 0; d < 8; ++d) acc[d] = fmaf(p, f[d], acc[d]);
  }
  // whole-warp sums: row[0 .. 63] = unnormalised output, row[64] = maximum, row[65] = sum
  __device__ __forceinline__ void store(float* row, int lane) {
    l = warp_sum(l);
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 8);
      acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 16);
    }
    if (lane < 8) {
#pragma unroll
      for (int d = 0; d < 8; ++d) row[lane * 8 + d] = acc[d];
    }
    if (lane == 0) {
      row[64] = m;
      row[65] = l;
    }
  }
};

// Sum of `n` stored parts (`stride` floats apart): this lane's two output dimensions, the maximum and the sum.
__device__ __forceinline__ void merge_parts(const float* rows, int n, int stride, int lane, float& o0, float& o1, float& mx, float& sum) {
  mx = -INFINITY;
  for (int w = 0; w < n; ++w) mx = fmaxf(mx, rows[w * stride + 64]);
  o0 = o1 = sum = 0.f;
  for (int w = 0; w < n; ++w) {
    const float e = exp_diff(rows[w * stride + 64], mx);
    sum += e * rows[w * stride + 65];
    o0 += e * rows[w * stride + 2 * lane];
    o1 += e * rows[w * stride + 2 * lane + 1];
  }
}

constexpr int kStepWarps = 8;        // at most
template <int KB> __host__ __device__ constexpr int keys_of() { return KB <= 2 ? 8 : 4; }

// One block of keys for the queries k0 .. k1 - 1: `kr` / `vr` are this lane's rows (null: none), `in` whether the lane's own key is
// one of them.
template <int KB, int K0, int K1, int KU>
__device__ __forceinline__ void attend_block(Running (&run)[KB], const float (&qs)[KB][64], const uint4 (&kv)[KU], const uint4 (&vv)[KU],
                                             bool in, int lane) {
  const int eighth = lane & 7;
  float d[K1 - K0][KU];
#pragma unroll
  for (int u = 0; u < KU; ++u) {
    float f[8];
    unpack8(kv[u], f);
#pragma unroll
    for (int k = K0; k < K1; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&qs[k][eighth * 8]), c = *reinterpret_cast<const float4*>(&qs[k][eighth * 8 + 4]);
      const float q8[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
      d[k - K0][u] = dot8(f, q8);
    }
  }
  float p[K1 - K0];
#pragma unroll
  for (int k = K0; k < K1; ++k) {
    const float s = fold_scores<KU>(d[k - K0], eighth);
    p[k - K0] = run[k].weigh(in ? s : -INFINITY, KU == 8 || !(lane & 1));
  }
#pragma unroll
  for (int u = 0; u < KU; ++u) {
    float f[8];
    unpack8(vv[u], f);
#pragma unroll
    for (int k = K0; k < K1; ++k) run[k].add(__shfl_sync(0xffffffffu, p[k - K0], owner_of<KU>(lane, u)), f);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// self-attention.  The hypotheses of a sentence share most of their past (they differ in the last words), so a block whose
// ancestor rows agree is read once for all of them, the others once per hypothesis.
// ---------------------------------------------------------------------------------------------------------------------
template <int KB, int K0>
__device__ __forceinline__ void attend_apart(Running (&run)[KB], const float (&qs)[KB][64], const int (&at)[KB], const __nv_bfloat16* kc,
                                             const __nv_bfloat16* vc, int hid, int col, int beams, int lane) {
  if constexpr (K0 < KB) {
    constexpr int KU = keys_of<KB>();
    if (K0 < beams) {
      uint4 kv[KU], vv[KU];
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const int from = __shfl_sync(0xffffffffu, at[K0], owner_of<KU>(lane, u));
        const long e = static_cast<long>(from) * hid + col;
        kv[u] = from >= 0 ? *reinterpret_cast<const uint4*>(kc + e) : make_uint4(0u, 0u, 0u, 0u);
        vv[u] = from >= 0 ? *reinterpret_cast<const uint4*>(vc + e) : make_uint4(0u, 0u, 0u, 0u);
      }
      attend_block<KB, K0, K0 + 1, KU>(run, qs, kv, vv, at[K0] >= 0, lane);
    }
    attend_apart<KB, K0 + 1>(run, qs, at, kc, vc, hid, col, beams, lane);
  }
}

template <int KB>
__global__ void __launch_bounds__(32 * kStepWarps, 2)
decode_self_kernel(const __nv_bfloat16* __restrict__ qkv, long ld, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                   const int* __restrict__ anc, const long* __restrict__ pos_rows, __nv_bfloat16* __restrict__ out, int first, int K, int groups,
                   int heads, int cap, float scale) {
  constexpr int KU = keys_of<KB>();
  __shared__ __align__(16) float qs[KB][64];
  __shared__ float part[kStepWarps][KB][66];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int h = blockIdx.x, item = first + blockIdx.y;
  const int r0 = (item / groups) * K + (item % groups) * KB;
  const int beams = min(KB, K - (item % groups) * KB);
  const int hid = heads * 64;
  const int sub = lane >> 3, eighth = lane & 7, col = h * 64 + eighth * 8;
  pdl_trigger();
  pdl_wait();
  const long pos_l = pos_rows[r0];                     // the same for all hypotheses of a sentence
  const int pos = pos_l < 0 ? 0 : (pos_l >= cap ? cap - 1 : static_cast<int>(pos_l));
  for (int i = threadIdx.x; i < KB * 64; i += blockDim.x) {
    const int k = i >> 6;
    qs[k][i & 63] = k < beams ? __bfloat162float(qkv[(r0 + k) * ld + h * 64 + (i & 63)]) * scale : 0.f;
  }
  Running run[KB];
#pragma unroll
  for (int k = 0; k < KB; ++k) run[k].clear();
  __syncthreads();
  for (int j0 = warp * 4 * KU; j0 < pos; j0 += warps * 4 * KU) {
    const int j = j0 + slot_of<KU>(eighth) * 4 + sub;
    int at[KB];
    bool agree = true;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      at[k] = (j < pos && k < beams) ? anc[static_cast<long>(r0 + k) * cap + j] * cap + j : -1;
      if (k < beams) agree = agree && at[k] == at[0];
    }
    if (__all_sync(0xffffffffu, agree)) {
      uint4 kv[KU], vv[KU];
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const int from = __shfl_sync(0xffffffffu, at[0], owner_of<KU>(lane, u));
        const long e = static_cast<long>(from) * hid + col;
        kv[u] = from >= 0 ? *reinterpret_cast<const uint4*>(kc + e) : make_uint4(0u, 0u, 0u, 0u);
        vv[u] = from >= 0 ? *reinterpret_cast<const uint4*>(vc + e) : make_uint4(0u, 0u, 0u, 0u);
      }
      attend_block<KB, 0, KB, KU>(run, qs, kv, vv, at[0] >= 0, lane);
    } else {
      attend_apart<KB, 0>(run, qs, at, kc, vc, hid, col, beams, lane);
    }
  }
  // the new position itself, straight from the projection, and its place in the caches
#pragma unroll
  for (int k = 0; k < KB; ++k) {
    if (k % warps == warp && k < beams) {
      const __nv_bfloat16* row = qkv + (r0 + k) * ld + h * 64;
      const uint4 kn = reinterpret_cast<const uint4*>(row + hid)[eighth], vn = reinterpret_cast<const uint4*>(row + 2 * hid)[eighth];
      const long to = (static_cast<long>(r0 + k) * cap + pos) * hid + col;
      if (sub == 0) *reinterpret_cast<uint4*>(kc + to) = kn;
      if (sub == 1) *reinterpret_cast<uint4*>(vc + to) = vn;
      float f[8];
      unpack8(kn, f);
      float s = dot8(f, &qs[k][eighth * 8]);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      const float p = run[k].weigh(s, lane == 0);
      unpack8(vn, f);
      run[k].add(sub == 0 ? p : 0.f, f);
    }
  }
#pragma unroll
  for (int k = 0; k < KB; ++k) run[k].store(part[warp][k], lane);
  __syncthreads();
  for (int k = warp; k < beams; k += warps) {
    float o0, o1, mx, sum;
    merge_parts(part[0][k], warps, KB * 66, lane, o0, o1, mx, sum);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    *reinterpret_cast<__nv_bfloat162*>(out + (static_cast<long>(r0 + k) * heads + h) * 64 + 2 * lane) = __floats2bfloat162_rn(o0 * inv, o1 * inv);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// encoder-decoder attention.  CTA = (head, sentence and group of up to KB hypotheses, share of the keys); the shares of a sentence
// are one cluster and meet in distributed shared memory.
// ---------------------------------------------------------------------------------------------------------------------
template <int KB>
__global__ void __launch_bounds__(32 * kStepWarps, 2)
decode_cross_kernel(const __nv_bfloat16* __restrict__ q, long ld, const __nv_bfloat16* __restrict__ ck, const __nv_bfloat16* __restrict__ cv,
                    const int* __restrict__ lengths, __nv_bfloat16* __restrict__ out, int first, int K, int groups, int heads, int cap,
                    float scale, int splits) {
  constexpr int KU = keys_of<KB>();
  __shared__ __align__(16) float qs[KB][64];
  __shared__ float part[kStepWarps][KB][66];
  __shared__ __align__(16) float mine[KB][68];      // this CTA's sums, read by the whole cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int h = blockIdx.x, item = first + blockIdx.y;
  const int b = item / groups, k0 = (item % groups) * KB;
  const int beams = min(KB, K - k0);
  const int share = blockIdx.z;
  const int hid = heads * 64;
  const int sub = lane >> 3, eighth = lane & 7;
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i < KB * 64; i += blockDim.x) {
    const int k = i >> 6;
    qs[k][i & 63] = k < beams ? __bfloat162float(q[(static_cast<long>(b) * K + k0 + k) * ld + h * 64 + (i & 63)]) * scale : 0.f;
  }
  int len = lengths[b];
  len = len < 0 ? 0 : (len > cap ? cap : len);
  const int chunk = ((len + splits - 1) / splits + 31) & ~31;
  const int begin = share * chunk, end = min(len, begin + chunk);
  const __nv_bfloat16* kb = ck + static_cast<long>(b) * cap * hid + h * 64 + eighth * 8;
  const __nv_bfloat16* vb = cv + static_cast<long>(b) * cap * hid + h * 64 + eighth * 8;
  Running run[KB];
#pragma unroll
  for (int k = 0; k < KB; ++k) run[k].clear();
  __syncthreads();
  for (int j0 = begin + warp * 4 * KU; j0 < end; j0 += warps * 4 * KU) {
    uint4 kv[KU], vv[KU];
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      const int j = j0 + u * 4 + sub;
      kv[u] = j < end ? *reinterpret_cast<const uint4*>(kb + static_cast<long>(j) * hid) : make_uint4(0u, 0u, 0u, 0u);
      vv[u] = j < end ? *reinterpret_cast<const uint4*>(vb + static_cast<long>(j) * hid) : make_uint4(0u, 0u, 0u, 0u);
    }
    attend_block<KB, 0, KB, KU>(run, qs, kv, vv, j0 + slot_of<KU>(eighth) * 4 + sub < end, lane);
  }
#pragma unroll
  for (int k = 0; k < KB; ++k) run[k].store(part[warp][k], lane);
  __syncthreads();
  for (int k = warp; k < KB; k += warps) {
    float o0, o1, mx, sum;
    merge_parts(part[0][k], warps, KB * 66, lane, o0, o1, mx, sum);
    if (splits == 1) {
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      if (k < beams)
        *reinterpret_cast<__nv_bfloat162*>(out + ((static_cast<long>(b) * K + k0 + k) * heads + h) * 64 + 2 * lane) =
            __floats2bfloat162_rn(o0 * inv, o1 * inv);
    } else {
      mine[k][2 * lane] = o0;
      mine[k][2 * lane + 1] = o1;
      if (lane == 0) {
        mine[k][64] = mx;
        mine[k][65] = sum;
      }
    }
  }
  if (splits == 1) return;
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int k = share + splits * warp; k < beams; k += splits * warps) {
    const uint32_t base = smem_u32(&mine[k][0]);
    float mx = -INFINITY, o0 = 0.f, o1 = 0.f, sum = 0.f;
    for (int s = 0; s < splits; ++s) {
      uint32_t remote;
      float v0, v1, pm, pl;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(base), "r"(s));
      asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v0), "=f"(v1) : "r"(remote + lane * 8) : "memory");
      asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(pm), "=f"(pl) : "r"(remote + 256) : "memory");
      const float mn = fmaxf(mx, pm), a = exp_diff(mx, mn), e = exp_diff(pm, mn);
      mx = mn;
      sum = sum * a + pl * e;
      o0 = o0 * a + v0 * e;
      o1 = o1 * a + v1 * e;
    }
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    *reinterpret_cast<__nv_bfloat162*>(out + ((static_cast<long>(b) * K + k0 + k) * heads + h) * 64 + 2 * lane) =
        __floats2bfloat162_rn(o0 * inv, o1 * inv);
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------------------------------
// best continuations
// ---------------------------------------------------------------------------------------------------------------------
// order-preserving map of floats to unsigned; NaN is below everything (never chosen before a number)
__device__ __forceinline__ uint32_t rank_of(float v) {
  const uint32_t u = __float_as_uint(v);
  return v != v ? 0u : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }

constexpr uint32_t kNone = 0xffffffffu;

// A candidate as one number: larger value first, then smaller index; 0 = none.
typedef unsigned long long Cand;
__device__ __forceinline__ Cand cand_of(float v, uint32_t index) { return (static_cast<Cand>(rank_of(v)) << 32) | (kNone - index); }
__device__ __forceinline__ float value_in(Cand c) { return value_of(static_cast<uint32_t>(c >> 32)); }
__device__ __forceinline__ uint32_t index_in(Cand c) { return kNone - static_cast<uint32_t>(c); }
__device__ __forceinline__ Cand warp_best(Cand c) {
  const uint32_t hi = __reduce_max_sync(0xffffffffu, static_cast<uint32_t>(c >> 32));
  const uint32_t lo = __reduce_max_sync(0xffffffffu, static_cast<uint32_t>(c >> 32) == hi ? static_cast<uint32_t>(c) : 0u);
  return (static_cast<Cand>(hi) << 32) | lo;
}
// The best `want` of n candidates, in order, given to emit(place, candidate).  Few of them: every thread counts how many beat its own
// (all reads are broadcasts, nothing is serial).  Many (equal logits, wide beams): one warp takes them one by one.
template <typename Emit>
__device__ __forceinline__ void take_best(const Cand* list, int n, int want, int threads, Emit emit) {
  if (n <= 1024) {
    for (int t = threadIdx.x; t < n; t += threads) {
      const Cand mine = list[t];
      int place = 0;
      for (int u = 0; u < n; ++u) place += list[u] > mine ? 1 : 0;
      if (mine != 0 && place < want) emit(place, mine);
    }
  } else if (threadIdx.x < 32) {
    Cand last = ~0ull;
    for (int j = 0; j < want && last != 0; ++j) {
      Cand best = 0;
      for (int t = threadIdx.x; t < n; t += 32)
        if (list[t] < last && list[t] > best) best = list[t];
      last = warp_best(best);
      if (threadIdx.x == 0 && last != 0) emit(j, last);
    }
  }
}

constexpr int kPartThreads = 256, kPartEach = 16, kPartCols = kPartThreads * kPartEach;

template <typename T>
__device__ __forceinline__ float as_float(T v);
template <> __device__ __forceinline__ float as_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float as_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// One piece of 4096 logits of one hypothesis, 16 in the registers of every thread.  The former kernel passed 2K + 2 times over the whole row
// in shared memory, one CTA per row: 43 us for 4 rows of 32000, which one pass over eight pieces does in a tenth.
template <typename T>
__global__ void __launch_bounds__(kPartThreads)
beam_part_kernel(const T* __restrict__ logits, long ld, const uint8_t* __restrict__ force, float2* __restrict__ part_lse,
                 Cand* __restrict__ part, int first, int K2, int V, int pad, int eos, int vec) {
  __shared__ Cand list[kPartCols];
  __shared__ float red[2][kPartThreads / 32];
  __shared__ int count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kPartThreads / 32;
  const int r = first + blockIdx.y, piece = blockIdx.x;
  const int c0 = piece * kPartCols;
  pdl_trigger();
  pdl_wait();
  const T* x = logits + static_cast<long>(r) * ld + c0;
  constexpr int kPer = 16 / sizeof(T);
  const int cols = min(kPartCols, V - c0);
  float f[kPartEach];
  int col[kPartEach / kPer];
#pragma unroll
  for (int i = 0; i < kPartEach / kPer; ++i) {
    col[i] = (i * kPartThreads + threadIdx.x) * kPer;
    if (vec && col[i] + kPer <= cols) {
      const uint4 u = *reinterpret_cast<const uint4*>(x + col[i]);
      const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
      for (int j = 0; j < kPer; ++j) f[i * kPer + j] = as_float<T>(e[j]);
    } else {
#pragma unroll
      for (int j = 0; j < kPer; ++j) f[i * kPer + j] = col[i] + j < cols ? as_float<T>(x[col[i] + j]) : -INFINITY;
    }
  }
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < kPartEach; ++i) mx = fmaxf(mx, f[i]);
  mx = warp_max(mx);
  if (lane == 0) red[0][warp] = mx;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < warps; ++w) mx = fmaxf(mx, red[0][w]);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kPartEach; ++i)
    if (col[i / kPer] + i % kPer < cols) sum += exp_diff(f[i], mx);
  sum = warp_sum(sum);
  if (lane == 0) red[1][warp] = sum;
  // masks: the padding word, and EOS where the control byte bans it
  const bool ban = force != nullptr && force[r] == 2;
  uint32_t key[kPartEach];
#pragma unroll
  for (int i = 0; i < kPartEach; ++i) {
    const int c = c0 + col[i / kPer] + i % kPer;
    key[i] = rank_of((c == pad || (ban && c == eos)) ? -INFINITY : f[i]);
  }
  // The K2-th largest of the 32 lanes' maxima is a lower bound of the warp's K2-th largest value, so only what reaches it can be
  // chosen: a handful of candidates, collected in shared memory (all of them where K2 exceeds the lanes).
  uint32_t high = 0;
#pragma unroll
  for (int i = 0; i < kPartEach; ++i)
    if (col[i / kPer] + i % kPer < cols) high = max(high, key[i]);
  uint32_t bar = 0;
  if (K2 <= 32) {
    uint32_t rest = high;
    for (int j = 0; j < K2; ++j) {
      bar = __reduce_max_sync(0xffffffffu, rest);
      const uint32_t who = __ballot_sync(0xffffffffu, rest == bar);
      if (lane == __ffs(who) - 1) rest = 0;
    }
  }
  uint32_t takes = 0;
#pragma unroll
  for (int i = 0; i < kPartEach; ++i)
    if (col[i / kPer] + i % kPer < cols && key[i] >= bar) takes |= 1u << i;
  const int mine = __popc(takes);
  int before = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += t;
  }
  int at = 0;
  if (lane == 31) at = atomicAdd(&count, before);
  at = __shfl_sync(0xffffffffu, at, 31) + before - mine;
#pragma unroll
  for (int i = 0; i < kPartEach; ++i)
    if ((takes >> i) & 1u) list[at++] = (static_cast<Cand>(key[i]) << 32) | (kNone - static_cast<uint32_t>(c0 + col[i / kPer] + i % kPer));
  __syncthreads();
  const long o = static_cast<long>(r) * gridDim.x + piece;
  if (threadIdx.x == kPartThreads - 1) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += red[1][w];
    part_lse[o] = make_float2(mx, s);
  }
  const int n = count;
  for (int j = n + threadIdx.x; j < K2; j += kPartThreads) part[o * K2 + j] = 0;
  take_best(list, n, K2, kPartThreads, [&](int place, Cand c) { part[o * K2 + place] = c; });
}

// Everything that the search does between two steps, one CTA per sentence.
//   ctl = {T, min_len, normalize}; inv_norm[n] = 1 / n^alpha for n = 1 .. T + 1 (1 without normalisation or with alpha <= 0).
//   `normalize` chooses the stop rule: with it a sentence goes on until its best active hypothesis, at the longest length, cannot beat the
//   worst finished one; without it the first K finished hypotheses end it
__global__ void __launch_bounds__(256)
beam_advance_kernel(const NmtgBeam s, const void* logits, int bf16, long ld, const float2* __restrict__ part_lse,
                    const Cand* __restrict__ part, int pieces, int V, int staged) {
  extern __shared__ __align__(16) uint8_t shared[];
  __shared__ int verdict;
  const int K = s.K, K2 = 2 * K, n = K * K2, m = pieces * K2;
  Cand* list = reinterpret_cast<Cand*>(shared);             // [K][K2] candidates of the sentence
  Cand* cands = list + n;                                    // [K][pieces][K2] if `staged`
  float* row_val = reinterpret_cast<float*>(cands + (staged ? K * m : 0));   // [K][K2] best of each hypothesis, scores added
  int* row_tok = reinterpret_cast<int*>(row_val + n);
  float* top_val = reinterpret_cast<float*>(row_tok + n);    // [K2]
  int* top_c = reinterpret_cast<int*>(top_val + K2);         // [K2]
  int* parent = top_c + K2;                                  // [K]
  int* column = parent + K;                                  // [K][256]: one column of the ancestor table per thread
  float* base = reinterpret_cast<float*>(column + K * 256);  // [K] score minus log-sum-exp
  float* old_score = base + K;                               // [K] what the tables hold, fetched in one round trip
  float* fs = old_score + K;
  float* f_last = fs + K;
  int* f_step = reinterpret_cast<int*>(f_last + K);
  int* f_row = f_step + K;
  int* plain = f_row + K;                                    // [K] the hypothesis is searched (not dead, not bound to end)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x;
  pdl_trigger();
  pdl_wait();
  const int step = static_cast<int>(s.pos_rows[b * K]);
  const int T = s.ctl[0], min_len = s.ctl[1], normalize = s.ctl[2];
  const int count0 = s.fin_count[b], done0 = s.done[b], limit = s.max_rows[b];
  if (threadIdx.x < K) {
    const int i = b * K + threadIdx.x;
    old_score[threadIdx.x] = s.scores[i];
    fs[threadIdx.x] = s.fin_score[i];
    f_last[threadIdx.x] = s.fin_last[i];
    f_step[threadIdx.x] = s.fin_step[i];
    f_row[threadIdx.x] = s.fin_row[i];
  }
  if (staged)
    for (int i = threadIdx.x; i < K * m; i += 256) cands[i] = part[static_cast<long>(b) * K * m + i];
  for (int k = warp; k < K; k += 8) {
    const int r = b * K + k;
    const float2* pl = part_lse + static_cast<long>(r) * pieces;
    float mx = -INFINITY;
    for (int i = lane; i < pieces; i += 32) mx = fmaxf(mx, pl[i].x);
    mx = warp_max(mx);
    float sum = 0.f;
    for (int i = lane; i < pieces; i += 32) sum += pl[i].y * exp_diff(pl[i].x, mx);
    sum = warp_sum(sum);
    const float add = s.scores[r] - (mx + __logf(sum));
    const bool only_eos = s.force[r] == 1;
    if (lane == 0) {
      base[k] = add;
      plain[k] = !(only_eos || add == -INFINITY);
    }
    for (int j = lane; j < K2; j += 32) {
      const bool live = only_eos && j == 0 && add != -INFINITY;
      float v = -INFINITY;
      if (live) {
        const long at = static_cast<long>(r) * ld + s.eos;
        v = (bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(logits)[at]) : static_cast<const float*>(logits)[at]) + add;
      }
      row_val[k * K2 + j] = v;
      row_tok[k * K2 + j] = live ? s.eos : (j == s.eos ? (s.eos + K2) % V : j);
    }
  }
  __syncthreads();
  // ---- the best 2K of every hypothesis
  if (staged) {
    for (int i = threadIdx.x; i < K * m; i += 256) {
      const int k = i / m;
      const Cand mine = cands[i];
      if (!plain[k] || mine == 0) continue;
      const Cand* row = cands + k * m;
      int place = 0;
      for (int u = 0; u < m; ++u) place += row[u] > mine ? 1 : 0;
      if (place < K2) {
        row_val[k * K2 + place] = value_in(mine) + base[k];
        row_tok[k * K2 + place] = static_cast<int>(index_in(mine));
      }
    }
  } else {
    for (int k = warp; k < K; k += 8) {
      if (!plain[k]) continue;
      const Cand* row = part + (static_cast<long>(b) * K + k) * m;
      Cand last = ~0ull;
      for (int j = 0; j < K2 && last != 0; ++j) {
        Cand best = 0;
        for (int t = lane; t < m; t += 32)
          if (row[t] < last && row[t] > best) best = row[t];
        last = warp_best(best);
        if (lane == 0 && last != 0) {
          row_val[k * K2 + j] = value_in(last) + base[k];
          row_tok[k * K2 + j] = static_cast<int>(index_in(last));
        }
      }
    }
  }
  __syncthreads();
  // ---- the best 2K of the sentence, best first
  for (int c = threadIdx.x; c < n; c += 256) list[c] = cand_of(row_val[c], c);
  __syncthreads();
  take_best(list, n, K2, 256, [&](int place, Cand c) {
    top_c[place] = static_cast<int>(index_in(c));
    top_val[place] = row_val[index_in(c)];
  });
  __syncthreads();
  if (warp == 0) {
    if (lane == 0) {
      const float inv_here = s.inv_norm[step + 1], inv_end = s.inv_norm[T + 1];
      int count = count0, dead = done0;
      // hypotheses that end here, if their EOS is among the best K
      if (step >= min_len && !dead) {
        int ended = 0;
        for (int j = 0; j < K; ++j) {
          const int k = top_c[j] / K2;
          const float v = top_val[j];
          if (row_tok[top_c[j]] != s.eos || !isfinite(v)) continue;
          ++ended;
          const float score = v * inv_here;
          int at = K;
          while (at > 0 && fs[at - 1] < score) --at;              // behind its equals
          if (at == K) continue;
          for (int t = K - 1; t > at; --t) {
            fs[t] = fs[t - 1];
            f_step[t] = f_step[t - 1];
            f_row[t] = f_row[t - 1];
            f_last[t] = f_last[t - 1];
          }
          fs[at] = score;
          f_step[at] = step;
          f_row[at] = k;
          f_last[at] = v - old_score[k];
        }
        count = min(count + ended, K);
      }
      // the next K hypotheses: the best continuations that do not end (EOS continues a hypothesis once at most, so there are K)
      int got = 0;
      for (int j = 0; j < K2 && got < K; ++j) {
        const int c = top_c[j];
        if (row_tok[c] == s.eos) continue;
        top_c[got] = c;                                           // got <= j
        top_val[got] = top_val[j];
        parent[got++] = c / K2;
      }
      for (; got < K; ++got) {
        top_c[got] = 0;
        top_val[got] = -INFINITY;
        parent[got] = 0;
      }
      const float best = top_val[0];
      const bool enough = count >= K && (!normalize || best * inv_end <= fs[K - 1]);
      dead = dead || enough || !isfinite(best);
      s.fin_count[b] = count;
      s.done[b] = static_cast<uint8_t>(dead);
      verdict = dead;
    }
    __syncwarp();
    const int next = step + 1;
    for (int k = lane; k < K; k += 32) {
      const int r = b * K + k, tok = row_tok[top_c[k]];
      const long at = static_cast<long>(step) * s.R + r;          // this step's record
      s.hist_tok[at] = tok;
      s.hist_par[at] = parent[k];
      s.hist_score[at] = top_val[k] - old_score[parent[k]];
      s.scores[r] = verdict ? -INFINITY : top_val[k];
      s.tok[r] = tok;
      s.pos_rows[r] = next;
      s.force[r] = next >= limit ? 1 : (next < min_len ? 2 : 0);
      s.fin_score[r] = fs[k];
      s.fin_last[r] = f_last[k];
      s.fin_step[r] = f_step[k];
      s.fin_row[r] = f_row[k];
    }
  }
  __syncthreads();
  // ---- the ancestor table follows the hypotheses; position `step` was written by the parent itself
  for (int j = threadIdx.x; j <= step && j < s.cap; j += 256) {
    for (int k = 0; k < K; ++k) column[k * 256 + threadIdx.x] = s.anc[static_cast<long>(b * K + k) * s.cap + j];
    for (int k = 0; k < K; ++k)
      s.anc[static_cast<long>(b * K + k) * s.cap + j] = j == step ? b * K + parent[k] : column[parent[k] * 256 + threadIdx.x];
  }
}

// One thread per finished hypothesis: its words and their scores, last to first.
__global__ void beam_trace_kernel(const NmtgBeam s, int B, int n_best, long* __restrict__ words, float* __restrict__ word_scores, int width) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * n_best) return;
  const int b = i / n_best, f = b * s.K + i % n_best;
  if (s.fin_score[f] == -INFINITY) return;
  const int last = s.fin_step[f];
  long* w = words + static_cast<long>(i) * width;
  float* ws = word_scores + static_cast<long>(i) * width;
  if (last < 0 || last >= width) return;
  w[last] = s.eos;
  ws[last] = s.fin_last[f];
  int k = s.fin_row[f];
  for (int t = last - 1; t >= 0; --t) {
    const long at = static_cast<long>(t) * s.R + b * s.K + k;
    w[t] = s.hist_tok[at];
    ws[t] = s.hist_score[at];
    k = s.hist_par[at];
  }
}

// Warps to a CTA: enough for a block of keys each, fewer where the CTAs are many.  Measured (us): 64 sentences x 4 hypotheses x 16
// heads, 80 words of past: two warps 11.2, eight 22.8; source of 60 words: two warps 7.2, eight 21.5; one sentence: eight warps 4.0
// and 3.2, and more with fewer.
int step_warps(long ctas, int blocks, int sms) {
  int w = ctas > 4L * sms ? 2 : ctas > 2L * sms ? 4 : 8;
  while (w > 1 && w > blocks) w >>= 1;
  return w;
}

// go(first, n) for runs of at most 65535 rows, the most that a grid holds along its second dimension (rows and heads in one
// dimension instead made the attention over 1500 frames take 52 us for 46, the wait for the kernel before it included)
template <typename Go>
const char* by_rows(int rows, Go go) {
  for (int first = 0; first < rows; first += 65535)
    if (const char* e = go(first, rows - first < 65535 ? rows - first : 65535)) return e;
  return nullptr;
}

template <int KB>
const char* launch_self(const void* qkv, long ld, void* kc, void* vc, const int* anc, const long* pos_rows, void* out, int B, int K, int heads,
                        int cap, float scale, int sms, cudaStream_t stream) {
  const int groups = (K + KB - 1) / KB;
  const int warps = step_warps(static_cast<long>(heads) * B * groups, cap, sms);
  return by_rows(B * groups, [&](int first, int n) {
    return launch(decode_self_kernel<KB>, dim3(heads, n), dim3(32 * warps), 0, 1, stream, static_cast<const __nv_bfloat16*>(qkv), ld,
                  static_cast<__nv_bfloat16*>(kc), static_cast<__nv_bfloat16*>(vc), anc, pos_rows, static_cast<__nv_bfloat16*>(out), first, K,
                  groups, heads, cap, scale);
  });
}

template <int KB>
const char* launch_cross(const void* q, long ld, const void* ck, const void* cv, const int* lengths, void* out, int B, int K, int heads,
                         int cap, float scale, int sms, cudaStream_t stream) {
  const int groups = (K + KB - 1) / KB;
  // shares of at least 128 keys until there are four CTAs to an SM.  8 sentences x 4 hypotheses x 20 heads x 1500 keys take 27 us
  // (bytes at the copy rate: 9.5), one sentence 9.6: what is left is the arithmetic of the dot products, folds and weights (about
  // 560 instructions per 16 keys and warp); two, four or eight shares make no difference
  const long ctas = static_cast<long>(heads) * B * groups;
  int splits = 1;
  while (splits < 8 && ctas * splits < 4L * sms && cap >= splits * 2 * 128) splits *= 2;
  const int blocks = (cap / splits + 4 * keys_of<KB>() - 1) / (4 * keys_of<KB>());
  const int warps = cap > 512 ? 4 : step_warps(ctas * splits, blocks, sms);
  return by_rows(B * groups, [&](int first, int n) {
    return launch(decode_cross_kernel<KB>, dim3(heads, n, splits), dim3(32 * warps), 0, splits, stream,
                  static_cast<const __nv_bfloat16*>(q), ld, static_cast<const __nv_bfloat16*>(ck), static_cast<const __nv_bfloat16*>(cv),
                  lengths, static_cast<__nv_bfloat16*>(out), first, K, groups, heads, cap, scale, splits);
  });
}

}  // namespace

int num_sms();

}  // namespace b200

using namespace b200;

extern "C" {

const char* nmtg_decode_self(const void* qkv, long ld, void* k_cache, void* v_cache, const int* anc, const long* pos_rows, void* out,
                             int B, int K, int heads, int cap, float scale, cudaStream_t stream) {
  if (B <= 0 || K <= 0 || heads <= 0 || cap <= 0) return "decode_self: bad geometry";
  if (ld % 8) return "decode_self: row stride must be a multiple of 8 elements";
  const int sms = num_sms();
  if (K == 1) return launch_self<1>(qkv, ld, k_cache, v_cache, anc, pos_rows, out, B, K, heads, cap, scale, sms, stream);
  if (K == 2) return launch_self<2>(qkv, ld, k_cache, v_cache, anc, pos_rows, out, B, K, heads, cap, scale, sms, stream);
  return launch_self<4>(qkv, ld, k_cache, v_cache, anc, pos_rows, out, B, K, heads, cap, scale, sms, stream);
}

const char* nmtg_decode_cross(const void* q, long ld, const void* ck, const void* cv, const int* lengths, void* out, int B, int K,
                              int heads, int cap, float scale, cudaStream_t stream) {
  if (B <= 0 || K <= 0 || heads <= 0 || cap <= 0) return "decode_cross: bad geometry";
  if (ld % 8) return "decode_cross: row stride must be a multiple of 8 elements";
  const int sms = num_sms();
  if (K == 1) return launch_cross<1>(q, ld, ck, cv, lengths, out, B, K, heads, cap, scale, sms, stream);
  if (K == 2) return launch_cross<2>(q, ld, ck, cv, lengths, out, B, K, heads, cap, scale, sms, stream);
  return launch_cross<4>(q, ld, ck, cv, lengths, out, B, K, heads, cap, scale, sms, stream);
}

const char* nmtg_beam_step(const NmtgBeam* s, const void* logits, long ld, int dtype, void* part_lse, void* part, int B, int V,
                           cudaStream_t stream) {
  const int K = s->K, K2 = 2 * K, pieces = (V + kPartCols - 1) / kPartCols, R = B * K;
  if (B <= 0 || K <= 0 || K > 32) return "beam_step: 1 to 32 hypotheses per sentence";
  if (K2 > V) return "beam_step: vocabulary smaller than twice the beam";
  if (ld < V) return "beam_step: row stride smaller than the vocabulary";
  const int vec = (ld * (dtype == 0 ? 4 : 2)) % 16 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  float2* lse = static_cast<float2*>(part_lse);
  Cand* cand = static_cast<Cand*>(part);
  const char* e = by_rows(R, [&](int first, int n) {
    if (dtype == 0)
      return launch(beam_part_kernel<float>, dim3(pieces, n), dim3(kPartThreads), 0, 1, stream, static_cast<const float*>(logits), ld, s->force,
                    lse, cand, first, K2, V, s->pad, s->eos, vec);
    return launch(beam_part_kernel<__nv_bfloat16>, dim3(pieces, n), dim3(kPartThreads), 0, 1, stream, static_cast<const __nv_bfloat16*>(logits),
                  ld, s->force, lse, cand, first, K2, V, s->pad, s->eos, vec);
  });
  if (e) return e;
  // the pieces' candidates are staged in shared memory unless a wide beam over a large vocabulary makes them many
  const size_t tables = static_cast<size_t>(K) * K2 * 16 + 4 * (2 * K2 + K + K * 256 + 7 * K), cands = static_cast<size_t>(K) * pieces * K2 * 8;
  const int staged = cands <= 32 * 1024;
  const size_t smem = tables + (staged ? cands : 0);                               // 32 hypotheses: 100 KB
  if (smem > 48 * 1024) {
    cudaError_t err = cudaFuncSetAttribute(beam_advance_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    if (err != cudaSuccess) return cudaGetErrorString(err);
  }
  return launch(beam_advance_kernel, dim3(B), dim3(256), smem, 1, stream, *s, logits, dtype, ld, static_cast<const float2*>(lse),
                static_cast<const Cand*>(cand), pieces, V, staged);
}

const char* nmtg_beam_trace(const NmtgBeam* s, int B, int n_best, long* words, float* word_scores, int width, cudaStream_t stream) {
  if (n_best < 1 || n_best > s->K) return "beam_trace: n_best must be between 1 and the beam";
  const int n = B * n_best;
  beam_trace_kernel<<<(n + 63) / 64, 64, 0, stream>>>(*s, B, n_best, words, word_scores, width);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // extern "C"
