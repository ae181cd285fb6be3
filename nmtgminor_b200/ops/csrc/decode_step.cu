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
// exp(a - b) with exp(-inf - -inf) = 0: an empty part has no weight
__device__ __forceinline__ float exp_diff(float a, float b) { return a == -INFINITY ? 0.f : __expf(a - b); }

// ---------------------------------------------------------------------------------------------------------------------
// Attention of one new position.  Both kernels serve the hypotheses of a sentence, up to eight, from one CTA (head, sentence), whose
// warps take blocks of 16 keys.  The products run on the tensor cores (m16n8k16): with dot products, folds and weights in ordinary
// instructions a block cost 560 of them, about 180 this way, and attention over 1500 frames was bound by that.  tcgen05 would want
// 128 rows; here the keys are the 16 rows of the first product, the dimensions those of the second, and the queries the 8 columns.
//   * The weights of the softmax are 32-bit numbers, and the product with the values takes 16-bit ones: it runs three times, with
//     the weights' rounding to bf16, the rounding of the rest, and the rest of that, which add up to all 24 bits.
//   * No operand passes through shared memory.  The order in which a contraction runs is free, so a lane takes eight consecutive
//     dimensions of a key (one 16-byte load) where the instruction wants four scattered pairs, as long as keys and queries do the
//     same; of the values it takes eight dimensions of four keys and pairs them with byte permutations, so that rows g and g + 8 of
//     tile j are dimensions 8 g + 2 j and 8 g + 2 j + 1.  The weights change from a row per key to a row per query with movmatrix.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kStepWarps = 8;        // at most
constexpr int kQueries = 8;          // to a CTA
constexpr int kRowLd = 68;           // 64 dimensions, maximum, sum, padding

__device__ __forceinline__ uint32_t transpose8(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// x, or the largest number with some sign for what is none
__device__ __forceinline__ float in_range(float x) {
  float y;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(3.402823466e38f));
  return y;
}
__device__ __forceinline__ uint4 zero4() { return make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

struct Keys { uint4 x[2][2]; };      // [i][c]: key g + 8 i, dimensions 32 c + 8 t ..   (g = lane / 4, t = lane % 4)
struct Values { uint4 x[2][2]; };    // [i][e]: key 8 i + 2 t + e, dimensions 8 g ..
struct Weights { uint32_t x[3][2]; };      // [part][i]: keys 8 i + 2 t, + 1 of query g

struct WarpTile {
  uint4 q[2];                        // query g, dimensions 32 c + 8 t ..
  float m[2], l[2];                  // queries 2 t + e
  float o[4][4];                     // [j][2 f + e]: dimension 8 g + 2 j + f of query 2 t + e

  // base: first query row of this head
  __device__ __forceinline__ void init(const __nv_bfloat16* base, long ld, int queries, int lane) {
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    const int g = lane >> 2;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const __nv_bfloat16* p = base + g * ld + 32 * c + 8 * (lane & 3);
      q[c] = zero4();
      if (g < queries) {
        if ((reinterpret_cast<uintptr_t>(base) & 15) == 0) q[c] = load8(p);
        else {
          __nv_bfloat16 e[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) e[j] = p[j];
          memcpy(&q[c], e, 16);
        }
      }
    }
  }
  // scores of the block's 16 keys: s[2 i + e] = key g + 8 i, query 2 t + e
  __device__ __forceinline__ void scores(const Keys& k, float (&s)[4]) const {
    s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      mma_bf16(s, k.x[0][c].x, k.x[1][c].x, k.x[0][c].y, k.x[1][c].y, q[c].x, q[c].y);
      mma_bf16(s, k.x[0][c].z, k.x[1][c].z, k.x[0][c].w, k.x[1][c].w, q[c].z, q[c].w);
    }
  }
  // Scores (`keys` of the 16 exist) -> weights; the output so far is brought to the new maximum.
  __device__ __forceinline__ void weigh(const float (&s)[4], Weights& w, int keys, float scale, int lane) {
    const int g = lane >> 2;
    float p[4], corr[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float x0 = g < keys ? s[e] * scale : -INFINITY, x1 = g + 8 < keys ? s[2 + e] * scale : -INFINITY;
      float mx = fmaxf(x0, x1);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float mn = fmaxf(m[e], mx);
      corr[e] = mn == m[e] ? 1.f : exp_diff(m[e], mn);
      m[e] = mn;
      p[e] = exp_diff(x0, mn);
      p[2 + e] = exp_diff(x1, mn);
      l[e] = l[e] * corr[e] + (p[e] + p[2 + e]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float a = p[2 * i], b = p[2 * i + 1];
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        const float2 f = __bfloat1622float2(h);
        a -= f.x;
        b -= f.y;
        w.x[part][i] = transpose8(*reinterpret_cast<const uint32_t*>(&h));
      }
    }
    if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        o[j][0] *= corr[0];
        o[j][1] *= corr[1];
        o[j][2] *= corr[0];
        o[j][3] *= corr[1];
      }
    }
  }
  // output += values x weights.  kOne: the values are those of query `only`, and the other queries' columns stay as they are, whatever
  // its values hold (0 x NaN).  A block's sum, smallest parts first, meets the output in an ordinary addition, which rounds to nearest; the
  // instruction cuts off, and summed through it alone outputs were 1.5 to 3 times as far from 64 bits (1500 keys 1.5e-8, 4.1e-9 so).
  // The smaller parts of a weight are often zero, and under an infinite value their sum is then no number: it is brought into range,
  // and what the largest part makes of such a value counts.
  template <bool kOne>
  __device__ __forceinline__ void add(const Values& v, const Weights& w, int only, int lane) {
    const uint32_t* v0 = reinterpret_cast<const uint32_t*>(&v.x[0][0]);
    const uint32_t* v1 = reinterpret_cast<const uint32_t*>(&v.x[0][1]);
    const uint32_t* v2 = reinterpret_cast<const uint32_t*>(&v.x[1][0]);
    const uint32_t* v3 = reinterpret_cast<const uint32_t*>(&v.x[1][1]);
    const int t = lane & 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t a0 = __byte_perm(v0[j], v1[j], 0x5410), a1 = __byte_perm(v0[j], v1[j], 0x7632);
      const uint32_t a2 = __byte_perm(v2[j], v3[j], 0x5410), a3 = __byte_perm(v2[j], v3[j], 0x7632);
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(d, a0, a1, a2, a3, w.x[2][0], w.x[2][1]);
      mma_bf16(d, a0, a1, a2, a3, w.x[1][0], w.x[1][1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) d[i] = in_range(d[i]);
      mma_bf16(d, a0, a1, a2, a3, w.x[0][0], w.x[0][1]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!kOne || 2 * t + (i & 1) == only) o[j][i] += d[i];
    }
  }
  // rows of this warp: [query][kRowLd] = unnormalised output, maximum, sum
  __device__ __forceinline__ void store(float* rows, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) l[e] += __shfl_xor_sync(0xffffffffu, l[e], o);
      float* row = rows + (2 * t + e) * kRowLd;
      *reinterpret_cast<float4*>(row + 8 * g) = make_float4(o[0][e], o[0][2 + e], o[1][e], o[1][2 + e]);
      *reinterpret_cast<float4*>(row + 8 * g + 4) = make_float4(o[2][e], o[2][2 + e], o[3][e], o[3][2 + e]);
      if (g == 0) {
        row[64] = m[e];
        row[65] = l[e];
      }
    }
  }
};

// Sum of `n` warps' rows of one query: this lane's two output dimensions, the maximum and the sum.
__device__ __forceinline__ void merge_rows(const float* rows, int n, int query, int lane, float& o0, float& o1, float& mx, float& sum) {
  mx = -INFINITY;
  for (int w = 0; w < n; ++w) mx = fmaxf(mx, rows[(w * kQueries + query) * kRowLd + 64]);
  o0 = o1 = sum = 0.f;
  for (int w = 0; w < n; ++w) {
    const float* row = rows + (w * kQueries + query) * kRowLd;
    const float e = exp_diff(row[64], mx);
    const float2 a = *reinterpret_cast<const float2*>(row + 2 * lane);
    sum += e * row[65];
    o0 += e * a.x;
    o1 += e * a.y;
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// self-attention.  The hypotheses of a sentence share the beginning of their past: a block whose ancestor rows agree is read once for
// all of them.  In the others every hypothesis has keys of its own: their scores are computed one hypothesis at a time, each column
// of the tile keeps those of its own query, and the softmax is again one for all.  The loads of four hypotheses are in flight together;
// one after the other they had a warp wait for memory four times a block.  Within a search step (`early`) the ancestors, and what
// the caches hold of earlier positions, come from earlier steps, and a step begins with a launch that waits for all before it: they
// are staged, and the keys and values fetched into L2, while the projection before this kernel still runs.  Back to back (us, dot
// products in ordinary instructions / this): 64 sentences x 4 hypotheses x 16 heads, 80 words 23.4 / 20.3; with the projection before it, one
// sentence 10.3 / 8.6, 8 x 4 with 20 heads, 50 words 14.7 / 11.8.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kPast = 256;           // positions whose ancestors are staged at a time

template <int kOpen>
__global__ void __launch_bounds__(32 * kStepWarps, kOpen == 4 ? 2 : 3)
decode_self_kernel(const __nv_bfloat16* __restrict__ qkv, long ld, __nv_bfloat16* __restrict__ kc, __nv_bfloat16* __restrict__ vc,
                   const int* __restrict__ anc, const long* __restrict__ pos_rows, __nv_bfloat16* __restrict__ out, int first, int K, int groups,
                   int per, int heads, int cap, float scale, int early) {
  extern __shared__ __align__(16) float rows[];          // [warps][kQueries][kRowLd]
  __shared__ int at[kQueries][kPast];                    // cache row of every hypothesis and position
  __shared__ int shared_by_all[kPast / 16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int h = blockIdx.x, item = first + blockIdx.y;
  const int k0 = (item % groups) * per, r0 = (item / groups) * K + k0;
  const int queries = min(per, K - k0);
  const int hid = heads * 64;
  const int g = lane >> 2, t = lane & 3;
  let_next_start();
  if (!early) wait_for_previous();
  const long pos_l = pos_rows[r0];                     // the same for all hypotheses of a sentence
  const int pos = pos_l < 0 ? 0 : (pos_l >= cap ? cap - 1 : static_cast<int>(pos_l));
  WarpTile tile;
  for (int c0 = 0; c0 <= pos; c0 += kPast) {
    if (c0 > 0) __syncthreads();
    // the table is read beyond `pos` too, so that it does not wait for it
    const int limit = (cap + 31) & ~31;
    for (int i = threadIdx.x; i < kPast && c0 + i < limit; i += blockDim.x) {
      const int j = c0 + i;
      int row[kQueries];
#pragma unroll
      for (int k = 0; k < kQueries; ++k) row[k] = j < cap && k < queries ? anc[static_cast<long>(r0 + k) * cap + j] : 0;
      bool agree = true;
#pragma unroll
      for (int k = 0; k < kQueries; ++k) {
        at[k][i] = row[k] * cap + j;
        if (k < queries) agree = agree && row[k] == row[0];
      }
      const uint32_t all = __ballot_sync(0xffffffffu, (agree && j != pos) || j > pos);      // the new position is everyone's own
      if (lane == 0) shared_by_all[i / 16] = (all & 0xffffu) == 0xffffu;
      if (lane == 16) shared_by_all[i / 16] = (all >> 16) == 0xffffu;
    }
    __syncthreads();
    if (early)
      for (int i = threadIdx.x; i < min(kPast, pos - c0); i += blockDim.x)
        for (int k = 0; k < queries; ++k)
          if (k == 0 || at[k][i] != at[0][i]) {
            const long e = static_cast<long>(at[k][i]) * hid + h * 64;
            prefetch_l2(kc + e);
            prefetch_l2(vc + e);
          }
    if (c0 == 0) {
      if (early) wait_for_previous();
      tile.init(qkv + r0 * ld + h * 64, ld, queries, lane);
    }
    for (int blk = warp; blk < kPast / 16 && c0 + blk * 16 <= pos; blk += warps) {
      const int j0 = c0 + blk * 16, keys = pos + 1 - j0;
      // row of position j of hypothesis k; the new position comes straight from the projection
      auto load_keys = [&](Keys& ks, int k) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const int j = j0 + 8 * n + g;
          const __nv_bfloat16* src = j == pos ? qkv + (r0 + k) * ld + hid + h * 64 : kc + static_cast<long>(at[k & (kQueries - 1)][j - c0]) * hid + h * 64;
#pragma unroll
          for (int c = 0; c < 2; ++c) ks.x[n][c] = k < queries && j <= pos ? load8(src + 32 * c + 8 * t) : zero4();
        }
      };
      auto load_values = [&](Values& vs, int k) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = j0 + 8 * n + 2 * t + e;
            const __nv_bfloat16* src = j == pos ? qkv + (r0 + k) * ld + 2 * hid + h * 64 : vc + static_cast<long>(at[k & (kQueries - 1)][j - c0]) * hid + h * 64;
            vs.x[n][e] = k < queries && j <= pos ? load8(src + 8 * g) : zero4();
          }
      };
      float s[4];
      Weights w;
      if (shared_by_all[blk]) {
        Keys ks;
        Values vs;
        load_keys(ks, 0);
        load_values(vs, 0);
        tile.scores(ks, s);
        tile.weigh(s, w, keys, scale, lane);
        tile.add<false>(vs, w, 0, lane);
      } else {
        s[0] = s[1] = s[2] = s[3] = 0.f;
        for (int first = 0; first < queries; first += kOpen) {
          Keys ks[kOpen];
#pragma unroll
          for (int i = 0; i < kOpen; ++i) load_keys(ks[i], first + i);
#pragma unroll
          for (int i = 0; i < kOpen; ++i) {
            float d[4];
            tile.scores(ks[i], d);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (2 * t + (e & 1) == first + i) s[e] = d[e];
          }
        }
        Values vs[kOpen];
#pragma unroll
        for (int i = 0; i < kOpen; ++i) load_values(vs[i], i);
        tile.weigh(s, w, keys, scale, lane);
        for (int first = 0; first < queries; first += kOpen) {
#pragma unroll
          for (int i = 0; i < kOpen; ++i)
            if (first + i < queries) tile.add<true>(vs[i], w, first + i, lane);
          if (first + kOpen < queries) {
#pragma unroll
            for (int i = 0; i < kOpen; ++i) load_values(vs[i], first + kOpen + i);
          }
        }
      }
    }
  }
  // the new position's place in the caches (other CTAs' heads and hypotheses write theirs; nobody reads it before the next step)
  for (int i = threadIdx.x; i < queries * 16; i += blockDim.x) {
    const int k = i >> 4, half = (i >> 3) & 1, c = i & 7;
    const uint4 u = load8(qkv + (r0 + k) * ld + (1 + half) * hid + h * 64 + 8 * c);
    *reinterpret_cast<uint4*>((half ? vc : kc) + (static_cast<long>(r0 + k) * cap + pos) * hid + h * 64 + 8 * c) = u;
  }
  tile.store(rows + warp * kQueries * kRowLd, lane);
  __syncthreads();
  for (int k = warp; k < queries; k += warps) {
    float o0, o1, mx, sum;
    merge_rows(rows, warps, k, lane, o0, o1, mx, sum);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    *reinterpret_cast<__nv_bfloat162*>(out + (static_cast<long>(r0 + k) * heads + h) * 64 + 2 * lane) = __floats2bfloat162_rn(o0 * inv, o1 * inv);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// encoder-decoder attention.  CTA = (head, sentence and group of hypotheses, share of the keys); the shares of a sentence are one
// cluster and meet in distributed shared memory.  Within a search step (`early`) nothing that may still run writes the encoder's
// keys, values and lengths: each warp loads its first block, and has the rest of its share fetched into L2, while the previous
// kernels of the step run.  Back to back (us, dot products in ordinary instructions / this): 8 sentences x 1500 frames x 20 heads 22.9 / 13.9
// (62 MB: 9.4 at the copy rate), 64 sentences of 60 words 7.5 / 5.9, one sentence 4.3 / 3.5.
// ---------------------------------------------------------------------------------------------------------------------
// (320 x 2 threads: 96 registers, so that five CTAs of four warps fit an SM; with 102 the 640 CTAs of 8 sentences are two waves, 19.3 us for 13.4)
__global__ void __launch_bounds__(320, 2)
decode_cross_kernel(const __nv_bfloat16* __restrict__ q, long ld, const __nv_bfloat16* __restrict__ ck, const __nv_bfloat16* __restrict__ cv,
                    const int* __restrict__ lengths, __nv_bfloat16* __restrict__ out, int first, int K, int groups, int per, int heads, int cap,
                    float scale, int splits, int early) {
  extern __shared__ __align__(16) float rows[];          // [warps][kQueries][kRowLd]
  __shared__ __align__(16) float mine[kQueries][kRowLd];      // this CTA's sums, read by the whole cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int h = blockIdx.x, item = first + blockIdx.y;
  const int b = item / groups, k0 = (item % groups) * per;
  const int queries = min(per, K - k0);
  const int share = blockIdx.z;
  const int hid = heads * 64;
  const int g = lane >> 2, t = lane & 3;
  let_next_start();
  if (!early) wait_for_previous();
  int len = lengths[b];
  len = len < 0 ? 0 : (len > cap ? cap : len);
  const int chunk = ((len + splits - 1) / splits + 15) & ~15;
  const int begin = share * chunk, end = min(len, begin + chunk);
  const __nv_bfloat16* kb = ck + static_cast<long>(b) * cap * hid + h * 64 + 8 * t;
  const __nv_bfloat16* vb = cv + static_cast<long>(b) * cap * hid + h * 64 + 8 * g;
  Keys ks;
  Values vs;
  auto load_keys = [&](int j0) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int j = j0 + 8 * n + g;
        ks.x[n][c] = j < end ? load8(kb + static_cast<long>(j) * hid + 32 * c) : zero4();
      }
  };
  auto load_values = [&](int j0) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = j0 + 8 * n + 2 * t + e;
        vs.x[n][e] = j < end ? load8(vb + static_cast<long>(j) * hid) : zero4();
      }
  };
  int j0 = begin + warp * 16;
  load_keys(j0);
  load_values(j0);
  if (early) {
    for (int j = begin + warps * 16 + threadIdx.x; j < end; j += blockDim.x) {
      const long at = (static_cast<long>(b) * cap + j) * hid + h * 64;
      prefetch_l2(ck + at);
      prefetch_l2(cv + at);
    }
    wait_for_previous();
  }
  WarpTile tile;
  tile.init(q + (static_cast<long>(b) * K + k0) * ld + h * 64, ld, queries, lane);
  for (; j0 < end; j0 += warps * 16) {
    float s[4];
    Weights w;
    tile.scores(ks, s);
    load_keys(j0 + warps * 16);
    tile.weigh(s, w, end - j0, scale, lane);
    tile.add<false>(vs, w, 0, lane);
    load_values(j0 + warps * 16);
  }
  tile.store(rows + warp * kQueries * kRowLd, lane);
  __syncthreads();
  for (int k = warp; k < queries; k += warps) {
    float o0, o1, mx, sum;
    merge_rows(rows, warps, k, lane, o0, o1, mx, sum);
    if (splits == 1) {
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
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
  for (int k = share + splits * warp; k < queries; k += splits * warps) {
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
// in shared memory, one CTA per row: 43 us for 4 rows of 32000, which one pass over eight pieces does in a tenth.  256 rows of 32000 are
// bound by instructions: comparing floats against the highest of the warps' bounds takes 14.1 us, where every column was ranked as an
// integer, masked and checked against the end, and each warp used its own bound, 21.9.
template <typename T, bool kWarm>
__global__ void __launch_bounds__(kPartThreads)
beam_part_kernel(const T* __restrict__ logits, long ld, const uint8_t* __restrict__ force, float2* __restrict__ part_lse,
                 Cand* __restrict__ part, int first, int K2, int V, int pad, int eos, int vec) {
  __shared__ Cand list[kPartCols];
  __shared__ float red[3][kPartThreads / 32];
  __shared__ int count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = kPartThreads / 32;
  const int r = first + blockIdx.y, piece = blockIdx.x;
  const int c0 = piece * kPartCols;
  let_next_start();
  const T* x = logits + static_cast<long>(r) * ld + c0;
  constexpr int kPer = 16 / sizeof(T);
  // kWarm: once over no columns, storing nothing, before the wait; a step runs these instructions once, and fetching them took longer than
  // running them (4 rows of 32000 in a search 6.6 us, 4.3 so; not where the blocks are several waves: 256 rows 13.5 and 16.5)
#pragma unroll 1
  for (int pass = kWarm ? 0 : 1; pass < 2; ++pass) {
    if (pass == 1) wait_for_previous();
    const int cols = pass == 1 ? min(kPartCols, V - c0) : 0;
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
    float top = -INFINITY;                                   // of this thread
#pragma unroll
    for (int i = 0; i < kPartEach; ++i) top = fmaxf(top, f[i]);
    float mx = warp_max(top);
    if (lane == 0) red[0][warp] = mx;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < warps; ++w) mx = fmaxf(mx, red[0][w]);
    float sum = 0.f;
    if (mx != -INFINITY) {                                   // columns past the end hold -inf, whose weight is zero
#pragma unroll
      for (int i = 0; i < kPartEach; ++i) sum += __expf(f[i] - mx);
    } else {
#pragma unroll
      for (int i = 0; i < kPartEach; ++i)
        if (f[i] != f[i]) sum = f[i];                        // no number here: NaN stays NaN
    }
    sum = warp_sum(sum);
    if (lane == 0) red[1][warp] = sum;
    // masks: the padding word, and EOS where the control byte bans it
    const bool ban = pass == 1 && force != nullptr && force[r] == 2;
    auto owns = [&](int word) { return word >= c0 && word - c0 < cols && (word - c0) / kPer % kPartThreads == threadIdx.x; };
    if (owns(pad) || (ban && owns(eos))) {
      top = -INFINITY;
#pragma unroll
      for (int i = 0; i < kPartEach; ++i) {
        const int c = c0 + col[i / kPer] + i % kPer;
        if (c == pad || (ban && c == eos)) f[i] = -INFINITY;
        top = fmaxf(top, f[i]);
      }
    }
    // The K2-th largest of a warp's 32 lane maxima is a lower bound of the piece's K2-th largest value, so only what reaches the highest of
    // these bounds can be chosen: a handful of candidates, collected in shared memory (all of them where K2 exceeds the lanes, or where the
    // bound excludes nothing: then NaN may be wanted too).
    float bar = -INFINITY;
    if (K2 <= 32) {
      uint32_t rest = rank_of(top), best = 0;
      for (int j = 0; j < K2; ++j) {
        best = __reduce_max_sync(0xffffffffu, rest);
        const uint32_t who = __ballot_sync(0xffffffffu, rest == best);
        if (lane == __ffs(who) - 1) rest = 0;
      }
      if (best != 0) bar = value_of(best);
      if (lane == 0) red[2][warp] = bar;
      __syncthreads();
#pragma unroll
      for (int w = 0; w < warps; ++w) bar = fmaxf(bar, red[2][w]);
    }
    uint32_t takes = 0;
    if (bar != -INFINITY) {
      if (top >= bar) {
#pragma unroll
        for (int i = 0; i < kPartEach; ++i)
          if (f[i] >= bar) takes |= 1u << i;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPartEach; ++i)
        if (col[i / kPer] + i % kPer < cols) takes |= 1u << i;
    }
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
      if ((takes >> i) & 1u) list[at++] = cand_of(f[i], c0 + col[i / kPer] + i % kPer);
    __syncthreads();
    const long o = static_cast<long>(r) * gridDim.x + piece;
    if (threadIdx.x == kPartThreads - 1 && pass == 1) {
      float s = 0.f;
      for (int w = 0; w < warps; ++w) s += red[1][w];
      part_lse[o] = make_float2(mx, s);
    }
    const int n = count;
    for (int j = n + threadIdx.x; j < K2 && pass == 1; j += kPartThreads) part[o * K2 + j] = 0;
    take_best(list, n, K2, kPartThreads, [&](int place, Cand c) { part[o * K2 + place] = c; });
    if (kWarm && pass == 0) __syncthreads();
  }
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
  let_next_start();
  wait_for_previous();
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

// go(first, n) for runs of at most 65535 rows, the most that a grid holds along its second dimension (rows and heads in one
// dimension instead made the attention over 1500 frames take 52 us for 46, the wait for the kernel before it included)
template <typename Go>
const char* by_rows(int rows, Go go) {
  for (int first = 0; first < rows; first += 65535)
    if (const char* e = go(first, rows - first < 65535 ? rows - first : 65535)) return e;
  return nullptr;
}

// hypotheses of a sentence -> groups of at most eight, evenly
struct Groups {
  int count, per;
  explicit Groups(int K) : count((K + kQueries - 1) / kQueries), per((K + count - 1) / count) {}
};

const char* launch_self(const void* qkv, long ld, void* kc, void* vc, const int* anc, const long* pos_rows, void* out, int B, int K, int heads,
                        int cap, float scale, int sms, cudaStream_t stream) {
  const Groups of(K);
  const long ctas = static_cast<long>(heads) * B * of.count;
  // as many warps to a CTA as the GPU holds at once, 16 to an SM with several hypotheses (128 registers): 64 sentences x 4 hypotheses x 16
  // heads, 80 words of past of their own: two warps 24.6 us, four 30.2, one 33.5 (memory: 13.4); 8 sentences x 20 heads, 50 words:
  // eight warps 6.7.  24 to an SM with one hypothesis, and a block of keys for every warp (us, with the product before it, two warps / by
  // this rule: 32 sentences x 20 heads, 186 words 23.1 / 18.1; 61 x 12, 106 words 18.1 / 14.5; four warps: 20 x 16, 80 words 10.8 / 10.1)
  int warps = kStepWarps;
  while (warps > 2 && (ctas * warps > (K == 1 ? 24L : 16L) * sms || (K == 1 && 16 * warps > cap))) warps >>= 1;
  return by_rows(B * of.count, [&](int first, int n) {
    return launch(K == 1 ? decode_self_kernel<1> : decode_self_kernel<4>, dim3(heads, n), dim3(32 * warps), warps * kQueries * kRowLd * sizeof(float), 1, stream,
                  static_cast<const __nv_bfloat16*>(qkv), ld, static_cast<__nv_bfloat16*>(kc), static_cast<__nv_bfloat16*>(vc), anc, pos_rows,
                  static_cast<__nv_bfloat16*>(out), first, K, of.count, of.per, heads, cap, scale, step_overlap() ? 1 : 0);
  });
}

const char* launch_cross(const void* q, long ld, const void* ck, const void* cv, const int* lengths, void* out, int B, int K, int heads,
                         int cap, float scale, int sms, cudaStream_t stream) {
  const Groups of(K);
  // shares of at least 128 keys until there are four CTAs to an SM
  const long ctas = static_cast<long>(heads) * B * of.count;
  int splits = 1;
  while (splits < 8 && ctas * splits < 4L * sms && cap >= splits * 2 * 128) splits *= 2;
  const int blocks = (cap / splits + 15) / 16;
  // a block for every warp, and no more warps than the GPU holds at once (8 sentences x 20 heads x 1500 frames, 640 CTAs: two warps
  // 21.6 us, four 16.3, the kernel alone)
  int warps = kStepWarps;
  while (warps > 1 && (warps > blocks || ctas * splits * warps > 24L * sms)) warps >>= 1;
  return by_rows(B * of.count, [&](int first, int n) {
    return launch(decode_cross_kernel, dim3(heads, n, splits), dim3(32 * warps), warps * kQueries * kRowLd * sizeof(float), splits, stream,
                  static_cast<const __nv_bfloat16*>(q), ld, static_cast<const __nv_bfloat16*>(ck), static_cast<const __nv_bfloat16*>(cv),
                  lengths, static_cast<__nv_bfloat16*>(out), first, K, of.count, of.per, heads, cap, scale, splits, step_overlap() ? 1 : 0);
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
  return launch_self(qkv, ld, k_cache, v_cache, anc, pos_rows, out, B, K, heads, cap, scale, sms, stream);
}

const char* nmtg_decode_cross(const void* q, long ld, const void* ck, const void* cv, const int* lengths, void* out, int B, int K,
                              int heads, int cap, float scale, cudaStream_t stream) {
  if (B <= 0 || K <= 0 || heads <= 0 || cap <= 0) return "decode_cross: bad geometry";
  if (ld % 8) return "decode_cross: row stride must be a multiple of 8 elements";
  const int sms = num_sms();
  return launch_cross(q, ld, ck, cv, lengths, out, B, K, heads, cap, scale, sms, stream);
}

const char* nmtg_beam_step(const NmtgBeam* s, const void* logits, long ld, int dtype, void* part_lse, void* part, int B, int V,
                           cudaStream_t stream) {
  const int K = s->K, K2 = 2 * K, pieces = (V + kPartCols - 1) / kPartCols, R = B * K;
  if (B <= 0 || K <= 0 || K > 32) return "beam_step: 1 to 32 hypotheses per sentence";
  if (K2 > V) return "beam_step: vocabulary smaller than twice the beam";
  if (ld < V) return "beam_step: row stride smaller than the vocabulary";
  const int vec = (ld * (dtype == 0 ? 4 : 2)) % 16 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  const bool warm = step_overlap() && static_cast<long>(pieces) * R <= 2L * num_sms();      // blocks that wait together
  float2* lse = static_cast<float2*>(part_lse);
  Cand* cand = static_cast<Cand*>(part);
  const char* e = by_rows(R, [&](int first, int n) {
    if (dtype == 0)
      return launch(warm ? beam_part_kernel<float, true> : beam_part_kernel<float, false>, dim3(pieces, n), dim3(kPartThreads), 0, 1, stream, static_cast<const float*>(logits), ld, s->force,
                    lse, cand, first, K2, V, s->pad, s->eos, vec);
    return launch(warm ? beam_part_kernel<__nv_bfloat16, true> : beam_part_kernel<__nv_bfloat16, false>, dim3(pieces, n), dim3(kPartThreads), 0, 1, stream, static_cast<const __nv_bfloat16*>(logits),
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
