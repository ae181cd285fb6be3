// Shared pieces of the tcgen05 GEMM kernels (single-CTA and CTA-pair variants): argument block and the
// fused epilogue applied to one 32-column chunk of an accumulator row.
#pragma once
#include "b200_ptx.cuh"
#include "ops_api.h"

namespace b200 {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kEpilogueWarps = 8;   // two warps per TMEM lane quarter, interleaved over 32-column chunks

struct GemmArgs {
  int M, N, K;
  int a_mn_major, b_mn_major;
  int split_k;             // >= 1; > 1 requires out_fp32, and atomic accumulation or part_rows
  int stream_k;            // CTA-pair kernel, fp32 accumulating output: equal runs of (tile, k-block) pairs per cluster
  float alpha;
  const __nv_bfloat16* bias;      // [N] or null
  const __nv_bfloat16* residual;  // [M, ld_res] or null, added last
  int ld_res;
  const __nv_bfloat16* aux;       // [M, ld_aux] activation-backward operand or null
  int ld_aux;
  void* out;
  int ld_out;
  int out_fp32;
  int accumulate;          // fp32 output only: out += result
  __nv_bfloat16* preact;   // optional [M, ld_out]: value after bias, before activation
  uint32_t* mask;          // optional [M, ld_mask] sign bits of the output (written, or read by kActMaskBwd)
  int ld_mask;
  float* colsum;           // optional fp32 [N]: += column sums of the stored bf16 output (from the staging tiles, or from registers: sum_here)
  int act;
  float dropout_p;
  unsigned long long seed, stream_id;
  const unsigned long long* seed_dev;
  int* status;
  int by_element;          // an epilogue operand is not on a 16-byte boundary: nothing of it moves as vectors
  int tma_store;           // bf16 output leaves through shared memory and TMA stores (CTA-pair kernel)
  int tma_second;          // so does the pre-activation, and the aux operand comes in that way (see two_stagings)
  int ablate;              // profiling aid: 1 = read the accumulator but skip arithmetic and stores, 2 = skip the epilogue body,
                           // 3 (traced kernel only) = also skip the MMAs: operand streaming alone
  int part_rows;           // > 0: part s of the sum over K is stored at row s * part_rows of the output, by itself (kernels with kEpiParts)
  long long* trace;        // profiling aid: when set, the CTA-pair kernel writes up to 16 cycle counters per cluster (see gemm2cta_tcgen05.cu)
};

// In-kernel gather of the B operand (fully sharded parameters), CTA-pair kernel.  The matrix is `units` blocks of
// 4 KB, claimed four at a time through the cursor counters[1]; block u belongs to segment u / seg_units, and the TMA
// producer loads tiles of a segment only after counters[2 + segment] has reached the segment's block count.
// n_seg == 0: no gather.
constexpr int kGatherBlockBytes = 4096;
constexpr int kGatherMaxSegs = 128;
struct GatherArgs {
  int n_seg;
  int rank, world;
  const unsigned short* shards[16];
  long shard_off, piece_len, unit_off;
  unsigned short* dst;      // local staging address of the matrix
  long units;               // 4 KB blocks in the matrix
  int seg_units;            // blocks per segment (the last segment may have fewer)
  int* counters;            // [0]: CTAs that have left the kernel, [1]: next unclaimed block, [2 + s]: finished blocks of segment s
};

// Distribution function of the normal distribution, and exp(-x^2 / 2) beside it, without a branch: in the middle (|x| < 1.25) 1/2 + x P(x^2),
// outside exp(-x^2 / 2) t Q(t) with t = 1 / (1 + 0.35 |x|) for the lower tail and one minus it above.  P and Q are minimax fits to the error
// function (iteratively reweighted least squares in 64 bits against erf and the scaled erfc; 2e-9 absolute and, down to the smallest
// normal float, 1.5e-8 relative).  Measured over 4 million points against 64 bits, largest and root mean square error, (1 + erff(x / sqrt 2)) / 2 in
// brackets:  |x| < 0.5 4.0e-8, 1.4e-8 (5.1e-8, 1.5e-8);  to 1.25 5.3e-8, 1.5e-8 (6.3e-8, 1.8e-8);  1.25 to 3 6.1e-8, 1.8e-8 (6.3e-8, 2.4e-8);
// relative in the lower tail 6e-7 at -3 (3e-5) and 2e-6 at -6 (all of it); the square in the exponent sets that.
// The two ranges of erff, a branch, cost an epilogue of 32 unrolled elements 16 us of 44 (6144 x 2048 x 512 with the GELU gradient).
__device__ __forceinline__ float normal_cdf(float x, float& bell) {
  const float z = x * x, a = fabsf(x);
  bell = exp2f(-0.72134752f * z);
  const float t = __fdividef(1.f, fmaf(0.35f, a, 1.f));
  float q = fmaf(t, 0.0444524474f, -0.111576788f);
  q = fmaf(t, q, 0.0438466556f);
  q = fmaf(t, q, 0.0324914902f);
  q = fmaf(t, q, 0.0890091509f);
  q = fmaf(t, q, 0.122769959f);
  q = fmaf(t, q, 0.139575362f);
  q = fmaf(t, q, 0.139633134f);
  const float tail = q * t * bell;
  float p = fmaf(z, -6.6448597e-06f, 0.000110327455f);
  p = fmaf(z, p, -0.00118270959f);
  p = fmaf(z, p, 0.00997150037f);
  p = fmaf(z, p, -0.0664899871f);
  p = fmaf(z, p, 0.398942262f);
  return a < 1.25f ? fmaf(x, p, 0.5f) : x < 0.f ? tail : 1.f - tail;
}
__device__ __forceinline__ float gelu_f(float x) {
  float bell;
  return x * normal_cdf(x, bell);
}
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + __expf(-x)); }

// Two elements at a time: the 32-bit pairs of sm_100 (one instruction, both halves rounded as the single one rounds).
struct Pair {
  uint64_t v;
  __device__ __forceinline__ Pair() {}
  __device__ __forceinline__ Pair(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
  __device__ __forceinline__ explicit Pair(float both) : Pair(both, both) {}
  __device__ __forceinline__ float2 split() const {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
  }
};
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
// normal_cdf of two values, the same operations
__device__ __forceinline__ Pair normal_cdf2(Pair x, Pair& bell) {
  const float2 f = x.split();
  const float a0 = fabsf(f.x), a1 = fabsf(f.y);
  const Pair z = mul2(x, x);
  const float2 e = mul2(z, Pair(-0.72134752f)).split();
  bell = Pair(exp2f(e.x), exp2f(e.y));
  const float2 d = fma2(Pair(0.35f), Pair(a0, a1), Pair(1.f)).split();
  const Pair t(__fdividef(1.f, d.x), __fdividef(1.f, d.y));
  Pair q = fma2(t, Pair(0.0444524474f), Pair(-0.111576788f));
  q = fma2(t, q, Pair(0.0438466556f));
  q = fma2(t, q, Pair(0.0324914902f));
  q = fma2(t, q, Pair(0.0890091509f));
  q = fma2(t, q, Pair(0.122769959f));
  q = fma2(t, q, Pair(0.139575362f));
  q = fma2(t, q, Pair(0.139633134f));
  const float2 tail = mul2(mul2(q, t), bell).split();
  Pair p = fma2(z, Pair(-6.6448597e-06f), Pair(0.000110327455f));
  p = fma2(z, p, Pair(-0.00118270959f));
  p = fma2(z, p, Pair(0.00997150037f));
  p = fma2(z, p, Pair(-0.0664899871f));
  p = fma2(z, p, Pair(0.398942262f));
  const float2 mid = fma2(x, p, Pair(0.5f)).split();
  return Pair(a0 < 1.25f ? mid.x : f.x < 0.f ? tail.x : 1.f - tail.x, a1 < 1.25f ? mid.y : f.y < 0.f ? tail.y : 1.f - tail.y);
}

// One thread = one accumulator row; processes columns [col0, col0 + 32) read from TMEM address `taddr`:
// alpha, bias, optional pre-activation store, activation or activation gradient, dropout, residual, store
// (bf16, fp32, fp32 accumulate, or fp32 red.add for split-K).  Warp-collective (contains a tcgen05.ld).
// `pre_row`: the same for the pre-activation; `aux_staged`: the aux operand has been copied into the staging row.
// `stage_row` (optional): instead of writing bf16 results to global memory, place the 64-byte row fragment in a
// shared-memory staging row laid out for a 128-byte-swizzled TMA store (logical 16-byte chunk j of row r sits at
// chunk j ^ (r & 7)); `stage_half` selects the left / right 32 columns of the 64-column staging tile.
// Feature bits of the epilogue.  A kernel instantiated with a mask contains only the code of those features (the
// run-time checks inside still apply), which keeps the epilogue a short straight-line sequence: with everything
// compiled in, each 32-column chunk jumps over a dozen large unused blocks and the warps wait on instruction fetch
// rather than on arithmetic.  kEpiAll is the general kernel.
constexpr uint32_t kEpiBias = 1u, kEpiPreact = 2u, kEpiActFwd = 4u, kEpiActBwd = 8u, kEpiMaskBwd = 16u, kEpiDrop = 32u,
                   kEpiMaskOut = 64u, kEpiRes = 128u, kEpiF32 = 256u, kEpiBf16 = 512u,
                   kEpiRagged = 1024u /* N not a multiple of 64, or unaligned operands: column chunks element by element */,
                   kEpiColsum = 2048u /* column sums of the output */, kEpiAll = 4095u,
                   kEpiParts = 4096u /* GemmArgs::part_rows; in kernels of its own */;

// Features a problem needs (host side).
inline uint32_t gemm_epilogue_features(const GemmArgs& a) {
  uint32_t f = 0;
  if (a.bias) f |= kEpiBias;
  if (a.preact) f |= kEpiPreact;
  if (a.act == kActMaskBwd) f |= kEpiMaskBwd;
  else if (a.act >= kActReluBwd) f |= kEpiActBwd;
  else if (a.act != 0) f |= kEpiActFwd;
  if (a.dropout_p > 0.f) f |= kEpiDrop;
  if (a.mask && a.act != kActMaskBwd) f |= kEpiMaskOut;
  if (a.residual) f |= kEpiRes;
  f |= a.out_fp32 ? kEpiF32 : kEpiBf16;
  if (a.N % 64 || a.by_element) f |= kEpiRagged;
  if (a.colsum) f |= kEpiColsum;
  return f;
}

template <uint32_t kFeat = kEpiAll>
__device__ __forceinline__ void gemm_epilogue_chunk(const GemmArgs& p, const DropRng& rng, const bool do_drop, const int row,
                                                    const bool row_ok, const int col0, const uint32_t taddr,
                                                    uint8_t* stage_row = nullptr, const int stage_half = 0,
                                                    const int stage_r = 0, uint8_t* pre_row = nullptr,
                                                    const bool aux_staged = false) {
    const bool full_cols = !(kFeat & kEpiRagged) || (!p.by_element && col0 + 32 <= p.N);
    // global operands of the epilogue are requested BEFORE the TMEM load so their latency overlaps it
    uint4 aux_v[4], res_v[4];
    const bool aux_vec = (kFeat & kEpiActBwd) && !aux_staged && row_ok && full_cols && p.act >= kActReluBwd && p.act != kActMaskBwd && (p.ld_aux & 7) == 0;
    uint32_t mask_word = 0;
    if ((kFeat & kEpiMaskBwd) && p.act == kActMaskBwd && row_ok) mask_word = p.mask[static_cast<size_t>(row) * p.ld_mask + (col0 >> 5)];
    const bool res_vec = (kFeat & kEpiRes) && row_ok && full_cols && p.residual != nullptr && (p.ld_res & 7) == 0;
    if (aux_vec) {
      const uint4* ap4 = reinterpret_cast<const uint4*>(p.aux + static_cast<size_t>(row) * p.ld_aux + col0);
#pragma unroll
      for (int g = 0; g < 4; ++g) aux_v[g] = ap4[g];
    }
    if (res_vec) {
      const uint4* rp4 = reinterpret_cast<const uint4*>(p.residual + static_cast<size_t>(row) * p.ld_res + col0);
#pragma unroll
      for (int g = 0; g < 4; ++g) res_v[g] = rp4[g];
    }
    uint32_t r[32];
    tmem_ld32(taddr, r);
    tmem_ld_wait();
    const bool live = row_ok && p.ablate != 1;
    // Column sums straight from registers (single-CTA kernel) need every lane of the warp, so that the lanes of rows past M go on to them.
    // They must meet no operand or output of their row on the way: the host sends column sums here with the mask epilogue at most.
    const bool sum_here = (kFeat & kEpiColsum) && p.colsum != nullptr && stage_row == nullptr;
    if (!live && !sum_here) return;
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
    if ((kFeat & kEpiBias) && p.bias) {
      if (full_cols) {
        const uint4* bp = reinterpret_cast<const uint4*>(p.bias + col0);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 b = __ldg(bp + g);
          const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = __bfloat1622float2(b2[j]);
            v[g * 8 + 2 * j] += f.x;
            v[g * 8 + 2 * j + 1] += f.y;
          }
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
      }
    }
    if ((kFeat & kEpiPreact) && p.preact) {
      __nv_bfloat16* pp = p.preact + static_cast<size_t>(row) * p.ld_out + col0;
      if (pre_row != nullptr) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 o;
          __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[g * 8 + 2 * j], v[g * 8 + 2 * j + 1]);
          *reinterpret_cast<uint4*>(pre_row + (((stage_half * 4 + g) ^ (stage_r & 7)) << 4)) = o;
        }
      } else if (full_cols) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 o;
          __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[g * 8 + 2 * j], v[g * 8 + 2 * j + 1]);
          reinterpret_cast<uint4*>(pp)[g] = o;
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) pp[j] = __float2bfloat16(v[j]);
      }
    }
    // activation (forward) or activation-gradient (backward; aux holds h or z)
    if ((kFeat & kEpiMaskBwd) && p.act == kActMaskBwd) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = ((mask_word >> j) & 1u) ? v[j] : 0.f;
    } else if ((kFeat & kEpiActBwd) && p.act >= kActReluBwd) {
      const __nv_bfloat16* ap = p.aux + static_cast<size_t>(row) * p.ld_aux + col0;
      float av[32];
      if (aux_staged) {       // the operand's row fragment lies where the result will be put
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) aux_v[g4] = *reinterpret_cast<const uint4*>(stage_row + (((stage_half * 4 + g4) ^ (stage_r & 7)) << 4));
      }
      if (aux_vec || aux_staged) {
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) {
          uint4 u = aux_v[g4];
          const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = __bfloat1622float2(u2[j]);
            av[g4 * 8 + 2 * j] = f.x;
            av[g4 * 8 + 2 * j + 1] = f.y;
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) av[j] = (col0 + j < p.N) ? __bfloat162float(ap[j]) : 0.f;
      }
      // one loop per activation: decided per element, the 32 copies of every branch overran the instruction cache (6144 x 2048 x 512
      // with the ReLU gradient 45.8 us, 23.3 so)
      if (p.act == kActReluBwd) {          // aux = relu output (after dropout)
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= av[j] > 0.f ? 1.f : 0.f;
      } else if (p.act == kActGeluBwd) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const Pair x(av[j], av[j + 1]);
          Pair bell;
          const Pair cdf = normal_cdf2(x, bell);
          const float2 d = fma2(x, mul2(Pair(0.3989422804014327f), bell), cdf).split();
          v[j] *= d.x;
          v[j + 1] *= d.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float s = sigmoid_f(av[j]);
          v[j] *= s * (1.f + av[j] * (1.f - s));
        }
      }
    } else if ((kFeat & kEpiActFwd) && p.act == kActRelu) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
    } else if ((kFeat & kEpiActFwd) && p.act == kActGelu) {
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const Pair x(v[j], v[j + 1]);
        Pair bell;
        const float2 f = mul2(x, normal_cdf2(x, bell)).split();
        v[j] = f.x;
        v[j + 1] = f.y;
      }
    } else if ((kFeat & kEpiActFwd) && p.act == kActSilu) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = v[j] * sigmoid_f(v[j]);
    }
    if ((kFeat & kEpiDrop) && do_drop) {
      // element index = row * N + col; 4 consecutive elements share one hash word (one byte each)
      const unsigned long long w0 = (static_cast<unsigned long long>(row) * p.N + col0) >> 2;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const uint32_t w = rng.word(w0 + g);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[g * 4 + j] = rng.keep(w, j) ? v[g * 4 + j] * rng.scale : 0.f;
      }
    }
    if ((kFeat & kEpiMaskOut) && p.mask && p.act != kActMaskBwd) {
      uint32_t bits = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) bits |= (v[j] > 0.f ? 1u : 0u) << j;
      p.mask[static_cast<size_t>(row) * p.ld_mask + (col0 >> 5)] = bits;
    }
    if ((kFeat & kEpiRes) && p.residual) {
      const __nv_bfloat16* rp = p.residual + static_cast<size_t>(row) * p.ld_res + col0;
      if (res_vec) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 b = res_v[g];
          const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = __bfloat1622float2(b2[j]);
            v[g * 8 + 2 * j] += f.x;
            v[g * 8 + 2 * j + 1] += f.y;
          }
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) v[j] += __bfloat162float(rp[j]);
      }
    }
    if ((kFeat & kEpiF32) && (p.out_fp32 || !(kFeat & kEpiBf16))) {
      float* op = reinterpret_cast<float*>(p.out) + static_cast<size_t>(row) * p.ld_out + col0;
      // accumulation into an existing fp32 buffer goes through the L2 reduction unit as well: no read round trip
      if ((p.split_k > 1 && !(kFeat & kEpiParts)) || p.accumulate || p.stream_k) {
        if (full_cols) {
#pragma unroll
          for (int g = 0; g < 8; ++g)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(op + g * 4), "f"(v[g * 4]),
                         "f"(v[g * 4 + 1]), "f"(v[g * 4 + 2]), "f"(v[g * 4 + 3])
                         : "memory");
        } else {
          for (int j = 0; j < 32; ++j)
            if (col0 + j < p.N) atomicAdd(op + j, v[j]);
        }
      } else if (full_cols) {
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float4 o = make_float4(v[g * 4], v[g * 4 + 1], v[g * 4 + 2], v[g * 4 + 3]);
          if (p.accumulate) {
            float4 old = reinterpret_cast<float4*>(op)[g];
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
          }
          reinterpret_cast<float4*>(op)[g] = o;
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) op[j] = p.accumulate ? op[j] + v[j] : v[j];
      }
    } else if (!(kFeat & kEpiBf16)) {
      // fp32-only kernel asked for bf16 output: the host never selects this combination
    } else if (stage_row != nullptr) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint4 o;
        __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[g * 8 + 2 * j], v[g * 8 + 2 * j + 1]);
        *reinterpret_cast<uint4*>(stage_row + (((stage_half * 4 + g) ^ (stage_r & 7)) << 4)) = o;
      }
    } else {
      if (sum_here) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = live ? __bfloat162float(__float2bfloat16(v[j])) : 0.f;
        float t[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) t[j] = v[j];
        // 32 rows x 32 columns: the lanes halve their lists while they add, lane l ends with column l
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const bool hi = (threadIdx.x & o) != 0;
#pragma unroll
          for (int j = 0; j < o; ++j) {
            const float keep = hi ? t[j + o] : t[j], give = hi ? t[j] : t[j + o];
            t[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        }
        const int c = col0 + static_cast<int>(threadIdx.x & 31);
        if (c < p.N) atomicAdd(p.colsum + c, t[0]);
        if (!live) return;
      }
      __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(row) * p.ld_out + col0;
      if (full_cols) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 o;
          __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(v[g * 8 + 2 * j], v[g * 8 + 2 * j + 1]);
          reinterpret_cast<uint4*>(op)[g] = o;
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) op[j] = __float2bfloat16(v[j]);
      }
    }
}

}  // namespace b200
