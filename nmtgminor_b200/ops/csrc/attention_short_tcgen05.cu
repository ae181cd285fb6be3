// Persistent, warp-specialised, software-pipelined attention for sequences that fit ONE 128-row tile
// (query and key length <= 128: every sentence-level translation batch).  A work item is one
// (sequence, head) pair; each CTA (one per SM) walks a strided list of items and overlaps, across items,
//   TMA loads of Q / K / V (/ dO)        - producer warp, multi-slot shared-memory ring
//   tcgen05 MMAs into TMEM               - MMA warp, issues S(i+1) before the second-stage MMAs of item i
//   softmax / dS math and the epilogues  - 128-thread groups, thread t = tile row t = TMEM lane t
// so that per-item latencies (global loads, MMA completion, TMEM reads) are hidden instead of summed, which
// is what dominates when a sentence has only 20..100 tokens.
//
// forward : four items in flight, each with a Q/K/V slot, 128 TMEM columns (S, then O) and a softmax group of its own.
// backward: 256 math threads (query row x half of the key columns) on one item, a warpgroup that prepares D / log-sum-exp
//           of the next item and writes dQ, dK, dV of the previous one; TMEM holds two sets (S dP, reused for dV dQ dK),
//           two Q/K/V/dO slots; P and dS are staged once in shared memory and consumed K-major (dQ = dS K) and MN-major
//           (dV = P^T dO, dK = dS^T Q).
// MMA reduction lengths are trimmed to the real sequence lengths (multiples of 16).
// The fetching of instructions bound these kernels when each had 157 KB of code: all roles run at once, each in code of its own, and the SMs
// of a GPC share what their own caches cannot hold (CTAs on a GPC with fewer of them ran 1.4 times as fast).  So a loop body is there once: one
// 32-column chunk a turn, dropout a template argument, MMA steps and gradient matrices in loops that are not unrolled (unrolling the
// backward pass's MMA steps alone cost 12 us).  With 39 and 70 KB a scheduler waits 0.5 cycles an instruction for the next one and 5 to 9 for
// tensor memory, barriers and loads: the chain of an item.  135 sentences of 20 to 100 words x 16 heads, us back to back, 157 KB / now:
// forward 38.8 / 22.6, with dropout 49.9 / 29.7, backward 74.4 / 61.0, with dropout 83.8 / 66.7.
// Same numerics, dropout counters and interfaces as the general kernels in attention_tcgen05.cu.
#include "attention_common.cuh"
#include "bounds_check.cuh"
#include "launch.cuh"

namespace b200 {

int num_sms();

struct Item {
  int q0 = 0, q_len = 0, k0 = 0, k_len = 0, h = 0;
  bool valid = false;
};

// `report`: this thread's look-ups are the ones that the debug build counts bad offsets in (one thread of a CTA that looks at every item)
__device__ __forceinline__ Item get_item(const AttnArgs& p, int item, bool report = false) {
  Item it;
  const int b = item / p.num_heads;
  it.h = item - b * p.num_heads;
  it.q0 = p.cu_q[b];
  it.q_len = p.cu_q[b + 1] - it.q0;
  it.k0 = p.cu_k[b];
  it.k_len = p.cu_k[b + 1] - it.k0;
  it.valid = it.q_len > 0 && it.k_len > 0 && it.q_len <= kTile && it.k_len <= kTile;
  // a sequence that does not fit one tile (or offsets that run backwards) is skipped by every role of the kernel; the host
  // dispatch sends such batches to the general kernels, so meeting one here means the offsets are wrong
  if (!it.valid && (it.q_len < 0 || it.k_len < 0 || it.q_len > kTile || it.k_len > kTile) && report) NMTG_BOUNDS_HIT();
  return it;
}

// ---------------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------------
// Four items are in flight, each in a slot and with a softmax group of its own: an item is a chain of waits (S, two passes over it, P,
// O, about 5500 cycles for 60 keys with dropout) that one or two warps of a scheduler cannot fill.  To fit, P overwrites the Q and K
// tiles (S = Q K^T is complete when a group starts) and O the columns of S.  Only the producer looks items up: the look-up is a
// round trip to memory, and in the MMA warp it took 1300 of the 3260 cycles that an item took with two groups.  Two groups took
// 38.8 us where four take 22.6, with dropout 49.9 and 29.7 (figures above).
constexpr int kFwdSlotBytes = 3 * kTileBytes;
constexpr int fwd_short_threads(int groups) { return groups * 128 + 64; }   // softmax groups, TMA producer warp, MMA warp
constexpr int fwd_short_smem(int groups) { return groups * kFwdSlotBytes + 512 + 1024 > kOwnSm ? groups * kFwdSlotBytes + 512 + 1024 : kOwnSm; }

// Up to 64 queries leave two of a group's four warps without work, and a warp's number decides both its rows (TMEM lanes) and its
// scheduler: odd groups take such items in rows 64 .. 127 (the tile starts 64 rows early; a load may start before the matrix).
__device__ __forceinline__ int row_shift(int group, int q_len) { return (group & 1) && q_len <= 64 ? 64 : 0; }

template <int kFwdGroups, bool kDrop>
__global__ void __launch_bounds__(fwd_short_threads(kFwdGroups), 1)
attn_fwd_short_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const AttnArgs p, const int num_items) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sSlots = smem;            // [4][Q K V]; P over Q and K
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kFwdGroups * kFwdSlotBytes);
  uint64_t* slot_full = bars;                       // TMA (and the item's descriptor) -> everybody
  uint64_t* slot_empty = bars + kFwdGroups;         // P V done -> TMA
  uint64_t* s_full = bars + 2 * kFwdGroups;         // S ready -> softmax group
  uint64_t* p_full = bars + 3 * kFwdGroups;         // P staged -> MMA
  uint64_t* o_full = bars + 4 * kFwdGroups;         // O ready -> softmax group
  uint64_t* o_read = bars + 5 * kFwdGroups;         // O read -> MMA may write the next S
  int4* desc = reinterpret_cast<int4*>(bars + 6 * kFwdGroups);      // q0, k0, head, (q_len << 8) | k_len; 0 lengths: no more items
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(desc + kFwdGroups);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kFwdGroups; ++i) {
      mbar_init(&slot_full[i], 1);
      mbar_init(&slot_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_read[i], 128);
    }
    *abort_word = 0;
    mbar_fence_init();
  }
  constexpr int kProducer = kFwdGroups * 4, kMma = kProducer + 1;
  wait_for_previous();
  zero_tail_fwd(p);
  if (warp == kMma) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  let_next_start();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kProducer) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      Item nxt = static_cast<int>(blockIdx.x) < num_items ? get_item(p, blockIdx.x, true) : Item{};
      for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        const Item w = nxt;
        if (item + static_cast<int>(gridDim.x) < num_items) nxt = get_item(p, item + gridDim.x, true);
        if (!w.valid) continue;
        const int slot = it % kFwdGroups;
        if (!mbar_wait(&slot_empty[slot], ((it / kFwdGroups) & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty)) { ok = false; break; }
        desc[slot] = make_int4(w.q0, w.k0, w.h, (w.q_len << 8) | w.k_len);
        uint8_t* s = sSlots + slot * kFwdSlotBytes;
        mbar_expect_tx(&slot_full[slot], kFwdSlotBytes);
        tma_load_2d(s, &tmap_q, &slot_full[slot], w.h * kHd, w.q0 - row_shift(slot, w.q_len));
        tma_load_2d(s + kTileBytes, &tmap_k, &slot_full[slot], w.h * kHd, w.k0);
        tma_load_2d(s + 2 * kTileBytes, &tmap_v, &slot_full[slot], w.h * kHd, w.k0);
        ++it;
      }
      for (int e = 0; e < kFwdGroups && ok; ++e, ++it) {
        const int slot = it % kFwdGroups;
        if (!mbar_wait(&slot_empty[slot], ((it / kFwdGroups) & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty)) break;
        desc[slot] = make_int4(0, 0, 0, 0);
        mbar_arrive(&slot_full[slot]);
      }
    }
  } else if (warp == kMma) {
    const uint32_t idesc_s = make_idesc_bf16(kTile, kTile, 0, 0);
    const uint32_t idesc_o = make_idesc_bf16(kTile, kHd, 0, 1);
    const uint32_t tmem = uniform(tmem_base), slots = uniform(smem_u32(sSlots));
    // two queues, served in whichever order their inputs arrive: S of item s_it, P V of item o_it
    int s_it = 0, o_it = 0;
    uint32_t steps = 0;                       // 16-key steps of the items in flight, 4 bits each
    bool more = true;
    uint32_t idle = 0;
    while (more || o_it < s_it) {
      bool progressed = false;
      if (o_it < s_it && all_lanes(mbar_test_wait(&p_full[o_it % kFwdGroups], (o_it / kFwdGroups) & 1))) {
        tc_fence_after_sync();
        const int g = o_it % kFwdGroups;
        const uint32_t pa = slots + g * kFwdSlotBytes, tO = tmem + g * kTile;
        const uint64_t ad = make_smem_desc_sw128(pa, 16, 1024), bd = make_smem_desc_sw128(pa + 2 * kTileBytes, 8192, 1024);
        const int nk = static_cast<int>((steps >> (4 * g)) & 15u);
        umma_slabs_warp(tO, ad, bd, idesc_o, nk);
        if (elect_one()) {
          umma_commit(&o_full[g]);
          umma_commit(&slot_empty[g]);
        }
        ++o_it;
        progressed = true;
      }
      if (more && s_it - o_it < kFwdGroups && all_lanes(mbar_test_wait(&slot_full[s_it % kFwdGroups], (s_it / kFwdGroups) & 1) &&
                                                        mbar_test_wait(&o_read[s_it % kFwdGroups], ((s_it / kFwdGroups) & 1) ^ 1))) {
        tc_fence_after_sync();
        const int g = s_it % kFwdGroups;
        const int lens = uniform(desc[g].w);
        if (lens == 0) more = false;
        else {
          const uint32_t qa = slots + g * kFwdSlotBytes;
          umma_steps_warp<32, 32>(tmem + g * kTile, make_smem_desc_sw128(qa, 16, 1024), make_smem_desc_sw128(qa + kTileBytes, 16, 1024), idesc_s, kHd / 16);
          if (elect_one()) umma_commit(&s_full[g]);
          steps = (steps & ~(15u << (4 * g))) | (static_cast<uint32_t>(((lens & 255) + 15) >> 4) << (4 * g));
          ++s_it;
        }
        progressed = true;
      }
      if (progressed) idle = 0;
      else if (!all_lanes(keep_polling(idle, abort_word, p.status))) break;
    }
  } else {
    const int g = warp >> 2;
    const int t = (warp & 3) * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem_base + g * kTile + lane_sel;      // S, then O in its first 64 columns
    uint8_t* myP = sSlots + g * kFwdSlotBytes;
    const float scale_log2 = p.scale * 1.4426950408889634f;
    const unsigned long long seed = p.seed + ((kDrop && p.seed_dev) ? *p.seed_dev : 0ull);
    for (uint32_t ph = 0;; ph ^= 1) {
      if (!mbar_wait(&slot_full[g], ph, abort_word, p.status, kTimeoutTmaFull)) break;
      const int4 d = desc[g];
      const int q_len = d.w >> 8, k_len = d.w & 255;
      if (d.w == 0) break;
      if (!mbar_wait(&s_full[g], ph, abort_word, p.status, kTimeoutTmemFull)) break;
      tc_fence_after_sync();
      const int tq = t - row_shift(g, q_len);               // this thread's query
      const int first = (warp & 3) * 32 - row_shift(g, q_len);
      const bool warp_active = first >= 0 && first < q_len;
      const int nchunks = (k_len + 31) >> 5;
      float row_sum = 0.f, row_max = kNegBig;
      if (warp_active) {
        const DropRng rng(seed, (p.stream_id << 16) | static_cast<unsigned long long>(d.z), p.dropout_p);
        // raw-score maximum (scale > 0: scaling commutes with the maximum)
        const int limit = p.causal ? min(k_len, tq + 1) : k_len;
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
          uint32_t r[32];
          tmem_ld32(tS + c * 32, r);
          tmem_ld_wait();
          const int left = limit - c * 32;
#pragma unroll
          for (int j = 0; j < 32; ++j) row_max = fmaxf(row_max, j < left ? __uint_as_float(r[j]) : kNegBig);
        }
        row_max *= scale_log2;         // from here on in the base-2 domain: P = 2^(S * scale * log2 e - row_max)
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
          uint32_t r[32];
          tmem_ld32(tS + c * 32, r);
          tmem_ld_wait();
          float pv[32];
          const int left = limit - c * 32;
          if (!p.causal && left >= 32) {            // no per-element test
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              pv[j] = ex2_approx(fmaf(__uint_as_float(r[j]), scale_log2, -row_max));
              pv[j + 1] = ex2_approx(fmaf(__uint_as_float(r[j + 1]), scale_log2, -row_max));
              pv[j + 2] = ex2_approx(fmaf(__uint_as_float(r[j + 2]), scale_log2, -row_max));
              pv[j + 3] = ex2_approx(fmaf(__uint_as_float(r[j + 3]), scale_log2, -row_max));
              s0 += pv[j];
              s1 += pv[j + 1];
              s2 += pv[j + 2];
              s3 += pv[j + 3];
            }
            row_sum += (s0 + s1) + (s2 + s3);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float e = j < left ? ex2_approx(fmaf(__uint_as_float(r[j]), scale_log2, -row_max)) : 0.f;
              row_sum += e;
              pv[j] = e;
            }
          }
          if constexpr (kDrop) apply_dropout32(rng, static_cast<unsigned long long>(d.x + tq) * p.kstride + c * 32, pv);
#pragma unroll
          for (int g4 = 0; g4 < 4; ++g4) {
            uint4 o;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(pv[g4 * 8 + 2 * j], pv[g4 * 8 + 2 * j + 1]);
            const int chunk = c * 4 + g4;
            *reinterpret_cast<uint4*>(myP + (chunk >> 3) * kTileBytes + sw128_offset(t, chunk & 7)) = o;
          }
        }
      }
      tc_fence_before_sync();
      fence_async_smem();
      mbar_arrive(&p_full[g]);
      if (!mbar_wait(&o_full[g], ph, abort_word, p.status, kTimeoutTmemFull)) break;
      tc_fence_after_sync();
      if (warp_active) {
        const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
        __nv_bfloat16* orow = p.out + static_cast<size_t>(d.x + tq) * p.ld_out + d.z * kHd;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tmem_ld32(tS + half * 32, r);
          tmem_ld_wait();
          if (tq < q_len) {
#pragma unroll
            for (int g4 = 0; g4 < 4; ++g4) {
              uint4 o;
              __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
              for (int j = 0; j < 4; ++j)
                o2[j] = __floats2bfloat162_rn(__uint_as_float(r[g4 * 8 + 2 * j]) * inv, __uint_as_float(r[g4 * 8 + 2 * j + 1]) * inv);
              reinterpret_cast<uint4*>(orow)[half * 4 + g4] = o;
            }
          }
        }
        if (p.lse && tq < q_len)
          p.lse[static_cast<size_t>(d.z) * p.lse_stride + d.x + tq] = row_sum > 0.f ? (row_max + __log2f(row_sum)) * 0.6931471805599453f : 0.f;
      }
      tc_fence_before_sync();
      mbar_arrive(&o_read[g]);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_word) {
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kMma) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------------
// Roles (448 threads):
//   warps 0-3 / 4-7   math: thread = (query row, half); half h owns key columns [32 c + 16 h, 32 c + 16 h + 16) of every
//                     32-column chunk c, so all 256 threads work on the SAME item and each holds few values at a time
//                     (the math is issue-bound: with one warp per scheduler and most registers tied up in TMEM chunks the
//                     compiler could not interleave independent elements, which is what made the one-group version slow)
//   warps 8-11        D = rowsum(dO * O) (dO from its tile, O from one loaded for this) and the log-sum-exp of item i+1 into shared memory,
//                     then dQ / dK / dV of item i-1
//   warp 12           TMA producer          warp 13   MMA issuer
// TMEM holds two sets of 256 columns, set = item & 1:
//   columns   0..127  S  = Q K^T          later  dV (0..63) and dQ (64..127)
//   columns 128..255  dP = dO V^T         later  dK (128..191)
// so the S / dP MMAs of item i+1 run while the gradients of item i-1 are still being read out of the other set.
// P and dS are staged in ONE pair of shared-memory tiles; the math threads wait for the gradient MMAs of the previous
// item (pds_free) only right before their first store, after the exponentials of the new item are done.
constexpr int kBwdSlots = 2;
constexpr int kBwdSlotBytes = 4 * kTileBytes;   // Q, K, V, dO
constexpr int kBwdShortThreads = 448;
constexpr int kBwdRowBytes = 2 * 2 * kTile * 4; // D and log-sum-exp of two items in flight
constexpr int kBwdShortSmem = kBwdSlots * kBwdSlotBytes + 2 * kPBytes + kTileBytes + kBwdRowBytes + 256 + 1024;

// One gradient row per thread (64 fp32 accumulator columns of its TMEM lane) scaled, packed to bf16 and stored.
__device__ __forceinline__ void bwd_store_rows(uint32_t taddr, __nv_bfloat16* base, int ld, int rows, float osc, int lane) {
  uint32_t r0[32], r1[32];
  tmem_ld32(taddr, r0);
  tmem_ld32(taddr + 32, r1);
  tmem_ld_wait();
  if (lane < rows) {
    __nv_bfloat16* drow = base + static_cast<size_t>(lane) * ld;
#pragma unroll
    for (int g4 = 0; g4 < 8; ++g4) {
      uint4 o;
      __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = (g4 & 3) * 8 + 2 * j;
        o2[j] = __floats2bfloat162_rn(__uint_as_float(g4 < 4 ? r0[e] : r1[e]) * osc, __uint_as_float(g4 < 4 ? r0[e + 1] : r1[e + 1]) * osc);
      }
      reinterpret_cast<uint4*>(drow)[g4] = o;
    }
  }
}

template <bool kDrop>
__global__ void __launch_bounds__(kBwdShortThreads, 1)
attn_bwd_short_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                      const __grid_constant__ CUtensorMap tmap_o, const AttnArgs p, const int num_items, const int ablate) {
  // `ablate` (0 in production) switches parts of the work off while keeping every barrier hand-shake, so that a timing run
  // can tell which role bounds the item rate (results are then meaningless):
  //   1 no P / dS math   2 no gradient read-out   4 no gradient MMAs   8 no S / dP MMAs   16 no TMA loads
  //   32 no D / log-sum-exp loads   64 no dropout masks
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sSlots = smem;
  uint8_t* sP = smem + kBwdSlots * kBwdSlotBytes;
  uint8_t* sDS = sP + kPBytes;
  uint8_t* sO = sDS + kPBytes;                           // O of the item whose D comes next
  float* sD = reinterpret_cast<float*>(sO + kTileBytes);   // [2][128] rowsum(dO * O) of the items in flight
  float* sL = sD + 2 * kTile;                            // [2][128] log-sum-exp * log2 e (+inf for rows past the sequence)
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + kTileBytes + kBwdRowBytes);
  uint64_t* slot_full = bars;        // [2] TMA -> MMA
  uint64_t* slot_empty = bars + 2;   // [2] gradient MMAs done -> TMA
  uint64_t* sdp_full = bars + 4;     // [2] S / dP ready -> math group
  uint64_t* set_free = bars + 6;     // [2] gradients read out -> MMA may overwrite the set
  uint64_t* grads_full = bars + 8;   // [2] gradient MMAs done -> epilogue group
  uint64_t* pds_full = bars + 10;    // P / dS staged -> MMA
  uint64_t* pds_free = bars + 11;    // gradient MMAs done -> math threads may overwrite P / dS
  uint64_t* d_full = bars + 12;      // [2] D / log-sum-exp rows written -> math threads
  uint64_t* d_free = bars + 14;      // [2] rows read -> may be overwritten
  uint64_t* o_full = bars + 16;      // O loaded -> D
  uint64_t* o_free = bars + 17;      // O read -> TMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&slot_full[i], 1);
      mbar_init(&slot_empty[i], 1);
      mbar_init(&sdp_full[i], 1);
      mbar_init(&set_free[i], 128);
      mbar_init(&grads_full[i], 1);
      mbar_init(&d_full[i], 128);
      mbar_init(&d_free[i], 256);
    }
    mbar_init(pds_full, 256);
    mbar_init(pds_free, 1);
    mbar_init(o_full, 1);
    mbar_init(o_free, 128);
    *abort_word = 0;
    mbar_fence_init();
  }
  wait_for_previous();
  zero_tail_bwd(p);
  if (warp == 13) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  let_next_start();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 12) {
    if (lane == 0) {
      int it = 0;
      for (int item = blockIdx.x; item < num_items; item += gridDim.x) {
        const Item w = get_item(p, item, true);
        if (!w.valid) continue;
        const int slot = it & 1;
        if (!mbar_wait(&slot_empty[slot], ((it >> 1) & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty)) break;
        uint8_t* s = sSlots + slot * kBwdSlotBytes;
        if (ablate & 16) {
          mbar_arrive(&slot_full[slot]);
          if (!mbar_wait(o_free, (it & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty)) break;
          mbar_arrive(o_full);
          ++it;
          continue;
        }
        mbar_expect_tx(&slot_full[slot], kBwdSlotBytes);
        tma_load_2d(s, &tmap_q, &slot_full[slot], w.h * kHd, w.q0);
        tma_load_2d(s + kTileBytes, &tmap_k, &slot_full[slot], w.h * kHd, w.k0);
        tma_load_2d(s + 3 * kTileBytes, &tmap_do, &slot_full[slot], w.h * kHd, w.q0);
        tma_load_2d(s + 2 * kTileBytes, &tmap_v, &slot_full[slot], w.h * kHd, w.k0);
        if (!mbar_wait(o_free, (it & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty)) break;
        mbar_expect_tx(o_full, kTileBytes);
        tma_load_2d(sO, &tmap_o, o_full, w.h * kHd, w.q0);
        ++it;
      }
    }
  } else if (warp == 13) {
    const uint32_t idesc_s = make_idesc_bf16(kTile, kTile, 0, 0);
    const uint32_t idesc_dq = make_idesc_bf16(kTile, kHd, 0, 1);
    const uint32_t idesc_dkv = make_idesc_bf16(kTile, kHd, 1, 1);
    const uint32_t tmem = uniform(tmem_base), slots = uniform(smem_u32(sSlots)), pa = uniform(smem_u32(sP)), dsa = uniform(smem_u32(sDS));
    // Two queues served in whichever order their inputs arrive: S / dP of item s_it (needs its tiles and a free TMEM
    // set) and the gradients of item g_it (needs P / dS).  Blocking on one would hold back the other: the tiles of item
    // i + 1 land about a TMA round trip after the gradients of item i - 1 completed.
    int s_it = 0, g_it = 0;
    uint32_t steps = 0;            // 16-row steps of queries (low 4 bits) and keys of the items in flight, a byte each
    int item = blockIdx.x;
    Item nxt = item < num_items ? get_item(p, item) : Item{};        // of `item`; fetched one ahead, a round trip to memory otherwise
    auto next_valid = [&]() {
      while (item < num_items) {
        const Item w = nxt;
        if (item + static_cast<int>(gridDim.x) < num_items) nxt = get_item(p, item + gridDim.x);
        const int lens = uniform(w.valid ? (w.q_len << 8) | w.k_len : 0);
        if (lens != 0) {
          const int sh = (s_it & 3) * 8;
          steps = (steps & ~(0xffu << sh)) | (static_cast<uint32_t>((((lens >> 8) + 15) >> 4) | ((((lens & 255) + 15) >> 4) << 4)) << sh);
          return true;
        }
        item += gridDim.x;
      }
      return false;
    };
    bool more = next_valid();
    uint32_t idle = 0;
    while (more || g_it < s_it) {
      bool progressed = false;
      if (g_it < s_it && all_lanes(mbar_test_wait(pds_full, g_it & 1))) {
        tc_fence_after_sync();
        const int s = g_it & 1;
        const uint32_t set = tmem + s * 256;
        const uint32_t qa = slots + s * kBwdSlotBytes, ka = qa + kTileBytes, doa = qa + 3 * kTileBytes;
        const uint32_t lw = (steps >> ((g_it & 3) * 8)) & 0xffu;
        const int nkq = lw & 15, nkk = lw >> 4;
        if (!(ablate & 4)) {
          // dV = P^T dO, dK = dS^T Q : A read MN-major (keys = M, two 64-key slabs), reduction over query rows
          umma_steps_warp<2048, 2048>(set, make_smem_desc_sw128(pa, kTileBytes, 1024), make_smem_desc_sw128(doa, 8192, 1024), idesc_dkv, nkq);
          umma_steps_warp<2048, 2048>(set + 128, make_smem_desc_sw128(dsa, kTileBytes, 1024), make_smem_desc_sw128(qa, 8192, 1024), idesc_dkv, nkq);
          // dQ = dS K : A K-major (slab per 64 keys), B = K tile MN-major, reduction over keys
          const uint64_t ad = make_smem_desc_sw128(dsa, 16, 1024), bd = make_smem_desc_sw128(ka, 8192, 1024);
          umma_slabs_warp(set + 64, ad, bd, idesc_dq, nkk);
        }
        if (elect_one()) {
          umma_commit(pds_free);
          umma_commit(&grads_full[s]);
          umma_commit(&slot_empty[s]);
        }
        ++g_it;
        progressed = true;
      }
      if (more && s_it - g_it < 2 && all_lanes(mbar_test_wait(&slot_full[s_it & 1], (s_it >> 1) & 1) &&
                                               mbar_test_wait(&set_free[s_it & 1], ((s_it >> 1) & 1) ^ 1))) {
        tc_fence_after_sync();
        const int s = s_it & 1;
        const uint32_t set = tmem + s * 256;
        const uint32_t base = slots + s * kBwdSlotBytes;
        if (!(ablate & 8)) {
          umma_steps_warp<32, 32>(set, make_smem_desc_sw128(base, 16, 1024), make_smem_desc_sw128(base + kTileBytes, 16, 1024), idesc_s, kHd / 16);   // Q K^T
          umma_steps_warp<32, 32>(set + 128, make_smem_desc_sw128(base + 3 * kTileBytes, 16, 1024),
                                  make_smem_desc_sw128(base + 2 * kTileBytes, 16, 1024), idesc_s, kHd / 16);                                          // dO V^T
        }
        if (elect_one()) umma_commit(&sdp_full[s]);
        ++s_it;
        item += gridDim.x;
        more = next_valid();
        progressed = true;
      }
      if (progressed) idle = 0;
      else if (!all_lanes(keep_polling(idle, abort_word, p.status))) break;
    }
  } else if (warp < 8) {
    // ---- math threads: P and dS of every item, 16 of every 32 key columns each ---------------------------------------
    const int half = warp >> 2;
    const int t = (warp & 3) * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float scale_log2 = p.scale * 1.4426950408889634f;
    const unsigned long long seed = p.seed + ((kDrop && p.seed_dev) ? *p.seed_dev : 0ull);
    int it = 0;
    int item = blockIdx.x;
    Item nxt = item < num_items ? get_item(p, item) : Item{};
    while (item < num_items) {
      const Item w = nxt;
      item += gridDim.x;
      if (item < num_items) nxt = get_item(p, item);   // the next item's descriptor is fetched under this item's work
      if (!w.valid) continue;
      const int s = it & 1;
      const uint32_t set = tmem_base + s * 256 + lane_sel + half * 16;
      if (!__all_sync(0xffffffffu, mbar_wait(&d_full[s], (it >> 1) & 1, abort_word, p.status, kTimeoutTmemFull))) break;
      const float Drow = sD[s * kTile + t], lse2 = sL[s * kTile + t];
      mbar_arrive(&d_free[s]);
      if (!__all_sync(0xffffffffu, mbar_wait(&sdp_full[s], (it >> 1) & 1, abort_word, p.status, kTimeoutTmemFull))) break;
      tc_fence_after_sync();
      const int nchunks = (w.k_len + 31) >> 5;
      const int q_rows16 = ((w.q_len + 15) >> 4) << 4;   // rows the MN-major MMAs will read
      const bool warp_writes = (warp & 3) * 32 < q_rows16 && !(ablate & 1);
      bool may_store = it == 0, ok = true;
      if (warp_writes) {
        const DropRng rng(seed, (p.stream_id << 16) | static_cast<unsigned long long>(w.h), p.dropout_p);
        const unsigned long long row_base = static_cast<unsigned long long>(w.q0 + t) * p.kstride + half * 16;
#pragma unroll 1
        for (int c = 0; c < nchunks; ++c) {
          uint32_t sc[16], dp[16];
          tmem_ld16(set + c * 32, sc);
          tmem_ld16(set + 128 + c * 32, dp);
          uint32_t km = 0xffffu;
          if constexpr (kDrop) km = drop_mask16(rng, row_base + c * 32);     // hashed while the TMEM loads are in flight
          tmem_ld_wait();
          // the arithmetic comes before the wait for the staging tiles: it overlaps the previous item's gradient MMAs
          uint4 pr[2], ds[2];
          bwd_compute16(sc, dp, km, kDrop, rng.scale, Drow, scale_log2, lse2, c * 32 + half * 16, w.k_len, p.causal != 0, c * 32 + half * 16, t, pr, ds);
          if (!may_store) {   // the gradient MMAs of the previous item still read the staging tiles
            ok = __all_sync(0xffffffffu, mbar_wait(pds_free, (it - 1) & 1, abort_word, p.status, kTimeoutSmemEmpty));
            if (!ok) break;
            may_store = true;
          }
          bwd_store16(pr, ds, c * 32 + half * 16, t, sP, sDS);
        }
      }
      if (ok && !may_store) {
        // No thread may run ahead: S / dP and the D rows are double-buffered, so without this wait a thread with nothing to
        // write could reach its arrival for the NEXT item while the others still write this one, and complete the phase
        // early.  pds_free(it - 1) implies that phase it - 1 of pds_full is complete.
        ok = __all_sync(0xffffffffu, mbar_wait(pds_free, (it - 1) & 1, abort_word, p.status, kTimeoutSmemEmpty));
      }
      if (!ok) break;
      tc_fence_before_sync();
      fence_async_smem();
      mbar_arrive(pds_full);
      ++it;
    }
  } else if (warp < 12) {
    // ---- D / log-sum-exp rows of item i, then dQ row t (queries) and dK / dV row t (keys) of item i - 1 --------------
    const int wq = warp - 8;
    const int t = wq * 32 + lane;
    const uint32_t lane_sel = static_cast<uint32_t>(wq * 32) << 16;
    const float kInf = __int_as_float(0x7f800000);
    int it = 0;
    int item = blockIdx.x;
    Item nxt = item < num_items ? get_item(p, item) : Item{};
    Item prev{};
    bool ok = true;
    auto read_out = [&](const Item& w, int j) -> bool {
      const int s = j & 1;
      const uint32_t set = tmem_base + s * 256 + lane_sel;
      if (!__all_sync(0xffffffffu, mbar_wait(&grads_full[s], (j >> 1) & 1, abort_word, p.status, kTimeoutTmemFull))) return false;
      tc_fence_after_sync();
      if (!(ablate & 2)) {
        // dQ, dK, dV; dQ and dK carry the softmax scale that dS left out
        const int row0 = wq * 32;
#pragma unroll 1
        for (int m = 0; m < 3; ++m) {
          const int len = m == 0 ? w.q_len : w.k_len, first = m == 0 ? w.q0 : w.k0;
          if (row0 >= len) continue;
          __nv_bfloat16* base = m == 0 ? p.dq : m == 1 ? p.dk : p.dv;
          const int ld = m == 0 ? p.ld_dq : m == 1 ? p.ld_dk : p.ld_dv;
          bwd_store_rows(set + (m == 0 ? 64 : m == 1 ? 128 : 0), base + static_cast<size_t>(first + row0) * ld + static_cast<size_t>(w.h) * kHd, ld,
                         len - row0, m == 2 ? 1.f : p.scale, lane);
        }
      }
      tc_fence_before_sync();
      mbar_arrive(&set_free[s]);
      return true;
    };
    while (item < num_items && ok) {
      const Item w = nxt;
      item += gridDim.x;
      if (item < num_items) nxt = get_item(p, item);
      if (!w.valid) continue;
      const int s = it & 1;
      float Drow = 0.f, lse2 = kInf;
      if (t < w.q_len) lse2 = (ablate & 32) ? 0.f : p.lse[static_cast<size_t>(w.h) * p.lse_stride + w.q0 + t] * 1.4426950408889634f;
      if (!__all_sync(0xffffffffu, mbar_wait(o_full, it & 1, abort_word, p.status, kTimeoutTmaFull) &&
                                       mbar_wait(&slot_full[s], (it >> 1) & 1, abort_word, p.status, kTimeoutTmaFull))) { ok = false; break; }
      if (t < w.q_len && !(ablate & 32)) {
        const uint8_t* so = sO;
        const uint8_t* sdo = sSlots + s * kBwdSlotBytes + 3 * kTileBytes;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int g4 = 0; g4 < 8; ++g4) {
          const uint4 a = *reinterpret_cast<const uint4*>(so + sw128_offset(t, g4)), d = *reinterpret_cast<const uint4*>(sdo + sw128_offset(t, g4));
          const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
          const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&d);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 x = __bfloat1622float2(a2[j]), y = __bfloat1622float2(d2[j]);
            acc[j] = fmaf(x.x, y.x, fmaf(x.y, y.y, acc[j]));
          }
        }
        Drow = (acc[0] + acc[1]) + (acc[2] + acc[3]);
      }
      mbar_arrive(o_free);
      // the rows of item it - 2 have been read by every math thread
      if (!__all_sync(0xffffffffu, mbar_wait(&d_free[s], ((it >> 1) & 1) ^ 1, abort_word, p.status, kTimeoutSmemEmpty))) { ok = false; break; }
      sD[s * kTile + t] = Drow;
      sL[s * kTile + t] = lse2;
      mbar_arrive(&d_full[s]);
      if (it > 0) ok = read_out(prev, it - 1);
      prev = w;
      ++it;
    }
    if (ok && it > 0) read_out(prev, it - 1);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_word) {
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 13) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

static int g_attn_bwd_ablate = 0;
void set_attn_bwd_ablation(int bits) { g_attn_bwd_ablate = bits; }
int get_attn_bwd_ablation() { return g_attn_bwd_ablate; }

template <int kGroups, bool kDrop>
static const char* launch_fwd_short(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnArgs& a, int num_items,
                                    cudaStream_t stream) {
  auto kern = attn_fwd_short_kernel<kGroups, kDrop>;
  static bool configured = false;
  if (!configured) {
    cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd_short_smem(kGroups));
    if (ce != cudaSuccess) return cudaGetErrorString(ce);
    configured = true;
  }
  const int grid = num_items < num_sms() ? num_items : num_sms();
  return launch_overlapped(kern, grid, fwd_short_threads(kGroups), fwd_short_smem(kGroups), stream, tq, tk, tv, a, num_items);
}

const char* launch_attn_fwd_short(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnArgs& a,
                                  int num_items, cudaStream_t stream) {
  const bool drop = a.dropout_p > 0.f;
  // up to two items to a CTA: two groups
  if (num_items <= 2 * num_sms())
    return drop ? launch_fwd_short<2, true>(tq, tk, tv, a, num_items, stream) : launch_fwd_short<2, false>(tq, tk, tv, a, num_items, stream);
  return drop ? launch_fwd_short<4, true>(tq, tk, tv, a, num_items, stream) : launch_fwd_short<4, false>(tq, tk, tv, a, num_items, stream);
}

template <bool kDrop>
static const char* launch_bwd_short(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                    const CUtensorMap& to, const AttnArgs& a, int num_items, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t ce = cudaFuncSetAttribute(attn_bwd_short_kernel<kDrop>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdShortSmem);
    if (ce != cudaSuccess) return cudaGetErrorString(ce);
    configured = true;
  }
  const int grid = num_items < num_sms() ? num_items : num_sms();
  return launch_overlapped(attn_bwd_short_kernel<kDrop>, grid, kBwdShortThreads, kBwdShortSmem, stream, tq, tk, tv, tdo, to, a, num_items,
                           g_attn_bwd_ablate);
}

const char* launch_attn_bwd_short(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                  const CUtensorMap& to, const AttnArgs& a, int num_items, cudaStream_t stream) {
  const bool drop = a.dropout_p > 0.f && !(g_attn_bwd_ablate & 64);
  return drop ? launch_bwd_short<true>(tq, tk, tv, tdo, to, a, num_items, stream) : launch_bwd_short<false>(tq, tk, tv, tdo, to, a, num_items, stream);
}

}  // namespace b200

NMTG_BOUNDS_READER(nmtg_bounds_attention_short)

void nmtg_set_attn_bwd_ablation(int bits) { b200::set_attn_bwd_ablation(bits); }
