// bf16 GEMM for few rows (incremental decoding: 1 to 512 activation rows): out[M, N] = epilogue(alpha * X W^T).
//
// What bounds it is latency: the weight matrix is read once (2 MB for 1024 x 1024, a third of a microsecond of HBM
// time), so the time is one memory round trip plus the chain load -> MMA -> reduction -> store, as long as enough SMs
// pull on the matrix at once.  Therefore
//   * the WEIGHTS are the 128-row A operand of tcgen05.mma and the activations its N operand (16, 32 or 64 columns), so a
//     handful of rows costs a handful of MMA columns instead of a 128-row tile of padding;
//   * K is cut over the CTAs of a cluster (up to 8): 1024 x 1024 runs on 64 SMs, two k-blocks each, instead of on the 16 CTAs
//     with 16 k-blocks each that 64-column tiles give.  The partial tiles meet in shared memory: every CTA writes
//     its fp32 accumulator as [row][128 features], and after one cluster barrier CTA r sums the rows r, r + S, ... over
//     its peers with distributed-shared-memory loads, in rank order, and runs the epilogue on them;
//   * with programmatic launch (nmtg_set_step_overlap, decoding steps only) barriers, TMEM and the first weight tiles
//     are set up while the previous kernel of the step is still running; everything that a previous kernel wrote is
//     touched only after griddepcontrol.wait.
#include "gemm_common.cuh"

namespace b200 {

// See nmtg_set_step_overlap.
static thread_local int t_step_overlap = 0;
bool step_overlap() { return t_step_overlap != 0; }

bool cached_tmap(CUtensorMap* out, const void* base, long rows, long cols, long ld, int br, int bc);

constexpr int kSkinnyThreads = 192;   // 4 epilogue warps (TMEM lanes), 1 TMA warp, 1 MMA warp
constexpr int kSkinnyFeat = 128;      // weight rows per tile

template <int NT>
struct SkinnySmem {
  static constexpr int kWBytes = kSkinnyFeat * BK * 2;
  static constexpr int kXBytes = NT * BK * 2;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = NT <= 32 ? 5 : 4;               // below 100 KB: two CTAs to an SM
  static constexpr int kRedBytes = NT * kSkinnyFeat * 4;          // overlays the stages once the MMAs are done
  static constexpr int kBody = kStages * kStageBytes > kRedBytes ? kStages * kStageBytes : kRedBytes;
  static constexpr int kTotal = kBody + 256 + 1024;
};

struct SkinnyArgs {
  int M, N, kb, split;
  float alpha;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int ld_res;
  __nv_bfloat16* out;
  int ld_out;
  int act;
  int early;        // weights may be read before the previous kernel has finished
  int* status;
};


__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

__device__ __forceinline__ float4 unpack4(uint2 u) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Not inlined: in every row of every unrolled split it made the kernel fetch instructions longer than it computes (transcription's
// products 1 % slower).
__device__ __noinline__ float4 skinny_gelu(float4 v) { return make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w)); }

__device__ __forceinline__ float4 skinny_act(float4 v, int act) {
  if (act == kActRelu) return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
  if (act == kActGelu) return skinny_gelu(v);
  if (act == kActSilu) return make_float4(v.x * sigmoid_f(v.x), v.y * sigmoid_f(v.y), v.z * sigmoid_f(v.z), v.w * sigmoid_f(v.w));
  return v;
}

// Sum of the partial tiles and epilogue of this CTA's rows (rank, rank + S, ...): a warp takes 128 features of a row, four per
// lane, and kRows rows at a time, all of whose loads (peers' partial sums, residual) are in flight together: row by row, the
// latency of the residual load alone made 512 x 512 with 256 rows take 18 us.
template <int kSplit, int kRows>
__device__ __forceinline__ void skinny_finish(const SkinnyArgs& p, const uint8_t* smem, int rank, int warp, int lane, int rows, int m0, int n0) {
  const int col = n0 + lane * 4;
  const bool col_ok = col < p.N, four = col + 4 <= p.N;
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.bias && four) bias = unpack4(*reinterpret_cast<const uint2*>(p.bias + col));
  else if (p.bias && col_ok) {
    bias.x = __bfloat162float(p.bias[col]);
    if (col + 1 < p.N) bias.y = __bfloat162float(p.bias[col + 1]);
    if (col + 2 < p.N) bias.z = __bfloat162float(p.bias[col + 2]);
  }
  const uint32_t red = smem_u32(smem) + lane * 16;
  for (int j0 = rank + kSplit * kRows * warp; j0 < rows; j0 += kSplit * kRows * 4) {
    float4 acc[kRows];
    uint2 res[kRows];
    float4 part[kRows][kSplit];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int j = j0 + i * kSplit;
      if (j >= rows) break;
      if (p.residual && col_ok) res[i] = *reinterpret_cast<const uint2*>(p.residual + static_cast<size_t>(m0 + j) * p.ld_res + col);
#pragma unroll
      for (int s = 0; s < kSplit; ++s)
        part[i][s] = kSplit == 1 ? *reinterpret_cast<const float4*>(smem + j * (kSkinnyFeat * 4) + lane * 16)
                                 : ld_cluster_f4(red + j * (kSkinnyFeat * 4), s);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int j = j0 + i * kSplit;
      if (j >= rows || !col_ok) break;
      acc[i] = part[i][0];
#pragma unroll
      for (int s = 1; s < kSplit; ++s) {
        acc[i].x += part[i][s].x; acc[i].y += part[i][s].y; acc[i].z += part[i][s].z; acc[i].w += part[i][s].w;
      }
      float4 v = skinny_act(make_float4(acc[i].x * p.alpha + bias.x, acc[i].y * p.alpha + bias.y, acc[i].z * p.alpha + bias.z,
                                        acc[i].w * p.alpha + bias.w), p.act);
      if (p.residual) {
        const float4 r = unpack4(res[i]);
        v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w;
      }
      uint2 o;
      __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      o.x = *reinterpret_cast<uint32_t*>(&lo);
      o.y = *reinterpret_cast<uint32_t*>(&hi);
      __nv_bfloat16* to = p.out + static_cast<size_t>(m0 + j) * p.ld_out + col;
      if (four) *reinterpret_cast<uint2*>(to) = o;
      else {                                     // N is no multiple of 4 (no residual then)
        to[0] = lo.x;
        if (col + 1 < p.N) to[1] = lo.y;
        if (col + 2 < p.N) to[2] = hi.x;
      }
    }
  }
}

template <int NT>
__global__ void __launch_bounds__(kSkinnyThreads)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SkinnyArgs p) {
  using S = SkinnySmem<NT>;
  constexpr uint32_t kCols = NT < 32 ? 32 : NT;
  constexpr int kLd = NT < 32 ? 16 : 32;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kBody);
  uint64_t* empty_bar = full_bar + S::kStages;
  uint64_t* done_bar = empty_bar + S::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.split;                 // the cluster is p.split consecutive blocks
  const int n0 = (blockIdx.x / p.split) * kSkinnyFeat;
  const int m0 = blockIdx.y * NT;
  const int rows = min(NT, p.M - m0);
  const int kb0 = rank * p.kb / p.split, kb1 = (rank + 1) * p.kb / p.split;    // never empty: split <= kb

  if (warp == 4 && lane == 0) {
    for (int i = 0; i < S::kStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(done_bar, 1);
    *abort_word = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 5) tmem_alloc(tmem_slot, kCols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();

  if (warp == 4) {
    if (lane == 0) {
      const int n_kb = kb1 - kb0;
      const int first = n_kb < S::kStages ? n_kb : S::kStages;
      if (!p.early) wait_for_previous();
      for (int i = 0; i < first; ++i) {
        mbar_expect_tx(&full_bar[i], S::kStageBytes);
        tma_load_2d(smem + i * S::kStageBytes, &tmap_w, &full_bar[i], (kb0 + i) * BK, n0);
      }
      // (Fetching the rest of the weights into L2 meanwhile gained nothing between the kernels of a step, and took traffic from the product that
      // was still running: 32000 x 2048, 8 rows, back to back 22.4 us without, 26.9 with it; 6944 x 5120, 256 rows 30.2, 42.3.)
      if (p.early) wait_for_previous();
      for (int i = 0; i < first; ++i)
        tma_load_2d(smem + i * S::kStageBytes + S::kWBytes, &tmap_x, &full_bar[i], (kb0 + i) * BK, m0);
      int stage = 0;
      uint32_t phase = 0;              // phase of the release that a refill waits for
      for (int i = first; i < n_kb; ++i) {
        if (!mbar_wait(&empty_bar[stage], phase, abort_word, p.status, kTimeoutSmemEmpty)) break;
        uint8_t* sw = smem + stage * S::kStageBytes;
        mbar_expect_tx(&full_bar[stage], S::kStageBytes);
        tma_load_2d(sw, &tmap_w, &full_bar[stage], (kb0 + i) * BK, n0);
        tma_load_2d(sw + S::kWBytes, &tmap_x, &full_bar[stage], (kb0 + i) * BK, m0);
        if (++stage == S::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 5) {                // all lanes: see elect_one
    constexpr uint32_t idesc = make_idesc_bf16(kSkinnyFeat, NT, 0, 0);
    const uint32_t tmem = uniform(tmem_base), smem0 = uniform(smem_u32(smem));
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!all_lanes(mbar_wait(&full_bar[stage], phase, abort_word, p.status, kTimeoutTmaFull))) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t sw = smem0 + stage * S::kStageBytes;
      const uint64_t wdesc = make_smem_desc_sw128(sw, 16, 1024);
      const uint64_t xdesc = make_smem_desc_sw128(sw + S::kWBytes, 16, 1024);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_bf16(tmem, wdesc + static_cast<uint64_t>(k * 2), xdesc + static_cast<uint64_t>(k * 2), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
      }
      if (++stage == S::kStages) { stage = 0; phase ^= 1; }
    }
    if (ok && elect_one()) umma_commit(done_bar);
  } else {
    wait_for_previous();        // the residual is an earlier kernel's output, and so may be the buffer that is written
    const bool ok = mbar_wait(done_bar, 0, abort_word, p.status, kTimeoutTmemFull);
    if (ok) {
      tc_fence_after_sync();
      // accumulator lane = feature, column = row of X  ->  red[row][feature]
      float* red = reinterpret_cast<float*>(smem);
#pragma unroll 1
      for (int c = 0; c < NT && c < rows; c += kLd) {
        uint32_t r[kLd];
        if constexpr (kLd == 32) tmem_ld32(tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + c, r);
        else tmem_ld16(tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kLd; ++j) red[(c + j) * kSkinnyFeat + warp * 32 + lane] = __uint_as_float(r[j]);
      }
    }
    tc_fence_before_sync();
  }
  __syncwarp();
  if (p.split > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else __syncthreads();
  if (warp < 4 && !*abort_word) {
    switch (p.split) {
      case 1: skinny_finish<1, 8>(p, smem, rank, warp, lane, rows, m0, n0); break;
      case 2: skinny_finish<2, 4>(p, smem, rank, warp, lane, rows, m0, n0); break;
      case 4: skinny_finish<4, 4>(p, smem, rank, warp, lane, rows, m0, n0); break;
      default: skinny_finish<8, 2>(p, smem, rank, warp, lane, rows, m0, n0); break;
    }
  }
  __syncwarp();
  // nobody leaves while a peer may still read its partial sums
  if (p.split > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else __syncthreads();
  if (*abort_word) {
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);      // copies in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kCols);
  }
}

template <int NT>
static const char* launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyArgs& a, int tiles_n, int tiles_m, bool pdl,
                                 cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnySmem<NT>::kTotal);
    if (e != cudaSuccess) return cudaGetErrorString(e);
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles_n * a.split, tiles_m);
  cfg.blockDim = dim3(kSkinnyThreads);
  cfg.dynamicSmemBytes = SkinnySmem<NT>::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<NT>, tw, tx, a);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

static int skinny_rows(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }

// Whether the few-row kernel takes this problem: plain Linear products (both operands K-major) with bias, activation and
// residual whose 128-feature x 64-row tiles fit the GPU at once (two CTAs to an SM), where the caller lets the sum over K be split:
// decoding steps do; training, scoring and encoding keep one order of their forward sums whatever the batch size.  Measured (us, this kernel back to back
// with programmatic launch / the tiled kernel): 1024 x 1024, 4 rows
// 3.6 / 8.4, 256 rows 7.2 / 9.3, 512 rows 7.5 / 9.3; 4096 x 1024, 64 rows 6.0 / 8.6; 1024 x 4096, 4 rows 5.4 / 22.8; 32000 x
// 1024, 33 rows 13.9 / 20.3.  Beyond one wave (32000 x 1024 with 128 rows: 25 us against 19) the tiled kernel is the better one; up to 32 rows
// two waves are no slower (51865 x 1280, four matrices in turn, 1 row 24.0 / 32.2, 8 rows 26.6 / 31.8, 32 rows 27.5 / 31.8).
bool skinny_takes(const GemmDesc* d, int sms) {
  const long tiles = static_cast<long>((d->N + kSkinnyFeat - 1) / kSkinnyFeat) * ((d->M + skinny_rows(d->M) - 1) / skinny_rows(d->M));
  return d->allow_split_k && d->M <= 512 && tiles <= (d->M <= 32 ? 4L : 2L) * sms && !d->out_fp32 && !d->a_mn_major && !d->b_mn_major && !d->gather && !d->preact && !d->mask &&
         !d->colsum && !d->aux && d->act >= 0 && d->act <= kActSilu && d->dropout_p <= 0.f && d->split_k <= 1 && d->force_bn == 0 &&
         (!d->residual || (d->N % 4 == 0 && d->ld_res % 4 == 0 && (reinterpret_cast<uintptr_t>(d->residual) & 7) == 0)) &&
         (reinterpret_cast<uintptr_t>(d->bias) & 7) == 0;
}

// `weights_settled`: no kernel that may still run writes the weights.  A gathered weight is not: the copy right before this launch
// writes it, so that it is read after griddepcontrol.wait like everything else.
const char* launch_gemm_skinny(const GemmDesc* d, int sms, bool weights_settled, cudaStream_t stream) {
  const bool pdl = step_overlap();
  const int nt = skinny_rows(d->M);
  CUtensorMap tw, tx;
  if (!cached_tmap(&tw, d->b, d->N, d->K, d->ldb, kSkinnyFeat, BK)) return "gemm: cuTensorMapEncodeTiled failed for B";
  if (!cached_tmap(&tx, d->a, d->M, d->K, d->lda, nt, BK)) return "gemm: cuTensorMapEncodeTiled failed for A";
  SkinnyArgs a;
  a.M = d->M; a.N = d->N; a.kb = (d->K + BK - 1) / BK;
  a.alpha = d->alpha;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(d->bias);
  a.residual = reinterpret_cast<const __nv_bfloat16*>(d->residual); a.ld_res = d->ld_res;
  a.out = reinterpret_cast<__nv_bfloat16*>(d->out); a.ld_out = d->ld_out;
  a.act = d->act; a.status = d->status;
  a.early = pdl && weights_settled ? 1 : 0;
  const int tiles_n = (d->N + kSkinnyFeat - 1) / kSkinnyFeat, tiles_m = (d->M + nt - 1) / nt;
  // as many K slices as keep one wave of CTAs, at least two k-blocks each
  int split = 8;
  while (split > 1 && (static_cast<long>(tiles_n) * tiles_m * split > 2L * sms || a.kb < 2 * split)) split >>= 1;
  a.split = split;
  if (nt == 16) return launch_skinny<16>(tw, tx, a, tiles_n, tiles_m, pdl, stream);
  if (nt == 32) return launch_skinny<32>(tw, tx, a, tiles_n, tiles_m, pdl, stream);
  return launch_skinny<64>(tw, tx, a, tiles_n, tiles_m, pdl, stream);
}

}  // namespace b200

void nmtg_set_step_overlap(int on) { b200::t_step_overlap = on; }
