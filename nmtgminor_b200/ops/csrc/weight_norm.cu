// Weight normalisation along the last dimension: w = v * g / |v|, the norm of every column of v [rows, cols] over all its rows (the
// positional convolutions of the audio encoders: 1024 x 64 rows, 128 columns).
//
// Bound by memory.  Tensor operations gave a column of a row-major matrix to a block, 4 bytes of every 512: 728 us forward and 922 backward
// for 33.5 MB.  Here a warp reads whole rows, a thread keeps the sums of four columns, and the blocks' partial sums, added in one order by
// each block of the second pass, meet in a table of `blocks` x cols; the second pass finds most of the matrix in L2.
#include "b200_ptx.cuh"
#include "seq_api.h"

namespace b200 {

int num_sms();

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float4 fma4(float4 a, float4 b, float4 c) {
  return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// columns 4 c .. of this thread, summed over the block's row slots; slot 0 has the sums
__device__ __forceinline__ float4 over_slots(float4 s, float4* shared, int lanes, int slots) {
  shared[threadIdx.x] = s;
  for (int n = slots >> 1; n > 0; n >>= 1) {
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < n * lanes) shared[threadIdx.x] = add4(shared[threadIdx.x], shared[threadIdx.x + n * lanes]);
  }
  __syncthreads();
  return shared[threadIdx.x % lanes];
}

// partial[block][cols] = sum over the block's rows of a * b
__global__ void __launch_bounds__(kThreads) column_dot_kernel(const float4* __restrict__ a, const float4* __restrict__ b, float4* __restrict__ partial,
                                                              long rows, int lanes) {
  __shared__ float4 shared[kThreads];
  const int slots = kThreads / lanes, c = threadIdx.x % lanes, slot = threadIdx.x / lanes;
  const long step = static_cast<long>(gridDim.x) * slots;
  float4 s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long r = static_cast<long>(blockIdx.x) * slots + slot; r < rows; r += 4 * step)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (r + i * step < rows) {
        const long at = (r + i * step) * lanes + c;
        s[i] = fma4(a[at], b[at], s[i]);
      }
  const float4 sum = over_slots(add4(add4(s[0], s[1]), add4(s[2], s[3])), shared, lanes, slots);
  if (slot == 0) partial[static_cast<long>(blockIdx.x) * lanes + c] = sum;
}

__device__ __forceinline__ float4 all_blocks(const float4* __restrict__ partial, int blocks, float4* shared, int lanes) {
  const int slots = kThreads / lanes, c = threadIdx.x % lanes, slot = threadIdx.x / lanes;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int i = slot; i < blocks; i += slots) s = add4(s, partial[static_cast<long>(i) * lanes + c]);
  return over_slots(s, shared, lanes, slots);
}

__global__ void __launch_bounds__(kThreads) weight_norm_kernel(const float4* __restrict__ v, const float4* __restrict__ gain,
                                                               const float4* __restrict__ partial, int blocks, float4* __restrict__ w,
                                                               float4* __restrict__ norm, long rows, int lanes) {
  __shared__ float4 shared[kThreads];
  const int slots = kThreads / lanes, c = threadIdx.x % lanes, slot = threadIdx.x / lanes;
  const float4 s = all_blocks(partial, blocks, shared, lanes), g = gain[c];
  const float4 n = make_float4(sqrtf(s.x), sqrtf(s.y), sqrtf(s.z), sqrtf(s.w));
  if (blockIdx.x == 0 && slot == 0) norm[c] = n;
  const float4 f = make_float4(__fdiv_rn(g.x, n.x), __fdiv_rn(g.y, n.y), __fdiv_rn(g.z, n.z), __fdiv_rn(g.w, n.w));
  for (long r = static_cast<long>(blockIdx.x) * slots + slot; r < rows; r += static_cast<long>(gridDim.x) * slots) {
    const float4 x = v[r * lanes + c];
    w[r * lanes + c] = make_float4(x.x * f.x, x.y * f.y, x.z * f.z, x.w * f.w);
  }
}

// dg = sum(dw v) / |v|, dv = g / |v| (dw - v sum(dw v) / |v|^2)
__global__ void __launch_bounds__(kThreads) weight_norm_bwd_kernel(const float4* __restrict__ dw, const float4* __restrict__ v,
                                                                   const float4* __restrict__ gain, const float4* __restrict__ norm,
                                                                   const float4* __restrict__ partial, int blocks, float4* __restrict__ dv,
                                                                   float4* __restrict__ dg, long rows, int lanes) {
  __shared__ float4 shared[kThreads];
  const int slots = kThreads / lanes, c = threadIdx.x % lanes, slot = threadIdx.x / lanes;
  const float4 s = all_blocks(partial, blocks, shared, lanes), g = gain[c], n = norm[c];
  const float4 d = make_float4(__fdiv_rn(s.x, n.x), __fdiv_rn(s.y, n.y), __fdiv_rn(s.z, n.z), __fdiv_rn(s.w, n.w));
  if (blockIdx.x == 0 && slot == 0) dg[c] = d;
  const float4 f = make_float4(__fdiv_rn(g.x, n.x), __fdiv_rn(g.y, n.y), __fdiv_rn(g.z, n.z), __fdiv_rn(g.w, n.w));
  const float4 e = make_float4(__fdiv_rn(-d.x, n.x), __fdiv_rn(-d.y, n.y), __fdiv_rn(-d.z, n.z), __fdiv_rn(-d.w, n.w));
  for (long r = static_cast<long>(blockIdx.x) * slots + slot; r < rows; r += static_cast<long>(gridDim.x) * slots) {
    const float4 y = fma4(v[r * lanes + c], e, dw[r * lanes + c]);
    dv[r * lanes + c] = make_float4(y.x * f.x, y.y * f.y, y.z * f.z, y.w * f.w);
  }
}

// blocks for `rows` rows: at most two to an SM, and no more than the table has room for
int blocks_for(long rows, int lanes, int table) {
  const long need = (rows + kThreads / lanes - 1) / (kThreads / lanes), most = 2L * num_sms();
  long n = need < most ? need : most;
  if (n > table) n = table;
  return static_cast<int>(n);
}
const char* sizes(long rows, int cols, int table) {
  const int lanes = cols / 4;
  return rows < 1 || table < 1 || cols < 4 || cols % 4 != 0 || lanes > kThreads || (lanes & (lanes - 1)) != 0 ? "weight_norm: sizes out of range" : nullptr;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" {

const char* nmtg_weight_norm(const float* v, const float* gain, float* w, float* norm, float* table, int table_rows, long rows, int cols,
                             cudaStream_t stream) {
  if (const char* bad = sizes(rows, cols, table_rows)) return bad;
  const int lanes = cols / 4, blocks = blocks_for(rows, lanes, table_rows);
  const float4* x = reinterpret_cast<const float4*>(v);
  float4* t = reinterpret_cast<float4*>(table);
  column_dot_kernel<<<blocks, kThreads, 0, stream>>>(x, x, t, rows, lanes);
  weight_norm_kernel<<<blocks, kThreads, 0, stream>>>(x, reinterpret_cast<const float4*>(gain), t, blocks, reinterpret_cast<float4*>(w),
                                                      reinterpret_cast<float4*>(norm), rows, lanes);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

const char* nmtg_weight_norm_bwd(const float* dw, const float* v, const float* gain, const float* norm, float* dv, float* dg, float* table,
                                 int table_rows, long rows, int cols, cudaStream_t stream) {
  if (const char* bad = sizes(rows, cols, table_rows)) return bad;
  const int lanes = cols / 4, blocks = blocks_for(rows, lanes, table_rows);
  const float4 *d = reinterpret_cast<const float4*>(dw), *x = reinterpret_cast<const float4*>(v);
  float4* t = reinterpret_cast<float4*>(table);
  column_dot_kernel<<<blocks, kThreads, 0, stream>>>(d, x, t, rows, lanes);
  weight_norm_bwd_kernel<<<blocks, kThreads, 0, stream>>>(d, x, reinterpret_cast<const float4*>(gain), reinterpret_cast<const float4*>(norm), t, blocks,
                                                          reinterpret_cast<float4*>(dv), reinterpret_cast<float4*>(dg), rows, lanes);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // extern "C"
