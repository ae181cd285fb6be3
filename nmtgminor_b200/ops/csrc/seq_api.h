// C launch API of the sequence-model kernels (transducer joint / loss, linear-recurrence scan, Cauchy kernel
// coefficients, row softmax with mask and dropout, beam-search step, single-query decode attention).
// Every launcher returns nullptr on success or a static error string; nothing allocates.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

extern "C" {

// ---- front end of raw audio, without gradients (frontend.cu): 256 or 512 channels, rows of utterance b at b * out_rows ----------
// wav fp32 [B, samples] (row stride wav_stride), w fp32 [channels][taps], bias optional; out bf16 frames t < T
const char* nmtg_conv_norm_gelu(const float* wav, long wav_stride, const float* w, const float* bias, const float* gamma, const float* beta,
                                float eps, void* out, int B, int samples, int T, int out_rows, int channels, int taps, int stride,
                                cudaStream_t stream);
const char* nmtg_norm_gelu(const void* x, const float* gamma, const float* beta, float eps, void* out, int B, int T, int in_rows, int out_rows,
                           int channels, cudaStream_t stream);

// ---- weight normalisation of the columns of v fp32 [rows, cols], cols / 4 a power of two up to 256 (weight_norm.cu) ----------------
// table: fp32 [table_rows, cols] of partial sums; norm [cols] is kept for the gradient; all pointers 16-byte aligned
const char* nmtg_weight_norm(const float* v, const float* gain, float* w, float* norm, float* table, int table_rows, long rows, int cols,
                             cudaStream_t stream);
const char* nmtg_weight_norm_bwd(const float* dw, const float* v, const float* gain, const float* norm, float* dv, float* dg, float* table,
                                 int table_rows, long rows, int cols, cudaStream_t stream);

// ---- transducer joint: h[b,t,u,:] = act(f[b,t,:] + g[b,u,:]) ------------------------------------------------
// dtype: 0 = fp32, 1 = bf16.  packed: rows of sentence b start at (b ? batch_offset[b-1] : 0) and are laid
// out [t][u] with u running over g_len[b]; dense: [B, T, U, H] with rows outside the lengths zeroed.
// relu / dropout are applied in that order; the dropout mask is a pure function of (seed, stream_id, element).
const char* nmtg_transducer_joint_fwd(const void* f, const void* g, const int* f_len, const int* g_len,
                                      const long* batch_offset, void* out, int B, int T, int U, int H, int dtype,
                                      int packed, int relu, float p, unsigned long long seed,
                                      unsigned long long stream_id, cudaStream_t stream);
// df[b,t,:] = sum_u d(out)  dg[b,u,:] = sum_t d(out); `out` (the forward result) is needed when relu or dropout is on.
const char* nmtg_transducer_joint_bwd(const void* dout, const void* out, const int* f_len, const int* g_len,
                                      const long* batch_offset, void* df, void* dg, int B, int T, int U, int H,
                                      int dtype, int packed, int relu, float p, unsigned long long seed,
                                      unsigned long long stream_id, float scale, cudaStream_t stream);

// ---- transducer loss on fp32 log-probabilities x[b,t,u,v] (dense [B,T,U,V] or packed as above) ----------------
// alpha / beta: fp32 [B, T, U]; loss[b] = -log p(label_b | audio_b).
const char* nmtg_transducer_loss_fwd(const float* x, const int* label, const int* f_len, const int* y_len,
                                     const long* batch_offset, float* alpha, float* beta, float* loss, int B, int T,
                                     int U, int V, int blank, int packed, cudaStream_t stream);
// dx has the layout of x.  fuse_softmax: x = log_softmax(z) and dx is the gradient with respect to z.
const char* nmtg_transducer_loss_bwd(const float* x, const float* loss_grad, const float* alpha, const float* beta,
                                     const int* label, const int* f_len, const int* y_len, const long* batch_offset,
                                     float* dx, int B, int T, int U, int V, int blank, int packed, int fuse_softmax,
                                     cudaStream_t stream);

// ---- diagonal linear recurrence on complex64 rows: h_t = lambda_n * h_(t-1) + x_t ------------------------------
// x, h: [B, N, L] (time innermost, interleaved re/im); lambda: [N]; lengths: [B].  direction 0 = left to right,
// 1 = right to left (starting at lengths[b]-1), 2 = first N/2 channels left to right, the rest right to left.
// Positions >= lengths[b] are written as zero.
const char* nmtg_lru_scan_fwd(const float2* lambda, const float2* x, const int* lengths, float2* h, int B, int N, int L,
                              int direction, cudaStream_t stream);
// PyTorch complex-gradient convention: dx_t = sum_s conj(lambda)^(|s-t|) g_s; dlambda[n] += sum conj(h_prev) * dx_t.
const char* nmtg_lru_scan_bwd(const float2* lambda, const float2* grad_h, const float2* h, const int* lengths,
                              float2* dx, float2* dlambda, int B, int N, int L, int direction, cudaStream_t stream);

// ---- Cauchy kernel coefficients: out[i,q,l,h] = sum_n a[i,q,h,n] / (b[q,l,h] - c[q,n])  (complex64) ------------
const char* nmtg_cauchy_fwd(const float2* a, const float2* b, const float2* c, float2* out, int I, int Q, int L, int H,
                            int N, cudaStream_t stream);
// da / db / dc must be zero on entry (db and dc are accumulated with atomics).
const char* nmtg_cauchy_bwd(const float2* a, const float2* b, const float2* c, const float2* dout, float2* da, float2* db,
                            float2* dc, int I, int Q, int L, int H, int N, cudaStream_t stream);

// ---- row softmax (+ additive/boolean key mask, + dropout) over x[rows, cols] ---------------------------------
// dtype 0 = fp32, 1 = bf16 (in and out).  pad_mask: uint8 [rows / rows_per_mask, cols], nonzero = masked out.
// y = softmax(x * scale + mask); yd = dropout(y) (yd may be null when p == 0).
const char* nmtg_softmax_dropout_fwd(const void* x, const uint8_t* pad_mask, void* y, void* yd, int rows, int cols,
                                     int rows_per_mask, int dtype, float scale, float p, unsigned long long seed,
                                     unsigned long long stream_id, cudaStream_t stream);
// dx = scale * y * (dyd_masked - sum(dyd_masked * y)) with dyd_masked = dropout-mask * dyd / (1-p)
const char* nmtg_softmax_dropout_bwd(const void* dyd, const void* y, void* dx, int rows, int cols, int dtype, float scale,
                                     float p, unsigned long long seed, unsigned long long stream_id,
                                     cudaStream_t stream);

// ---- beam search step ---------------------------------------------------------------------------------------
// logits: [R = B*K, V], rows `ld` elements apart (dtype 0 fp32 / 1 bf16).  For every row: lp = log_softmax(logits) with pad -> -inf,
// eos -> -inf when step < min_len, everything but eos -> -inf when force_eos[r]; then per sentence the best
// 2K of (scores[r] + lp[r, v]) over its K rows.  out_scores / out_index: [B, 2K]; index = k * V + v.
// row_lse: fp32 [R] scratch, cand_*: scratch [R, 2K].
const char* nmtg_beam_topk(const void* logits, long ld, int dtype, const float* scores, const uint8_t* force_eos,
                           float* row_lse, float* cand_val, int* cand_idx, float* out_scores, long* out_index, int B, int K,
                           int V, int pad, int eos, int ban_eos, cudaStream_t stream);
// dst[r, 0:copy_bytes] = src[index[r], 0:copy_bytes] for rows `row_stride_bytes` apart (both multiples of 16).
const char* nmtg_gather_rows(const void* src, void* dst, const long* index, int rows, int src_rows, long row_stride_bytes,
                             long copy_bytes, cudaStream_t stream);

// ---- single-query attention over a preallocated cache ------------------------------------------------------
// q: bf16 [R, heads, 64]; k_cache / v_cache: bf16 [R / kv_div, cap, heads, 64] (kv_div > 1 shares one cache row
// between the hypotheses of a sentence, as for encoder-decoder attention); lengths: int32 [R / kv_div] or null
// (= all rows use `len`); out: bf16 [R, heads, 64].
const char* nmtg_decode_attn(const void* q, long q_ld, const void* k_cache, const void* v_cache, const int* lengths,
                             void* out, int R, int heads, int cap, int len, int kv_div, float scale, cudaStream_t stream);
// cache[r, pos, :] = new[r, :] for k and v (new rows `ld` elements apart, heads * 64 elements each).
const char* nmtg_cache_append(const void* k_new, const void* v_new, long ld, void* k_cache, void* v_cache, int R, int heads,
                              int cap, int pos, cudaStream_t stream);

// ---- one replayable beam-search step (decode_step.cu) -------------------------------------------------------------
// Tables of a search over B sentences x K hypotheses (R = B K rows), all on the device.
struct NmtgBeam {
  int K, R, cap, pad, eos;
  const int* ctl;          // {T, min_len, normalize}
  const float* inv_norm;   // [n] = 1 / n^alpha for lengths up to T + 1
  const int* max_rows;     // [B] step at which only EOS may follow
  float* scores;           // [R] sums of log-probabilities
  uint8_t* force;          // [R] 1 = only EOS may follow, 2 = EOS is banned, 0 = free
  uint8_t* done;           // [B]
  long* tok;               // [R] last word of every hypothesis
  long* pos_rows;          // [R] its position = the current step
  int* anc;                // [R, cap] cache row that holds position j of hypothesis r
  int* fin_count;          // [B]
  float* fin_score;        // [B, K] finished hypotheses, best first; -inf = none
  int* fin_step;           // [B, K] step of the EOS
  int* fin_row;            // [B, K] hypothesis (0 .. K-1) that it ended
  float* fin_last;         // [B, K] log-probability of the EOS
  int* hist_tok;           // [steps, R] word chosen at a step, its parent (0 .. K-1) and its log-probability
  int* hist_par;
  float* hist_score;
};
// qkv: bf16 [R, 3 * heads * 64]; the new keys / values go to row r, position pos_rows[r] of the caches [R, cap, heads * 64]
const char* nmtg_decode_self(const void* qkv, long ld, void* k_cache, void* v_cache, const int* anc, const long* pos_rows, void* out,
                             int B, int K, int heads, int cap, float scale, cudaStream_t stream);
// q: bf16 [B K, heads * 64]; ck / cv: bf16 [B, cap, heads * 64], lengths int32 [B]
const char* nmtg_decode_cross(const void* q, long ld, const void* ck, const void* cv, const int* lengths, void* out, int B, int K,
                              int heads, int cap, float scale, cudaStream_t stream);
// logits [R, V] (dtype 0 = fp32, 1 = bf16); workspaces: part_lse 8 bytes x [R, pieces], part 8 bytes x [R, pieces, 2K] with
// pieces = ceil(V / 4096).  Advances every table by one step.
const char* nmtg_beam_step(const NmtgBeam* s, const void* logits, long ld, int dtype, void* part_lse, void* part, int B, int V,
                           cudaStream_t stream);
// words / word_scores [B, n_best, width]: the finished hypotheses, fin_step + 1 entries each
const char* nmtg_beam_trace(const NmtgBeam* s, int B, int n_best, long* words, float* word_scores, int width, cudaStream_t stream);

// ---- relative-position (Transformer-XL) self-attention on packed sequences of at most 128 tokens ---------------
// qkv: bf16 [N, 3 * heads * 64]; r: bf16 [L, heads * 64], row r_center - d = projected embedding of distance d;
// u / w: fp32 [heads, 64] content / position biases; cu: int32 [B + 1]; out: bf16 [N, heads * 64]; lse: fp32 [heads, N].
const char* nmtg_rel_attn_fwd(const void* qkv, const void* r, const float* u, const float* w, const int* cu, void* out, float* lse,
                              int B, int N, int heads, int max_len, int r_center, int L, int causal, float scale, float p,
                              unsigned long long seed, unsigned long long stream_id, cudaStream_t stream);
// dqkv: bf16 [N, 3H] (rows of the sequences are overwritten); dr [L, H], du, dw [heads, 64]: fp32, ACCUMULATED into.
const char* nmtg_rel_attn_bwd(const void* qkv, const void* r, const float* u, const float* w, const int* cu, const float* lse,
                              const void* dctx, void* dqkv, float* dr, float* du, float* dw, int B, int N, int heads, int max_len,
                              int r_center, int L, int causal, float scale, float p, unsigned long long seed,
                              unsigned long long stream_id, cudaStream_t stream);
}
