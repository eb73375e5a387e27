// Routing, row movement, gating and balancing kernels (SIMT; bandwidth or latency bound).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmoe {

// counts[tot] (int32), rank[n_slots] (int32, -1 for dropped slots), optional offs[tot + 1]
// (exclusive prefix of counts) and optional pos[n_slots] (slot ids sorted by expert, then by
// rank: pos[offs[e] + rank[s]] = s; entries past offs[tot] are not written).  Deterministic:
// slots of one expert are ranked by slot id.
// `part` (optional): int32 scratch of route_blocks(n_slots, tot) * tot entries; with it, more than
// 64 K slots (32 K with more experts than the cluster takes) are ranked by many CTAs in two
// launches instead of by one cluster or CTA.
int route_blocks(int n_slots, int tot);
cudaError_t launch_route(const int64_t* idx, int n_slots, int tot, int* counts, int* rank,
                         int* offs, int* pos, int* part, cudaStream_t stream);

// new_idx[s] = (idx[s] >= 0 && rank[s] < cap[idx[s]]) ? idx[s] : -1
cudaError_t launch_prune(const int64_t* idx, const int* rank, const int* cap, int n_slots, int tot,
                         int64_t* new_idx, cudaStream_t stream);

// SWIPE reassignment of one choice column (idx: global expert ids; rank: slot rank of every
// token inside its worker; count / quota: int32 [n_worker] tokens routed to / accepted by every
// worker).  `mark` writes key 0 for tokens beyond their worker's quota and -1 otherwise; after
// ranking the moved tokens (mrank), `assign` writes the balanced ids.
cudaError_t launch_swipe_mark(const int64_t* idx, const int* rank, const int* quota, int n,
                              int n_expert, int n_worker, int64_t* key, cudaStream_t stream);
cudaError_t launch_swipe_assign(const int64_t* idx, const int64_t* key, const int* mrank,
                                const int* count, const int* quota, int n, int n_expert,
                                int n_worker, int bias, int64_t* out, cudaStream_t stream);

// Rank-ordered capacity grant; ec/eca are [n_worker, n_expert] int64, cap[n_expert] int32 (in/out).
cudaError_t launch_limit_by_capacity(const int64_t* ec, int* cap, int64_t* eca, int n_expert,
                                     int n_worker, cudaStream_t stream);

// pos[base_excl[idx[s]] + rank[s]] = s   (the reference's `pos` array)
cudaError_t launch_fill_pos(const int64_t* idx, const int* rank, const int* cum_incl, int n_slots,
                            int tot, int64_t* pos, cudaStream_t stream);

// dst[base[idx[s]] + rank[s], :] = scale[s] * src[s / k, :]   (16-bit element types)
// `row_slot` (optional) receives the slot id of every written row.
cudaError_t launch_scatter_rows(int dtype, const void* src, const int64_t* idx, const int* rank,
                                const int* base, const void* scale, int n_slots, int k, int d,
                                void* dst, int* row_slot, cudaStream_t stream);

// out[t, :] = sum_j w[t, j] * rows[base[idx[t, j]] + rank[t, j], :]   (w = 1 when null)
cudaError_t launch_gather_combine(int dtype, const void* rows, const int64_t* idx, const int* rank,
                                  const int* base, const void* weight, int n_tokens, int k, int d,
                                  void* out, cudaStream_t stream);

// Backward of the weighted combine:  dscore[t, j] = <dout[t], rows[dest(t, j)]>  and
// drows[dest(t, j), :] = w[t, j] * dout[t, :].
cudaError_t launch_combine_bwd(int dtype, const void* dout, const void* rows, const int64_t* idx,
                               const int* rank, const int* base, const void* weight, int n_tokens,
                               int k, int d, void* drows, void* dscore, cudaStream_t stream);

// out[g, :] += column sums of x[offs[g] : offs[g + 1], :]  (fp32 accumulation buffer, pre-zeroed)
cudaError_t launch_colsum(int dtype, const void* x, const int* offs, int num_groups, long rows_cap,
                          int n, float* out, cudaStream_t stream);

// Top-k of each logits row (descending) with softmax over the selected values.
// logit_dtype: 0 bf16, 1 f16, 2 f32; prob has the dtype of the logits.  `zero` (here and below,
// optional) is set to 0 unless there are no rows.
cudaError_t launch_gate_topk_softmax(int logit_dtype, const void* logits, int n_rows, int n_experts,
                                     int k, int64_t* idx, void* prob, float* zero, cudaStream_t stream);
cudaError_t launch_gate_topk_softmax_bwd(int logit_dtype, const void* dprob, const int64_t* idx,
                                         const void* prob, int n_rows, int n_experts, int k,
                                         void* dlogits, cudaStream_t stream);

// Balance losses of the capacity-limited gates and Switch's choice (logit_dtype as above, `pitch`
// elements between rows of logits, tot <= 64, n >= 1).  part: fp32 [balance_blocks(n)][2 * tot];
// loss fp32 scalar; weight fp32 [tot], handed to the backward with the same is_switch and scale.
// ids[t * id_stride] is the expert a token counts for (-1: none).  The backward takes dloss (device
// scalar or null) and, for a score that is the softmax probability of expert win[t], dscore (or
// null; Switch only); dlogits is [n, tot].
bool balance_supported(int tot);
int balance_blocks(int n);
cudaError_t launch_balance_loss(int logit_dtype, const void* logits, long pitch, const int64_t* ids, int id_stride, int n,
                                int tot, bool is_switch, float scale, float* part, float* loss, float* weight,
                                cudaStream_t stream);
cudaError_t launch_balance_bwd(int logit_dtype, const void* logits, long pitch, const float* weight, const float* dloss,
                               const int64_t* win, const void* dscore, int n, int tot, bool is_switch, float scale,
                               void* dlogits, cudaStream_t stream);
cudaError_t launch_switch_top1(int logit_dtype, const void* logits, int n, int tot, int64_t* win, void* score,
                               cudaStream_t stream);

// Weight [tot, d] and bias [tot] (or null) of a 16-bit gate followed by rows of zeros and a bias that no top-k
// selects, up to `padded` experts.  d % 8 == 0, 16-byte aligned.
cudaError_t launch_gate_pad(int dtype, const void* w, const void* bias, int tot, int padded, int d, void* w_out, void* bias_out,
                            cudaStream_t stream);

// dst[i] = values[i] for host values, i < n <= kMaxHostOffsets.
constexpr int kMaxHostOffsets = 960;
cudaError_t launch_host_offsets(const int* values, int n, int* dst, cudaStream_t stream);

// new_idx[s] = (idx[s] in range && rank[s] < cap) ? idx[s] : -1
cudaError_t launch_prune_scalar(const int64_t* idx, const int* rank, int cap, int n_slots, int tot, int64_t* new_idx,
                                cudaStream_t stream);

// Fused gate (dtype: 0 bf16, 1 f16, 2 f32): logits = x W^T + b (tot <= 64 experts; f32: 8), top-k ids (descending) and
// softmax over the selected logits; one pass over x.
bool gate_fused_supported(int tot, int d, int k);
cudaError_t launch_gate_linear_topk(int dtype, const void* x, const void* w, const void* bias,
                                    int n_rows, int d, int tot, int k, void* logits, int64_t* idx,
                                    void* prob, float* zero, cudaStream_t stream);
// The same result for a few tokens (one block each), 16 bits.
cudaError_t launch_gate_linear_topk_few(int dtype, const void* x, const void* w, const void* bias, int n_rows, int d,
                                        int tot, int k, void* logits, int64_t* idx, void* prob, float* zero,
                                        cudaStream_t stream);
// Backward of the fused gate.  dl_scratch: fp32 [n_rows, tot]; dx (optional) [n_rows, d].
// part (optional, tot <= 16): fp32 scratch of gate_bwd_ranges() * (tot * d + tot) entries; with it
// dw_db receives dW [tot, d] followed by db [tot] in the layer's type.  Above 16 experts pass
// part = nullptr and form dW = dl^T x from dl_scratch with a library GEMM.
int gate_bwd_ranges(int dtype, int n_rows, int d);
cudaError_t launch_gate_bwd(int dtype, const void* dprob, const int64_t* idx, const void* prob,
                            const void* dlogits_in, const void* x, const void* w, int n_rows, int d,
                            int tot, int k, float* dl_scratch, void* dx, float* part, void* dw_db,
                            cudaStream_t stream);

// Reference-precision grouped GEMM for fp32 / fp64 and for shapes the tensor-core kernel
// does not take (elem: 0 bf16, 1 f16, 2 f32, 3 f64).  Same modes as the tcgen05 kernel; the row
// modes zero the rows past the last expert.
cudaError_t launch_simt_grouped_gemm(int mode, int elem, int num_groups, long rows_cap, int m, int n,
                                     int k, const void* a, const void* b, const int* offs,
                                     const void* bias, void* out, cudaStream_t stream);

// fp32 with 16-byte aligned rows (see sgemm.cu).  `psum` (weight gradient, optional): fp32
// [num_groups, m] column sums of `a` per group.
bool sgemm_applies(int mode, int num_groups, int m, int n, int k, const void* a, const void* b, const void* bias,
                   const void* out);
cudaError_t launch_sgemm(int mode, int num_groups, long rows_cap, int m, int n, int k, const float* a, const float* b,
                         const int* offs, const float* bias, float* out, float* psum, cudaStream_t stream);

}  // namespace fmoe
