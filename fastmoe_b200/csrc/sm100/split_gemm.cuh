// Host interface of the fp32 grouped GEMM on the tensor cores (split_gemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmoe {

// An fp32 matrix as three bf16 planes, one behind the other: h, m 2^7 and l 2^14, where h + m + l is the value (to
// 2^-148 where it is below 2^-124).
// Matrices of token rows are padded: rows of expert e begin at split_row(offs[e], e), and the rows
// from its last one to the next multiple of 64 are zero.
__host__ __device__ inline long split_row(long off, long e) { return ((off + 63) / 64 + e) * 64; }
inline long split_rows_cap(long rows, int num_groups) { return split_row(rows, num_groups); }

enum SplitOut : int {
  kSplitPlain = 0,   // fp32 rows (+ bias) or weight gradients; row modes zero the rows past the last expert
  kSplitAct = 1,     // planes of act(acc + bias); optionally `pre` = acc + bias
  kSplitDAct = 2,    // planes of acc * act'(pre)
};

struct SplitGemmArgs {
  int mode = 0;                 // GemmMode
  int num_groups = 0;
  long rows_cap = 0;            // rows of the fp32 matrices; the planes have split_rows_cap of them
  int m = 0, n = 0, k = 0;      // as in GroupedGemmArgs
  const void* a = nullptr;      // planes [3][padded rows][k], or P [3][padded rows][m]
  const void* b = nullptr;      // planes [3][num_groups][..][..] of the weights, or Q [3][padded rows][n]
  const int* offs = nullptr;    // device, [num_groups + 1]
  int kind = kSplitPlain;
  int act = 0;                  // ActKind
  const float* bias = nullptr;  // [num_groups, n]
  float* out = nullptr;         // kSplitPlain
  void* planes = nullptr;       // kSplitAct, kSplitDAct: [3][padded rows][n]
  float* pre = nullptr;         // [rows_cap, n]: written by kSplitAct (optional), read by kSplitDAct
  float* psum = nullptr;        // weight gradient, optional: [num_groups, m] column sums of P
  // scratch for tiles that CTA pairs share: split_work_floats floats, and split_num_flags flags that
  // are zero before the launch (null: no tile is shared)
  float* work = nullptr;
  int* flags = nullptr;
  // scratch of `psum`: split_sum_floats floats, and split_num_counts counts that are zero before
  float* sums = nullptr;
  int* sum_counts = nullptr;
  int* status = nullptr;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
};

// Widths are multiples of 8 and at least 16, at most 256 groups, 32-byte aligned matrices.
bool split_gemm_supported(int mode, int m, int n, int k, int num_groups, long rows_cap);
cudaError_t launch_split_gemm(const SplitGemmArgs& args);
long split_work_floats(int num_sms);
int split_num_flags(int num_sms);
long split_sum_floats(long rows_cap, int num_groups, int m);
int split_num_counts(int num_groups, int m);

// planes[3][num_groups][per_expert] of the weights of experts with rows (per_expert a multiple of 8).
cudaError_t launch_split_weight(const float* src, const int* offs, int num_groups, long per_expert, void* planes,
                                cudaStream_t stream);
// The kernels below also zero `num_flags` flags (for GEMMs that follow in the stream).
// planes of token rows [rows_cap, width] grouped by expert.
cudaError_t launch_split_rows(const float* src, const int* offs, int num_groups, long rows_cap, int width, void* planes,
                              int* flags, int num_flags, cudaStream_t stream);
// planes of src[s / k] in the row of slot s, for all kept slots.
cudaError_t launch_split_scatter(const float* src, const int64_t* idx, const int* rank, const int* offs, int num_groups,
                                 long n_slots, int k, int width, void* planes, int* flags, int num_flags,
                                 cudaStream_t stream);
// Backward of the weighted combine: planes of score[s] * dout[s / k] in the row of slot s, and
// dscore[s] = <dout[s / k], rows[offs[e] + rank[s]]>.
cudaError_t launch_split_combine_bwd(const float* dout, const float* rows, const int64_t* idx, const int* rank,
                                     const int* offs, const float* score, int num_groups, long n_slots, int k, int width,
                                     void* planes, float* dscore, int* flags, int num_flags, cudaStream_t stream);
// out[t] = sum over the slots of token t of weight[s] * rows[offs[e] + rank[s]] (weights null: 1), and
// its backward: drows[offs[e] + rank[s]] = score[s] * dout[s / k], dscore as above.
cudaError_t launch_combine_f32(const float* rows, const int64_t* idx, const int* rank, const int* offs,
                               const float* weight, long n_tokens, int k, int width, float* out, cudaStream_t stream);
cudaError_t launch_combine_bwd_f32(const float* dout, const float* rows, const int64_t* idx, const int* rank,
                                   const int* offs, const float* score, long n_slots, int k, int width, float* drows,
                                   float* dscore, cudaStream_t stream);

}  // namespace fmoe
