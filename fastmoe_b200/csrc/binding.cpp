// Python bindings of the native extension.
//
// The reference exposes 13 functions from one pybind module (cuda/fmoe_cuda.cpp:104-125).
// Their counterparts are bound here under the same names where the calling convention could
// be kept (expert_count, assign_pos, limit_by_capacity, prune_gate_by_capacity); the rest of
// the surface is the device-count-driven API the fused layer uses (route, grouped_gemm,
// scatter_rows, gather_combine, combine_bwd, colsum, gate_topk_softmax, ...).  Errors raise
// Python exceptions; nothing calls exit().
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/extension.h>

#include <atomic>
#include <map>
#include <mutex>

#include "cpu/cpu_ops.h"
#include "sm100/grouped_gemm.cuh"
#include "sm100/routing.cuh"
#include "sm100/split_gemm.cuh"
#include "sm100/tile_walk.cuh"
#include "sm100/p2p.cuh"

namespace {

#define FMOE_CUDA_CHECK(expr)                                                       \
  do {                                                                              \
    cudaError_t _e = (expr);                                                        \
    TORCH_CHECK(_e == cudaSuccess, "fastmoe_b200: ", #expr, " failed: ",            \
                cudaGetErrorString(_e));                                            \
  } while (0)

// Number of kernels of this library launched by this process (benchmarks report it).
std::atomic<int64_t> g_launches{0};

}  // namespace

// Called by the exchange bindings (other translation unit) for every kernel they launch.
void fmoe_count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

namespace {

cudaStream_t cur_stream() {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return at::cuda::getCurrentCUDAStream().stream();
}

int dtype16(const torch::Tensor& t) {
  if (t.scalar_type() == torch::kBFloat16) return fmoe::kBF16;
  TORCH_CHECK(t.scalar_type() == torch::kHalf, "expected a bf16 or fp16 tensor");
  return fmoe::kF16;
}

int elem_code(const torch::Tensor& t) {
  switch (t.scalar_type()) {
    case torch::kBFloat16: return 0;
    case torch::kHalf: return 1;
    case torch::kFloat: return 2;
    case torch::kDouble: return 3;
    default: TORCH_CHECK(false, "unsupported dtype for the grouped GEMM"); return -1;
  }
}

void check_cuda_contig(const torch::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
}

// For kernels that read or write rows 16 bytes at a time: a contiguous view into a flat buffer may
// start anywhere.
void check_rows(const torch::Tensor& t, const char* name) {
  check_cuda_contig(t, name);
  TORCH_CHECK(reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0, name, " must be 16-byte aligned");
}

// One int32 status word per device; kernels write a non-zero code when a bounded wait ran out.
std::mutex g_status_mu;
std::map<int, torch::Tensor> g_status;

torch::Tensor status_tensor(int device) {
  std::lock_guard<std::mutex> lock(g_status_mu);
  auto it = g_status.find(device);
  if (it != g_status.end()) return it->second;
  auto t = torch::zeros({4}, torch::dtype(torch::kInt32).device(torch::kCUDA, device));
  g_status[device] = t;
  return t;
}

int num_sms(int device) {
  static std::map<int, int> cache;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(device);
  if (it != cache.end()) return it->second;
  int n = 148;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
  cache[device] = n;
  return n;
}

// ------------------------------------------------------------------------------ routing
std::vector<torch::Tensor> route(torch::Tensor idx, int64_t tot, bool want_offs, bool want_pos = false) {
  check_cuda_contig(idx, "idx");
  TORCH_CHECK(idx.scalar_type() == torch::kLong, "idx must be int64");
  c10::cuda::CUDAGuard guard(idx.device());
  const int n_slots = static_cast<int>(idx.numel());
  auto opt = torch::dtype(torch::kInt32).device(idx.device());
  auto counts = torch::empty({tot}, opt);
  auto rank = torch::empty({n_slots}, opt);
  torch::Tensor offs;
  int* offs_ptr = nullptr;
  if (want_offs || want_pos) {
    offs = torch::empty({tot + 1}, opt);
    offs_ptr = offs.data_ptr<int>();
  }
  torch::Tensor pos;
  int* pos_ptr = nullptr;
  if (want_pos) {
    pos = torch::empty({n_slots > 0 ? n_slots : 1}, opt);
    pos_ptr = pos.data_ptr<int>();
  }
  torch::Tensor part;
  int* part_ptr = nullptr;
  const int nb = fmoe::route_blocks(n_slots, static_cast<int>(tot));
  if (nb > 1) {
    part = torch::empty({static_cast<int64_t>(nb) * tot}, opt);
    part_ptr = part.data_ptr<int>();
    g_launches.fetch_add(1, std::memory_order_relaxed);  // the second launch of the pair
  }
  FMOE_CUDA_CHECK(fmoe::launch_route(idx.data_ptr<int64_t>(), n_slots, static_cast<int>(tot),
                                     counts.data_ptr<int>(), rank.data_ptr<int>(), offs_ptr,
                                     pos_ptr, part_ptr, cur_stream()));
  if (want_pos) return {counts, rank, offs, pos};
  if (want_offs) return {counts, rank, offs};
  return {counts, rank};
}

void expert_count(torch::Tensor idx, torch::Tensor counts_inout) {
  auto res = route(idx.contiguous().view({-1}), counts_inout.numel(), false);
  counts_inout.add_(res[0]);
}

void assign_pos(torch::Tensor cum_count, torch::Tensor idx, torch::Tensor pos) {
  check_cuda_contig(cum_count, "cum_count");
  check_cuda_contig(pos, "pos");
  auto flat = idx.contiguous().view({-1});
  const int tot = static_cast<int>(cum_count.numel());
  auto res = route(flat, tot, false);
  c10::cuda::CUDAGuard guard(idx.device());
  FMOE_CUDA_CHECK(fmoe::launch_fill_pos(flat.data_ptr<int64_t>(), res[1].data_ptr<int>(),
                                        cum_count.data_ptr<int>(), static_cast<int>(flat.numel()),
                                        tot, pos.data_ptr<int64_t>(), cur_stream()));
}

torch::Tensor limit_by_capacity(torch::Tensor ec, torch::Tensor cap, int64_t n_expert,
                                int64_t n_worker) {
  check_cuda_contig(ec, "expert_count");
  check_cuda_contig(cap, "capacity");
  TORCH_CHECK(ec.scalar_type() == torch::kLong && cap.scalar_type() == torch::kInt,
              "limit_by_capacity: expert_count int64, capacity int32");
  c10::cuda::CUDAGuard guard(ec.device());
  auto eca = torch::empty_like(ec);
  FMOE_CUDA_CHECK(fmoe::launch_limit_by_capacity(ec.data_ptr<int64_t>(), cap.data_ptr<int>(),
                                                 eca.data_ptr<int64_t>(), static_cast<int>(n_expert),
                                                 static_cast<int>(n_worker), cur_stream()));
  return eca;
}

torch::Tensor prune_gate_by_capacity(torch::Tensor idx, torch::Tensor cap, int64_t n_expert,
                                     int64_t n_worker) {
  check_cuda_contig(idx, "gate_idx");
  check_cuda_contig(cap, "expert_count");
  TORCH_CHECK(cap.scalar_type() == torch::kInt, "prune_gate_by_capacity: capacity must be int32");
  const int tot = static_cast<int>(n_expert * n_worker);
  auto flat = idx.view({-1});
  auto res = route(flat, tot, false);
  c10::cuda::CUDAGuard guard(idx.device());
  auto out = torch::empty_like(idx);
  FMOE_CUDA_CHECK(fmoe::launch_prune(flat.data_ptr<int64_t>(), res[1].data_ptr<int>(),
                                     cap.data_ptr<int>(), static_cast<int>(flat.numel()), tot,
                                     out.data_ptr<int64_t>(), cur_stream()));
  cap.sub_(res[0]);
  return out;
}

// SWIPE on the device: balanced ids of one choice column from the quota the exchange kernel
// computed.  No count reaches the host.
torch::Tensor swipe_reassign(torch::Tensor idx, torch::Tensor quota, int64_t n_expert, int64_t bias) {
  check_cuda_contig(idx, "idx");
  check_cuda_contig(quota, "quota");
  TORCH_CHECK(idx.scalar_type() == torch::kLong && quota.scalar_type() == torch::kInt,
              "swipe_reassign: int64 ids, int32 quota");
  c10::cuda::CUDAGuard guard(idx.device());
  const int n = static_cast<int>(idx.numel());
  const int n_worker = static_cast<int>(quota.numel());
  auto worker = torch::div(idx, n_expert, "floor");
  auto r1 = route(worker.contiguous(), n_worker, false);          // counts per worker, slot ranks
  auto key = torch::empty_like(idx);
  FMOE_CUDA_CHECK(fmoe::launch_swipe_mark(idx.data_ptr<int64_t>(), r1[1].data_ptr<int>(),
                                          quota.data_ptr<int>(), n, static_cast<int>(n_expert),
                                          n_worker, key.data_ptr<int64_t>(), cur_stream()));
  auto r2 = route(key, 1, false);                                  // ordinal among the moved tokens
  auto out = torch::empty_like(idx);
  FMOE_CUDA_CHECK(fmoe::launch_swipe_assign(idx.data_ptr<int64_t>(), key.data_ptr<int64_t>(),
                                            r2[1].data_ptr<int>(), r1[0].data_ptr<int>(),
                                            quota.data_ptr<int>(), n, static_cast<int>(n_expert),
                                            n_worker, static_cast<int>(bias),
                                            out.data_ptr<int64_t>(), cur_stream()));
  return out;
}

// ------------------------------------------------------------------------------ grouped GEMM
// Generic entry: see sm100/grouped_gemm.cuh for the meaning of mode / act / epi.  Without `offs`
// there is one group, which all rows belong to.
void grouped_gemm(int64_t mode, torch::Tensor a, torch::Tensor b, c10::optional<torch::Tensor> offs,
                  torch::Tensor out, c10::optional<torch::Tensor> bias,
                  c10::optional<torch::Tensor> pre_out, c10::optional<torch::Tensor> aux,
                  int64_t act, int64_t epi, bool accumulate,
                  c10::optional<torch::Tensor> psum) {
  check_cuda_contig(a, "a");
  check_cuda_contig(b, "b");
  check_cuda_contig(out, "out");
  if (offs.has_value()) {
    check_cuda_contig(*offs, "offs");
    TORCH_CHECK(offs->scalar_type() == torch::kInt, "offs must be int32");
  }
  c10::cuda::CUDAGuard guard(a.device());
  fmoe::GroupedGemmArgs g;
  g.mode = static_cast<int>(mode);
  g.dtype = dtype16(a);
  TORCH_CHECK(b.scalar_type() == a.scalar_type(), "operand dtypes differ");
  g.num_groups = offs.has_value() ? static_cast<int>(offs->numel() - 1) : 1;
  g.rows_cap = a.size(0);
  if (mode == fmoe::kWgrad) {
    // a = P [rows, m], b = Q [rows, n], out [G, m, n]
    TORCH_CHECK(b.size(0) == a.size(0), "wgrad operands need the same number of rows");
    g.m = static_cast<int>(a.size(1));
    g.n = static_cast<int>(b.size(1));
    g.k = 0;
    TORCH_CHECK(out.numel() == static_cast<int64_t>(g.num_groups) * g.m * g.n, "wgrad out shape");
    g.out_fp32 = out.scalar_type() == torch::kFloat ? 1 : 0;
    TORCH_CHECK(g.out_fp32 || out.scalar_type() == a.scalar_type(), "wgrad out dtype");
  } else {
    g.k = static_cast<int>(a.size(1));
    if (mode == fmoe::kRowsNT) {
      TORCH_CHECK(b.dim() == 3 && b.size(2) == g.k, "weight must be [G, n, k]");
      g.n = static_cast<int>(b.size(1));
    } else {
      TORCH_CHECK(b.dim() == 3 && b.size(1) == g.k, "weight must be [G, k, n]");
      g.n = static_cast<int>(b.size(2));
    }
    TORCH_CHECK(b.size(0) == g.num_groups, "weight group count");
    TORCH_CHECK(out.size(0) == a.size(0) && out.size(1) == g.n, "out shape");
    TORCH_CHECK(out.scalar_type() == a.scalar_type(), "out dtype");
  }
  auto aligned32 = [](const torch::Tensor& t) {
    return reinterpret_cast<uintptr_t>(t.data_ptr()) % 32 == 0;
  };
  TORCH_CHECK(aligned32(a) && aligned32(b) && aligned32(out),
              "grouped_gemm: operands must be 32-byte aligned");
  g.a = a.data_ptr();
  g.b = b.data_ptr();
  g.offs = offs.has_value() ? offs->data_ptr<int>() : nullptr;
  g.out = out.data_ptr();
  if (bias.has_value() && bias->defined()) {
    check_cuda_contig(*bias, "bias");
    TORCH_CHECK(bias->scalar_type() == a.scalar_type(), "bias dtype");
    TORCH_CHECK(aligned32(*bias), "grouped_gemm: bias must be 32-byte aligned");
    g.bias = bias->data_ptr();
  }
  // The pre-activation (written as pre_out, read back as aux) is tile-blocked: one 128 x 256
  // block per output tile, (ceil(rows / 128) + groups) * ceil(n / 256) blocks at most.
  const int64_t pre_elems = mode == fmoe::kWgrad ? 0
      : ((a.size(0) + 127) / 128 + g.num_groups) * ((g.n + 255) / 256) * (128 * 256);
  if (pre_out.has_value() && pre_out->defined()) {
    check_cuda_contig(*pre_out, "pre_out");
    TORCH_CHECK(aligned32(*pre_out) && pre_out->numel() >= pre_elems &&
                    pre_out->scalar_type() == a.scalar_type(),
                "grouped_gemm: pre_out must be a 32-byte aligned tile-blocked buffer of ", pre_elems,
                " elements");
    g.pre_out = pre_out->data_ptr();
  }
  if (aux.has_value() && aux->defined()) {
    check_cuda_contig(*aux, "aux");
    TORCH_CHECK(aligned32(*aux) && aux->numel() >= pre_elems && aux->scalar_type() == a.scalar_type(),
                "grouped_gemm: aux must be a 32-byte aligned tile-blocked buffer of ", pre_elems,
                " elements");
    g.aux = aux->data_ptr();
  }
  if (psum.has_value() && psum->defined()) {
    TORCH_CHECK(mode == fmoe::kWgrad, "psum is an output of the weight-gradient mode");
    check_cuda_contig(*psum, "psum");
    TORCH_CHECK(psum->scalar_type() == a.scalar_type() &&
                    psum->numel() == static_cast<int64_t>(g.num_groups) * g.m,
                "psum must be [groups, m] in the operands' dtype");
    TORCH_CHECK(reinterpret_cast<uintptr_t>(psum->data_ptr()) % 16 == 0, "psum must be 16-byte aligned");
    g.psum = psum->data_ptr();
  }
  g.act = static_cast<int>(act);
  g.epi = static_cast<int>(epi);
  g.accumulate = accumulate ? 1 : 0;
  g.status = status_tensor(a.device().index()).data_ptr<int>();
  g.num_sms = num_sms(a.device().index());
  g.stream = cur_stream();
  TORCH_CHECK(fmoe::grouped_gemm_supported(g.mode, g.m, g.n, g.k, g.num_groups),
              "grouped_gemm: shape not supported by the tcgen05 kernel (m=", g.m, " n=", g.n,
              " k=", g.k, " groups=", g.num_groups, ")");
  FMOE_CUDA_CHECK(fmoe::launch_grouped_gemm(g));
}

bool grouped_gemm_supported(int64_t mode, int64_t m, int64_t n, int64_t k, int64_t groups) {
  return fmoe::grouped_gemm_supported(static_cast<int>(mode), static_cast<int>(m),
                                      static_cast<int>(n), static_cast<int>(k),
                                      static_cast<int>(groups));
}

// Whether the weight-gradient mode of simt_grouped_gemm can return the column sums of `a` too.
bool simt_column_sums(const torch::Tensor& a, const torch::Tensor& b, const torch::Tensor& out) {
  return a.scalar_type() == torch::kFloat && a.is_contiguous() && b.is_contiguous() && out.is_contiguous() &&
         fmoe::sgemm_applies(fmoe::kWgrad, static_cast<int>(out.size(0)), static_cast<int>(a.size(1)),
                             static_cast<int>(b.size(1)), 0, a.data_ptr(), b.data_ptr(), nullptr, out.data_ptr());
}

void simt_grouped_gemm(int64_t mode, torch::Tensor a, torch::Tensor b, torch::Tensor offs,
                       torch::Tensor out, c10::optional<torch::Tensor> bias,
                       c10::optional<torch::Tensor> psum) {
  check_cuda_contig(a, "a");
  check_cuda_contig(b, "b");
  check_cuda_contig(out, "out");
  c10::cuda::CUDAGuard guard(a.device());
  const int groups = static_cast<int>(offs.numel() - 1);
  int m = 0, n = 0, k = 0;
  if (mode == fmoe::kWgrad) {
    m = static_cast<int>(a.size(1));
    n = static_cast<int>(b.size(1));
  } else {
    k = static_cast<int>(a.size(1));
    n = static_cast<int>(mode == fmoe::kRowsNT ? b.size(1) : b.size(2));
  }
  const void* bias_ptr = nullptr;
  if (bias.has_value() && bias->defined()) bias_ptr = bias->data_ptr();
  if (psum.has_value() && psum->defined()) {
    // the column sums of `a` come with the fp32 kernel: the caller asked simt_column_sums first
    check_cuda_contig(*psum, "psum");
    TORCH_CHECK(mode == fmoe::kWgrad && psum->scalar_type() == torch::kFloat &&
                    psum->numel() == static_cast<int64_t>(groups) * m && simt_column_sums(a, b, out),
                "simt_grouped_gemm: no column sums for these operands");
    FMOE_CUDA_CHECK(fmoe::launch_sgemm(static_cast<int>(mode), groups, a.size(0), m, n, k, a.data_ptr<float>(),
                                       b.data_ptr<float>(), offs.data_ptr<int>(), nullptr,
                                       out.data_ptr<float>(), psum->data_ptr<float>(), cur_stream()));
    return;
  }
  FMOE_CUDA_CHECK(fmoe::launch_simt_grouped_gemm(static_cast<int>(mode), elem_code(a), groups,
                                                 a.size(0), m, n, k, a.data_ptr(), b.data_ptr(),
                                                 offs.data_ptr<int>(), bias_ptr, out.data_ptr(),
                                                 cur_stream()));
}

// ------------------------------------------------------------------------------ fp32 on the tensor cores
torch::Tensor plane_rows(long rows, int64_t groups, int64_t width, const torch::Tensor& like) {
  return torch::empty({3, fmoe::split_rows_cap(rows, static_cast<int>(groups)), width}, like.options().dtype(torch::kBFloat16));
}

torch::Tensor split_weight(const torch::Tensor& w, const torch::Tensor& offs) {
  auto planes = torch::empty({3, w.numel()}, w.options().dtype(torch::kBFloat16));
  FMOE_CUDA_CHECK(fmoe::launch_split_weight(w.data_ptr<float>(), offs.data_ptr<int>(), static_cast<int>(w.size(0)),
                                            w.numel() / w.size(0), planes.data_ptr(), cur_stream()));
  return planes;
}

// Scratch of split GEMMs that follow one another in a stream; its flags are zeroed by the kernel
// that splits the token rows before them.  `sums_of`: the widths whose column sums are wanted.
struct SplitScratch {
  torch::Tensor work, flags, sums;
  int per_gemm, gemms, groups;
  SplitScratch(const torch::Tensor& like, int n_gemms, int64_t rows, int64_t n_groups, std::initializer_list<int64_t> sums_of)
      : gemms(n_gemms), groups(static_cast<int>(n_groups)) {
    const int sms = num_sms(like.device().index());
    per_gemm = fmoe::split_num_flags(sms);
    int64_t n = static_cast<int64_t>(gemms) * per_gemm, widest = 0;
    for (int64_t m : sums_of) {
      n += fmoe::split_num_counts(groups, static_cast<int>(m));
      widest = std::max(widest, m);
    }
    work = torch::empty({fmoe::split_work_floats(sms)}, like.options().dtype(torch::kFloat));
    flags = torch::empty({n}, like.options().dtype(torch::kInt));
    if (widest > 0) {
      sums = torch::empty({fmoe::split_sum_floats(rows, groups, static_cast<int>(widest))}, like.options().dtype(torch::kFloat));
    }
    next_count = flags.data_ptr<int>() + static_cast<int64_t>(gemms) * per_gemm;
  }
  int* all() { return flags.data_ptr<int>(); }
  int count() { return static_cast<int>(flags.numel()); }
  void give(fmoe::SplitGemmArgs& g) {
    g.work = work.data_ptr<float>();
    g.flags = all() + (given++) * per_gemm;
  }
  void give_sums(fmoe::SplitGemmArgs& g, float* psum) {
    g.psum = psum;
    g.sums = sums.data_ptr<float>();
    g.sum_counts = next_count;
    next_count += fmoe::split_num_counts(groups, g.m);
  }

 private:
  int given = 0;
  int* next_count;
};

torch::Tensor split_token_rows(const torch::Tensor& x, const torch::Tensor& offs, SplitScratch* scratch) {
  const int groups = static_cast<int>(offs.numel() - 1);
  auto planes = plane_rows(x.size(0), groups, x.size(1), x);
  FMOE_CUDA_CHECK(fmoe::launch_split_rows(x.data_ptr<float>(), offs.data_ptr<int>(), groups, x.size(0),
                                          static_cast<int>(x.size(1)), planes.data_ptr(),
                                          scratch != nullptr ? scratch->all() : nullptr,
                                          scratch != nullptr ? scratch->count() : 0, cur_stream()));
  return planes;
}

fmoe::SplitGemmArgs split_args(int64_t mode, int64_t rows, int64_t m, int64_t n, int64_t k, const torch::Tensor& a,
                               const torch::Tensor& b, const torch::Tensor& offs) {
  fmoe::SplitGemmArgs g;
  g.mode = static_cast<int>(mode);
  g.num_groups = static_cast<int>(offs.numel() - 1);
  g.rows_cap = rows;
  g.m = static_cast<int>(m);
  g.n = static_cast<int>(n);
  g.k = static_cast<int>(k);
  g.a = a.data_ptr();
  g.b = b.data_ptr();
  g.offs = offs.data_ptr<int>();
  g.status = status_tensor(a.device().index()).data_ptr<int>();
  g.num_sms = num_sms(a.device().index());
  g.stream = cur_stream();
  return g;
}

struct GemmSizes {
  int groups, m, n, k;
};
GemmSizes gemm_sizes(int64_t mode, const torch::Tensor& a, const torch::Tensor& b, const torch::Tensor& offs) {
  const int groups = static_cast<int>(offs.numel() - 1), inner = static_cast<int>(a.size(1));
  if (mode == fmoe::kWgrad) return {groups, inner, static_cast<int>(b.size(1)), 0};
  return {groups, 0, static_cast<int>(mode == fmoe::kRowsNT ? b.size(1) : b.size(2)), inner};
}

// The three products of a grouped linear in fp32, each operand split by a launch of its own.
void split_grouped_gemm(int64_t mode, torch::Tensor a, torch::Tensor b, torch::Tensor offs, torch::Tensor out,
                        c10::optional<torch::Tensor> bias, c10::optional<torch::Tensor> psum) {
  const GemmSizes z = gemm_sizes(mode, a, b, offs);
  for (const auto& t : {a, b, out}) {
    check_rows(t, "operand");
    TORCH_CHECK(t.scalar_type() == torch::kFloat, "split_grouped_gemm: fp32 operands");
  }
  TORCH_CHECK(reinterpret_cast<uintptr_t>(out.data_ptr()) % 32 == 0, "split_grouped_gemm: out must be 32-byte aligned");
  TORCH_CHECK(fmoe::split_gemm_supported(static_cast<int>(mode), z.m, z.n, z.k, z.groups, a.size(0)),
              "split_grouped_gemm: shape not supported");
  c10::cuda::CUDAGuard guard(a.device());
  const bool sums = psum.has_value() && psum->defined();
  SplitScratch scratch = sums ? SplitScratch(a, 1, a.size(0), z.groups, {z.m}) : SplitScratch(a, 1, a.size(0), z.groups, {});
  const torch::Tensor pa = split_token_rows(a, offs, &scratch);
  const torch::Tensor pb = mode == fmoe::kWgrad ? split_token_rows(b, offs, nullptr) : split_weight(b, offs);
  auto g = split_args(mode, a.size(0), z.m, z.n, z.k, pa, pb, offs);
  scratch.give(g);
  g.out = out.data_ptr<float>();
  if (bias.has_value() && bias->defined()) {
    check_rows(*bias, "bias");
    g.bias = bias->data_ptr<float>();
  }
  if (sums) {
    check_rows(*psum, "psum");
    scratch.give_sums(g, psum->data_ptr<float>());
  }
  FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
}

// When one product by itself is faster split than on the FMA units.  Those take the larger of the operations
// at 47 TFLOP/s and their serial chain (one sum over k, or over an expert's rows: 0.066 us per element).
// Split, the operands are read and written first (16 bytes an element in all), the weight gradient is stored
// by few tiles, and the chain is short.  Taken where the estimate is 25 us lower, which is what issuing the
// other launches costs an eager program (8 experts, 277 rows each, 160 -> 320, eager, forward and backward:
// 203 us split, 183 not).  us measured, split against FMA, forward / input gradient / weight gradient: 8
// experts, 512 rows each, 512 -> 2048: 94, 113, 108 against 203, 220, 177; 16 experts, 64 rows each: 92, 110,
// 74 against 83, 152, 54; 8 experts, 128 rows each, 128 -> 512: 17, 26, 27 against 12, 37, 12; 4 experts,
// 7500 rows each, 64 -> 64: 20, 17, 43 against 17, 15, 544.
bool split_worth_it(int64_t mode, int64_t rows, const GemmSizes& z) {
  const bool wgrad = mode == fmoe::kWgrad;
  const double r = static_cast<double>(rows), n = z.n, k = wgrad ? z.m : z.k, weights = n * k * z.groups;
  const double flops = 2 * r * n * k, chain = wgrad ? r / z.groups : k;
  const double fma = 4 + std::max(0.066 * chain, flops / 47e6);
  const double split = 14 + ((wgrad ? 8 : 16) * weights + 16 * r * (wgrad ? n + k : k)) / 6.5e6 + 6 * flops / 1.1e9;
  return split + 25 < fma;
}

// fp32, fp64 and what the 16-bit tensor-core kernel does not take.
void wide_grouped_gemm(int64_t mode, torch::Tensor a, torch::Tensor b, torch::Tensor offs, torch::Tensor out,
                       c10::optional<torch::Tensor> bias, c10::optional<torch::Tensor> psum) {
  const GemmSizes z = gemm_sizes(mode, a, b, offs);
  auto usable = [](const torch::Tensor& t) {
    return t.scalar_type() == torch::kFloat && t.is_cuda() && t.is_contiguous() &&
           reinterpret_cast<uintptr_t>(t.data_ptr()) % 32 == 0;
  };
  auto usable_or_none = [&](const c10::optional<torch::Tensor>& t) { return !t.has_value() || !t->defined() || usable(*t); };
  if (usable(a) && usable(b) && usable(out) && usable_or_none(bias) && usable_or_none(psum) &&
      fmoe::split_gemm_supported(static_cast<int>(mode), z.m, z.n, z.k, z.groups, a.size(0)) &&
      split_worth_it(mode, a.size(0), z)) {
    return split_grouped_gemm(mode, a, b, offs, out, bias, psum);
  }
  simt_grouped_gemm(mode, a, b, offs, out, bias, psum);
}

// ------------------------------------------------------------------------------ row movement
// The kernels read the tables of the slots, and a weight per slot in the type of the rows, through plain pointers.
void check_slots(const torch::Tensor& rows, int64_t tokens, int64_t k, const torch::Tensor& idx, const torch::Tensor& rank,
                 const torch::Tensor& base) {
  for (const auto& t : {idx, rank, base}) {
    check_cuda_contig(t, "slot table");
    TORCH_CHECK(t.device() == rows.device(), "slot table on another device than the rows");
  }
  TORCH_CHECK(rows.dim() == 2 && k > 0 && idx.numel() == tokens * k && rank.numel() == idx.numel(), "slot tables do not fit the rows");
}
void check_weight(const torch::Tensor& rows, const torch::Tensor& idx, const torch::Tensor& weight) {
  check_cuda_contig(weight, "slot weights");
  TORCH_CHECK(weight.device() == rows.device() && weight.scalar_type() == rows.scalar_type() && weight.numel() == idx.numel(),
              "slot weights: one per slot, in the type of the rows");
}
const void* weight_ptr(const torch::Tensor& rows, const torch::Tensor& idx, const c10::optional<torch::Tensor>& weight) {
  if (!weight.has_value() || !weight->defined()) return nullptr;
  check_weight(rows, idx, *weight);
  return weight->data_ptr();
}

void scatter_rows(torch::Tensor src, torch::Tensor idx, torch::Tensor rank, torch::Tensor base,
                  c10::optional<torch::Tensor> scale, int64_t k, torch::Tensor dst,
                  c10::optional<torch::Tensor> row_slot) {
  check_rows(src, "src");
  check_rows(dst, "dst");
  c10::cuda::CUDAGuard guard(src.device());
  check_slots(src, src.size(0), k, idx, rank, base);
  const void* sc = weight_ptr(src, idx, scale);
  int* rs = (row_slot.has_value() && row_slot->defined()) ? row_slot->data_ptr<int>() : nullptr;
  // unscaled fp32 rows are moved as 16-bit rows of twice the width
  const bool wide = src.scalar_type() == torch::kFloat;
  TORCH_CHECK(!wide || sc == nullptr, "scatter_rows: only 16-bit rows are scaled");
  FMOE_CUDA_CHECK(fmoe::launch_scatter_rows(wide ? fmoe::kBF16 : dtype16(src), src.data_ptr(), idx.data_ptr<int64_t>(),
                                            rank.data_ptr<int>(), base.data_ptr<int>(), sc,
                                            static_cast<int>(idx.numel()), static_cast<int>(k),
                                            static_cast<int>(src.size(1)) * (wide ? 2 : 1), dst.data_ptr(), rs,
                                            cur_stream()));
}

void gather_combine(torch::Tensor rows, torch::Tensor idx, torch::Tensor rank, torch::Tensor base,
                    c10::optional<torch::Tensor> weight, int64_t k, torch::Tensor out) {
  check_rows(rows, "rows");
  check_rows(out, "out");
  c10::cuda::CUDAGuard guard(rows.device());
  check_slots(rows, out.size(0), k, idx, rank, base);
  const void* w = weight_ptr(rows, idx, weight);
  if (rows.scalar_type() == torch::kFloat) {
    TORCH_CHECK(rows.size(1) % 8 == 0, "fp32 rows of a multiple of 8 columns");
    FMOE_CUDA_CHECK(fmoe::launch_combine_f32(rows.data_ptr<float>(), idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                             base.data_ptr<int>(), static_cast<const float*>(w), out.size(0),
                                             static_cast<int>(k), static_cast<int>(rows.size(1)), out.data_ptr<float>(),
                                             cur_stream()));
    return;
  }
  FMOE_CUDA_CHECK(fmoe::launch_gather_combine(dtype16(rows), rows.data_ptr(),
                                              idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                              base.data_ptr<int>(), w,
                                              static_cast<int>(out.size(0)), static_cast<int>(k),
                                              static_cast<int>(rows.size(1)), out.data_ptr(),
                                              cur_stream()));
}

void combine_bwd(torch::Tensor dout, torch::Tensor rows, torch::Tensor idx, torch::Tensor rank,
                 torch::Tensor base, torch::Tensor weight, int64_t k, torch::Tensor drows,
                 torch::Tensor dscore) {
  check_rows(dout, "dout");
  check_rows(rows, "rows");
  check_rows(drows, "drows");
  c10::cuda::CUDAGuard guard(dout.device());
  check_slots(rows, dout.size(0), k, idx, rank, base);
  check_weight(rows, idx, weight);
  check_weight(rows, idx, dscore);
  if (dout.scalar_type() == torch::kFloat) {
    TORCH_CHECK(dout.size(1) % 8 == 0, "fp32 rows of a multiple of 8 columns");
    FMOE_CUDA_CHECK(fmoe::launch_combine_bwd_f32(dout.data_ptr<float>(), rows.data_ptr<float>(), idx.data_ptr<int64_t>(),
                                                 rank.data_ptr<int>(), base.data_ptr<int>(), weight.data_ptr<float>(),
                                                 idx.numel(), static_cast<int>(k), static_cast<int>(dout.size(1)),
                                                 drows.data_ptr<float>(), dscore.data_ptr<float>(), cur_stream()));
    return;
  }
  FMOE_CUDA_CHECK(fmoe::launch_combine_bwd(dtype16(dout), dout.data_ptr(), rows.data_ptr(),
                                           idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                           base.data_ptr<int>(), weight.data_ptr(),
                                           static_cast<int>(dout.size(0)), static_cast<int>(k),
                                           static_cast<int>(dout.size(1)), drows.data_ptr(),
                                           dscore.data_ptr(), cur_stream()));
}

// ------------------------------------------------------------------------------ whole layer
// One GPU, both expert linears with a fused activation: the launches of a layer's forward, and of
// its backward, issued by one call each.  For a small layer the calls from Python between the
// kernels, and not the kernels, were what a training step waited for.
torch::Tensor aligned(const torch::Tensor& t, uintptr_t bytes) {
  torch::Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % bytes == 0 ? c : c.clone();
}
torch::Tensor aligned32(const torch::Tensor& t) { return aligned(t, 32); }

bool moe_mlp_supported(int64_t experts, int64_t d, int64_t h) {
  const int g = static_cast<int>(experts), id = static_cast<int>(d), ih = static_cast<int>(h);
  return d % 64 == 0 && h % 64 == 0 && fmoe::grouped_gemm_supported(fmoe::kRowsNT, 0, ih, id, g) &&
         fmoe::grouped_gemm_supported(fmoe::kRowsNT, 0, id, ih, g);
}

// Whether the fp32 layer runs on the tensor cores: `rows` are tokens times choices.  What it replaces,
// the general path with its host read and three dozen launches, takes about 0.7 ms of host time, as
// long as splitting 280 M weights, so only a layer of many weights needs rows to be worth it.
bool moe_mlp_supported_f32(int64_t experts, int64_t d, int64_t h, int64_t rows) {
  const int g = static_cast<int>(experts), id = static_cast<int>(d), ih = static_cast<int>(h);
  return fmoe::split_gemm_supported(fmoe::kRowsNT, 0, ih, id, g, rows) &&
         fmoe::split_gemm_supported(fmoe::kRowsNT, 0, id, ih, g, rows) &&
         (rows >= 64 * experts || 2 * experts * d * h <= 80000000);
}

// As moe_mlp_forward for fp32: xs and a are planes.
std::vector<torch::Tensor> moe_mlp_forward_f32(const torch::Tensor& x, const torch::Tensor& idx, const torch::Tensor& score,
                                               const torch::Tensor& w1, const torch::Tensor& b1, const torch::Tensor& w2,
                                               const torch::Tensor& b2, int64_t act, bool keep) {
  const int64_t groups = w1.size(0), h = w1.size(1), d = w1.size(2), rows = idx.numel(), k = rows / x.size(0);
  auto r = route(idx, groups, true);
  const torch::Tensor rank = r[1], offs = r[2];
  auto xs = plane_rows(rows, groups, d, x);
  SplitScratch scratch(x, 2, rows, groups, {});
  FMOE_CUDA_CHECK(fmoe::launch_split_scatter(x.data_ptr<float>(), idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                             offs.data_ptr<int>(), static_cast<int>(groups), rows, static_cast<int>(k),
                                             static_cast<int>(d), xs.data_ptr(), scratch.all(), scratch.count(), cur_stream()));
  auto a = plane_rows(rows, groups, h, x);
  torch::Tensor pre;
  if (keep && act != fmoe::kActNone) pre = torch::empty({rows, h}, x.options());
  {
    const torch::Tensor planes = split_weight(w1, offs);
    auto g = split_args(fmoe::kRowsNT, rows, 0, h, d, xs, planes, offs);
    scratch.give(g);
    g.kind = fmoe::kSplitAct;
    g.act = static_cast<int>(act);
    g.bias = b1.data_ptr<float>();
    g.planes = a.data_ptr();
    g.pre = pre.defined() ? pre.data_ptr<float>() : nullptr;
    FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
  }
  auto ys = torch::empty({rows, d}, x.options());
  {
    const torch::Tensor planes = split_weight(w2, offs);
    auto g = split_args(fmoe::kRowsNT, rows, 0, d, h, a, planes, offs);
    scratch.give(g);
    g.bias = b2.data_ptr<float>();
    g.out = ys.data_ptr<float>();
    FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
  }
  auto out = torch::empty_like(x);
  FMOE_CUDA_CHECK(fmoe::launch_combine_f32(ys.data_ptr<float>(), idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                           offs.data_ptr<int>(), score.data_ptr<float>(), x.size(0),
                                           static_cast<int>(k), static_cast<int>(d), out.data_ptr<float>(), cur_stream()));
  return {out, xs, pre, a, ys, rank, offs, score, idx};
}

std::vector<torch::Tensor> moe_mlp_backward_f32(const torch::Tensor& dout, const torch::Tensor& xs,
                                                const c10::optional<torch::Tensor>& pre, const torch::Tensor& a,
                                                const torch::Tensor& ys, const torch::Tensor& rank, const torch::Tensor& offs,
                                                const torch::Tensor& score, const torch::Tensor& idx, const torch::Tensor& w1,
                                                const torch::Tensor& w2, int64_t act, bool need_dx, bool need_w1, bool need_w2) {
  const int64_t groups = w1.size(0), h = w1.size(1), d = w1.size(2), n_tok = dout.size(0), rows = idx.numel(), k = rows / n_tok;
  auto dys = plane_rows(rows, groups, d, dout);
  auto dscore = torch::empty_like(score);
  SplitScratch scratch(dout, 4, rows, groups, {d, h});
  FMOE_CUDA_CHECK(fmoe::launch_split_combine_bwd(dout.data_ptr<float>(), ys.data_ptr<float>(), idx.data_ptr<int64_t>(),
                                                 rank.data_ptr<int>(), offs.data_ptr<int>(), score.data_ptr<float>(),
                                                 static_cast<int>(groups), rows, static_cast<int>(k), static_cast<int>(d),
                                                 dys.data_ptr(), dscore.data_ptr<float>(), scratch.all(),
                                                 scratch.count(), cur_stream()));
  auto wgrad = [&](const torch::Tensor& p, const torch::Tensor& q, int64_t m, int64_t n, torch::Tensor& dw, torch::Tensor& db) {
    dw = torch::empty({groups, m, n}, dout.options());
    db = torch::empty({groups, m}, dout.options());
    auto g = split_args(fmoe::kWgrad, rows, m, n, 0, p, q, offs);
    scratch.give(g);
    scratch.give_sums(g, db.data_ptr<float>());
    g.out = dw.data_ptr<float>();
    FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
  };
  torch::Tensor dw1, db1, dw2, db2, dx;
  if (need_w2) wgrad(dys, a, d, h, dw2, db2);
  if (need_dx || need_w1) {
    auto da = plane_rows(rows, groups, h, dout);
    {
      const torch::Tensor planes = split_weight(w2, offs);
      auto g = split_args(fmoe::kRowsNN, rows, 0, h, d, dys, planes, offs);
      scratch.give(g);
      g.kind = fmoe::kSplitDAct;
      g.act = pre.has_value() ? static_cast<int>(act) : fmoe::kActNone;
      g.planes = da.data_ptr();
      g.pre = pre.has_value() ? pre->data_ptr<float>() : nullptr;
      FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
    }
    if (need_w1) wgrad(da, xs, h, d, dw1, db1);
    if (need_dx) {
      auto dxs = torch::empty_like(ys);
      const torch::Tensor planes = split_weight(w1, offs);
      auto g = split_args(fmoe::kRowsNN, rows, 0, d, h, da, planes, offs);
      scratch.give(g);
      g.out = dxs.data_ptr<float>();
      FMOE_CUDA_CHECK(fmoe::launch_split_gemm(g));
      dx = torch::empty({n_tok, d}, dout.options());
      FMOE_CUDA_CHECK(fmoe::launch_combine_f32(dxs.data_ptr<float>(), idx.data_ptr<int64_t>(), rank.data_ptr<int>(),
                                               offs.data_ptr<int>(), nullptr, n_tok,
                                               static_cast<int>(k), static_cast<int>(d), dx.data_ptr<float>(), cur_stream()));
    }
  }
  return {dx, dscore, dw1, db1, dw2, db2};
}

// {out, xs, pre (empty when not kept), a, ys, rank, offs, score in the layer's type, idx}
std::vector<torch::Tensor> moe_mlp_forward(torch::Tensor x_in, torch::Tensor idx_in, torch::Tensor score_in,
                                           torch::Tensor w1_in, torch::Tensor b1_in, torch::Tensor w2_in,
                                           torch::Tensor b2_in, int64_t act, bool keep) {
  c10::cuda::CUDAGuard guard(x_in.device());
  TORCH_CHECK(x_in.dim() == 2 && idx_in.device() == x_in.device() && score_in.device() == x_in.device() &&
              x_in.size(0) > 0 && idx_in.numel() % x_in.size(0) == 0 && idx_in.numel() > 0 && score_in.numel() == idx_in.numel(),
              "moe_mlp: ids and scores do not fit the rows");
  const torch::Tensor x = aligned(x_in, 16);
  const torch::Tensor idx = idx_in.contiguous().view({-1});
  const torch::Tensor score = score_in.reshape({-1}).to(x.scalar_type()).contiguous();
  const torch::Tensor w1 = aligned32(w1_in), b1 = aligned32(b1_in), w2 = aligned32(w2_in), b2 = aligned32(b2_in);
  if (x.scalar_type() == torch::kFloat) return moe_mlp_forward_f32(aligned32(x), idx, score, w1, b1, w2, b2, act, keep);
  const int64_t groups = w1.size(0), h = w1.size(1), d = w1.size(2), rows = idx.numel(), k = rows / x.size(0);
  auto r = route(idx, groups, true);
  const torch::Tensor rank = r[1], offs = r[2];
  auto xs = torch::empty({rows, d}, x.options());
  scatter_rows(x, idx, rank, offs, c10::nullopt, k, xs, c10::nullopt);
  auto a = torch::empty({rows, h}, x.options());
  c10::optional<torch::Tensor> pre;
  if (keep && act != fmoe::kActNone) {
    pre = torch::empty({((rows + 127) / 128 + groups) * ((h + 255) / 256) * (128 * 256)}, x.options());
  }
  grouped_gemm(fmoe::kRowsNT, xs, w1, offs, a, b1, pre, c10::nullopt, act, fmoe::kEpiBiasAct, false, c10::nullopt);
  auto ys = torch::empty({rows, d}, x.options());
  grouped_gemm(fmoe::kRowsNT, a, w2, offs, ys, b2, c10::nullopt, c10::nullopt, fmoe::kActNone, fmoe::kEpiBiasAct,
               false, c10::nullopt);
  auto out = torch::empty_like(x);
  gather_combine(ys, idx, rank, offs, score, k, out);
  return {out, xs, pre.has_value() ? *pre : torch::Tensor(), a, ys, rank, offs, score, idx};
}

// {dx, dscore, dw1, db1, dw2, db2}; what `need_*` leaves out is empty.  Saved tensors may have been
// through hooks of the caller, which need not return them where they were.
std::vector<torch::Tensor> moe_mlp_backward(torch::Tensor dout_in, torch::Tensor xs_in, c10::optional<torch::Tensor> pre,
                                            torch::Tensor a_in, torch::Tensor ys_in, torch::Tensor rank, torch::Tensor offs,
                                            torch::Tensor score, torch::Tensor idx, torch::Tensor w1_in,
                                            torch::Tensor w2_in, int64_t act, bool need_dx, bool need_w1, bool need_w2) {
  c10::cuda::CUDAGuard guard(xs_in.device());
  const torch::Tensor dout = aligned(dout_in, 16), xs = aligned32(xs_in), a = aligned32(a_in), ys = aligned(ys_in, 16);
  if (pre.has_value()) pre = aligned32(*pre);
  const torch::Tensor w1 = aligned32(w1_in), w2 = aligned32(w2_in);
  if (ys.scalar_type() == torch::kFloat) {
    return moe_mlp_backward_f32(dout, xs, pre, a, ys, rank, offs, score, idx, w1, w2, act, need_dx, need_w1, need_w2);
  }
  const int64_t groups = w1.size(0), h = w1.size(1), d = w1.size(2), n_tok = dout.size(0), k = idx.numel() / n_tok;
  auto dys = torch::empty_like(ys);
  auto dscore = torch::empty_like(score);
  combine_bwd(dout, ys, idx, rank, offs, score, k, dys, dscore);
  torch::Tensor dw1, db1, dw2, db2, dx;
  if (need_w2) {
    dw2 = torch::empty({groups, d, h}, xs.options());
    db2 = torch::empty({groups, d}, xs.options());
    grouped_gemm(fmoe::kWgrad, dys, a, offs, dw2, c10::nullopt, c10::nullopt, c10::nullopt, 0, 0, false, db2);
  }
  if (need_dx || need_w1) {
    auto da = torch::empty_like(a);
    grouped_gemm(fmoe::kRowsNN, dys, w2, offs, da, c10::nullopt, c10::nullopt, pre, pre.has_value() ? act : 0,
                 pre.has_value() ? fmoe::kEpiDAct : fmoe::kEpiBiasAct, false, c10::nullopt);
    if (need_w1) {
      dw1 = torch::empty({groups, h, d}, xs.options());
      db1 = torch::empty({groups, h}, xs.options());
      grouped_gemm(fmoe::kWgrad, da, xs, offs, dw1, c10::nullopt, c10::nullopt, c10::nullopt, 0, 0, false, db1);
    }
    if (need_dx) {
      auto dxs = torch::empty_like(xs);
      grouped_gemm(fmoe::kRowsNN, da, w1, offs, dxs, c10::nullopt, c10::nullopt, c10::nullopt, 0, fmoe::kEpiBiasAct,
                   false, c10::nullopt);
      dx = torch::empty({n_tok, d}, xs.options());
      gather_combine(dxs, idx, rank, offs, c10::nullopt, k, dx);
    }
  }
  return {dx, dscore, dw1, db1, dw2, db2};
}

torch::Tensor colsum(torch::Tensor x, torch::Tensor offs) {
  check_rows(x, "x");
  c10::cuda::CUDAGuard guard(x.device());
  const int groups = static_cast<int>(offs.numel() - 1);
  auto out = torch::zeros({groups, x.size(1)}, torch::dtype(torch::kFloat).device(x.device()));
  FMOE_CUDA_CHECK(fmoe::launch_colsum(dtype16(x), x.data_ptr(), offs.data_ptr<int>(), groups,
                                      x.size(0), static_cast<int>(x.size(1)),
                                      out.data_ptr<float>(), cur_stream()));
  return out;
}

// ------------------------------------------------------------------------------ gate
int logit_code(const torch::Tensor& t) {
  if (t.scalar_type() == torch::kBFloat16) return 0;
  if (t.scalar_type() == torch::kHalf) return 1;
  TORCH_CHECK(t.scalar_type() == torch::kFloat, "gate logits must be bf16, fp16 or fp32");
  return 2;
}

// A one-element fp32 tensor of the caller that the kernel is to zero, or null.
float* zero_of(const c10::optional<torch::Tensor>& zero) {
  if (!zero.has_value() || !zero->defined()) return nullptr;
  TORCH_CHECK(zero->is_cuda() && zero->scalar_type() == torch::kFloat && zero->numel() == 1, "zero: one fp32 element");
  return zero->data_ptr<float>();
}

std::vector<torch::Tensor> gate_topk_softmax(torch::Tensor logits, int64_t k,
                                             c10::optional<torch::Tensor> zero = c10::nullopt) {
  check_cuda_contig(logits, "logits");
  c10::cuda::CUDAGuard guard(logits.device());
  const int rows = static_cast<int>(logits.size(0));
  const int ne = static_cast<int>(logits.size(1));
  auto idx = torch::empty({rows, k}, torch::dtype(torch::kLong).device(logits.device()));
  auto prob = torch::empty({rows, k}, logits.options());
  FMOE_CUDA_CHECK(fmoe::launch_gate_topk_softmax(logit_code(logits), logits.data_ptr(), rows, ne,
                                                 static_cast<int>(k), idx.data_ptr<int64_t>(),
                                                 prob.data_ptr(), zero_of(zero), cur_stream()));
  return {idx, prob};
}

torch::Tensor gate_topk_softmax_bwd(torch::Tensor dprob, torch::Tensor idx, torch::Tensor prob,
                                    int64_t n_experts) {
  check_cuda_contig(dprob, "dprob");
  c10::cuda::CUDAGuard guard(dprob.device());
  const int rows = static_cast<int>(dprob.size(0));
  const int k = static_cast<int>(dprob.size(1));
  auto dlogits = torch::empty({rows, n_experts}, dprob.options());
  FMOE_CUDA_CHECK(fmoe::launch_gate_topk_softmax_bwd(
      logit_code(dprob), dprob.data_ptr(), idx.data_ptr<int64_t>(), prob.data_ptr(), rows,
      static_cast<int>(n_experts), k, dlogits.data_ptr(), cur_stream()));
  return dlogits;
}

// ------------------------------------------------------------------------------ balanced gates
bool balance_supported(int64_t tot) { return fmoe::balance_supported(static_cast<int>(tot)); }

// Slots of every expert beyond the first `cap` (in slot order) become -1.
torch::Tensor prune_gate_scalar(torch::Tensor idx, int64_t cap, int64_t tot) {
  check_cuda_contig(idx, "gate_idx");
  auto flat = idx.view({-1});
  auto res = route(flat, tot, false);
  c10::cuda::CUDAGuard guard(idx.device());
  auto out = torch::empty_like(idx);
  FMOE_CUDA_CHECK(fmoe::launch_prune_scalar(flat.data_ptr<int64_t>(), res[1].data_ptr<int>(),
                                            static_cast<int>(std::min<int64_t>(cap, INT32_MAX)),
                                            static_cast<int>(flat.numel()), static_cast<int>(tot),
                                            out.data_ptr<int64_t>(), cur_stream()));
  return out;
}

// {[1, padded, d], [1, padded]}: see routing.cuh.
std::vector<torch::Tensor> gate_pad(torch::Tensor w, c10::optional<torch::Tensor> bias, int64_t padded) {
  check_rows(w, "w");
  TORCH_CHECK(w.dim() == 2 && padded >= w.size(0), "gate weight");
  TORCH_CHECK(!bias.has_value() || (bias->device() == w.device() && bias->scalar_type() == w.scalar_type() &&
                                    bias->is_contiguous() && bias->numel() == w.size(0)), "gate bias does not fit");
  c10::cuda::CUDAGuard guard(w.device());
  auto wp = torch::empty({1, padded, w.size(1)}, w.options());
  auto bp = torch::empty({1, padded}, w.options());
  FMOE_CUDA_CHECK(fmoe::launch_gate_pad(dtype16(w), w.data_ptr(), bias.has_value() ? bias->data_ptr() : nullptr,
                                        static_cast<int>(w.size(0)), static_cast<int>(padded), static_cast<int>(w.size(1)),
                                        wp.data_ptr(), bp.data_ptr(), cur_stream()));
  return {wp, bp};
}

// int32 [groups + 1] exclusive prefix of host counts, on `device` (-1: the current one).
torch::Tensor host_offsets(torch::Tensor counts_in, int64_t device) {
  TORCH_CHECK(counts_in.device().is_cpu() && counts_in.scalar_type() == torch::kLong && counts_in.dim() == 1 &&
              counts_in.numel() < fmoe::kMaxHostOffsets, "host counts");
  const torch::Tensor counts = counts_in.contiguous();
  c10::cuda::OptionalCUDAGuard guard;
  if (device >= 0) guard.set_index(static_cast<c10::DeviceIndex>(device));
  const int n = static_cast<int>(counts.numel());
  int values[fmoe::kMaxHostOffsets];
  const int64_t* c = counts.data_ptr<int64_t>();
  int64_t sum = 0;
  values[0] = 0;
  for (int i = 0; i < n; ++i) values[i + 1] = static_cast<int>(sum += c[i]);
  auto offs = torch::empty({n + 1}, torch::dtype(torch::kInt32).device(torch::kCUDA, c10::cuda::current_device()));
  FMOE_CUDA_CHECK(fmoe::launch_host_offsets(values, n + 1, offs.data_ptr<int>(), cur_stream()));
  return offs;
}

void check_logits(const torch::Tensor& logits) {
  TORCH_CHECK(logits.is_cuda() && logits.dim() == 2 && logits.stride(1) == 1 && logits.size(0) > 0,
              "logits must be a non-empty CUDA matrix with contiguous rows");
}

// {loss, weight}: see routing.cuh.  `ids` is [n, ...]: its first column counts.
std::vector<torch::Tensor> balance_loss(torch::Tensor logits, torch::Tensor ids, bool is_switch, double scale) {
  check_logits(logits);
  check_cuda_contig(ids, "ids");
  TORCH_CHECK(ids.scalar_type() == torch::kLong && ids.size(0) == logits.size(0), "ids must be int64 [n, k]");
  c10::cuda::CUDAGuard guard(logits.device());
  const int n = static_cast<int>(logits.size(0)), tot = static_cast<int>(logits.size(1));
  auto f32 = torch::dtype(torch::kFloat).device(logits.device());
  auto part = torch::empty({static_cast<long>(fmoe::balance_blocks(n)) * 2 * tot}, f32);
  auto loss = torch::empty({}, f32);
  auto weight = torch::empty({tot}, f32);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  FMOE_CUDA_CHECK(fmoe::launch_balance_loss(logit_code(logits), logits.data_ptr(), logits.stride(0),
                                            ids.data_ptr<int64_t>(), static_cast<int>(ids.numel() / n), n, tot,
                                            is_switch, static_cast<float>(scale), part.data_ptr<float>(),
                                            loss.data_ptr<float>(), weight.data_ptr<float>(), cur_stream()));
  return {loss, weight};
}

torch::Tensor balance_bwd(torch::Tensor logits, torch::Tensor weight, c10::optional<torch::Tensor> dloss,
                          c10::optional<torch::Tensor> win, c10::optional<torch::Tensor> dscore, bool is_switch,
                          double scale) {
  check_logits(logits);
  c10::cuda::CUDAGuard guard(logits.device());
  const int n = static_cast<int>(logits.size(0)), tot = static_cast<int>(logits.size(1));
  TORCH_CHECK(!dloss.has_value() || (dloss->scalar_type() == torch::kFloat && dloss->numel() == 1), "dloss");
  TORCH_CHECK(!dscore.has_value() || (dscore->scalar_type() == logits.scalar_type() && dscore->numel() == n &&
                                      dscore->is_contiguous() && win.has_value() && is_switch), "dscore");
  auto dlogits = torch::empty({n, tot}, logits.options());
  FMOE_CUDA_CHECK(fmoe::launch_balance_bwd(
      logit_code(logits), logits.data_ptr(), logits.stride(0), weight.data_ptr<float>(),
      dloss.has_value() ? dloss->data_ptr<float>() : nullptr, win.has_value() ? win->data_ptr<int64_t>() : nullptr,
      dscore.has_value() ? dscore->data_ptr() : nullptr, n, tot, is_switch, static_cast<float>(scale),
      dlogits.data_ptr(), cur_stream()));
  return dlogits;
}

std::vector<torch::Tensor> switch_top1(torch::Tensor logits) {
  check_logits(logits);
  check_cuda_contig(logits, "logits");
  c10::cuda::CUDAGuard guard(logits.device());
  const int n = static_cast<int>(logits.size(0)), tot = static_cast<int>(logits.size(1));
  auto win = torch::empty({n, 1}, torch::dtype(torch::kLong).device(logits.device()));
  auto score = torch::empty({n, 1}, logits.options());
  FMOE_CUDA_CHECK(fmoe::launch_switch_top1(logit_code(logits), logits.data_ptr(), n, tot, win.data_ptr<int64_t>(),
                                           score.data_ptr(), cur_stream()));
  return {win, score};
}

bool gate_fused_supported(int64_t tot, int64_t d, int64_t k) {
  return fmoe::gate_fused_supported(static_cast<int>(tot), static_cast<int>(d), static_cast<int>(k));
}

// logits [B, tot], idx [B, k] and prob [B, k] of a linear gate in one pass over x.
std::vector<torch::Tensor> gate_forward(const torch::Tensor& x, const torch::Tensor& w,
                                        const c10::optional<torch::Tensor>& bias, int64_t k, bool few, float* zero) {
  check_rows(x, "x");
  check_rows(w, "w");
  TORCH_CHECK(x.scalar_type() == w.scalar_type(), "gate input and weight dtypes differ");
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1) && x.device() == w.device(),
              "gate input and weight do not fit");
  const torch::Tensor b = bias.has_value() && bias->defined() ? bias->contiguous() : torch::Tensor();
  TORCH_CHECK(!b.defined() || (b.device() == x.device() && b.scalar_type() == x.scalar_type() && b.numel() == w.size(0)),
              "gate bias does not fit");
  c10::cuda::CUDAGuard guard(x.device());
  const int rows = static_cast<int>(x.size(0));
  const int d = static_cast<int>(x.size(1));
  const int tot = static_cast<int>(w.size(0));
  auto logits = torch::empty({rows, tot}, x.options());
  auto idx = torch::empty({rows, k}, torch::dtype(torch::kLong).device(x.device()));
  auto prob = torch::empty({rows, k}, x.options());
  FMOE_CUDA_CHECK((few ? fmoe::launch_gate_linear_topk_few : fmoe::launch_gate_linear_topk)(
      logit_code(x), x.data_ptr(), w.data_ptr(), b.defined() ? b.data_ptr() : nullptr, rows, d,
      tot, static_cast<int>(k), logits.data_ptr(), idx.data_ptr<int64_t>(), prob.data_ptr(),
      zero, cur_stream()));
  return {logits, idx, prob};
}

std::vector<torch::Tensor> gate_linear_topk(torch::Tensor x, torch::Tensor w, c10::optional<torch::Tensor> bias, int64_t k,
                                            bool few, c10::optional<torch::Tensor> zero) {
  return gate_forward(x, w, bias, k, few, zero_of(zero));
}

// Returns {dx or empty, dw (layer dtype) or empty, db or empty, dl fp32 [B, tot]}.  Without `x` no dw and db are
// formed, without `w` (of which `tot` is the rows then) no dx.
std::vector<torch::Tensor> gate_linear_topk_bwd(c10::optional<torch::Tensor> dprob, torch::Tensor idx,
                                                torch::Tensor prob,
                                                c10::optional<torch::Tensor> dlogits,
                                                c10::optional<torch::Tensor> x, c10::optional<torch::Tensor> w,
                                                bool need_dx, bool need_db, int64_t tot_without_w) {
  const bool need_dw = x.has_value() && x->defined(), has_w = w.has_value() && w->defined();
  if (need_dw) check_rows(*x, "x");
  if (has_w) check_rows(*w, "w");
  TORCH_CHECK((need_dw || has_w) && (has_w || (!need_dx && tot_without_w > 0)) && (need_dw || !need_db), "gate gradient: operands missing");
  const torch::Tensor& like = need_dw ? *x : *w;
  c10::cuda::CUDAGuard guard(like.device());
  const int rows = static_cast<int>(idx.size(0));
  const int d = static_cast<int>(like.size(1));
  const int tot = static_cast<int>(has_w ? w->size(0) : tot_without_w);
  const int k = static_cast<int>(idx.size(1));
  TORCH_CHECK(!need_dw || (x->size(0) == rows && (!has_w || x->size(1) == w->size(1))), "gate gradient: operands do not fit");
  auto f32 = torch::dtype(torch::kFloat).device(like.device());
  auto dl = torch::empty({rows, tot}, f32);
  torch::Tensor dx = need_dx ? torch::empty({rows, d}, like.options()) : torch::Tensor();
  const bool fused_dw = need_dw && tot <= 16;
  torch::Tensor part, dw_db;
  if (fused_dw) {
    const long elems = static_cast<long>(tot) * d + tot;
    // without rows nothing is launched: the sums over no tokens are zero
    dw_db = rows > 0 ? torch::empty({elems}, like.options()) : torch::zeros({elems}, like.options());
    part = torch::empty({fmoe::gate_bwd_ranges(logit_code(like), rows, d) * elems}, f32);
  }
  FMOE_CUDA_CHECK(fmoe::launch_gate_bwd(
      logit_code(like), dprob.has_value() ? dprob->data_ptr() : nullptr, idx.data_ptr<int64_t>(),
      prob.data_ptr(), dlogits.has_value() ? dlogits->data_ptr() : nullptr, need_dw ? x->data_ptr() : nullptr,
      has_w ? w->data_ptr() : nullptr, rows, d, tot, k, dl.data_ptr<float>(), need_dx ? dx.data_ptr() : nullptr,
      fused_dw ? part.data_ptr<float>() : nullptr, fused_dw ? dw_db.data_ptr() : nullptr, cur_stream()));
  torch::Tensor dw, db;
  if (fused_dw) {
    g_launches.fetch_add(2, std::memory_order_relaxed);  // the weight-gradient and merge kernels
    dw = dw_db.narrow(0, 0, static_cast<long>(tot) * d).view({tot, d});
    if (need_db) db = dw_db.narrow(0, static_cast<long>(tot) * d, tot);
  } else if (need_dw) {
    auto dl16 = dl.to(like.scalar_type());
    dw = dl16.t().matmul(*x);
    if (need_db) db = dl.sum(0).to(like.scalar_type());
  }
  return {dx, dw, db, dl};
}

// ------------------------------------------------------------------------------ autograd nodes
// The layer behind the gate and the linear gate as nodes of the native engine: their backward runs
// without the interpreter, and a forward costs one call from Python.
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// The fp32 layer's inputs that its backward does not read, for a gradient of the gradient.  Looked at only
// there: until then they may be changed in place.
struct SecondOrder : torch::CustomClassHolder {
  torch::autograd::SavedVariable x, score, b1, b2;
};

// The layer behind the gate as operations, experts one after the other.
torch::Tensor moe_mlp_operations(const torch::Tensor& x, const torch::Tensor& score, const torch::Tensor& w1, const torch::Tensor& b1,
                                 const torch::Tensor& w2, const torch::Tensor& b2, const torch::Tensor& rank,
                                 const torch::Tensor& offs, const torch::Tensor& idx, int64_t act) {
  const torch::Tensor ends = offs.cpu();
  const int* end = ends.data_ptr<int>();
  const int64_t groups = w1.size(0), k = idx.numel() / x.size(0), rows = end[groups];
  const torch::Tensor kept = rank.ge(0).nonzero().squeeze(1), expert = idx.index_select(0, kept);
  const torch::Tensor row = (offs.index_select(0, expert) + rank.index_select(0, kept)).to(torch::kLong);
  const torch::Tensor slot = torch::empty({rows}, idx.options()).index_copy_(0, row, kept);
  const torch::Tensor token = torch::floor_divide(slot, k), xs = x.index_select(0, token);
  std::vector<torch::Tensor> ys;
  for (int64_t e = 0; e < groups; ++e) {
    if (end[e + 1] == end[e]) continue;
    torch::Tensor hid = torch::linear(xs.slice(0, end[e], end[e + 1]), w1.select(0, e), b1.select(0, e));
    if (act == fmoe::kActRelu) hid = torch::relu(hid);
    if (act == fmoe::kActGelu || act == fmoe::kActGeluTanh) hid = at::gelu(hid, act == fmoe::kActGelu ? "none" : "tanh");
    ys.push_back(torch::linear(hid, w2.select(0, e), b2.select(0, e)));
  }
  const torch::Tensor w = score.reshape({-1}).index_select(0, slot).to(x.scalar_type()).unsqueeze(1);
  return torch::zeros_like(x).index_add(0, token, torch::cat(ys) * w);
}

struct MoEMLPSaved {
  torch::Tensor xs, pre, a, ys, rank, offs, score, slots;
};

// The fp32 layer's backward as a node of its own, for create_graph: its values are the kernels', its derivatives
// those of the operations.  Outputs: dx where wanted, dscore, dw1 and db1, dw2 and db2 where wanted.
class MoEMLPGrad : public torch::autograd::Function<MoEMLPGrad> {
 public:
  static variable_list forward(AutogradContext* ctx, const torch::Tensor& dout, const torch::Tensor& x, const torch::Tensor& score,
                               const torch::Tensor& w1, const torch::Tensor& b1, const torch::Tensor& w2, const torch::Tensor& b2,
                               const MoEMLPSaved* s, int64_t act, bool need_dx, bool need_w1, bool need_w2) {
    c10::optional<torch::Tensor> pre;
    if (s->pre.defined()) pre = s->pre;
    auto r = moe_mlp_backward(dout, s->xs, pre, s->a, s->ys, s->rank, s->offs, s->score, s->slots, w1, w2, act, need_dx,
                              need_w1, need_w2);
    variable_list out;
    std::vector<int64_t> of;   // which input each output is the gradient of (1: x, 2: score, ...)
    for (int64_t i = 0; i < 6; ++i) {
      if (!r[i].defined()) continue;
      out.push_back(r[i]);
      of.push_back(i + 1);
    }
    ctx->save_for_backward({dout, x, score, w1, b1, w2, b2, s->rank, s->offs, s->slots});
    ctx->saved_data["of"] = of;
    ctx->saved_data["act"] = act;
    ctx->set_materialize_grads(false);
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const std::vector<int64_t> of = ctx->saved_data["of"].toIntVector();
    const bool again = at::GradMode::is_enabled();
    at::AutoGradMode record(true);
    at::NoTF32Guard all_bits;
    variable_list in(s.begin(), s.begin() + 7), result(12);   // dout, x, score, w1, b1, w2, b2
    // variables of their own: dout depends on the other inputs, and the derivatives wanted are the partial ones
    for (auto& t : in) t = again ? t.view_as(t) : t.detach().set_requires_grad(true);
    const torch::Tensor y = moe_mlp_operations(in[1], in[2], in[3], in[4], in[5], in[6], s[7], s[8], s[9],
                                               ctx->saved_data["act"].toInt());
    variable_list wrt, seeds;
    for (size_t i = 0; i < grads.size(); ++i) {
      const torch::Tensor& t = in[of[i]];
      if (!grads[i].defined() || !t.requires_grad()) continue;
      wrt.push_back(t);
      seeds.push_back(grads[i].reshape(t.sizes()).to(t.scalar_type()));
    }
    if (wrt.empty()) return result;
    const variable_list first = torch::autograd::grad({y}, wrt, {in[0]}, true, true, true);
    variable_list outs, out_seeds, ins;
    std::vector<int64_t> at_input;
    for (size_t i = 0; i < first.size(); ++i) {
      if (!first[i].defined() || !first[i].requires_grad()) continue;
      outs.push_back(first[i]);
      out_seeds.push_back(seeds[i]);
    }
    for (int64_t i = 0; i < 7; ++i) {
      if (!ctx->needs_input_grad(i)) continue;
      ins.push_back(in[i]);
      at_input.push_back(i);
    }
    if (outs.empty() || ins.empty()) return result;
    const variable_list second = torch::autograd::grad(outs, ins, out_seeds, true, again, true);
    for (size_t i = 0; i < ins.size(); ++i) result[at_input[i]] = second[i];
    return result;
  }
};

class MoEMLP : public torch::autograd::Function<MoEMLP> {
 public:
  static torch::Tensor forward(AutogradContext* ctx, const torch::Tensor& x, const torch::Tensor& score,
                               const torch::Tensor& w1, const torch::Tensor& b1, const torch::Tensor& w2,
                               const torch::Tensor& b2, const torch::Tensor& idx, int64_t act, bool keep) {
    auto r = moe_mlp_forward(x, idx, score, w1, b1, w2, b2, act, keep);
    if (keep) ctx->save_for_backward({r[1], r[2], r[3], r[4], r[5], r[6], r[7], r[8], w1, w2});
    ctx->saved_data["act"] = act;
    ctx->saved_data["shape"] = score.sizes().vec();
    ctx->saved_data["dtype"] = static_cast<int64_t>(score.scalar_type());
    if (keep && x.scalar_type() == torch::kFloat) {
      auto second = c10::make_intrusive<SecondOrder>();
      second->x = torch::autograd::SavedVariable(x, false);
      second->score = torch::autograd::SavedVariable(score, false);
      second->b1 = torch::autograd::SavedVariable(b1, false);
      second->b2 = torch::autograd::SavedVariable(b2, false);
      ctx->saved_data["second"] = c10::IValue::make_capsule(second);
    }
    return r[0];
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();   // xs, pre, a, ys, rank, offs, score, slots, w1, w2
    const bool need_dx = ctx->needs_input_grad(0), need_score = ctx->needs_input_grad(1);
    const bool need_w1 = ctx->needs_input_grad(2) || ctx->needs_input_grad(3);
    const bool need_w2 = ctx->needs_input_grad(4) || ctx->needs_input_grad(5);
    const int64_t act = ctx->saved_data["act"].toInt();
    variable_list r;   // dx, dscore, dw1, db1, dw2, db2
    if (at::GradMode::is_enabled() && s[3].scalar_type() == torch::kFloat) {
      auto second = c10::static_intrusive_pointer_cast<SecondOrder>(ctx->saved_data["second"].toCapsule());
      const MoEMLPSaved saved{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7]};
      const variable_list out = MoEMLPGrad::apply(grads[0], second->x.unpack(), second->score.unpack(), s[8], second->b1.unpack(),
                                                  s[9], second->b2.unpack(), &saved, act, need_dx, need_w1, need_w2);
      size_t next = 0;
      auto take = [&](bool there) { return there ? out[next++] : torch::Tensor(); };
      for (bool there : {need_dx, true, need_w1, need_w1, need_w2, need_w2}) r.push_back(take(there));
    } else {
      c10::optional<torch::Tensor> pre;
      if (s[1].defined()) pre = s[1];
      r = moe_mlp_backward(grads[0], s[0], pre, s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], act, need_dx, need_w1, need_w2);
    }
    if (!torch::autograd::get_current_graph_task_keep_graph()) ctx->saved_data.erase("second");   // as the saved variables
    torch::Tensor dscore;
    if (need_score) {
      dscore = r[1].to(static_cast<torch::ScalarType>(ctx->saved_data["dtype"].toInt()))
                   .view(ctx->saved_data["shape"].toIntVector());
    }
    return {r[0], dscore, r[2], r[3], r[4], r[5], torch::Tensor(), torch::Tensor(), torch::Tensor()};
  }
};

class GateLinearTopk : public torch::autograd::Function<GateLinearTopk> {
 public:
  static variable_list forward(AutogradContext* ctx, const torch::Tensor& x, const torch::Tensor& w,
                               const c10::optional<torch::Tensor>& bias, int64_t k, int64_t zero) {
    // `zero`: address of the caller's one-element tensor, which is not an input of the node
    // The kernels load 16 bytes at a time.  Saved are the inputs, which a gradient of the gradient goes
    // on to: the graph does not know of copies made here.
    auto r = gate_forward(aligned(x, 16), aligned(w, 16), bias, k, false, reinterpret_cast<float*>(zero));
    const bool has_bias = bias.has_value() && bias->defined();
    // each operand where the other's gradient is wanted (what is not saved may be changed in place)
    ctx->save_for_backward({w.requires_grad() || (has_bias && bias->requires_grad()) ? x : torch::Tensor(),
                            x.requires_grad() ? w : torch::Tensor(), r[1], r[2]});
    ctx->saved_data["bias"] = has_bias;
    ctx->saved_data["tot"] = w.size(0);
    ctx->mark_non_differentiable({r[1]});
    ctx->set_materialize_grads(false);
    return {r[0], r[1], r[2]};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined() && !grads[2].defined()) return variable_list(5);
    const variable_list s = ctx->get_saved_variables();
    const bool has_bias = ctx->saved_data["bias"].toBool();
    const bool need_dx = ctx->needs_input_grad(0), need_dw = ctx->needs_input_grad(1);
    const bool need_db = has_bias && ctx->needs_input_grad(2);
    if (at::GradMode::is_enabled() && (!grads[2].defined() || s[3].scalar_type() == torch::kFloat)) {
      // a gradient of the gradient is wanted: the linear's, in operations that have one (the scores'
      // counts as a constant)
      torch::Tensor dl = grads[0];
      if (grads[2].defined()) {
        auto through = gate_topk_softmax_bwd(grads[2].contiguous(), s[2], s[3], ctx->saved_data["tot"].toInt());
        dl = dl.defined() ? dl + through : through;
      }
      return {need_dx ? dl.matmul(s[1]) : torch::Tensor(), need_dw ? dl.t().matmul(s[0]) : torch::Tensor(),
              need_db ? dl.sum(0) : torch::Tensor(), torch::Tensor(), torch::Tensor()};
    }
    auto given = [](const torch::Tensor& g) {
      return g.defined() ? c10::optional<torch::Tensor>(g.contiguous()) : c10::nullopt;
    };
    // (at any address: the caller's, or where hooks on saved tensors put them)
    auto rows = [](const torch::Tensor& t) { return t.defined() ? c10::optional<torch::Tensor>(aligned(t, 16)) : c10::nullopt; };
    auto r = gate_linear_topk_bwd(given(grads[2]), s[2], s[3], given(grads[0]), rows(s[0]), rows(s[1]), need_dx, need_db,
                                  ctx->saved_data["tot"].toInt());
    return {need_dx ? r[0] : torch::Tensor(), need_dw ? r[1] : torch::Tensor(), need_db ? r[2] : torch::Tensor(),
            torch::Tensor(), torch::Tensor()};
  }
};

torch::Tensor moe_mlp(torch::Tensor x, torch::Tensor score, torch::Tensor w1, torch::Tensor b1, torch::Tensor w2,
                      torch::Tensor b2, torch::Tensor idx, int64_t act, bool keep) {
  return MoEMLP::apply(x, score, w1, b1, w2, b2, idx, act, keep);
}

variable_list gate_linear_topk_node(torch::Tensor x, torch::Tensor w, c10::optional<torch::Tensor> bias, int64_t k,
                                    c10::optional<torch::Tensor> zero) {
  return GateLinearTopk::apply(x, w, bias, k, reinterpret_cast<int64_t>(zero_of(zero)));
}

// ------------------------------------------------------------------------------ status
int64_t read_status(int64_t device) {
  auto t = status_tensor(static_cast<int>(device));
  return t.cpu().data_ptr<int>()[0];
}

void clear_status(int64_t device) { status_tensor(static_cast<int>(device)).zero_(); }

torch::Tensor status_word(int64_t device) { return status_tensor(static_cast<int>(device)); }

}  // namespace

namespace {
// The parts {group, tile, kb0, kb1, num_kb, last_piece} that one pair of a persistent GEMM walks (host).
std::vector<std::vector<int>> tile_walk(std::vector<int> tiles, std::vector<int> units, int pair, int pairs, int min_kb) {
  TORCH_CHECK(tiles.size() >= 2 && tiles.size() == units.size() && pair >= 0 && pair < pairs, "tile_walk");
  fmoe::TileWalk walk(tiles.data(), units.data(), static_cast<int>(tiles.size()) - 1, pair, pairs, min_kb);
  std::vector<std::vector<int>> parts;
  fmoe::WalkPart p;
  while (walk.next(p)) parts.push_back({p.group, p.tile, p.kb0, p.kb1, p.num_kb, p.last_piece});
  return parts;
}
}  // namespace

void bind_p2p(pybind11::module& m);  // sm100/p2p_binding.cpp

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "fastmoe_b200 native ops (sm_100a kernels + C++ host runtime)";
  // reference-compatible names
  m.def("expert_count", &expert_count);
  m.def("assign_pos", &assign_pos);
  m.def("limit_by_capacity", &limit_by_capacity);
  m.def("prune_gate_by_capacity", &prune_gate_by_capacity);
  // device-count-driven API
  m.def("route", [](torch::Tensor idx, int64_t tot) { return route(idx, tot, false); });
  m.def("route_offs", [](torch::Tensor idx, int64_t tot) { return route(idx, tot, true); });
  // counts, rank, offs and pos (slot ids sorted by expert then rank: the send order of the
  // fused dispatch)
  m.def("route_pos", [](torch::Tensor idx, int64_t tot) { return route(idx, tot, true, true); });
  m.def("swipe_reassign", &swipe_reassign);
  m.def("grouped_gemm", &grouped_gemm, py::arg("mode"), py::arg("a"), py::arg("b"), py::arg("offs"),
        py::arg("out"), py::arg("bias") = py::none(), py::arg("pre_out") = py::none(),
        py::arg("aux") = py::none(), py::arg("act") = 0, py::arg("epi") = 0,
        py::arg("accumulate") = false, py::arg("psum") = py::none());
  m.def("grouped_gemm_supported", &grouped_gemm_supported);
  m.def("simt_grouped_gemm", &simt_grouped_gemm, py::arg("mode"), py::arg("a"), py::arg("b"),
        py::arg("offs"), py::arg("out"), py::arg("bias") = py::none(), py::arg("psum") = py::none());
  m.def("simt_column_sums", &simt_column_sums);
  m.def("split_grouped_gemm", &split_grouped_gemm, py::arg("mode"), py::arg("a"), py::arg("b"),
        py::arg("offs"), py::arg("out"), py::arg("bias") = py::none(), py::arg("psum") = py::none());
  m.def("wide_grouped_gemm", &wide_grouped_gemm, py::arg("mode"), py::arg("a"), py::arg("b"),
        py::arg("offs"), py::arg("out"), py::arg("bias") = py::none(), py::arg("psum") = py::none());
  m.def("tile_walk", &tile_walk);
  m.def("moe_mlp_supported_f32", &moe_mlp_supported_f32);
  m.def("scatter_rows", &scatter_rows, py::arg("src"), py::arg("idx"), py::arg("rank"),
        py::arg("base"), py::arg("scale"), py::arg("k"), py::arg("dst"),
        py::arg("row_slot") = py::none());
  m.def("gather_combine", &gather_combine);
  m.def("combine_bwd", &combine_bwd);
  m.def("colsum", &colsum);
  m.def("moe_mlp_supported", &moe_mlp_supported);
  m.def("moe_mlp_forward", &moe_mlp_forward);
  m.def("moe_mlp_backward", &moe_mlp_backward);
  m.def("gate_topk_softmax", &gate_topk_softmax, py::arg("logits"), py::arg("k"), py::arg("zero") = py::none());
  m.def("moe_mlp", &moe_mlp);
  m.def("gate_linear_topk_node", &gate_linear_topk_node, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("k"),
        py::arg("zero") = py::none());
  m.def("gate_topk_softmax_bwd", &gate_topk_softmax_bwd);
  m.def("balance_supported", &balance_supported);
  m.def("prune_gate_scalar", &prune_gate_scalar);
  m.def("host_offsets", &host_offsets);
  m.def("gate_pad", &gate_pad);
  m.def("balance_loss", &balance_loss);
  m.def("balance_bwd", &balance_bwd);
  m.def("switch_top1", &switch_top1);
  m.def("gate_fused_supported", &gate_fused_supported);
  m.def("gate_linear_topk", &gate_linear_topk, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("k"),
        py::arg("few") = false, py::arg("zero") = py::none());
  m.def("gate_linear_topk_bwd", &gate_linear_topk_bwd, py::arg("dprob"), py::arg("idx"), py::arg("prob"), py::arg("dlogits"),
        py::arg("x"), py::arg("w"), py::arg("need_dx"), py::arg("need_db"), py::arg("tot") = 0);
  m.def("launch_count", []() { return g_launches.load(); });
  m.def("read_status", &read_status);
  m.def("clear_status", &clear_status);
  m.def("status_word", &status_word);
  // C++ CPU ops
  m.def("cpu_route", &fmoe::cpu::route);
  m.def("cpu_limit_by_capacity", &fmoe::cpu::limit_by_capacity);
  m.def("cpu_prune_gate_by_capacity", &fmoe::cpu::prune_gate_by_capacity);
  m.def("cpu_linear_forward", &fmoe::cpu::linear_forward);
  m.def("cpu_linear_backward", &fmoe::cpu::linear_backward);
  m.def("cpu_swipe_plan", &fmoe::cpu::swipe_plan);
  m.def("cpu_smart_schedule_plan", &fmoe::cpu::smart_schedule_plan);
  bind_p2p(m);
}
