// Routing bookkeeping, row scatter / combine, gate top-k and balancing kernels.
//
// Replaces cuda/local_exchange.cuh (expert_count, assign_pos), cuda/balancing.cuh
// (limit_by_capacity, prune_gate_by_capacity), cuda/parallel_linear.cuh:8-53 (column_reduce)
// and the ATen index_select / index_copy_ / bmm / topk / softmax calls of the reference's layer.
// All kernels are deterministic: no result depends on the order in which atomics land.
#include "launch.cuh"
#include "ptx.cuh"
#include "routing.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace fmoe {
namespace {

namespace cg = cooperative_groups;

constexpr int kRouteThreads = 1024;
constexpr int kRouteSmemLimit = 200 * 1024;
constexpr int kRouteCluster = 8;
constexpr int kRouteClusterSlots = 65536;
constexpr int kRouteClusterExperts = 1024;
constexpr int kRouteCtaSlots = 32768;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// CTA b owns the contiguous slot range [b * cta_slots, (b + 1) * cta_slots), warp w of it the
// sub-range [w * chunk, (w + 1) * chunk): pass 1 builds per-warp histograms, the CTA turns them
// into exclusive prefixes over warps, pass 2 hands every slot its rank.  Within a warp slots
// are visited in order, 32 at a time.  The chain of these steps is what bounds the kernel (a
// match of 32 keys and an update of shared memory that the next step waits for), so up to
// kRouteClusterSlots slots are spread over a cluster of eight CTAs, which exchange their per-expert totals
// through distributed shared memory in the one launch: 16384 slots on 8 experts 19 -> 6.8 us, 8192 slots on
// 64 experts 17.9 -> 6.4 us.  For more slots the work is spread over more CTAs and two launches: the first
// (`part_out`) only writes every CTA's per-expert totals, the second (`part_in`) starts each CTA's prefixes
// at the sum of the totals of the CTAs before it.  Ranks are always those of a single ordered scan.
__global__ void __launch_bounds__(kRouteThreads, 1)
route_kernel(const int64_t* __restrict__ idx, int n_slots, int tot, int nw, int cta_slots, int in_cluster,
             const int* __restrict__ part_in, int* __restrict__ part_out, int* __restrict__ counts,
             int* __restrict__ rank, int* __restrict__ offs, int* __restrict__ pos) {
  ptx::chain_begin();
  extern __shared__ int hist[];  // [nw][tot], [tot + 1] expert offsets; in a cluster [tot] totals of this CTA
  int* eoff = hist + nw * tot;
  int* mine = in_cluster ? eoff + tot + 1 : eoff + 1;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < nw * tot; i += blockDim.x) hist[i] = 0;
  __syncthreads();

  const int cta_begin = blockIdx.x * cta_slots;
  const int cta_end = min(n_slots, cta_begin + cta_slots);
  int chunk = (cta_slots + nw - 1) / nw;
  chunk = (chunk + 31) & ~31;
  const int begin = cta_begin + warp * chunk;
  const int end = min(cta_end, begin + chunk);

  if (warp < nw) {
    int* h = hist + warp * tot;
    for (int s0 = begin; s0 < end; s0 += 32) {
      const int s = s0 + lane;
      long e = (s < end) ? idx[s] : -1;
      const bool valid = e >= 0 && e < tot;
      const int key = valid ? static_cast<int>(e) : tot + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, key);
      if (valid && (peers & lanemask_lt()) == 0) h[key] += __popc(peers);
      __syncwarp();
    }
  }
  __syncthreads();
  // exclusive prefixes over the warps, and this CTA's totals
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    int run = 0;
    for (int w0 = 0; w0 < nw; w0 += 8) {
      int t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = w0 + i < nw ? hist[(w0 + i) * tot + e] : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (w0 + i < nw) hist[(w0 + i) * tot + e] = run;
        run += t[i];
      }
    }
    mine[e] = run;
    if (part_out != nullptr) part_out[blockIdx.x * tot + e] = run;
  }
  if (part_out != nullptr) return;   // first launch of the two-launch scheme: totals, nothing else
  if (in_cluster) cg::this_cluster().sync(); else __syncthreads();
  for (int e = threadIdx.x; e < tot; e += blockDim.x) {
    int run = 0, total = 0;
    if (part_in != nullptr) {
      for (int b = 0; b < static_cast<int>(gridDim.x); ++b) {
        const int t = part_in[b * tot + e];
        if (b < static_cast<int>(blockIdx.x)) run += t;
        total += t;
      }
    } else if (in_cluster) {
#pragma unroll
      for (int b = 0; b < kRouteCluster; ++b) {
        const int t = *cg::this_cluster().map_shared_rank(mine + e, b);
        if (b < static_cast<int>(blockIdx.x)) run += t;
        total += t;
      }
    } else {
      total = mine[e];
    }
    if (run != 0) {
      for (int w = 0; w < nw; ++w) hist[w * tot + e] += run;
    }
    if (blockIdx.x == 0) counts[e] = total;
    eoff[e + 1] = total;
  }
  if (in_cluster) cg::this_cluster().sync(); else __syncthreads();   // nobody reads `mine` any more
  if (pos != nullptr || offs != nullptr) {
    // exclusive prefix of the counts: where the slots of every expert start in `pos`
    if (warp == 0) {
      int run = 0;
      if (lane == 0) eoff[0] = 0;
      for (int e0 = 0; e0 < tot; e0 += 32) {
        const int e = e0 + lane;
        int v = e < tot ? eoff[e + 1] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += up;
        }
        if (e < tot) eoff[e + 1] = run + v;
        run += __shfl_sync(0xffffffffu, v, 31);
      }
    }
    __syncthreads();
  }
  if (warp < nw) {
    int* h = hist + warp * tot;
    for (int s0 = begin; s0 < end; s0 += 32) {
      const int s = s0 + lane;
      long e = (s < end) ? idx[s] : -1;
      const bool valid = e >= 0 && e < tot;
      const int key = valid ? static_cast<int>(e) : tot + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, key);
      const int before = __popc(peers & lanemask_lt());
      int r = -1;
      if (valid) r = h[key] + before;
      __syncwarp();
      if (valid && before == 0) h[key] += __popc(peers);
      __syncwarp();
      if (s < end) rank[s] = r;
      if (pos != nullptr && valid) pos[eoff[key] + r] = s;
    }
  }
  if (offs != nullptr && blockIdx.x == 0) {
    for (int e = threadIdx.x; e <= tot; e += blockDim.x) offs[e] = eoff[e];
  }
}

__global__ void prune_kernel(const int64_t* __restrict__ idx, const int* __restrict__ rank,
                             const int* __restrict__ cap, int n_slots, int tot,
                             int64_t* __restrict__ out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const long e = idx[s];
  out[s] = (e >= 0 && e < tot && rank[s] < cap[e]) ? e : -1;
}

__global__ void limit_kernel(const int64_t* __restrict__ ec, int* __restrict__ cap,
                             int64_t* __restrict__ eca, int n_expert, int n_worker) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_expert) return;
  long left = cap[e];
  for (int w = 0; w < n_worker; ++w) {
    const long want = ec[w * n_expert + e];
    const long room = left > 0 ? left : 0;
    eca[w * n_expert + e] = want < room ? want : room;
    left -= want;
  }
  cap[e] = static_cast<int>(left);
}

__global__ void fill_pos_kernel(const int64_t* __restrict__ idx, const int* __restrict__ rank,
                                const int* __restrict__ cum_incl, int n_slots, int tot,
                                int64_t* __restrict__ pos) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const long e = idx[s];
  if (e < 0 || e >= tot) return;
  const int base = e == 0 ? 0 : cum_incl[e - 1];
  pos[base + rank[s]] = s;
}

// SWIPE reassignment, two passes around a ranking of the moved tokens.  A token keeps its
// expert while its worker's quota lasts (slot order); `swipe_mark` writes key 0 for the others
// (and -1 for the kept ones), the routing kernel ranks them, and `swipe_assign` sends the i-th
// moved token to expert `bias` of the worker that owns the i-th unit of spare quota.
__global__ void swipe_mark_kernel(const int64_t* __restrict__ idx, const int* __restrict__ rank,
                                  const int* __restrict__ quota, int n, int n_expert, int n_worker,
                                  int64_t* __restrict__ key) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const long e = idx[s];
  const int w = static_cast<int>(e / n_expert);
  const bool valid = e >= 0 && w < n_worker;
  key[s] = (valid && rank[s] >= quota[w]) ? 0 : -1;
}

__global__ void swipe_assign_kernel(const int64_t* __restrict__ idx, const int64_t* __restrict__ key,
                                    const int* __restrict__ mrank, const int* __restrict__ count,
                                    const int* __restrict__ quota, int n, int n_expert, int n_worker,
                                    int bias, int64_t* __restrict__ out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  if (key[s] < 0) {
    out[s] = idx[s];
    return;
  }
  const int o = mrank[s];
  int run = 0, target = -1;
  for (int j = 0; j < n_worker; ++j) {
    const int kept = count[j] < quota[j] ? count[j] : quota[j];
    run += quota[j] - kept;
    if (o < run) {
      target = j;
      break;
    }
  }
  out[s] = target < 0 ? -1 : static_cast<int64_t>(target) * n_expert + bias;
}

// ------------------------------------------------------------------------------ row movement
template <typename T> struct V2;
template <> struct V2<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ float2 to_f2(type v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ type from_f2(float a, float b) { return __floats2bfloat162_rn(a, b); }
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16(v); }
};
template <> struct V2<__half> {
  using type = __half2;
  static __device__ __forceinline__ float2 to_f2(type v) { return __half22float2(v); }
  static __device__ __forceinline__ type from_f2(float a, float b) { return __floats2half2_rn(a, b); }
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half(v); }
};
template <> struct V2<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& w, float (&f)[8]) {
  using P = typename V2<T>::type;
  const P* p = reinterpret_cast<const P*>(&w);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 v = V2<T>::to_f2(p[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  using P = typename V2<T>::type;
  uint4 w;
  P* p = reinterpret_cast<P*>(&w);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = V2<T>::from_f2(f[2 * i], f[2 * i + 1]);
  return w;
}

// The values of one 16-byte load: eight of 16 bits, four of 32.
template <typename T> constexpr int kPer16 = 16 / static_cast<int>(sizeof(T));
template <typename T>
__device__ __forceinline__ void unpack16(const uint4& w, float (&f)[kPer16<T>]) {
  if constexpr (sizeof(T) == 4) {
    f[0] = __uint_as_float(w.x);
    f[1] = __uint_as_float(w.y);
    f[2] = __uint_as_float(w.z);
    f[3] = __uint_as_float(w.w);
  } else {
    unpack8<T>(w, f);
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack16(const float (&f)[kPer16<T>]) {
  if constexpr (sizeof(T) == 4) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  } else {
    return pack8<T>(f);
  }
}

// One warp per slot; d % 8 == 0.
template <typename T>
__global__ void scatter_rows_kernel(const T* __restrict__ src, const int64_t* __restrict__ idx,
                                    const int* __restrict__ rank, const int* __restrict__ base,
                                    const T* __restrict__ scale, int n_slots, int k, int d,
                                    T* __restrict__ dst, int* __restrict__ row_slot) {
  ptx::chain_begin();
  const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (s >= n_slots) return;
  const int rk = rank[s];   // negative for dropped slots and for ids that name no expert
  if (rk < 0) return;
  const long row = static_cast<long>(base[idx[s]]) + rk;
  const uint4* in = reinterpret_cast<const uint4*>(src + static_cast<long>(s / k) * d);
  uint4* out = reinterpret_cast<uint4*>(dst + row * d);
  const int nv = d >> 3;
  const float sc = scale == nullptr ? 1.f : V2<T>::to_f(scale[s]);
  // Four 16-byte loads in flight per lane before the first store.
  for (int i0 = lane; i0 < nv; i0 += 128) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i0 + u * 32 < nv) v[u] = __ldg(in + i0 + u * 32);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i0 + u * 32 < nv) {
        if (scale != nullptr) {
          float f[8];
          unpack8<T>(v[u], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] *= sc;
          v[u] = pack8<T>(f);
        }
        out[i0 + u * 32] = v[u];
      }
    }
  }
  if (row_slot != nullptr && lane == 0) row_slot[row] = s;
}

// One warp per token; d % 8 == 0.  At most 64 registers, so that four blocks fit on an SM and a
// batch of 4096 tokens is one wave on 148 SMs.
template <typename T>
__global__ void __launch_bounds__(256, 4) gather_combine_kernel(const T* __restrict__ rows, const int64_t* __restrict__ idx,
                                      const int* __restrict__ rank, const int* __restrict__ base,
                                      const T* __restrict__ weight, int n_tokens, int k, int d,
                                      T* __restrict__ out) {
  ptx::chain_begin();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= n_tokens) return;
  const int nv = d >> 3;
  uint4* o = reinterpret_cast<uint4*>(out + static_cast<long>(t) * d);
  // Rows and weights of the k slots first, then four 16-byte chunks of every row in flight.
  constexpr int kMaxInline = 4;
  long rows_of[kMaxInline];
  float w_of[kMaxInline];
  const int kk = k < kMaxInline ? k : kMaxInline;
#pragma unroll
  for (int j = 0; j < kMaxInline; ++j) {
    rows_of[j] = -1;
    w_of[j] = 0.f;
    if (j < kk) {
      const int s = t * k + j;
      const int rk = rank[s];
      if (rk >= 0) {
        rows_of[j] = static_cast<long>(base[idx[s]]) + rk;
        w_of[j] = weight != nullptr ? V2<T>::to_f(weight[s]) : 1.f;
      }
    }
  }
  for (int i0 = lane; i0 < nv; i0 += 64) {
    float acc[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < kMaxInline; ++j) {
      if (j >= kk || rows_of[j] < 0) continue;
      const uint4* src = reinterpret_cast<const uint4*>(rows + rows_of[j] * d);
      uint4 v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (i0 + u * 32 < nv) v[u] = __ldg(src + i0 + u * 32);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (i0 + u * 32 < nv) {
          float f[8];
          unpack8<T>(v[u], f);
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[u][q] += w_of[j] * f[q];
        }
      }
    }
    for (int j = kk; j < k; ++j) {  // more than kMaxInline slots per token: plain path
      const int s = t * k + j;
      const int rk = rank[s];
      if (rk < 0) continue;
      const long row = static_cast<long>(base[idx[s]]) + rk;
      const float w = weight != nullptr ? V2<T>::to_f(weight[s]) : 1.f;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (i0 + u * 32 < nv) {
          float f[8];
          unpack8<T>(__ldg(reinterpret_cast<const uint4*>(rows + row * d) + i0 + u * 32), f);
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[u][q] += w * f[q];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (i0 + u * 32 < nv) o[i0 + u * 32] = pack8<T>(acc[u]);
    }
  }
}

// One warp per slot.
template <typename T>
__global__ void combine_bwd_kernel(const T* __restrict__ dout, const T* __restrict__ rows,
                                   const int64_t* __restrict__ idx, const int* __restrict__ rank,
                                   const int* __restrict__ base, const T* __restrict__ weight,
                                   int n_slots, int k, int d, T* __restrict__ drows,
                                   T* __restrict__ dscore) {
  ptx::chain_begin();
  const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (s >= n_slots) return;
  const int rk = rank[s];
  if (rk < 0) {
    if (lane == 0 && dscore != nullptr) dscore[s] = V2<T>::from_f(0.f);
    return;
  }
  const long row = static_cast<long>(base[idx[s]]) + rk;
  const uint4* g = reinterpret_cast<const uint4*>(dout + static_cast<long>(s / k) * d);
  const uint4* y = reinterpret_cast<const uint4*>(rows + row * d);
  uint4* dy = reinterpret_cast<uint4*>(drows + row * d);
  const float w = V2<T>::to_f(weight[s]);
  const int nv = d >> 3;
  float dot = 0.f;
  for (int i = lane; i < nv; i += 32) {
    float gf[8], yf[8];
    unpack8<T>(__ldg(g + i), gf);
    unpack8<T>(__ldg(y + i), yf);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      dot += gf[q] * yf[q];
      gf[q] *= w;
    }
    dy[i] = pack8<T>(gf);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (lane == 0 && dscore != nullptr) dscore[s] = V2<T>::from_f(dot);
}

// Column sums per group.  A block takes 128 rows x 256 columns; blockIdx.y enumerates the
// (group, 128-row chunk) pieces, found by scanning the offsets.
template <typename T>
__global__ void __launch_bounds__(256)
colsum_kernel(const T* __restrict__ x, const int* __restrict__ offs, int num_groups, int n,
              long rows_cap, float* __restrict__ out) {
  __shared__ float red[8][256 + 8];
  int piece = blockIdx.x;  // pieces on x (up to 2^31 - 1 blocks), column blocks on y
  int g = 0, r0 = 0, r1 = 0;
  bool found = false;
  for (; g < num_groups; ++g) {
    const int b = offs[g], e = offs[g + 1];
    const int pieces = (e - b + 127) >> 7;
    if (piece < pieces) {
      r0 = b + piece * 128;
      r1 = min(e, r0 + 128);
      if (r1 > rows_cap) r1 = static_cast<int>(rows_cap);  // offsets past the matrix are not followed
      found = true;
      break;
    }
    piece -= pieces;
  }
  if (!found) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.y * 256 + lane * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < n) {
    for (int r = r0 + warp; r < r1; r += 8) {
      float f[8];
      unpack8<T>(__ldg(reinterpret_cast<const uint4*>(x + static_cast<long>(r) * n + col)), f);
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] += f[q];
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) red[warp][lane * 8 + q] = acc[q];
  __syncthreads();
  const int c = blockIdx.y * 256 + threadIdx.x;
  if (c < n) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
    atomicAdd(out + static_cast<long>(g) * n + c, s);
  }
}

// ------------------------------------------------------------------------------ gate
template <typename T> struct Ld;
template <> struct Ld<float> {
  static __device__ __forceinline__ float get(const float* p, long i) { return p[i]; }
  static __device__ __forceinline__ void put(float* p, long i, float v) { p[i] = v; }
};
template <> struct Ld<__nv_bfloat16> {
  static __device__ __forceinline__ float get(const __nv_bfloat16* p, long i) { return __bfloat162float(p[i]); }
  static __device__ __forceinline__ void put(__nv_bfloat16* p, long i, float v) { p[i] = __float2bfloat16(v); }
};
template <> struct Ld<__half> {
  static __device__ __forceinline__ float get(const __half* p, long i) { return __half2float(p[i]); }
  static __device__ __forceinline__ void put(__half* p, long i, float v) { p[i] = __float2half(v); }
};

constexpr int kMaxK = 8;

// Top-k with softmax of one row of at most 64 logits without a NaN, two per lane (-inf where there is
// none): k rounds of a warp-wide maximum of keys that order as the logits do; ties go to the lower id.
// 4096 rows of 64, k = 2: 5.1 us with rounds of shuffles and the choices in local arrays, now 2.0.
__device__ __forceinline__ unsigned order_key(float v) {
  const unsigned u = __float_as_uint(v + 0.f);   // (-0 and +0 are a tie)
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
template <typename T>
__device__ __forceinline__ void topk_row64(float v0, float v1, bool on0, bool on1, int lane, int k, int64_t* idx, T* prob) {
  unsigned k0 = on0 ? order_key(v0) : 0u, k1 = on1 ? order_key(v1) : 0u;   // 0: taken, or none
  float top = 0.f, den = 0.f, my_ex = 0.f;
  int my_e = 0;
  for (int j = 0; j < k; ++j) {
    const unsigned m = __reduce_max_sync(0xffffffffu, k0 > k1 ? k0 : k1);
    const unsigned low = __ballot_sync(0xffffffffu, k0 == m), high = __ballot_sync(0xffffffffu, k1 == m);
    const int e = low != 0 ? __ffs(low) - 1 : 31 + __ffs(high);
    const float v = __uint_as_float(m & 0x80000000u ? m & 0x7fffffffu : ~m);
    if (j == 0) top = v;
    const float ex = __expf(v - top);
    den += ex;
    if (lane == j) {
      my_e = e;
      my_ex = ex;
    }
    if (e == lane) k0 = 0u;
    if (e == lane + 32) k1 = 0u;
  }
  if (lane < k) {
    idx[lane] = my_e;
    Ld<T>::put(prob, lane, my_ex / den);
  }
}

// The same for any number of experts, and with NaN: k rounds of warp arg-max.
template <typename T>
__device__ __noinline__ void topk_row(const T* in, int n_experts, int lane, int k, int64_t* idx, T* prob) {
  float sel_v[kMaxK];
  int sel_i[kMaxK];
  for (int j = 0; j < k; ++j) {
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int e = lane; e < n_experts; e += 32) {
      bool taken = false;
      for (int q = 0; q < j; ++q) taken |= (sel_i[q] == e);
      if (taken) continue;
      const float v = Ld<T>::get(in, e);
      if (v > best || (v == best && e < best_i) || best_i == 0x7fffffff) {
        best = v;
        best_i = e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (oi != 0x7fffffff && (best_i == 0x7fffffff || ov > best || (ov == best && oi < best_i))) {
        best = ov;
        best_i = oi;
      }
    }
    // (with NaN the lanes may disagree: all go by lane 0, so that k different experts are chosen)
    sel_v[j] = __shfl_sync(0xffffffffu, best, 0);
    sel_i[j] = __shfl_sync(0xffffffffu, best_i, 0);
  }
  if (lane == 0) {
    const float mx = sel_v[0];
    float den = 0.f;
    float ex[kMaxK];
    for (int j = 0; j < k; ++j) {
      ex[j] = __expf(sel_v[j] - mx);
      den += ex[j];
    }
    for (int j = 0; j < k; ++j) {
      idx[j] = sel_i[j];
      Ld<T>::put(prob, j, ex[j] / den);
    }
  }
}

// One warp per row.
template <typename T>
__global__ void gate_topk_softmax_kernel(const T* __restrict__ logits, int n_rows, int n_experts,
                                         int k, int64_t* __restrict__ idx, T* __restrict__ prob, float* zero) {
  ptx::chain_begin();
  if (zero != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero = 0.f;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const T* in = logits + static_cast<long>(row) * n_experts;
  idx += static_cast<long>(row) * k;
  prob += static_cast<long>(row) * k;
  if (n_experts <= 64) {
    const bool on0 = lane < n_experts, on1 = lane + 32 < n_experts;
    const float v0 = on0 ? Ld<T>::get(in, lane) : 0.f, v1 = on1 ? Ld<T>::get(in, lane + 32) : 0.f;
    if (!__any_sync(0xffffffffu, v0 != v0 || v1 != v1)) {
      topk_row64<T>(v0, v1, on0, on1, lane, k, idx, prob);
      return;
    }
  }
  topk_row<T>(in, n_experts, lane, k, idx, prob);
}

// dlogits[row, idx_j] = p_j * (g_j - sum_i g_i p_i), zero elsewhere.  One warp per row.
template <typename T>
__global__ void gate_topk_softmax_bwd_kernel(const T* __restrict__ dprob,
                                             const int64_t* __restrict__ idx,
                                             const T* __restrict__ prob, int n_rows, int n_experts,
                                             int k, T* __restrict__ dlogits) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  float g[kMaxK], p[kMaxK];
  int id[kMaxK];
  float dotp = 0.f;
  for (int j = 0; j < k; ++j) {
    g[j] = Ld<T>::get(dprob, static_cast<long>(row) * k + j);
    p[j] = Ld<T>::get(prob, static_cast<long>(row) * k + j);
    id[j] = static_cast<int>(idx[static_cast<long>(row) * k + j]);
    dotp += g[j] * p[j];
  }
  T* out = dlogits + static_cast<long>(row) * n_experts;
  for (int e = lane; e < n_experts; e += 32) {
    float v = 0.f;
    for (int j = 0; j < k; ++j) {
      if (id[j] == e) v = p[j] * (g[j] - dotp);
    }
    Ld<T>::put(out, e, v);
  }
}

// ------------------------------------------------------------------------------ balance losses
// GShard: loss = mean_e(c_e m_e) scale, c_e = share of the tokens whose first choice is e, m_e = mean
// softmax probability; Switch: loss = scale sum_e (f_e / K) (P_e / K) with f_e the kept tokens of e,
// P_e the sum of its probabilities and K = max(1, kept).  As PyTorch operations a loss and its
// gradient were about 25 launches of 1 to 17 us; here: partial sums per block, one block that adds
// them in order, and one pass for the gradient.  One thread per token, tot <= kBalanceMaxExperts.
// Sums are formed in fp32.  Switch holds everything else in fp32 too, as its PyTorch operations do;
// GShard's operations hold the probabilities, their mean and the gradients of both in the type T of
// the logits, and the kernels round where they round: with two experts in fp16 a gradient without
// those roundings moves the gate's bias gradient by up to 1e-2.
constexpr int kBalanceMaxExperts = 64;
constexpr int kBalanceThreads = 128;

// `v` as a tensor of type T holds it
template <typename T> __device__ __forceinline__ float rounded(float v) {
  T t;
  Ld<T>::put(&t, 0, v);
  return Ld<T>::get(&t, 0);
}

// Sum over the experts in the order of a butterfly over lanes, largest distance first, as softmax
// and its gradient form it: with 64 experts a sum in ascending order left the scores more than twice as
// far from 64 bits (2.1 against 0.86 units of 2^-24).  Zeros past the last expert change nothing.
template <int TOT> __device__ __forceinline__ float sum_experts(const float (&v)[TOT]) {
  float s[TOT];
#pragma unroll
  for (int e = 0; e < TOT; ++e) s[e] = v[e];
#pragma unroll
  for (int o = TOT / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int e = 0; e < o; ++e) s[e] += s[e + o];
  }
  return s[0];
}

// p[e] = softmax(logits[row])_e, zero from `tot` on
template <typename T, int TOT>
__device__ __forceinline__ void row_softmax(const T* in, int tot, float (&p)[TOT]) {
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    p[e] = e < tot ? Ld<T>::get(in, e) : -INFINITY;
    mx = fmaxf(mx, p[e]);
  }
#pragma unroll
  for (int e = 0; e < TOT; ++e) p[e] = e < tot ? expf(p[e] - mx) : 0.f;
  const float den = sum_experts<TOT>(p);
#pragma unroll
  for (int e = 0; e < TOT; ++e) p[e] = e < tot ? p[e] / den : 0.f;
}

// part[block][2 * tot]: kept tokens and probability sums of the block's tokens per expert.
template <typename T, bool SWITCH, int TOT>
__global__ void __launch_bounds__(kBalanceThreads)
balance_sums_kernel(const T* __restrict__ logits, long pitch, const int64_t* __restrict__ ids, int id_stride, int n,
                    int tot, float* __restrict__ part) {
  __shared__ float red[kBalanceThreads / 32][2 * kBalanceMaxExperts];
  const int t = blockIdx.x * kBalanceThreads + threadIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* in = logits + static_cast<long>(min(t, n - 1)) * pitch;
  const long id = t < n ? ids[static_cast<long>(t) * id_stride] : -1;
  float prob[TOT];
  row_softmax<T, TOT>(in, tot, prob);
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    if (e < tot) {
      float p = SWITCH ? prob[e] : rounded<T>(prob[e]);
      if (t >= n) p = 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
      const int c = __popc(__ballot_sync(0xffffffffu, id == e));
      if (lane == 0) {
        red[warp][e] = static_cast<float>(c);
        red[warp][tot + e] = p;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * tot; i += kBalanceThreads) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kBalanceThreads / 32; ++w) s += red[w][i];
    part[static_cast<long>(blockIdx.x) * 2 * tot + i] = s;
  }
}

// One block: adds the blocks' sums.  `weight` [tot] receives d loss / d P_e of Switch, the shares
// c_e of GShard.
template <typename T, bool SWITCH>
__global__ void __launch_bounds__(1024)
balance_finish_kernel(const float* __restrict__ part, int blocks, int n, int tot, float scale,
                      float* __restrict__ loss, float* __restrict__ weight) {
  __shared__ float red[32][2 * kBalanceMaxExperts];
  __shared__ float total[2 * kBalanceMaxExperts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = lane; i < 2 * tot; i += 32) {
    float s = 0.f;
    for (int b = warp; b < blocks; b += 32) s += part[static_cast<long>(b) * 2 * tot + i];
    red[warp][i] = s;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * tot; i += blockDim.x) {
    float s = 0.f;
    for (int w = 0; w < 32; ++w) s += red[w][i];
    total[i] = s;
  }
  __syncthreads();
  const float inv_n = 1.f / static_cast<float>(n);
  float factor = inv_n;
  if (SWITCH) {
    float kept = 0.f;
    for (int e = 0; e < tot; ++e) kept += total[e];
    kept = fmaxf(kept, 1.f);
    factor = scale / (kept * kept);
  }
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int e = 0; e < tot; ++e) {
      s += SWITCH ? total[e] * total[tot + e] : total[e] * inv_n * rounded<T>(total[tot + e] * inv_n);
    }
    *loss = SWITCH ? s * factor : s * (1.f / static_cast<float>(tot)) * scale;
  }
  for (int e = threadIdx.x; e < tot; e += blockDim.x) weight[e] = total[e] * factor;
}

// Switch: dlogits[t, e] = p_e g_e - p_e sum_i p_i g_i with g_e = dloss * weight_e, and, for a score
// that is the probability of expert win[t], dscore[t] added to g of that expert (win / dscore may
// be null).  GShard: the same with g_e = dloss scale / tot c_e / n, in the steps and roundings of
// the operations' backwards (mean, product, cast, mean over the tokens, softmax).
template <typename T, bool SWITCH, int TOT>
__global__ void __launch_bounds__(kBalanceThreads)
balance_bwd_kernel(const T* __restrict__ logits, long pitch, const float* __restrict__ weight,
                   const float* __restrict__ dloss, const int64_t* __restrict__ win, const T* __restrict__ dscore,
                   float scale, int n, int tot, T* __restrict__ dlogits) {
  const int t = blockIdx.x * kBalanceThreads + threadIdx.x;
  if (t >= n) return;
  T* out = dlogits + static_cast<long>(t) * tot;
  float p[TOT], pg[TOT];
  row_softmax<T, TOT>(logits + static_cast<long>(t) * pitch, tot, p);
  float gl = dloss != nullptr ? *dloss : 0.f;
  const float gs = dscore != nullptr ? Ld<T>::get(dscore, t) : 0.f;
  const long w = win != nullptr ? win[t] : -1;
  const float inv_n = 1.f / static_cast<float>(n);
  if (!SWITCH) gl = gl * scale * (1.f / static_cast<float>(tot));
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    pg[e] = 0.f;
    if (e < tot) {
      if (SWITCH) {
        pg[e] = p[e] * (gl * weight[e] + (e == w ? gs : 0.f));
      } else {
        p[e] = rounded<T>(p[e]);
        pg[e] = rounded<T>(rounded<T>(rounded<T>(gl * weight[e]) * inv_n) * p[e]);
      }
    }
  }
  const float sum = sum_experts<TOT>(pg);
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    if (e < tot) Ld<T>::put(out, e, pg[e] - p[e] * sum);
  }
}

// Switch: the most probable expert (the lower id wins a tie) and its softmax probability.
template <typename T, int TOT>
__global__ void __launch_bounds__(kBalanceThreads)
switch_top1_kernel(const T* __restrict__ logits, int n, int tot, int64_t* __restrict__ win, T* __restrict__ score) {
  const int t = blockIdx.x * kBalanceThreads + threadIdx.x;
  if (t >= n) return;
  float p[TOT];
  row_softmax<T, TOT>(logits + static_cast<long>(t) * tot, tot, p);
  // as torch.max over the probabilities: NaN counts as the largest, the first of equals wins
  int best = 0;
  float best_p = p[0];
#pragma unroll
  for (int e = 1; e < TOT; ++e) {
    if (e < tot && (p[e] > best_p || (p[e] != p[e] && best_p == best_p))) {
      best = e;
      best_p = p[e];
    }
  }
  win[t] = best;
  Ld<T>::put(score, t, best_p);
}

// What the tensor-core gate multiplies with when its experts are no multiple of 64: one launch where padding,
// filling and copying were four (a layer's step, eager, 16 experts, 1237 tokens, d 256: 472 -> 430 us).
template <typename T>
__global__ void __launch_bounds__(256)
gate_pad_kernel(const T* __restrict__ w, const T* __restrict__ bias, int tot, int padded, int d, T* __restrict__ w_out,
                T* __restrict__ bias_out) {
  ptx::chain_begin();
  const long held = static_cast<long>(tot) * d / 8, all = static_cast<long>(padded) * d / 8;
  for (long i = static_cast<long>(blockIdx.x) * 256 + threadIdx.x; i < all; i += static_cast<long>(gridDim.x) * 256) {
    reinterpret_cast<uint4*>(w_out)[i] = i < held ? reinterpret_cast<const uint4*>(w)[i] : make_uint4(0u, 0u, 0u, 0u);
  }
  if (blockIdx.x == 0) {
    for (int e = threadIdx.x; e < padded; e += 256) {
      // (-30000: representable in both types)
      bias_out[e] = e >= tot ? V2<T>::from_f(-30000.f) : bias != nullptr ? bias[e] : V2<T>::from_f(0.f);
    }
  }
}

// Host values that travel with the launch, in place of the operations that formed the prefix on the host and a
// copy from pageable memory: a grouped linear's forward and backward, 16 experts, 142 rows, d 320, 197 -> 162 us.
template <int N> struct HostValues {
  int v[N];
};
template <int N>
__global__ void host_offsets_kernel(const __grid_constant__ HostValues<N> values, int n, int* __restrict__ dst) {
  ptx::chain_begin();
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = values.v[i];
}

// out[s] = idx[s] when fewer than `cap` slots of its expert come before it, else -1
__global__ void prune_scalar_kernel(const int64_t* __restrict__ idx, const int* __restrict__ rank, int cap, int n_slots,
                                    int tot, int64_t* __restrict__ out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const long e = idx[s];
  out[s] = (e >= 0 && e < tot && rank[s] < cap) ? e : -1;
}

// ------------------------------------------------------------------------------ fused gate
// logits = x W^T + b for a handful of experts (tot <= kGateMaxExperts), top-k and softmax of the
// selected logits, one warp per token: x is read once, W comes from L1/L2, nothing but the
// [B, tot] logits and the [B, k] ids / probabilities is written.
constexpr int kGateMaxExperts = 64;

template <typename T, int TOT>
__global__ void __launch_bounds__(256)
gate_linear_topk_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias,
                        int n_rows, int d, int tot, int k, T* __restrict__ logits,
                        int64_t* __restrict__ idx, T* __restrict__ prob, float* zero) {
  if (zero != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero = 0.f;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  float acc[TOT];
#pragma unroll
  for (int e = 0; e < TOT; ++e) acc[e] = 0.f;
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<long>(row) * d);
  const int nv = d >> 3;
#pragma unroll 4
  for (int i = lane; i < nv; i += 32) {
    float xf[8];
    unpack8<T>(__ldg(xr + i), xf);
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      if (e < tot) {
        float wf[8];
        unpack8<T>(__ldg(reinterpret_cast<const uint4*>(w + static_cast<long>(e) * d) + i), wf);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[e] = fmaf(xf[q], wf[q], acc[e]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if (e < tot && bias != nullptr) acc[e] += V2<T>::to_f(bias[e]);
    // the logits leave in the layer's dtype; selection below uses the rounded values so that
    // ids and probabilities are consistent with what autograd consumers see
    if (e < tot) acc[e] = V2<T>::to_f(V2<T>::from_f(acc[e]));
  }
  if (lane < tot) {
    float mine = 0.f;
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      if (e == lane) mine = acc[e];
    }
    logits[static_cast<long>(row) * tot + lane] = V2<T>::from_f(mine);
  }
  if (TOT > 32 && lane + 32 < tot) {
    float mine = 0.f;
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      if (e == lane + 32) mine = acc[e];
    }
    logits[static_cast<long>(row) * tot + lane + 32] = V2<T>::from_f(mine);
  }
  if (lane == 0) {
    float sel_v[kMaxK];
    int sel_i[kMaxK];
    unsigned long long taken = 0ull;
    for (int j = 0; j < k; ++j) {
      float best = -INFINITY;
      int best_i = -1;
#pragma unroll
      for (int e = 0; e < TOT; ++e) {
        if (e < tot && !((taken >> e) & 1ull) && (best_i < 0 || acc[e] > best)) {
          best = acc[e];
          best_i = e;
        }
      }
      taken |= 1ull << best_i;
      sel_v[j] = best;
      sel_i[j] = best_i;
    }
    float den = 0.f, ex[kMaxK];
    for (int j = 0; j < k; ++j) {
      ex[j] = __expf(sel_v[j] - sel_v[0]);
      den += ex[j];
    }
    for (int j = 0; j < k; ++j) {
      idx[static_cast<long>(row) * k + j] = sel_i[j];
      prob[static_cast<long>(row) * k + j] = V2<T>::from_f(ex[j] / den);
    }
  }
}

// The same for a few tokens and 9 to 64 experts: one block per token, a warp for every eighth expert.
// All of W comes out of the L2 once per token, which at 64 experts, d = 1024 is 128 KB: 64 tokens 6.0
// us, where padding W and the bias, the tensor-core product and the top-k were five launches, 16.5 us.
template <typename T>
__global__ void __launch_bounds__(256)
gate_linear_topk_few_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias, int d, int tot,
                            int k, T* __restrict__ logits, int64_t* __restrict__ idx, T* __restrict__ prob, float* zero) {
  ptx::chain_begin();
  if (zero != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero = 0.f;
  __shared__ T row_logits[kGateMaxExperts];
  constexpr int PER = kGateMaxExperts / 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long row = blockIdx.x;
  float acc[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) acc[u] = 0.f;
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * d);
  const int nv = d >> 3;
  const int mine = (tot - warp + 7) / 8;   // experts warp, warp + 8, ...
  for (int i = lane; i < nv; i += 32) {
    uint4 wv[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (u < mine) wv[u] = __ldg(reinterpret_cast<const uint4*>(w + static_cast<long>(warp + 8 * u) * d) + i);
    }
    float xf[8];
    unpack8<T>(__ldg(xr + i), xf);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (u < mine) {
        float wf[8];
        unpack8<T>(wv[u], wf);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[u] = fmaf(xf[q], wf[q], acc[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (u < mine) {
      float v = acc[u];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      const int e = warp + 8 * u;
      if (bias != nullptr) v += V2<T>::to_f(bias[e]);
      if (lane == 0) {
        row_logits[e] = V2<T>::from_f(v);
        logits[row * tot + e] = V2<T>::from_f(v);
      }
    }
  }
  __syncthreads();
  if (warp != 0) return;
  // the choice and the probabilities follow the rounded logits
  const bool on0 = lane < tot, on1 = lane + 32 < tot;
  const float v0 = on0 ? V2<T>::to_f(row_logits[lane]) : 0.f, v1 = on1 ? V2<T>::to_f(row_logits[lane + 32]) : 0.f;
  if (!__any_sync(0xffffffffu, v0 != v0 || v1 != v1)) {
    topk_row64<T>(v0, v1, on0, on1, lane, k, idx + row * k, prob + row * k);
  } else {
    topk_row<T>(row_logits, tot, lane, k, idx + row * k, prob + row * k);
  }
}

// The same result for R tokens per warp, TOT <= 8 and R * TOT <= 32: a slice of W is loaded and
// unpacked once for R tokens, and the R * TOT sums over the lanes are formed together (each
// exchange step halves the number of values a lane still holds; the additions are those of the
// one-token kernel, in the same tree).  Loads carry no predicates: with `e < tot` around each the
// slices of W arrived one after the other.  Measured: 8192 tokens, d = 2048, 8 experts 34 -> 17.6
// us (4 tokens per warp; 25.5 with 2, 30.3 with 1), 11264 tokens, d = 512 18.8 -> 9.5 us, 8 tokens,
// d = 1024 10.5 -> 7.3 us; 3001 tokens are the same with 1, 2 or 4.
template <typename T, int TOT, int R>
__global__ void __launch_bounds__(256)
gate_linear_topk_rows_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ bias,
                             int n_rows, int d, int tot, int k, T* __restrict__ logits,
                             int64_t* __restrict__ idx, T* __restrict__ prob, float* zero) {
  ptx::chain_begin();
  if (zero != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *zero = 0.f;
  constexpr int V = R * TOT;
  const int row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
  const int lane = threadIdx.x & 31;
  if (row0 >= n_rows) return;
  float acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.f;
  constexpr int W = kPer16<T>;
  const int nv = d / W;
  const uint4* xr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) xr[r] = reinterpret_cast<const uint4*>(x + static_cast<long>(min(row0 + r, n_rows - 1)) * d);
#pragma unroll(R == 1 ? 4 : 2)
  for (int i = lane; i < nv; i += 32) {
    uint4 xv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) xv[r] = __ldg(xr[r] + i);
    uint4 wv[TOT];
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      // (past the last expert the last one again, for nothing: the loads need no predicate)
      wv[e] = __ldg(reinterpret_cast<const uint4*>(w + static_cast<long>(min(e, tot - 1)) * d) + i);
    }
    float xf[R][W];
#pragma unroll
    for (int r = 0; r < R; ++r) unpack16<T>(xv[r], xf[r]);
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      float wf[W];
      unpack16<T>(wv[e], wf);
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int q = 0; q < W; ++q) acc[r * TOT + e] = fmaf(xf[r][q], wf[q], acc[r * TOT + e]);
      }
    }
  }
  // value v of the warp ends in the lanes whose low bits, read from 16 down, spell v
  int held = V, at = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (held > 1) {
      held >>= 1;
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int v = 0; v < V / 2; ++v) {
        if (v < held) {
          const float send = up ? acc[v] : acc[v + held];
          const float keep = up ? acc[v + held] : acc[v];
          acc[v] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      if (up) at += held;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    }
  }
  const int r = at / TOT, e_of = at % TOT;
  float mine = acc[0];
  if (e_of < tot && bias != nullptr) mine += V2<T>::to_f(bias[e_of]);
  mine = V2<T>::to_f(V2<T>::from_f(mine));   // ids and probabilities follow the rounded logits
  constexpr int kStep = 32 / V;                 // lanes that hold the same value
  const bool row_ok = row0 + r < n_rows;
  if (row_ok && e_of < tot && (lane & (kStep - 1)) == 0) {
    logits[static_cast<long>(row0 + r) * tot + e_of] = V2<T>::from_f(mine);
  }
  // Every lane ranks its logit among those of its token (ties to the lower id) and writes the
  // entry of that rank: a handful of instructions where a selection loop unrolled into
  // registers was long enough to be bound by instruction fetch (8 tokens: 17 us).
  const int base = lane & ~(TOT * kStep - 1);   // first lane of this token's group
  const float key = (e_of < tot && mine == mine) ? mine : -INFINITY;
  int pos = 0;
  float top = -INFINITY;
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    const float other = __shfl_sync(0xffffffffu, key, base + e * kStep);
    pos += (other > key || (other == key && e < e_of)) ? 1 : 0;
    top = fmaxf(top, other);
  }
  const bool chosen = e_of < tot && pos < k;
  const float ex = chosen ? __expf(mine - top) : 0.f;
  float den = ex;
#pragma unroll
  for (int o = kStep; o < TOT * kStep; o <<= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
  const bool writes = row_ok && (lane & (kStep - 1)) == 0;
  const long out = static_cast<long>(row0 + r) * k;
  const bool nan = e_of < tot && mine != mine;
  if (!__any_sync(0xffffffffu, nan)) {
    if (writes && chosen) {
      idx[out + pos] = e_of;
      prob[out + pos] = V2<T>::from_f(ex / den);
    }
    return;
  }
  // With a NaN in the warp the choice is what k scans over the experts left give, in which only a
  // greater logit replaces the first one: a NaN that comes first is chosen, and makes all scores of
  // its token NaN.  (After the usual path, whose registers these loops would cost.)
  pos = TOT;
#pragma unroll 1
  for (int j = 0; j < k; ++j) {
    float best = 0.f;
    int best_e = -1;
#pragma unroll 1
    for (int e = 0; e < tot; ++e) {
      const float other = __shfl_sync(0xffffffffu, mine, base + e * kStep);
      const int taken = __shfl_sync(0xffffffffu, pos, base + e * kStep) < TOT;
      if (!taken && (best_e < 0 || other > best)) {
        best = other;
        best_e = e;
      }
    }
    if (best_e == e_of) pos = j;
  }
  const float again = pos < k ? __expf(mine - top) : 0.f;
  float sum = again;
#pragma unroll
  for (int o = kStep; o < TOT * kStep; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (writes && pos < k) {
    idx[out + pos] = e_of;
    prob[out + pos] = V2<T>::from_f(again / sum);
  }
}

// dl[t, e] = softmax backward of the selected logits scattered to their experts, plus the
// gradient that reached the logits directly (may be null).  dx[t, :] = sum_e dl[t, e] W[e, :].
// dl is written out (fp32) for the weight-gradient kernel.  One warp per token; every lane forms
// the dl of one expert and the warp shares them.  9 and more experts (fewer: below).
template <typename T, int TOT>
__global__ void __launch_bounds__(256)
gate_bwd_dx_kernel(const T* __restrict__ dprob, const int64_t* __restrict__ idx,
                   const T* __restrict__ prob, const T* __restrict__ dlogits_in,
                   const T* __restrict__ w, int n_rows, int d, int tot, int k,
                   float* __restrict__ dl_out, T* __restrict__ dx) {
  ptx::chain_begin();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  float dl[TOT];
#pragma unroll
  for (int e0 = 0; e0 < TOT; e0 += 32) {
    const int e = e0 + lane;
    float mine = 0.f;
    if (e < tot) {
      if (dlogits_in != nullptr) mine = V2<T>::to_f(dlogits_in[static_cast<long>(row) * tot + e]);
      if (dprob != nullptr) {
        const T* g = dprob + static_cast<long>(row) * k;
        const T* p = prob + static_cast<long>(row) * k;
        const int64_t* id = idx + static_cast<long>(row) * k;
        float dotp = 0.f;
        for (int j = 0; j < k; ++j) dotp += V2<T>::to_f(g[j]) * V2<T>::to_f(p[j]);
        for (int j = 0; j < k; ++j) {
          if (id[j] == e) mine += V2<T>::to_f(p[j]) * (V2<T>::to_f(g[j]) - dotp);
        }
      }
      dl_out[static_cast<long>(row) * tot + e] = mine;
    }
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      if (e0 + u < TOT) dl[e0 + u] = __shfl_sync(0xffffffffu, mine, u);
    }
  }
  if (dx == nullptr) return;
  uint4* out = reinterpret_cast<uint4*>(dx + static_cast<long>(row) * d);
  const int nv = d >> 3;
#pragma unroll 4
  for (int i = lane; i < nv; i += 32) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      if (e < tot && dl[e] != 0.f) {
        float wf[8];
        unpack8<T>(__ldg(reinterpret_cast<const uint4*>(w + static_cast<long>(e) * d) + i), wf);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fmaf(dl[e], wf[q], acc[q]);
      }
    }
    out[i] = pack8<T>(acc);
  }
}

// The same for R tokens per warp, TOT <= 8: a slice of W is loaded and unpacked once for R tokens, and
// its loads carry no predicates.  The sums are those of the one-token kernel.  All of the gate's
// backward, 8192 tokens, d = 2048, 8 experts: 35 us, 41 with gradients at all logits; with this kernel
// and dl in shared memory in the next one 30 and 33, with that one's sums of dl shared out and four
// chains in the merge 28 and 31 (16384 tokens, d = 256: 18.9 -> 17.1).
template <typename T, int TOT, int R>
__global__ void __launch_bounds__(256)
gate_bwd_dx_rows_kernel(const T* __restrict__ dprob, const int64_t* __restrict__ idx, const T* __restrict__ prob,
                        const T* __restrict__ dlogits_in, const T* __restrict__ w, int n_rows, int d, int tot, int k,
                        float* __restrict__ dl_out, T* __restrict__ dx) {
  ptx::chain_begin();
  const int row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * R;
  const int lane = threadIdx.x & 31;
  if (row0 >= n_rows) return;
  float mine = 0.f;
  {
    const int row = row0 + lane / TOT, e = lane % TOT;
    if (lane < R * TOT && row < n_rows && e < tot) {
      if (dlogits_in != nullptr) mine = V2<T>::to_f(dlogits_in[static_cast<long>(row) * tot + e]);
      if (dprob != nullptr) {
        const T* g = dprob + static_cast<long>(row) * k;
        const T* p = prob + static_cast<long>(row) * k;
        const int64_t* id = idx + static_cast<long>(row) * k;
        float dotp = 0.f;
        for (int j = 0; j < k; ++j) dotp += V2<T>::to_f(g[j]) * V2<T>::to_f(p[j]);
        for (int j = 0; j < k; ++j) {
          if (id[j] == e) mine += V2<T>::to_f(p[j]) * (V2<T>::to_f(g[j]) - dotp);
        }
      }
      dl_out[static_cast<long>(row) * tot + e] = mine;
    }
  }
  if (dx == nullptr) return;
  float dl[R][TOT];
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int e = 0; e < TOT; ++e) dl[r][e] = __shfl_sync(0xffffffffu, mine, r * TOT + e);
  }
  constexpr int W = kPer16<T>;
  const int nv = d / W;
#pragma unroll 2
  for (int i = lane; i < nv; i += 32) {
    uint4 wv[TOT];
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      // (past the last expert the last one again, for nothing)
      wv[e] = __ldg(reinterpret_cast<const uint4*>(w + static_cast<long>(min(e, tot - 1)) * d) + i);
    }
    float acc[R][W];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int q = 0; q < W; ++q) acc[r][q] = 0.f;
    }
#pragma unroll
    for (int e = 0; e < TOT; ++e) {
      float wf[W];
      unpack16<T>(wv[e], wf);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        // (the same for the whole warp; an expert without gradient adds nothing, but in 32 bits, where
        // 0 times an infinite weight is NaN, as a product makes it)
        if (sizeof(T) == 4 ? e < tot : dl[r][e] != 0.f) {
#pragma unroll
          for (int q = 0; q < W; ++q) acc[r][q] = fmaf(dl[r][e], wf[q], acc[r][q]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (row0 + r < n_rows) reinterpret_cast<uint4*>(dx + static_cast<long>(row0 + r) * d)[i] = pack16<T>(acc[r]);
    }
  }
}

// Partial sums of dW[e, c] = sum_t dl[t, e] x[t, c] and db[e] = sum_t dl[t, e] over one of
// `gridDim.y` token ranges: part[range][tot * d + tot] in fp32.  A block takes a strip of 256 columns
// (fp32: 128); a lane owns eight (four) of them, so that a token is one 16-byte load per lane (two columns per lane,
// as before, kept too few bytes in flight).  The ranges used to be merged with atomics on a
// zeroed buffer: 296 additions per address took most of the 20 us of 16384 tokens with d = 256,
// which take 6 us now and 5 in the merge; 8192 tokens, d = 2048, 8 experts 40 -> 18 us, 11264 tokens,
// d = 512 19 -> 10 us.  Two blocks per SM; with one 29 and 13 us.
template <typename T, int TOT>
__global__ void __launch_bounds__(256, TOT <= 8 ? 2 : 1)
gate_bwd_dw_kernel(const float* __restrict__ dl, const T* __restrict__ x, int n_rows, int d, int tot,
                   float* __restrict__ part) {
  ptx::chain_begin();
  constexpr int CHUNK = 128;   // tokens whose dl are held at a time: a multiple of the warps' step of 32
  constexpr int W = kPer16<T>, STRIP = 32 * W;
  __shared__ float red[8][STRIP];
  __shared__ __align__(16) float dls[CHUNK][TOT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * STRIP + lane * W;
  const int per = (n_rows + gridDim.y - 1) / gridDim.y;
  const int t0 = blockIdx.y * per, t1 = min(n_rows, t0 + per);
  const bool sums = blockIdx.x == 0;
  float* mine = part + static_cast<long>(blockIdx.y) * (static_cast<long>(tot) * d + tot);
  __shared__ float bred[8][TOT];
  float acc[TOT][W], bsum = 0.f;   // bsum: of expert threadIdx.x % TOT
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
#pragma unroll
    for (int q = 0; q < W; ++q) acc[e][q] = 0.f;
  }
  constexpr int U = 4;
  for (int c0 = t0; c0 < t1; c0 += CHUNK) {
    const int c1 = min(t1, c0 + CHUNK);
    __syncthreads();
    for (int i = threadIdx.x; i < CHUNK * TOT; i += 256) {
      const int t = c0 + i / TOT, e = i % TOT;
      const float v = t < c1 && e < tot ? __ldg(dl + static_cast<long>(t) * tot + e) : 0.f;
      dls[i / TOT][e] = v;
      if (sums) bsum += v;
    }
    __syncthreads();
    for (int t = c0 + warp; t < c1; t += 8 * U) {
      uint4 xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        xv[u] = (t + 8 * u < c1 && col < d) ? __ldg(reinterpret_cast<const uint4*>(x + static_cast<long>(t + 8 * u) * d + col))
                                            : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (t + 8 * u >= c1) break;
        float xf[W], g[TOT];
        unpack16<T>(xv[u], xf);
#pragma unroll
        for (int e = 0; e < TOT; e += 2) {
          const float2 two = *reinterpret_cast<const float2*>(&dls[t + 8 * u - c0][e]);
          g[e] = two.x;
          g[e + 1] = two.y;
        }
#pragma unroll
        for (int e = 0; e < TOT; ++e) {
#pragma unroll
          for (int q = 0; q < W; ++q) acc[e][q] = fmaf(g[e], xf[q], acc[e][q]);
        }
      }
    }
  }
  if (sums) {   // short chains: the sum of a softmax's gradients over the tokens cancels
#pragma unroll
    for (int o = 16; o >= TOT; o >>= 1) bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
    if (lane < TOT) bred[warp][lane] = bsum;
  }
#pragma unroll
  for (int e = 0; e < TOT; ++e) {
    if (e >= tot) break;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < W; ++q) red[warp][lane * W + q] = acc[e][q];
    __syncthreads();
    const int c = blockIdx.x * STRIP + threadIdx.x;
    if (threadIdx.x < STRIP && c < d) {
      float s = 0.f;
#pragma unroll
      for (int wv = 0; wv < 8; ++wv) s += red[wv][threadIdx.x];
      mine[static_cast<long>(e) * d + c] = s;
    }
    if (sums && threadIdx.x == 0) {
      float s[8];
#pragma unroll
      for (int wv = 0; wv < 8; ++wv) s[wv] = bred[wv][e];
      mine[static_cast<long>(tot) * d + e] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
    }
  }
}

// out[i] = sum over the ranges of part[range][i], in a fixed order, in the layer's type: eight
// lanes of ranges per 32 elements, in short chains (a gradient of the bias cancels).
template <typename T>
__global__ void __launch_bounds__(256)
gate_bwd_merge_kernel(const float* __restrict__ part, int ranges, long elems, T* __restrict__ out) {
  ptx::chain_begin();
  __shared__ float red[8][33];
  const int sub = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long i = static_cast<long>(blockIdx.x) * 32 + lane;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  if (i < elems) {
    int r = sub;
#pragma unroll 2
    for (; r + 24 < ranges; r += 32) {
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] += __ldg(part + static_cast<long>(r + 8 * u) * elems + i);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      if (r + 8 * u < ranges) s[u] += __ldg(part + static_cast<long>(r + 8 * u) * elems + i);
    }
  }
  red[sub][lane] = (s[0] + s[1]) + (s[2] + s[3]);
  __syncthreads();
  if (sub == 0 && i < elems) {
    float t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = red[u][lane];
    out[i] = V2<T>::from_f(((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7])));
  }
}

// ------------------------------------------------------------------------------ SIMT GEMM
template <typename T> struct Acc { using type = float; };
template <> struct Acc<double> { using type = double; };

template <typename T> __device__ __forceinline__ typename Acc<T>::type ldv(const T* p, long i) {
  return static_cast<typename Acc<T>::type>(p[i]);
}
template <> __device__ __forceinline__ float ldv<__nv_bfloat16>(const __nv_bfloat16* p, long i) {
  return __bfloat162float(p[i]);
}
template <> __device__ __forceinline__ float ldv<__half>(const __half* p, long i) {
  return __half2float(p[i]);
}
template <typename T> __device__ __forceinline__ void stv(T* p, long i, typename Acc<T>::type v) {
  p[i] = static_cast<T>(v);
}
template <> __device__ __forceinline__ void stv<__nv_bfloat16>(__nv_bfloat16* p, long i, float v) {
  p[i] = __float2bfloat16(v);
}
template <> __device__ __forceinline__ void stv<__half>(__half* p, long i, float v) {
  p[i] = __float2half(v);
}

// Shared-memory tiled SIMT GEMM for fp64, for fp32 with rows that are not 16-byte aligned (split_gemm.cu and
// sgemm.cu take the others) and for 16-bit shapes the tensor-core kernel does not take.  One CTA of 256
// threads computes a 64 x 64 tile of C = A B with a K step of 16; every thread owns a 4 x 4 block of the tile
// and accumulates in fp32 (fp64 for doubles).  The three products of a grouped linear differ only in where
// A(i, kk) and B(kk, j) live:
//   mode 0 (NT)   rows of expert g:  A = a[row, kk],   B = b[g, j, kk]
//   mode 1 (NN)   rows of expert g:  A = a[row, kk],   B = b[g, kk, j]
//   mode 2 (wgrad) out[g, i, j]:     A = p[r0 + kk, i], B = q[r0 + kk, j], K = rows of expert g
// (the reference calls cublasSgemm / cublasDgemm per expert here, cuda/utils/cublas_wrapper.h:51-72).
constexpr int kSimtTile = 64;
constexpr int kSimtK = 16;

template <typename T, int MODE>
__global__ void __launch_bounds__(256)
simt_tiled_kernel(int num_groups, long rows_cap, int m, int n, int k, const T* __restrict__ a, const T* __restrict__ b,
                  const int* __restrict__ offs, const T* __restrict__ bias, T* __restrict__ out) {
  using A = typename Acc<T>::type;
  __shared__ A As[kSimtK][kSimtTile + 4];
  __shared__ A Bs[kSimtK][kSimtTile + 4];
  int g, i0, rows_i, kk_total, row_base;
  const int j0 = blockIdx.y * kSimtTile;
  if (MODE == 2) {
    g = blockIdx.z;
    i0 = blockIdx.x * kSimtTile;
    rows_i = m;
    row_base = offs[g];
    kk_total = offs[g + 1] - row_base;
  } else {
    // blockIdx.x walks the 64-row pieces of all experts: find the expert this piece belongs to
    int piece = blockIdx.x;
    bool found = false;
    for (g = 0; g < num_groups; ++g) {
      const int cnt = offs[g + 1] - offs[g];
      const int pieces = (cnt + kSimtTile - 1) / kSimtTile;
      if (piece < pieces) {
        found = true;
        break;
      }
      piece -= pieces;
    }
    if (!found) {
      // no piece left: zero the rows past the last expert, so that what is applied to the whole
      // buffer afterwards meets no stale bits
      const long r0 = static_cast<long>(offs[num_groups]) + static_cast<long>(piece) * kSimtTile;
      for (int it = threadIdx.x; it < kSimtTile * kSimtTile; it += blockDim.x) {
        const long r = r0 + it / kSimtTile;
        const int j = j0 + it % kSimtTile;
        if (r < rows_cap && j < n) stv<T>(out, r * n + j, 0);
      }
      return;
    }
    row_base = offs[g];
    i0 = piece * kSimtTile;
    rows_i = offs[g + 1] - row_base;
    kk_total = k;
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  A acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0;
  }
  for (int kk0 = 0; kk0 < kk_total; kk0 += kSimtK) {
    // 16 x 64 elements of each operand, 4 per thread
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int e = threadIdx.x + l * 256;
      int kk, ii;
      if (MODE == 2) { kk = e / kSimtTile; ii = e % kSimtTile; }    // A is row-major over (kk, i)
      else { ii = e / kSimtK; kk = e % kSimtK; }                    // A is row-major over (i, kk)
      A va = 0;
      if (kk0 + kk < kk_total && i0 + ii < rows_i) {
        va = MODE == 2 ? ldv<T>(a, static_cast<long>(row_base + kk0 + kk) * m + i0 + ii)
                       : ldv<T>(a, static_cast<long>(row_base + i0 + ii) * k + kk0 + kk);
      }
      As[kk][ii] = va;
      int kb, jj;
      if (MODE == 0) { jj = e / kSimtK; kb = e % kSimtK; }          // B is row-major over (j, kk)
      else { kb = e / kSimtTile; jj = e % kSimtTile; }              // B is row-major over (kk, j)
      A vb = 0;
      if (kk0 + kb < kk_total && j0 + jj < n) {
        if (MODE == 0) vb = ldv<T>(b, (static_cast<long>(g) * n + j0 + jj) * k + kk0 + kb);
        else if (MODE == 1) vb = ldv<T>(b, (static_cast<long>(g) * k + kk0 + kb) * n + j0 + jj);
        else vb = ldv<T>(b, static_cast<long>(row_base + kk0 + kb) * n + j0 + jj);
      }
      Bs[kb][jj] = vb;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kSimtK; ++kk) {
      A ra[4], rb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) ra[u] = As[kk][ty * 4 + u];
#pragma unroll
      for (int v = 0; v < 4; ++v) rb[v] = Bs[kk][tx * 4 + v];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] += ra[u] * rb[v];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int ii = i0 + ty * 4 + u;
    if (ii >= rows_i) continue;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int jj = j0 + tx * 4 + v;
      if (jj >= n) continue;
      A val = acc[u][v];
      if (MODE != 2 && bias != nullptr) val += ldv<T>(bias, static_cast<long>(g) * n + jj);
      const long o = MODE == 2 ? (static_cast<long>(g) * m + ii) * n + jj
                               : static_cast<long>(row_base + ii) * n + jj;
      stv<T>(out, o, val);
    }
  }
}

template <typename T>
cudaError_t simt_typed(int mode, int num_groups, long rows_cap, int m, int n, int k, const void* a,
                       const void* b, const int* offs, const void* bias, void* out,
                       cudaStream_t stream) {
  const T* ap = static_cast<const T*>(a);
  const T* bp = static_cast<const T*>(b);
  const T* biasp = static_cast<const T*>(bias);
  T* op = static_cast<T*>(out);
  const unsigned nt = (n + kSimtTile - 1) / kSimtTile;
  if (mode == 2) {
    dim3 grid((m + kSimtTile - 1) / kSimtTile, nt, num_groups);
    simt_tiled_kernel<T, 2><<<grid, 256, 0, stream>>>(num_groups, rows_cap, m, n, k, ap, bp, offs, biasp, op);
  } else {
    if (rows_cap == 0) return cudaSuccess;
    dim3 grid(static_cast<unsigned>((rows_cap + kSimtTile - 1) / kSimtTile + num_groups), nt);
    if (mode == 0) {
      simt_tiled_kernel<T, 0><<<grid, 256, 0, stream>>>(num_groups, rows_cap, m, n, k, ap, bp, offs, biasp, op);
    } else {
      simt_tiled_kernel<T, 1><<<grid, 256, 0, stream>>>(num_groups, rows_cap, m, n, k, ap, bp, offs, biasp, op);
    }
  }
  return cudaGetLastError();
}

}  // namespace

// ------------------------------------------------------------------------------ launchers
int route_blocks(int n_slots, int tot) {
  // one launch up to what a cluster, or a single CTA where the cluster does not apply, holds; beyond
  // that 16 K slots per CTA (1025 experts: 40000 slots 58 us on three CTAs, 97 on one; 65536 slots 67
  // and 154; 65536 slots on 1024 experts 28 on the cluster)
  if (n_slots <= (tot <= kRouteClusterExperts ? kRouteClusterSlots : kRouteCtaSlots)) return 1;
  int nb = (n_slots + 16383) / 16384;
  return nb > 148 ? 148 : nb;
}

cudaError_t launch_route(const int64_t* idx, int n_slots, int tot, int* counts, int* rank,
                         int* offs, int* pos, int* part, cudaStream_t stream) {
  if (tot <= 0) return cudaErrorInvalidValue;
  int nw = (kRouteSmemLimit - 4 * (tot + 1)) / (4 * tot);
  if (nw < 1) return cudaErrorInvalidValue;
  if (nw > 32) nw = 32;
  const int nb = part != nullptr ? route_blocks(n_slots, tot) : 1;
  // below 1 K slots one CTA has at most one step per warp and pass: nothing to spread; with very
  // many experts the histograms of fewer warps fit beside the cluster's totals
  const bool cluster = nb == 1 && n_slots > 1024 && tot <= kRouteClusterExperts;
  const int ctas = cluster ? kRouteCluster : nb;
  int cta_slots = (n_slots + ctas - 1) / ctas;
  cta_slots = (cta_slots + 31) & ~31;
  if (cta_slots < 32) cta_slots = 32;
  const int by_work = (cta_slots + 31) / 32;
  if (nw > by_work) nw = by_work > 0 ? by_work : 1;
  const size_t smem = static_cast<size_t>(nw) * tot * 4 + static_cast<size_t>(cluster ? 2 * tot + 1 : tot + 1) * 4;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(route_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kRouteSmemLimit);
    if (e != cudaSuccess) return e;
  }
  const int* none_in = nullptr;
  int* none_out = nullptr;
  if (nb > 1) {
    const cudaError_t e = launch_chained(route_kernel, dim3(nb), dim3(kRouteThreads), smem, stream, idx, n_slots, tot, nw,
                                         cta_slots, 0, none_in, part, counts, rank, offs, pos);
    if (e != cudaSuccess) return e;
    return launch_chained(route_kernel, dim3(nb), dim3(kRouteThreads), smem, stream, idx, n_slots, tot, nw, cta_slots, 0,
                          static_cast<const int*>(part), none_out, counts, rank, offs, pos);
  }
  if (!cluster) {
    return launch_chained(route_kernel, dim3(1), dim3(kRouteThreads), smem, stream, idx, n_slots, tot, nw, cta_slots, 0,
                          none_in, none_out, counts, rank, offs, pos);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kRouteCluster);
  cfg.blockDim = dim3(kRouteThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kRouteCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, route_kernel, idx, n_slots, tot, nw, cta_slots, 1, none_in, none_out,
                                           counts, rank, offs, pos);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

cudaError_t launch_swipe_mark(const int64_t* idx, const int* rank, const int* quota, int n,
                              int n_expert, int n_worker, int64_t* key, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  swipe_mark_kernel<<<(n + 255) / 256, 256, 0, stream>>>(idx, rank, quota, n, n_expert, n_worker, key);
  return cudaGetLastError();
}

cudaError_t launch_swipe_assign(const int64_t* idx, const int64_t* key, const int* mrank,
                                const int* count, const int* quota, int n, int n_expert,
                                int n_worker, int bias, int64_t* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  swipe_assign_kernel<<<(n + 255) / 256, 256, 0, stream>>>(idx, key, mrank, count, quota, n, n_expert,
                                                          n_worker, bias, out);
  return cudaGetLastError();
}

cudaError_t launch_prune(const int64_t* idx, const int* rank, const int* cap, int n_slots, int tot,
                         int64_t* new_idx, cudaStream_t stream) {
  if (n_slots == 0) return cudaSuccess;
  prune_kernel<<<(n_slots + 255) / 256, 256, 0, stream>>>(idx, rank, cap, n_slots, tot, new_idx);
  return cudaGetLastError();
}

cudaError_t launch_limit_by_capacity(const int64_t* ec, int* cap, int64_t* eca, int n_expert,
                                     int n_worker, cudaStream_t stream) {
  limit_kernel<<<(n_expert + 127) / 128, 128, 0, stream>>>(ec, cap, eca, n_expert, n_worker);
  return cudaGetLastError();
}

cudaError_t launch_fill_pos(const int64_t* idx, const int* rank, const int* cum_incl, int n_slots,
                            int tot, int64_t* pos, cudaStream_t stream) {
  if (n_slots == 0) return cudaSuccess;
  fill_pos_kernel<<<(n_slots + 255) / 256, 256, 0, stream>>>(idx, rank, cum_incl, n_slots, tot, pos);
  return cudaGetLastError();
}

#define FMOE_DISPATCH_16(dtype, ...)                                  \
  if ((dtype) == 0) { using T = __nv_bfloat16; __VA_ARGS__; }         \
  else { using T = __half; __VA_ARGS__; }
#define FMOE_DISPATCH_ANY(dtype, ...)                                 \
  if ((dtype) == 2) { using T = float; __VA_ARGS__; }                 \
  else FMOE_DISPATCH_16(dtype, __VA_ARGS__)

cudaError_t launch_scatter_rows(int dtype, const void* src, const int64_t* idx, const int* rank,
                                const int* base, const void* scale, int n_slots, int k, int d,
                                void* dst, int* row_slot, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_slots == 0) return cudaSuccess;
  if (d % 8 != 0) return cudaErrorInvalidValue;
  const int wpb = 8;
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(scatter_rows_kernel<T>, dim3((n_slots + wpb - 1) / wpb), dim3(wpb * 32), 0, stream,
      static_cast<const T*>(src), idx, rank, base, static_cast<const T*>(scale), n_slots, k, d,
      static_cast<T*>(dst), row_slot)));
  return chained;
}

cudaError_t launch_gather_combine(int dtype, const void* rows, const int64_t* idx, const int* rank,
                                  const int* base, const void* weight, int n_tokens, int k, int d,
                                  void* out, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_tokens == 0) return cudaSuccess;
  if (d % 8 != 0) return cudaErrorInvalidValue;
  const int wpb = 8;
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(gather_combine_kernel<T>, dim3((n_tokens + wpb - 1) / wpb), dim3(wpb * 32), 0, stream,
      static_cast<const T*>(rows), idx, rank, base, static_cast<const T*>(weight), n_tokens, k, d,
      static_cast<T*>(out))));
  return chained;
}

cudaError_t launch_combine_bwd(int dtype, const void* dout, const void* rows, const int64_t* idx,
                               const int* rank, const int* base, const void* weight, int n_tokens,
                               int k, int d, void* drows, void* dscore, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  const int n_slots = n_tokens * k;
  if (n_slots == 0) return cudaSuccess;
  if (d % 8 != 0) return cudaErrorInvalidValue;
  const int wpb = 8;
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(combine_bwd_kernel<T>, dim3((n_slots + wpb - 1) / wpb), dim3(wpb * 32), 0, stream,
      static_cast<const T*>(dout), static_cast<const T*>(rows), idx, rank, base,
      static_cast<const T*>(weight), n_slots, k, d, static_cast<T*>(drows),
      static_cast<T*>(dscore))));
  return chained;
}

cudaError_t launch_colsum(int dtype, const void* x, const int* offs, int num_groups, long rows_cap,
                          int n, float* out, cudaStream_t stream) {
  if (rows_cap == 0) return cudaSuccess;
  if (n % 8 != 0) return cudaErrorInvalidValue;
  if ((n + 255) / 256 > 65535 || (rows_cap + 127) / 128 + num_groups > 2147483647L) {
    return cudaErrorInvalidValue;
  }
  dim3 grid(static_cast<unsigned>((rows_cap + 127) / 128 + num_groups), (n + 255) / 256);
  FMOE_DISPATCH_16(dtype, (colsum_kernel<T><<<grid, 256, 0, stream>>>(
      static_cast<const T*>(x), offs, num_groups, n, rows_cap, out)));
  return cudaGetLastError();
}

cudaError_t launch_gate_topk_softmax(int logit_dtype, const void* logits, int n_rows, int n_experts,
                                     int k, int64_t* idx, void* prob, float* zero, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_rows == 0) return cudaSuccess;
  if (k < 1 || k > kMaxK || k > n_experts) return cudaErrorInvalidValue;
  const int wpb = 8;
  const int grid = (n_rows + wpb - 1) / wpb;
  if (logit_dtype == 0) {
    chained = launch_chained(gate_topk_softmax_kernel<__nv_bfloat16>, dim3(grid), dim3(wpb * 32), 0, stream,
        static_cast<const __nv_bfloat16*>(logits), n_rows, n_experts, k, idx,
        static_cast<__nv_bfloat16*>(prob), zero);
  } else if (logit_dtype == 1) {
    chained = launch_chained(gate_topk_softmax_kernel<__half>, dim3(grid), dim3(wpb * 32), 0, stream,
        static_cast<const __half*>(logits), n_rows, n_experts, k, idx, static_cast<__half*>(prob), zero);
  } else {
    chained = launch_chained(gate_topk_softmax_kernel<float>, dim3(grid), dim3(wpb * 32), 0, stream,
        static_cast<const float*>(logits), n_rows, n_experts, k, idx, static_cast<float*>(prob), zero);
  }
  return chained;
}

cudaError_t launch_gate_topk_softmax_bwd(int logit_dtype, const void* dprob, const int64_t* idx,
                                         const void* prob, int n_rows, int n_experts, int k,
                                         void* dlogits, cudaStream_t stream) {
  if (n_rows == 0) return cudaSuccess;
  if (k < 1 || k > kMaxK) return cudaErrorInvalidValue;
  const int wpb = 8;
  const int grid = (n_rows + wpb - 1) / wpb;
  if (logit_dtype == 0) {
    gate_topk_softmax_bwd_kernel<__nv_bfloat16><<<grid, wpb * 32, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(dprob), idx, static_cast<const __nv_bfloat16*>(prob),
        n_rows, n_experts, k, static_cast<__nv_bfloat16*>(dlogits));
  } else if (logit_dtype == 1) {
    gate_topk_softmax_bwd_kernel<__half><<<grid, wpb * 32, 0, stream>>>(
        static_cast<const __half*>(dprob), idx, static_cast<const __half*>(prob), n_rows,
        n_experts, k, static_cast<__half*>(dlogits));
  } else {
    gate_topk_softmax_bwd_kernel<float><<<grid, wpb * 32, 0, stream>>>(
        static_cast<const float*>(dprob), idx, static_cast<const float*>(prob), n_rows, n_experts,
        k, static_cast<float*>(dlogits));
  }
  return cudaGetLastError();
}

#define FMOE_DISPATCH_LOGITS(code, ...)                                   \
  if ((code) == 0) { using T = __nv_bfloat16; __VA_ARGS__; }              \
  else if ((code) == 1) { using T = __half; __VA_ARGS__; }                \
  else { using T = float; __VA_ARGS__; }

bool balance_supported(int tot) { return tot >= 1 && tot <= kBalanceMaxExperts; }
int balance_blocks(int n) { return (n + kBalanceThreads - 1) / kBalanceThreads; }

// TOT: the width in registers that the experts fit in
#define FMOE_BALANCE_TOT(tot, ...)                                       \
  if ((tot) <= 8) { constexpr int TOT = 8; __VA_ARGS__ }                 \
  else if ((tot) <= 16) { constexpr int TOT = 16; __VA_ARGS__ }          \
  else if ((tot) <= 32) { constexpr int TOT = 32; __VA_ARGS__ }          \
  else { constexpr int TOT = kBalanceMaxExperts; __VA_ARGS__ }
#define FMOE_DISPATCH_BALANCE(code, is_switch, ...)                                                       \
  if (is_switch) { constexpr bool SWITCH = true; FMOE_DISPATCH_LOGITS(code, __VA_ARGS__) }               \
  else { constexpr bool SWITCH = false; FMOE_DISPATCH_LOGITS(code, __VA_ARGS__) }

cudaError_t launch_balance_loss(int code, const void* logits, long pitch, const int64_t* ids, int id_stride, int n,
                                int tot, bool is_switch, float scale, float* part, float* loss, float* weight,
                                cudaStream_t stream) {
  if (n < 1 || !balance_supported(tot)) return cudaErrorInvalidValue;
  const int blocks = balance_blocks(n);
  FMOE_BALANCE_TOT(tot, FMOE_DISPATCH_BALANCE(code, is_switch,
      (balance_sums_kernel<T, SWITCH, TOT><<<blocks, kBalanceThreads, 0, stream>>>(
           static_cast<const T*>(logits), pitch, ids, id_stride, n, tot, part))));
  FMOE_DISPATCH_BALANCE(code, is_switch,
      (balance_finish_kernel<T, SWITCH><<<1, 1024, 0, stream>>>(part, blocks, n, tot, scale, loss, weight)));
  return cudaGetLastError();
}

cudaError_t launch_balance_bwd(int code, const void* logits, long pitch, const float* weight, const float* dloss,
                               const int64_t* win, const void* dscore, int n, int tot, bool is_switch, float scale,
                               void* dlogits, cudaStream_t stream) {
  if (n < 1 || !balance_supported(tot)) return cudaErrorInvalidValue;
  FMOE_BALANCE_TOT(tot, FMOE_DISPATCH_BALANCE(code, is_switch,
      (balance_bwd_kernel<T, SWITCH, TOT><<<balance_blocks(n), kBalanceThreads, 0, stream>>>(
           static_cast<const T*>(logits), pitch, weight, dloss, win, static_cast<const T*>(dscore), scale, n, tot,
           static_cast<T*>(dlogits)))));
  return cudaGetLastError();
}

cudaError_t launch_switch_top1(int code, const void* logits, int n, int tot, int64_t* win, void* score,
                               cudaStream_t stream) {
  if (n < 1 || !balance_supported(tot)) return cudaErrorInvalidValue;
  FMOE_BALANCE_TOT(tot, FMOE_DISPATCH_LOGITS(code,
      (switch_top1_kernel<T, TOT><<<balance_blocks(n), kBalanceThreads, 0, stream>>>(
           static_cast<const T*>(logits), n, tot, win, static_cast<T*>(score)))));
  return cudaGetLastError();
}

cudaError_t launch_gate_pad(int dtype, const void* w, const void* bias, int tot, int padded, int d, void* w_out, void* bias_out,
                            cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (tot < 1 || padded < tot || d < 8 || d % 8 != 0) return cudaErrorInvalidValue;
  const long chunks = static_cast<long>(padded) * d / 8;
  const unsigned grid = static_cast<unsigned>(chunks < 148L * 4 * 256 ? (chunks + 255) / 256 : 148 * 4);
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(gate_pad_kernel<T>, dim3(grid), dim3(256), 0, stream, static_cast<const T*>(w),
      static_cast<const T*>(bias), tot, padded, d, static_cast<T*>(w_out), static_cast<T*>(bias_out))));
  return chained;
}

template <int N>
static cudaError_t host_offsets(const int* values, int n, int* dst, cudaStream_t stream) {
  HostValues<N> v;
  for (int i = 0; i < n; ++i) v.v[i] = values[i];
  return launch_chained(host_offsets_kernel<N>, dim3(1), dim3(128), 0, stream, v, n, dst);
}

cudaError_t launch_host_offsets(const int* values, int n, int* dst, cudaStream_t stream) {
  if (n < 1 || n > kMaxHostOffsets) return cudaErrorInvalidValue;
  // (launches copy all of their parameters)
  return n <= 80 ? host_offsets<80>(values, n, dst, stream) : host_offsets<kMaxHostOffsets>(values, n, dst, stream);
}

cudaError_t launch_prune_scalar(const int64_t* idx, const int* rank, int cap, int n_slots, int tot, int64_t* new_idx,
                                cudaStream_t stream) {
  if (n_slots == 0) return cudaSuccess;
  prune_scalar_kernel<<<(n_slots + 255) / 256, 256, 0, stream>>>(idx, rank, cap, n_slots, tot, new_idx);
  return cudaGetLastError();
}

bool gate_fused_supported(int tot, int d, int k) {
  return tot >= 1 && tot <= kGateMaxExperts && d % 8 == 0 && k >= 1 && k <= kMaxK && k <= tot;
}

// Tokens per warp: as many as leave every SM eight warps, up to what registers hold (measured with
// d = 2048, 8 experts: see the kernels).
int gate_rows_per_warp(int n_rows, int tot) {
  if (tot > 8 || n_rows < 148 * 8 * 2) return 1;
  return n_rows < 148 * 8 * 4 ? 2 : 4;
}

cudaError_t launch_gate_linear_topk(int dtype, const void* x, const void* w, const void* bias,
                                    int n_rows, int d, int tot, int k, void* logits, int64_t* idx,
                                    void* prob, float* zero, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_rows == 0) return cudaSuccess;
  if (!gate_fused_supported(tot, d, k) || (dtype == 2 && tot > 8)) return cudaErrorInvalidValue;
  const int per = gate_rows_per_warp(n_rows, tot);
  const int grid = (n_rows + 8 * per - 1) / (8 * per);
#define FMOE_GATE_ROWS(TOT, R)                                                                          \
  FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_linear_topk_rows_kernel<T, TOT, R>, dim3(grid), dim3(256), 0, stream,  \
      static_cast<const T*>(x), static_cast<const T*>(w), static_cast<const T*>(bias), n_rows, d, tot,  \
      k, static_cast<T*>(logits), idx, static_cast<T*>(prob), zero)))
  if (tot <= 8) {
    if (tot <= 2) {
      if (per == 1) { FMOE_GATE_ROWS(2, 1); } else if (per == 2) { FMOE_GATE_ROWS(2, 2); } else { FMOE_GATE_ROWS(2, 4); }
    } else if (tot <= 4) {
      if (per == 1) { FMOE_GATE_ROWS(4, 1); } else if (per == 2) { FMOE_GATE_ROWS(4, 2); } else { FMOE_GATE_ROWS(4, 4); }
    } else {
      if (per == 1) { FMOE_GATE_ROWS(8, 1); } else if (per == 2) { FMOE_GATE_ROWS(8, 2); } else { FMOE_GATE_ROWS(8, 4); }
    }
    return chained;
  }
#undef FMOE_GATE_ROWS
  // The layer's gates come here with at most 8 experts (above, the tensor-core gate is faster):
  // the wider instances, which spill from 16 experts on, serve direct calls of the gate's function.
#define FMOE_GATE_WIDE(TOT)                                                                             \
  FMOE_DISPATCH_16(dtype, (gate_linear_topk_kernel<T, TOT><<<grid, 256, 0, stream>>>(                   \
      static_cast<const T*>(x), static_cast<const T*>(w), static_cast<const T*>(bias), n_rows, d, tot,  \
      k, static_cast<T*>(logits), idx, static_cast<T*>(prob), zero)))
  if (tot <= 16) {
    FMOE_GATE_WIDE(16);
  } else if (tot <= 32) {
    FMOE_GATE_WIDE(32);
  } else {
    FMOE_GATE_WIDE(64);
  }
#undef FMOE_GATE_WIDE
  return cudaGetLastError();
}

cudaError_t launch_gate_linear_topk_few(int dtype, const void* x, const void* w, const void* bias, int n_rows, int d,
                                        int tot, int k, void* logits, int64_t* idx, void* prob, float* zero, cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_rows == 0) return cudaSuccess;
  if (!gate_fused_supported(tot, d, k) || dtype == 2) return cudaErrorInvalidValue;
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(gate_linear_topk_few_kernel<T>, dim3(n_rows), dim3(256), 0, stream,
      static_cast<const T*>(x), static_cast<const T*>(w), static_cast<const T*>(bias), d, tot, k,
      static_cast<T*>(logits), idx, static_cast<T*>(prob), zero)));
  return chained;
}

int gate_bwd_ranges(int dtype, int n_rows, int d) {
  // two blocks per SM over the strips and token ranges, a warp at least four tokens
  const int strip = dtype == 2 ? 128 : 256, strips = (d + strip - 1) / strip;
  int ranges = (2 * 148 + strips - 1) / strips;
  if (ranges > (n_rows + 31) / 32) ranges = (n_rows + 31) / 32;
  return ranges > 0 ? ranges : 1;
}

cudaError_t launch_gate_bwd(int dtype, const void* dprob, const int64_t* idx, const void* prob,
                            const void* dlogits_in, const void* x, const void* w, int n_rows, int d,
                            int tot, int k, float* dl_scratch, void* dx, float* part, void* dw_db,
                            cudaStream_t stream) {
  cudaError_t chained = cudaSuccess;
  if (n_rows == 0) return cudaSuccess;
  if (!gate_fused_supported(tot, d, k) || (dtype == 2 && tot > 8)) return cudaErrorInvalidValue;
  const int per = gate_rows_per_warp(n_rows, tot);
  const int grid = (n_rows + 8 * per - 1) / (8 * per);
#define FMOE_GATE_DX(TOT, R)                                                                            \
  FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_bwd_dx_rows_kernel<T, TOT, R>, dim3(grid), dim3(256), 0, stream,    \
      static_cast<const T*>(dprob), idx, static_cast<const T*>(prob), static_cast<const T*>(dlogits_in),                  \
      static_cast<const T*>(w), n_rows, d, tot, k, dl_scratch, static_cast<T*>(dx))))
  if (tot <= 2) {
    if (per == 1) { FMOE_GATE_DX(2, 1); } else if (per == 2) { FMOE_GATE_DX(2, 2); } else { FMOE_GATE_DX(2, 4); }
  } else if (tot <= 4) {
    if (per == 1) { FMOE_GATE_DX(4, 1); } else if (per == 2) { FMOE_GATE_DX(4, 2); } else { FMOE_GATE_DX(4, 4); }
  } else if (tot <= 8) {
    if (per == 1) { FMOE_GATE_DX(8, 1); } else if (per == 2) { FMOE_GATE_DX(8, 2); } else { FMOE_GATE_DX(8, 4); }
  } else {
#define FMOE_GATE_DX_WIDE(TOT)                                                                          \
  FMOE_DISPATCH_16(dtype, (chained = launch_chained(gate_bwd_dx_kernel<T, TOT>, dim3(grid), dim3(256), 0, stream,          \
      static_cast<const T*>(dprob), idx, static_cast<const T*>(prob), static_cast<const T*>(dlogits_in),                  \
      static_cast<const T*>(w), n_rows, d, tot, k, dl_scratch, static_cast<T*>(dx))))
    if (tot <= 16) { FMOE_GATE_DX_WIDE(16); } else if (tot <= 32) { FMOE_GATE_DX_WIDE(32); } else { FMOE_GATE_DX_WIDE(64); }
#undef FMOE_GATE_DX_WIDE
  }
#undef FMOE_GATE_DX
  if (chained != cudaSuccess) return chained;
  if (part == nullptr) return cudaSuccess;
  if (tot > 16) return cudaErrorInvalidValue;
  const int ranges = gate_bwd_ranges(dtype, n_rows, d), strip = dtype == 2 ? 128 : 256;
  dim3 g2((d + strip - 1) / strip, ranges);
  if (tot <= 2) {
    FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_bwd_dw_kernel<T, 2>, g2, dim3(256), 0, stream,
        dl_scratch, static_cast<const T*>(x), n_rows, d, tot, part)));
  } else if (tot <= 4) {
    FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_bwd_dw_kernel<T, 4>, g2, dim3(256), 0, stream,
        dl_scratch, static_cast<const T*>(x), n_rows, d, tot, part)));
  } else if (tot <= 8) {
    FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_bwd_dw_kernel<T, 8>, g2, dim3(256), 0, stream,
        dl_scratch, static_cast<const T*>(x), n_rows, d, tot, part)));
  } else {
    FMOE_DISPATCH_16(dtype, (chained = launch_chained(gate_bwd_dw_kernel<T, 16>, g2, dim3(256), 0, stream,
        dl_scratch, static_cast<const T*>(x), n_rows, d, tot, part)));
  }
  if (chained != cudaSuccess) return chained;
  const long elems = static_cast<long>(tot) * d + tot;
  FMOE_DISPATCH_ANY(dtype, (chained = launch_chained(gate_bwd_merge_kernel<T>, dim3(static_cast<unsigned>((elems + 31) / 32)), dim3(256), 0, stream,
      part, ranges, elems, static_cast<T*>(dw_db))));
  return chained;
}

cudaError_t launch_simt_grouped_gemm(int mode, int elem, int num_groups, long rows_cap, int m, int n,
                                     int k, const void* a, const void* b, const int* offs,
                                     const void* bias, void* out, cudaStream_t stream) {
  switch (elem) {
    case 0: return simt_typed<__nv_bfloat16>(mode, num_groups, rows_cap, m, n, k, a, b, offs, bias, out, stream);
    case 1: return simt_typed<__half>(mode, num_groups, rows_cap, m, n, k, a, b, offs, bias, out, stream);
    case 2:
      if (sgemm_applies(mode, num_groups, m, n, k, a, b, bias, out)) {
        return launch_sgemm(mode, num_groups, rows_cap, m, n, k, static_cast<const float*>(a),
                            static_cast<const float*>(b), offs, static_cast<const float*>(bias),
                            static_cast<float*>(out), nullptr, stream);
      }
      return simt_typed<float>(mode, num_groups, rows_cap, m, n, k, a, b, offs, bias, out, stream);
    case 3: return simt_typed<double>(mode, num_groups, rows_cap, m, n, k, a, b, offs, bias, out, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fmoe
