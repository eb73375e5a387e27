// fp32 grouped GEMM on the FMA units: the three products of a grouped linear at the full precision
// of fp32 (the tensor cores' tf32 would drop 13 bits of the inputs), for calls too small to be worth
// splitting for the tensor cores (split_gemm.cu).
//
// One CTA of 128 threads computes a 64 x 128 tile with a K step of 16; a thread owns 8 x 8 outputs
// and adds its products in ascending k, one fused multiply-add each (packed two to an instruction:
// every lane rounds like the scalar one).  Bound by the FMA pipe: 64 FMAs per thread and k against
// 4 shared-memory loads of 16 bytes; the next K step travels from global memory to registers
// during the math and into the other of two buffers after it.  64 rows per tile, and not 128,
// because an expert's last tile is ragged: 4096 rows on 8 experts with 512 outputs are 272 tiles
// for 148 SMs, with 128 x 128 they would be 144, many of them nearly empty.
// Measured, 16384 rows, 4 experts, 1024 <-> 2048: 49 to 53 TFLOP/s (43 to 48 with scalar FMAs);
// 4096 rows, 8 experts, 512 <-> 2048: forward 203 and 227, input gradient 192 and 218, weight
// gradient with the bias gradient 171 us, where the general kernel took 437, 347 and 283 us on
// average and the bias gradient a dozen more launches.
// Operands need 16-byte aligned rows; the general kernel of routing.cu takes the rest.
#include "ptx.cuh"
#include "routing.cuh"

namespace fmoe {
namespace {

constexpr int TM = 64;
constexpr int TN = 128;
constexpr int TK = 16;
constexpr int THREADS = 128;
constexpr int AP = TM + 4;   // pitches keep 16-byte alignment and spread the transposing stores
constexpr int BP = TN + 4;

__device__ __forceinline__ float4 ld4(const float* p, bool ok) {
  return ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Modes as in GemmMode: 0 rows x weight^T, 1 rows x weight, 2 weight gradient (`psum`, optional:
// [num_groups, m] column sums of `a` per group, formed by the CTAs of the first column block).
template <int MODE>
__global__ void __launch_bounds__(THREADS, MODE == 1 ? 4 : 3)   // 168 registers, 8 bytes spilled in mode 0; 128 and 16 in mode 1
sgemm_kernel(int num_groups, long rows_cap, int m, int n, int k, const float* __restrict__ a, const float* __restrict__ b,
             const int* __restrict__ offs, const float* __restrict__ bias, float* __restrict__ out,
             float* __restrict__ psum) {
  __shared__ __align__(16) float As[2][TK][AP];
  __shared__ __align__(16) float Bs[2][TK][BP];
  const int tid = threadIdx.x;
  const int j0 = blockIdx.y * TN;
  int g, i0, rows_i, kk_total, row_base;
  if (MODE == 2) {
    g = blockIdx.z;
    i0 = blockIdx.x * TM;
    rows_i = m;
    row_base = offs[g];
    kk_total = offs[g + 1] - row_base;
  } else {
    // blockIdx.x counts the 64-row pieces of all experts: every warp finds the expert of its
    // piece, 32 experts at a time
    const int lane = tid & 31;
    const int piece = blockIdx.x;
    int before = 0;
    g = -1;
    i0 = 0;
    row_base = 0;
    rows_i = 0;
    for (int g0 = 0; g0 < num_groups && g < 0; g0 += 32) {
      const int gl = g0 + lane;
      const int lo = gl < num_groups ? offs[gl] : 0;
      const int rows = gl < num_groups ? offs[gl + 1] - lo : 0;
      int incl = (rows + TM - 1) / TM;
      const int mine = incl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const int first = before + incl - mine;
      const unsigned hit = __ballot_sync(0xffffffffu, piece >= first && piece < first + mine);
      before += __shfl_sync(0xffffffffu, incl, 31);
      if (hit != 0) {
        const int src = __ffs(hit) - 1;
        g = g0 + src;
        row_base = __shfl_sync(0xffffffffu, lo, src);
        rows_i = __shfl_sync(0xffffffffu, rows, src);
        i0 = (piece - __shfl_sync(0xffffffffu, first, src)) * TM;
      }
    }
    if (g < 0) {
      // no piece left: the rows past the last expert are zeroed, so that what is applied to the
      // whole buffer afterwards meets no stale bits
      const long r0 = static_cast<long>(offs[num_groups]) + static_cast<long>(piece - before) * TM;
      for (int it = tid; it < TM * (TN / 4); it += THREADS) {
        const long r = r0 + it / (TN / 4);
        const int j = j0 + (it % (TN / 4)) * 4;
        if (r < rows_cap && j < n) *reinterpret_cast<float4*>(out + r * n + j) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      return;
    }
    kk_total = k;
  }

  float4 ra[2], rb[4];
  auto load = [&](int kk0) {
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      const int f = tid + l * THREADS;
      if (MODE == 2) {
        const int kk = kk0 + f / (TM / 4), i = i0 + (f % (TM / 4)) * 4;
        ra[l] = ld4(a + static_cast<long>(row_base + kk) * m + i, kk < kk_total && i < rows_i);
      } else {
        const int i = i0 + f / (TK / 4), kk = kk0 + (f % (TK / 4)) * 4;
        ra[l] = ld4(a + static_cast<long>(row_base + i) * k + kk, kk < kk_total && i < rows_i);
      }
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int f = tid + l * THREADS;
      if (MODE == 0) {
        const int j = j0 + f / (TK / 4), kk = kk0 + (f % (TK / 4)) * 4;
        rb[l] = ld4(b + (static_cast<long>(g) * n + j) * k + kk, kk < kk_total && j < n);
      } else {
        const int kk = kk0 + f / (TN / 4), j = j0 + (f % (TN / 4)) * 4;
        const long row = MODE == 1 ? static_cast<long>(g) * k + kk : static_cast<long>(row_base) + kk;
        rb[l] = ld4(b + row * n + j, kk < kk_total && j < n);
      }
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      const int f = tid + l * THREADS;
      if (MODE == 2) {
        *reinterpret_cast<float4*>(&As[buf][f / (TM / 4)][(f % (TM / 4)) * 4]) = ra[l];
      } else {
        const int i = f / (TK / 4), kk = (f % (TK / 4)) * 4;
        As[buf][kk][i] = ra[l].x;
        As[buf][kk + 1][i] = ra[l].y;
        As[buf][kk + 2][i] = ra[l].z;
        As[buf][kk + 3][i] = ra[l].w;
      }
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const int f = tid + l * THREADS;
      if (MODE == 0) {
        const int j = f / (TK / 4), kk = (f % (TK / 4)) * 4;
        Bs[buf][kk][j] = rb[l].x;
        Bs[buf][kk + 1][j] = rb[l].y;
        Bs[buf][kk + 2][j] = rb[l].z;
        Bs[buf][kk + 3][j] = rb[l].w;
      } else {
        *reinterpret_cast<float4*>(&Bs[buf][f / (TN / 4)][(f % (TN / 4)) * 4]) = rb[l];
      }
    }
  };

  const int tx = tid & 15, ty = tid >> 4;   // columns tx * 4 and 64 + tx * 4, rows ty * 4 and 32 + ty * 4
  ptx::f32x2 acc[8][4];   // outputs in pairs of neighbouring columns
#pragma unroll
  for (int u = 0; u < 8; ++u) {
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0ull;
  }
  const bool sums = MODE == 2 && psum != nullptr && blockIdx.y == 0;
  float col_sum = 0.f;   // of column i0 + tid (threads 0 .. 63), one partial sum per K step

  if (kk_total > 0) {
    load(0);
    store(0);
  }
  __syncthreads();
  int buf = 0;
  for (int kk0 = 0; kk0 < kk_total; kk0 += TK) {
    const bool more = kk0 + TK < kk_total;
    if (more) load(kk0 + TK);
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][32 + ty * 4]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][tx * 4]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][64 + tx * 4]);
      const float fa[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const ptx::f32x2 fb[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const ptx::f32x2 aa = ptx::pack2(fa[u], fa[u]);
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = ptx::fma2(aa, fb[v], acc[u][v]);
      }
    }
    if (sums && tid < TM) {
      float part = 0.f;
#pragma unroll
      for (int kk = 0; kk < TK; ++kk) part += As[buf][kk][tid];
      col_sum += part;
    }
    if (more) store(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  if (sums && tid < TM && i0 + tid < m) psum[static_cast<long>(g) * m + i0 + tid] = col_sum;

#pragma unroll
  for (int v4 = 0; v4 < 2; ++v4) {
    const int j = j0 + v4 * 64 + tx * 4;
    if (j >= n) continue;
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE != 2 && bias != nullptr) bv = __ldg(reinterpret_cast<const float4*>(bias + static_cast<long>(g) * n + j));
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + (u >> 2) * 32 + ty * 4 + (u & 3);
      if (i >= rows_i) continue;
      const long row = MODE == 2 ? static_cast<long>(g) * m + i : static_cast<long>(row_base) + i;
      float4 w;
      ptx::unpack2(acc[u][v4 * 2], w.x, w.y);
      ptx::unpack2(acc[u][v4 * 2 + 1], w.z, w.w);
      w.x += bv.x;
      w.y += bv.y;
      w.z += bv.z;
      w.w += bv.w;
      *reinterpret_cast<float4*>(out + row * n + j) = w;
    }
  }
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

bool sgemm_applies(int mode, int num_groups, int m, int n, int k, const void* a, const void* b, const void* bias,
                   const void* out) {
  const int inner = mode == 2 ? m : k;   // row length of `a`
  return inner % 4 == 0 && n % 4 == 0 && inner > 0 && n > 0 && num_groups <= 65535 && (n + TN - 1) / TN <= 65535 &&
         aligned16(a) && aligned16(b) && aligned16(out) && (bias == nullptr || aligned16(bias));
}

cudaError_t launch_sgemm(int mode, int num_groups, long rows_cap, int m, int n, int k, const float* a, const float* b,
                         const int* offs, const float* bias, float* out, float* psum, cudaStream_t stream) {
  const unsigned nt = (n + TN - 1) / TN;
  if (mode == 2) {
    dim3 grid((m + TM - 1) / TM, nt, num_groups);
    sgemm_kernel<2><<<grid, THREADS, 0, stream>>>(num_groups, rows_cap, m, n, k, a, b, offs, nullptr, out, psum);
  } else {
    if (rows_cap == 0) return cudaSuccess;
    dim3 grid(static_cast<unsigned>((rows_cap + TM - 1) / TM + num_groups), nt);
    if (mode == 0) {
      sgemm_kernel<0><<<grid, THREADS, 0, stream>>>(num_groups, rows_cap, m, n, k, a, b, offs, bias, out, nullptr);
    } else {
      sgemm_kernel<1><<<grid, THREADS, 0, stream>>>(num_groups, rows_cap, m, n, k, a, b, offs, bias, out, nullptr);
    }
  }
  return cudaGetLastError();
}

}  // namespace fmoe
