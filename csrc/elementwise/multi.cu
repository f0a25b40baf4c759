// Small-tensor work of the layer protocol in one launch each: finite checks, scaled copies and plain updates over a list
// of fp32 tensors, and the mean-squared-error loss.
//
// A training step of a small model through the layer API is bound by launches and host reads, not by bytes (a step of a
// 64-128-8 perceptron moves 0.3 MB in 170 launches and ten host reads, 2.3 ms): one check of one tensor was five launches
// and a host read.  Here a list of tensors is one grid, every tensor a run of blocks by its size, and what the host has to know (did every
// block see finite values) is written by the blocks straight into pinned host memory, so that a stream synchronisation
// is all that the check costs on top of its launch.
#include "../common/host.h"
#include "../common/ptx.cuh"

namespace {

constexpr int kMultiMax = 48;        // tensors per launch: the table travels as a kernel argument
constexpr int kMultiThreads = 256;

struct MultiTable {
  const float* src[kMultiMax];
  float* dst[kMultiMax];
  __nv_bfloat16* half[kMultiMax];      // STEP: receives the updated values rounded to bf16, or null
  long long n[kMultiMax];
  int first[kMultiMax + 1];            // blocks first[i] to first[i + 1] - 1 work on tensor i
};

enum MultiOp : int { MULTI_CHECK = 0, MULTI_DIV = 1, MULTI_STEP = 2 };

// CHECK: bad[tensor * slots + block of the tensor] = some src element is not finite, 0 in the slots past its blocks.  DIV: the
// same, and dst = src / value.  STEP: dst -= value * src, the product rounded before the difference.
// Large tensors get as many blocks as stay resident, and their bytes bound them: an update of 64 M elements takes 0.17 ms and a
// check 0.09; with 32 blocks, enough for the small ones, they took 4.2 and 0.96.
template <int OP>
__global__ void __launch_bounds__(kMultiThreads)
multi_kernel(const __grid_constant__ MultiTable t, float value, int* __restrict__ bad, int slots) {
  int which = 0;
#pragma unroll
  for (int step = 32; step > 0; step >>= 1)
    if (which + step < kMultiMax && t.first[which + step] <= static_cast<int>(blockIdx.x)) which += step;
  const int block = blockIdx.x - t.first[which], blocks = t.first[which + 1] - t.first[which];
  const float* __restrict__ src = t.src[which];      // the table is part of the arguments: no access to global memory yet
  st::chain_begin(src);
  float* dst = t.dst[which];
  __nv_bfloat16* half = OP == MULTI_STEP ? t.half[which] : nullptr;
  const long long n = t.n[which], stride = (long long)blocks * kMultiThreads;
  bool odd = false;
  for (long long i = block * (long long)kMultiThreads + threadIdx.x; i < n; i += 4 * stride) {
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = i + u * stride < n ? src[i + u * stride] : 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long at = i + u * stride;
      if (OP != MULTI_STEP) odd |= !isfinite(v[u]);
      if (at < n) {
        if (OP == MULTI_DIV) dst[at] = __fdiv_rn(v[u], value);
        if (OP == MULTI_STEP) {
          const float w = __fsub_rn(dst[at], __fmul_rn(value, v[u]));
          dst[at] = w;
          if (half) half[at] = __float2bfloat16(w);
        }
      }
    }
  }
  if (OP != MULTI_STEP) {
    odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) bad[which * slots + block] = odd;
    if (block == blocks - 1)
      for (int i = blocks + threadIdx.x; i < slots; i += kMultiThreads) bad[which * slots + i] = 0;
  }
}

// dst (bf16) = src (fp32) for a list of tensors, eight elements per thread and step; the tail element by element
__global__ void __launch_bounds__(kMultiThreads)
multi_cast_kernel(const __grid_constant__ MultiTable t) {
  const float* __restrict__ src = t.src[blockIdx.y];
  st::chain_begin(src);
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(t.dst[blockIdx.y]);
  const long long n = t.n[blockIdx.y], n8 = n / 8;
  for (long long i = blockIdx.x * (long long)kMultiThreads + threadIdx.x; i < n8; i += (long long)gridDim.x * kMultiThreads) {
    const float4 a = reinterpret_cast<const float4*>(src)[2 * i], b = reinterpret_cast<const float4*>(src)[2 * i + 1];
    reinterpret_cast<uint4*>(dst)[i] = make_uint4(st::pack_bf16x2(a.x, a.y), st::pack_bf16x2(a.z, a.w),
                                                  st::pack_bf16x2(b.x, b.y), st::pack_bf16x2(b.z, b.w));
  }
  if (blockIdx.x == 0 && n8 * 8 + threadIdx.x < n) dst[n8 * 8 + threadIdx.x] = __float2bfloat16(src[n8 * 8 + threadIdx.x]);
}

__device__ __forceinline__ float block_sum_256(float v, float* sh) {
  v = st::warp_sum(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < kMultiThreads / 32; ++i) s += sh[i];
  return s;
}

// value = mean((p - t)^2).  Blocks leave their sums in `part` and the last one to finish adds them in block order, so the
// result does not depend on scheduling.  bad[block]: a prediction or a target is not finite.
__global__ void __launch_bounds__(kMultiThreads)
mse_forward_kernel(const float* __restrict__ p, const float* __restrict__ t, long long n, float* __restrict__ value,
                   float* __restrict__ part, unsigned* __restrict__ arrived, int* __restrict__ bad) {
  st::chain_begin(p, t);
  __shared__ float sh[kMultiThreads / 32];
  __shared__ bool last;
  float s = 0.0f;
  bool odd = false;
  for (long long i = blockIdx.x * (long long)kMultiThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kMultiThreads) {
    const float a = p[i], b = t[i], d = a - b;
    odd |= !isfinite(a) || !isfinite(b);
    s += d * d;
  }
  odd = __syncthreads_or(odd);
  s = block_sum_256(s, sh);
  if (threadIdx.x == 0) {
    bad[blockIdx.x] = odd;
    last = false;
    if (gridDim.x == 1) {
      *value = s / (float)n;
    } else {
      part[blockIdx.x] = s;
      __threadfence();
      last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __syncthreads();
  float total = threadIdx.x < gridDim.x ? *reinterpret_cast<volatile float*>(part + threadIdx.x) : 0.0f;
  total = block_sum_256(total, sh);
  if (threadIdx.x == 0) *value = total / (float)n;
}

// g = (1 / n) * 2 (p - t)
__global__ void __launch_bounds__(kMultiThreads)
mse_backward_kernel(const float* __restrict__ p, const float* __restrict__ t, long long n, float inv_n, float* __restrict__ g,
                    int* __restrict__ bad) {
  st::chain_begin(p, t);
  bool odd = false;
  for (long long i = blockIdx.x * (long long)kMultiThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kMultiThreads) {
    const float a = p[i], b = t[i];
    odd |= !isfinite(a) || !isfinite(b);
    g[i] = inv_n * (2.0f * (a - b));
  }
  odd = __syncthreads_or(odd);
  if (threadIdx.x == 0) bad[blockIdx.x] = odd;
}

int blocks_for(long long n, int most) {
  const long long b = (n + 4 * kMultiThreads - 1) / (4 * kMultiThreads);
  return (int)(b < 1 ? 1 : (b > most ? most : b));
}
int multi_cap() { return 8 * st::sm_count(); }      // blocks of one tensor at most

}  // namespace

// Tensors per st_multi call, and ints of result a call over tensors of at most `most` elements writes per tensor.
ST_API int st_multi_max() { return kMultiMax; }
ST_API int st_multi_blocks(long long most) { return blocks_for(most, multi_cap()); }

namespace {
int run_multi(int op, int count, const void* const* src, void* const* dst, void* const* half, const long long* n, float value,
              int* bad, void* stream_v);
}

// op 0: finite check of src; 1: dst = src / value and finite check of src; 2: dst -= value * src.  `bad` (op 0 and 1):
// count * st_multi_blocks(largest n) ints, tensor by tensor, in memory that the device can write (pinned host memory).
ST_API int st_multi(int op, int count, const void* const* src, void* const* dst, const long long* n, float value, int* bad,
                    void* stream_v) {
  return run_multi(op, count, src, dst, nullptr, n, value, bad, stream_v);
}
// dst -= value * src, and where half[i] is not null the updated values as bf16 there.
ST_API int st_multi_step_bf16(int count, const void* const* src, void* const* dst, void* const* half, const long long* n, float value,
                              void* stream_v) {
  return run_multi(MULTI_STEP, count, src, dst, half, n, value, nullptr, stream_v);
}

namespace {
int run_multi(int op, int count, const void* const* src, void* const* dst, void* const* half, const long long* n, float value,
              int* bad, void* stream_v) {
  if (count <= 0) return ST_OK;
  if (count > kMultiMax) return st::fail(ST_ERR_TOO_LARGE, "multi: too many tensors for one launch");
  if (op < MULTI_CHECK || op > MULTI_STEP || !src || !n || (op != MULTI_CHECK && !dst) || (op != MULTI_STEP && !bad))
    return st::fail(ST_ERR_INVALID, "multi: bad arguments");
  MultiTable t;
  long long most = 0;
  const int cap = multi_cap();
  int grid = 0;
  for (int i = 0; i < count; ++i) {
    t.src[i] = static_cast<const float*>(src[i]);
    t.dst[i] = dst ? static_cast<float*>(dst[i]) : nullptr;
    t.half[i] = half ? static_cast<__nv_bfloat16*>(half[i]) : nullptr;
    t.n[i] = n[i];
    t.first[i] = grid;
    grid += blocks_for(n[i], cap);
    most = n[i] > most ? n[i] : most;
  }
  for (int i = count; i <= kMultiMax; ++i) t.first[i] = i == count ? grid : 0x7FFFFFFF;
  const int slots = blocks_for(most, cap);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  if (op == MULTI_CHECK) st::chained(multi_kernel<MULTI_CHECK>, grid, kMultiThreads, 0, s)(t, value, bad, slots);
  else if (op == MULTI_DIV) st::chained(multi_kernel<MULTI_DIV>, grid, kMultiThreads, 0, s)(t, value, bad, slots);
  else st::chained(multi_kernel<MULTI_STEP>, grid, kMultiThreads, 0, s)(t, value, bad, slots);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

}  // namespace

// bf16 copies of fp32 tensors; every pointer 16-byte aligned.
ST_API int st_multi_cast_bf16(int count, const void* const* src, void* const* dst, const long long* n, void* stream_v) {
  if (count <= 0) return ST_OK;
  if (count > kMultiMax) return st::fail(ST_ERR_TOO_LARGE, "multi_cast: too many tensors for one launch");
  if (!src || !dst || !n) return st::fail(ST_ERR_INVALID, "multi_cast: bad arguments");
  MultiTable t;
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    if ((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i])) & 15)
      return st::fail(ST_ERR_INVALID, "multi_cast: tensors must be 16-byte aligned");
    t.src[i] = static_cast<const float*>(src[i]);
    t.dst[i] = static_cast<float*>(dst[i]);
    t.n[i] = n[i];
    most = n[i] > most ? n[i] : most;
  }
  const dim3 grid(blocks_for(most / 2, 8 * st::sm_count()), count);
  st::chained(multi_cast_kernel, grid, kMultiThreads, 0, reinterpret_cast<cudaStream_t>(stream_v))(t);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// 32-bit words of workspace st_mse_forward wants, and blocks (ints of `bad`) that both directions write.
ST_API int st_mse_workspace() { return kMultiThreads + 1; }
ST_API int st_mse_blocks(long long n) { return blocks_for(n, kMultiThreads); }

ST_API int st_mse_forward(const float* p, const float* t, long long n, float* value, void* workspace, int* bad, void* stream_v) {
  if (!p || !t || !value || !workspace || !bad || n <= 0) return st::fail(ST_ERR_INVALID, "mse: bad arguments");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  float* part = static_cast<float*>(workspace);
  unsigned* arrived = reinterpret_cast<unsigned*>(part + kMultiThreads);
  const int blocks = blocks_for(n, kMultiThreads);
  if (blocks > 1) ST_CUDA_CHECK(cudaMemsetAsync(arrived, 0, sizeof(unsigned), s));
  st::chained(mse_forward_kernel, blocks, kMultiThreads, 0, s)(p, t, n, value, part, arrived, bad);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_mse_backward(const float* p, const float* t, long long n, float* g, int* bad, void* stream_v) {
  if (!p || !t || !g || !bad || n <= 0) return st::fail(ST_ERR_INVALID, "mse: bad arguments");
  st::chained(mse_backward_kernel, blocks_for(n, kMultiThreads), kMultiThreads, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      p, t, n, 1.0f / (float)n, g, bad);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
