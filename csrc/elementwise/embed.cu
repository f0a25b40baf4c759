// Elementwise steps of the contrastive embedding loss on one GPU: the two noisy views, row normalisation with its backward,
// and the softmax rows of the similarity matrix with their gradient in place.
//
// Each is one pass where the tensor-by-tensor statement needs five to eight; at a batch of 1024 a step is a few dozen
// launches of a few microseconds, so passes and launches are what it costs.
#include "../common/host.h"
#include "../common/ptx.cuh"

namespace {

constexpr int kThreads = 256;

// out[0 .. n) = bf16(base + noise * n1), out[n .. 2n) = bf16(base + noise * n2); product and sum rounded one after the other
__global__ void __launch_bounds__(kThreads)
views_kernel(const float4* __restrict__ base, const float4* __restrict__ n1, const float4* __restrict__ n2, float noise,
             uint2* __restrict__ out, long long n4) {
  st::chain_begin(base, n1, n2);
  for (long long i = blockIdx.x * (long long)kThreads + threadIdx.x; i < n4; i += (long long)gridDim.x * kThreads) {
    const float4 b = base[i], u = n1[i], v = n2[i];
    auto at = [noise](float x, float z) { return __fadd_rn(x, __fmul_rn(noise, z)); };
    out[i] = make_uint2(st::pack_bf16x2(at(b.x, u.x), at(b.y, u.y)), st::pack_bf16x2(at(b.z, u.z), at(b.w, u.w)));
    out[n4 + i] = make_uint2(st::pack_bf16x2(at(b.x, v.x), at(b.y, v.y)), st::pack_bf16x2(at(b.z, v.z), at(b.w, v.w)));
  }
}

constexpr float kTiny = 1e-12f;

// y = z / max(|z|, 1e-12) per row in fp32, and |z|; one warp per row
__global__ void __launch_bounds__(kThreads)
row_normalize_kernel(const __nv_bfloat16* __restrict__ z, float* __restrict__ y, float* __restrict__ norm, int rows, int d) {
  st::chain_begin(z);
  const int row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const __nv_bfloat16* zr = z + (size_t)row * d;
  float s = 0.0f;
  for (int c = lane; c < d; c += 32) {
    const float v = __bfloat162float(zr[c]);
    s += v * v;
  }
  const float n = sqrtf(st::warp_sum(s)), by = fmaxf(n, kTiny);
  for (int c = lane; c < d; c += 32) y[(size_t)row * d + c] = __bfloat162float(zr[c]) / by;
  if (lane == 0) norm[row] = n;
}

// dz = (g - y (y . g)) / |z| as bf16; below the clamp the norm has no gradient: dz = g / 1e-12
__global__ void __launch_bounds__(kThreads)
row_normalize_bwd_kernel(const float* __restrict__ g, const float* __restrict__ y, const float* __restrict__ norm,
                         __nv_bfloat16* __restrict__ dz, int rows, int d) {
  st::chain_begin(g, y, norm);
  const int row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t base = (size_t)row * d;
  const float n = norm[row];
  float dot = 0.0f;
  if (n >= kTiny) {
    for (int c = lane; c < d; c += 32) dot += g[base + c] * y[base + c];
    dot = st::warp_sum(dot);
  }
  const float by = fmaxf(n, kTiny);
  for (int c = lane; c < d; c += 32) dz[base + c] = __float2bfloat16((g[base + c] - y[base + c] * dot) / by);
}

// Row i of the similarities s: x = s / temperature, loss[i] = logsumexp(x) - x[i], and s := (softmax(x) - e_i) / (rows
// temperature), the gradient of the mean loss.  The row waits in shared memory between the passes.
__global__ void __launch_bounds__(kThreads)
nce_rows_kernel(float* __restrict__ s, float* __restrict__ loss, int rows, int cols, float temperature) {
  st::chain_begin();
  extern __shared__ float x[];
  __shared__ float sh[kThreads / 32];
  float* row = s + (size_t)blockIdx.x * cols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float m = -INFINITY;
  for (int c = threadIdx.x; c < cols; c += kThreads) {
    const float v = row[c] / temperature;
    x[c] = v;
    m = fmaxf(m, v);
  }
  m = st::warp_max(m);
  if (lane == 0) sh[warp] = m;
  __syncthreads();
  m = sh[0];
  for (int w = 1; w < kThreads / 32; ++w) m = fmaxf(m, sh[w]);
  __syncthreads();
  float sum = 0.0f;
  for (int c = threadIdx.x; c < cols; c += kThreads) sum += expf(x[c] - m);
  sum = st::warp_sum(sum);
  if (lane == 0) sh[warp] = sum;
  __syncthreads();
  sum = 0.0f;
  for (int w = 0; w < kThreads / 32; ++w) sum += sh[w];
  const float lse = m + logf(sum), by = 1.0f / (float)rows;
  for (int c = threadIdx.x; c < cols; c += kThreads)
    row[c] = (expf(x[c] - lse) - (c == (int)blockIdx.x ? 1.0f : 0.0f)) * by / temperature;
  if (threadIdx.x == 0) loss[blockIdx.x] = lse - x[blockIdx.x];
}

}  // namespace

// base, n1, n2: fp32 of n elements (n % 4 == 0), 16-byte aligned; out: bf16 of 2 n elements.
ST_API int st_contrastive_views(const float* base, const float* n1, const float* n2, float noise, void* out, long long n, void* stream_v) {
  if (!base || !n1 || !n2 || !out || n <= 0 || (n & 3)) return st::fail(ST_ERR_INVALID, "contrastive_views: bad arguments");
  if ((reinterpret_cast<uintptr_t>(base) | reinterpret_cast<uintptr_t>(n1) | reinterpret_cast<uintptr_t>(n2) | reinterpret_cast<uintptr_t>(out)) & 15)
    return st::fail(ST_ERR_INVALID, "contrastive_views: tensors must be 16-byte aligned");
  long long blocks = (n / 4 + kThreads - 1) / kThreads;
  if (blocks > 8ll * st::sm_count()) blocks = 8ll * st::sm_count();
  st::chained(views_kernel, (unsigned)blocks, kThreads, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      reinterpret_cast<const float4*>(base), reinterpret_cast<const float4*>(n1), reinterpret_cast<const float4*>(n2), noise,
      static_cast<uint2*>(out), n / 4);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_row_normalize(const void* z, float* y, float* norm, int rows, int d, void* stream_v) {
  if (!z || !y || !norm || rows <= 0 || d <= 0) return st::fail(ST_ERR_INVALID, "row_normalize: bad arguments");
  st::chained(row_normalize_kernel, (rows + 7) / 8, kThreads, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(z), y, norm, rows, d);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_row_normalize_bwd(const float* g, const float* y, const float* norm, void* dz, int rows, int d, void* stream_v) {
  if (!g || !y || !norm || !dz || rows <= 0 || d <= 0) return st::fail(ST_ERR_INVALID, "row_normalize_bwd: bad arguments");
  st::chained(row_normalize_bwd_kernel, (rows + 7) / 8, kThreads, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      g, y, norm, static_cast<__nv_bfloat16*>(dz), rows, d);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// s: fp32 [rows, rows] similarities, replaced by the gradient of the mean loss; loss: fp32 [rows].  At most 12000 rows.
ST_API int st_nce_rows(float* s, float* loss, int rows, float temperature, void* stream_v) {
  if (!s || !loss || rows <= 0 || !(temperature > 0.0f)) return st::fail(ST_ERR_INVALID, "nce_rows: bad arguments");
  if (rows > 12000) return st::fail(ST_ERR_TOO_LARGE, "nce_rows: the row does not fit in shared memory");
  st::chained(nce_rows_kernel, rows, kThreads, rows * sizeof(float), reinterpret_cast<cudaStream_t>(stream_v))(s, loss, rows, rows, temperature);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
