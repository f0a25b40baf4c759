// LayerNorm and RMSNorm, forward and backward, bf16 in / fp32 statistics.
//
// Forward: one CTA per row, 16-byte vector loads, the row stays in registers between the
// statistics pass and the normalisation pass (one HBM read, one write).
// Backward: a persistent grid; each CTA walks rows with a stride, writes dx and keeps its
// share of dgamma / dbeta in registers; per-CTA partials go to an fp32 scratch buffer that
// a second kernel reduces.  (The scratch is global memory beyond inputs and outputs.)
//
// Reference parity: layer_norm.wgsl (crates/st-tensor/src/wgpu_shaders) and the CPU
// layer_norm_affine (crates/st-tensor/src/pure.rs:3702-4058); RMSNorm is new (the
// reference has none).
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "norm.h"

namespace {
using namespace st;

constexpr int NT = 256;     // threads per CTA
constexpr int MAXV = 4;     // most 16-byte vectors per thread held in registers (d <= 8192)
// The kernels are instantiated for 1, 2 or 4 vectors per thread (d <= 2048 / 4096 / 8192): the
// per-thread arrays are sized by the template argument, so the common d = 2048 case needs a
// quarter of the registers and four times as many CTAs stay resident per SM.

__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) sh[0] = t;
  }
  __syncthreads();
  return sh[0];
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

// RMS: y = x * rstd * gamma.   LN: y = (x - mean) * rstd * gamma + beta.
// Optional fused residual: x := x + residual is written to `sum_out` before normalising.
template <bool RMS, int MV, bool GELU = false>
__global__ void __launch_bounds__(NT)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ beta,
                __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ sum_out,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int d,
                float eps) {
  chain_begin(x, residual, gamma, beta);
  __shared__ float sh[NT / 32];
  const int row = blockIdx.x;
  if (row >= rows) return;
  const int nvec = d >> 3;
  const __nv_bfloat16* xr = x + (size_t)row * d;
  float v[MV][8];
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = threadIdx.x + i * NT;
    if (vi < nvec) {
      load8(xr + vi * 8, v[i]);
      if (residual) {
        float r[8];
        load8(residual + (size_t)row * d + vi * 8, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] += r[j];
        if (sum_out) {
          store8(sum_out + (size_t)row * d + vi * 8, v[i]);
          // normalise what was stored (bf16-rounded) so forward and backward agree
          load8(sum_out + (size_t)row * d + vi * 8, v[i]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += RMS ? v[i][j] * v[i][j] : v[i][j];
    }
  }
  float mean = 0.0f, rstd;
  if (RMS) {
    const float ms = block_sum(s, sh) / d;
    rstd = rsqrtf(ms + eps);
  } else {
    mean = block_sum(s, sh) / d;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int vi = threadIdx.x + i * NT;
      if (vi < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float c = v[i][j] - mean;
          q += c * c;
        }
      }
    }
    const float var = block_sum(q, sh) / d;
    rstd = rsqrtf(var + eps);
  }
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = threadIdx.x + i * NT;
    if (vi < nvec) {
      float g[8], o[8];
      load8(gamma + vi * 8, g);
      if (!RMS && beta) {
        float b[8];
        load8(beta + vi * 8, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * g[j] + b[j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * g[j];
      }
      if (GELU) {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = gelu_tanh(__bfloat162float(__float2bfloat16(o[j])));
      }
      store8(y + (size_t)row * d + vi * 8, o);
    }
  }
}

// dx for one row and the CTA's running dgamma/dbeta.
template <bool RMS, int MV>
__global__ void __launch_bounds__(NT)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ mean_in,
                const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                __nv_bfloat16* __restrict__ dx, float* __restrict__ partial_dgamma,
                float* __restrict__ partial_dbeta, int rows, int d) {
  chain_begin(dy, x, gamma, mean_in, rstd_in, dres);
  __shared__ float sh[NT / 32];
  const int nvec = d >> 3;
  float g[MV][8], dg[MV][8], db[MV][8];
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = threadIdx.x + i * NT;
    if (vi < nvec) load8(gamma + vi * 8, g[i]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dg[i][j] = 0.0f;
      db[i][j] = 0.0f;
    }
  }
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float mean = RMS ? 0.0f : mean_in[row];
    const float rstd = rstd_in[row];
    float xh[MV][8], gy[MV][8], rr[MV][8];
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int vi = threadIdx.x + i * NT;
      if (vi < nvec) {
        float xv[8], dv[8];
        load8(x + (size_t)row * d + vi * 8, xv);
        load8(dy + (size_t)row * d + vi * 8, dv);
        // the residual-branch gradient is only needed after the row reduction: issue its load now so that the
        // reduction hides the latency
        if (dres) load8(dres + (size_t)row * d + vi * 8, rr[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[i][j] = (xv[j] - mean) * rstd;
          gy[i][j] = dv[j] * g[i][j];
          dg[i][j] += dv[j] * xh[i][j];
          db[i][j] += dv[j];
          s1 += gy[i][j] * xh[i][j];
          s2 += gy[i][j];
        }
      }
    }
    const float m1 = block_sum(s1, sh) / d;
    const float m2 = RMS ? 0.0f : block_sum(s2, sh) / d;
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      const int vi = threadIdx.x + i * NT;
      if (vi < nvec) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (gy[i][j] - m2 - xh[i][j] * m1);
        if (dres) {  // gradient arriving through the residual branch
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rr[i][j];
        }
        store8(dx + (size_t)row * d + vi * 8, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = threadIdx.x + i * NT;
    if (vi < nvec) {
      float* pg = partial_dgamma + (size_t)blockIdx.x * d + vi * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) pg[j] = dg[i][j];
      if (!RMS && partial_dbeta) {
        float* pb = partial_dbeta + (size_t)blockIdx.x * d + vi * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) pb[j] = db[i][j];
      }
    }
  }
}

// RMSNorm with one vector per thread (1024 < d <= 2048): the next row's loads are in flight during this row's reduction, which
// passes one barrier (alternating buffers) where block_sum passes three; operands stay as loaded, which leaves four CTAs their
// registers.  16384 rows of 2048 with a residual gradient: 58.7 -> 55.3 us back to back, 64.5 -> 58.2 inside a training step (41
// of bytes); 1536 features 51.8 -> 47.3; 2048 rows 15.5 -> 14.3.
__global__ void __launch_bounds__(NT, 4)
rms_bwd_ahead_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                     const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                     float* __restrict__ partial_dgamma, int rows, int d) {
  chain_begin(dy, x, gamma, rstd_in, dres);
  __shared__ __align__(16) float sh[2][NT / 32];
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const bool live = threadIdx.x < (d >> 3);
  const int col = threadIdx.x * 8, step = gridDim.x;
  auto at = [&](const __nv_bfloat16* p, int row) { return live && row < rows ? *reinterpret_cast<const uint4*>(p + (size_t)row * d + col) : zero; };
  auto get = [](const uint4& u, float (&f)[8]) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), e = unpack_bf16x2(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = e.x; f[7] = e.y;
  };
  const uint4 gv = live ? *reinterpret_cast<const uint4*>(gamma + col) : zero;
  float dg[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) dg[j] = 0.0f;
  int row = blockIdx.x, buf = 0;
  uint4 xv = at(x, row), yv = at(dy, row);
  for (; row < rows; row += step, buf ^= 1) {
    const uint4 rv = dres ? at(dres, row) : zero, xn = at(x, row + step), yn = at(dy, row + step);
    const float rstd = rstd_in[row];
    float g[8], xh[8], dv[8], s = 0.0f;
    get(gv, g); get(xv, xh); get(yv, dv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      xh[j] *= rstd;
      dg[j] += dv[j] * xh[j];
      dv[j] *= g[j];
      s += dv[j] * xh[j];
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sh[buf][threadIdx.x >> 5] = s;
    __syncthreads();
    const float4 a = reinterpret_cast<const float4*>(sh[buf])[0], b = reinterpret_cast<const float4*>(sh[buf])[1];
    const float m1 = ((a.x + a.y) + (a.z + a.w) + ((b.x + b.y) + (b.z + b.w))) / d;
    if (live) {
      float r[8], o[8];
      get(rv, r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = rstd * (dv[j] - xh[j] * m1);
        if (dres) o[j] += r[j];
      }
      store8(dx + (size_t)row * d + col, o);
    }
    xv = xn; yv = yn;
  }
  if (live) {
    float* pg = partial_dgamma + (size_t)blockIdx.x * d + col;
#pragma unroll
    for (int j = 0; j < 8; ++j) pg[j] = dg[j];
  }
}

// ---- rows of up to 1024 features: one warp per row --------------------------------------------------------------------
// A block per row leaves most of its 256 threads without a vector below 2048 features (96 busy at 768) and passes two to
// four block barriers per row; a warp keeps a row of up to 1024 in registers and needs shuffles only.  Forward of 16384 rows
// of 768 features: 36 us with a block per row, 19 now, 15 of bytes.
// T is bf16, or float for the layer protocol, whose tensors then need no conversion passes around the call.
constexpr int WARP_ROWS = NT / 32;      // rows in flight per CTA

__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void store8(float* p, const float (&f)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ float as_stored(float v, const __nv_bfloat16*) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ float as_stored(float v, const float*) { return v; }

// fp32 tensors whose values count as bf16: rounded when read and when written, so that the results are those of the bf16 form
// between two conversion passes.  The layer protocol takes this form: a pre-activation that keeps more bits may fall on the
// other side of the ReLU behind it, which a gradient summed over a few rows shows.
struct F32AsBf16 {
  float v;
};
__device__ __forceinline__ float as_stored(float v, const F32AsBf16*) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ void load8(const F32AsBf16* p, float (&f)[8]) {
  load8(reinterpret_cast<const float*>(p), f);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = as_stored(f[j], p);
}
__device__ __forceinline__ void store8(F32AsBf16* p, const float (&f)[8]) {
  float r[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = as_stored(f[j], p);
  store8(reinterpret_cast<float*>(p), r);
}

// Eight elements as they lie in memory
template <typename T>
struct Raw8;
template <>
struct Raw8<__nv_bfloat16> {
  uint4 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
  }
  __device__ __forceinline__ void set(const float (&f)[8]) {
    u = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
  }
};
template <>
struct Raw8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = reinterpret_cast<const float4*>(p)[0];
    b = reinterpret_cast<const float4*>(p)[1];
  }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
};
template <>
struct Raw8<F32AsBf16> {
  Raw8<float> raw;
  __device__ __forceinline__ void load(const F32AsBf16* p) { raw.load(reinterpret_cast<const float*>(p)); }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    raw.get(f);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = as_stored(f[j], static_cast<const F32AsBf16*>(nullptr));
  }
};

// GELU: the normalised row is rounded to T and goes through the activation before it is stored.
template <typename T, bool RMS, int MV, bool GELU = false>
__global__ void __launch_bounds__(NT)
norm_fwd_warp_kernel(const T* __restrict__ x, const T* __restrict__ residual, const T* __restrict__ gamma,
                     const T* __restrict__ beta, T* __restrict__ y, T* __restrict__ sum_out, float* __restrict__ mean_out,
                     float* __restrict__ rstd_out, int rows, int d, float eps) {
  chain_begin(x, residual, gamma, beta);
  const int row = blockIdx.x * WARP_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int nvec = d >> 3;
  const size_t base = (size_t)row * d;
  float v[MV][8];
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) load8(x + base + vi * 8, v[i]);
  }
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) {
      if (residual) {
        float r[8];
        load8(residual + base + vi * 8, r);
        // normalise what is stored (rounded to T) so forward and backward agree
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = sum_out ? as_stored(v[i][j] + r[j], x) : v[i][j] + r[j];
      }
      if (sum_out) store8(sum_out + base + vi * 8, v[i]);      // without a residual: a copy of x
#pragma unroll
      for (int j = 0; j < 8; ++j) s += RMS ? v[i][j] * v[i][j] : v[i][j];
    }
  }
  s = warp_sum(s) / d;
  float mean = 0.0f, rstd;
  if (RMS) {
    rstd = rsqrtf(s + eps);
  } else {
    mean = s;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < MV; ++i) {
      if (lane + i * 32 < nvec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float c = v[i][j] - mean;
          q += c * c;
        }
      }
    }
    rstd = rsqrtf(warp_sum(q) / d + eps);
  }
  if (lane == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < MV; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) {
      float g[8], o[8];
      load8(gamma + vi * 8, g);
      if (!RMS && beta) {
        float b[8];
        load8(beta + vi * 8, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * g[j] + b[j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * g[j];
      }
      if (GELU) {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = gelu_tanh(as_stored(o[j], x));
      }
      store8(y + base + vi * 8, o);
    }
  }
}

// Backward for up to 2048 features: thread t owns the 8 columns from 8 t, a persistent CTA of d / 8 threads takes ROWS rows
// per step.  The gradient sums of a column then need 16 registers, not 16 per vector of a whole row (a warp per row spilled
// at 1024 features and kept 16 rows in flight per SM), all loads of a step are issued together, and its row sums cost one
// barrier: two to four per row with a block per row.
// GELU: dy is the gradient behind an activation of the (rounded) normalised row, which is formed again from x here; the
// product with the activation's derivative is rounded to T as a pass of its own would store it.
template <typename T, bool RMS, int ROWS, bool GELU = false>
__global__ void __launch_bounds__(NT)
norm_bwd_rows_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, const T* __restrict__ dres,
                     T* __restrict__ dx, float* __restrict__ partial_dgamma, float* __restrict__ partial_dbeta, int rows, int d,
                     const T* __restrict__ beta = nullptr) {
  chain_begin(dy, x, gamma, mean_in, rstd_in, dres, beta);
  __shared__ float sh[2][NT / 32][2 * ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int c0 = threadIdx.x * 8;
  const bool live = c0 < d;
  float g[8], dg[8], db[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) g[j] = dg[j] = db[j] = 0.0f;
  if (live) load8(gamma + c0, g);
  float shift[GELU ? 8 : 1];
  if constexpr (GELU) {
#pragma unroll
    for (int j = 0; j < 8; ++j) shift[j] = 0.0f;
    if (live) load8(beta + c0, shift);
  }
  int buf = 0;
  for (long long row0 = (long long)blockIdx.x * ROWS; row0 < rows; row0 += (long long)gridDim.x * ROWS, buf ^= 1) {
    Raw8<T> xr[ROWS], yr[ROWS], rr[ROWS];
    float mean[ROWS], rstd[ROWS], sums[2 * ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (row0 + r < rows && live) {
        const size_t at = (size_t)(row0 + r) * d + c0;
        xr[r].load(x + at);
        yr[r].load(dy + at);
        if (dres) rr[r].load(dres + at);
      }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const bool in = row0 + r < rows;
      mean[r] = !RMS && in ? mean_in[row0 + r] : 0.0f;
      rstd[r] = in ? rstd_in[row0 + r] : 0.0f;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float s1 = 0.0f, s2 = 0.0f;
      if (row0 + r < rows && live) {
        float xv[8], dv[8];
        xr[r].get(xv);
        yr[r].get(dv);
        if constexpr (GELU) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            dv[j] = as_stored(dv[j] * gelu_tanh_grad(as_stored((xv[j] - mean[r]) * rstd[r] * g[j] + shift[j], x)), x);
          yr[r].set(dv);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (xv[j] - mean[r]) * rstd[r], gy = dv[j] * g[j];
          dg[j] += dv[j] * xh;
          if (!RMS) db[j] += dv[j];
          s1 += gy * xh;
          s2 += gy;
        }
      }
      sums[2 * r] = warp_sum(s1);
      sums[2 * r + 1] = RMS ? 0.0f : warp_sum(s2);
    }
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 2 * ROWS; ++i) sh[buf][warp][i] = sums[i];
    }
    __syncthreads();      // the other buffer's readers are past it: they arrive here only after reading
#pragma unroll
    for (int i = 0; i < 2 * ROWS; ++i) {
      float t = 0.0f;
      for (int w = 0; w < warps; ++w) t += sh[buf][w][i];
      sums[i] = t / d;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (row0 + r >= rows || !live) continue;
      float xv[8], dv[8], o[8];
      xr[r].get(xv);
      yr[r].get(dv);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        o[j] = rstd[r] * (dv[j] * g[j] - sums[2 * r + 1] - (xv[j] - mean[r]) * rstd[r] * sums[2 * r]);
      if (dres) {  // gradient arriving through the residual branch
        float q[8];
        rr[r].get(q);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += q[j];
      }
      store8(dx + (size_t)(row0 + r) * d + c0, o);
    }
  }
  if (!live) return;
  store8(partial_dgamma + (size_t)blockIdx.x * d + c0, dg);
  if (!RMS && partial_dbeta) store8(partial_dbeta + (size_t)blockIdx.x * d + c0, db);
}

// out[c] (+)= sum_p partial[p, c]; with out2, blockIdx.y = 1 does the same for the second set of partials.  A CTA owns
// 32 columns; its 32 thread rows sum every 32nd partial (each a coalesced 128-byte read) and are combined through shared
// memory.
__global__ void __launch_bounds__(1024)
reduce_partials_kernel(const float* __restrict__ partial, float* __restrict__ out, const float* __restrict__ partial2,
                       float* __restrict__ out2, int parts, int d, int accumulate) {
  chain_begin(partial, partial2);
  if (blockIdx.y) {
    partial = partial2;
    out = out2;
  }
  __shared__ float sh[32][33];
  const int cx = threadIdx.x & 31, k = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s0 = 0.0f, s1 = 0.0f;
  if (c < d) {
    int p = k;
    for (; p + 32 < parts; p += 64) {
      s0 += partial[(size_t)p * d + c];
      s1 += partial[(size_t)(p + 32) * d + c];
    }
    if (p < parts) s0 += partial[(size_t)p * d + c];
  }
  sh[k][cx] = s0 + s1;
  __syncthreads();
  const float t = warp_sum(sh[cx][k]);       // thread row k now holds column k's 32 sums
  const int cc = blockIdx.x * 32 + k;
  if (cx == 0 && cc < d) out[cc] = accumulate ? out[cc] + t : t;
}

constexpr int kWarpRowFeatures = 1024;   // forward, fp32 form
// Backward with a thread per 8 columns: 16384 rows of 768 / 1024 features in 31 / 38 us where a block per row took 62 / 67
// (15 / 21 of bytes); with 2048 features LayerNorm takes 73 instead of 88 us, but RMSNorm 73 instead of 63, because the
// block kernel keeps four CTAs resident without the offset's sums.  Two rows per step and 768 threads per SM are the best
// of {1, 2, 4} x {512, 768, 1024}.
constexpr int kRowsThreads = 768;
inline bool rows_kernel(int rms, int d) { return d <= kWarpRowFeatures || (!rms && d <= NT * 8); }
inline int bwd_threads(int d) { return (d + 255) / 256 * 32; }
inline int step_grid(int grid, int rows) { return grid < (rows + 1) / 2 ? grid : (rows + 1) / 2; }      // at most a CTA per step of two rows

template <typename T>
int fwd_warp(int rms, const T* x, const T* r, const T* g, const T* b, T* y, T* s, float* mean, float* rstd, int rows, int d,
             float eps, cudaStream_t stream) {
  const int grid = (rows + WARP_ROWS - 1) / WARP_ROWS;
#define ST_FWD_WARP(MVV) \
  if (rms) st::chained(norm_fwd_warp_kernel<T, true, MVV>, grid, NT, 0, stream)(x, r, g, b, y, s, mean, rstd, rows, d, eps); \
  else st::chained(norm_fwd_warp_kernel<T, false, MVV>, grid, NT, 0, stream)(x, r, g, b, y, s, mean, rstd, rows, d, eps)
  switch ((d + 255) / 256) {
    case 1: ST_FWD_WARP(1); break;
    case 2: ST_FWD_WARP(2); break;
    case 3: ST_FWD_WARP(3); break;
    default: ST_FWD_WARP(4); break;
  }
#undef ST_FWD_WARP
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

template <typename T>
int bwd_rows(int rms, const T* dy, const T* x, const T* g, const float* mean, const float* rstd, const T* dres, T* dx,
             float* pg, float* pb, int rows, int d, int grid, cudaStream_t stream) {
  constexpr int ROWS = 2;
  const int threads = bwd_threads(d);
  if (rms) st::chained(norm_bwd_rows_kernel<T, true, ROWS>, grid, threads, 0, stream)(dy, x, g, mean, rstd, dres, dx, pg, nullptr, rows, d, nullptr);
  else st::chained(norm_bwd_rows_kernel<T, false, ROWS>, grid, threads, 0, stream)(dy, x, g, mean, rstd, dres, dx, pg, pb, rows, d, nullptr);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

int reduce_param_grads(int rms, const float* pg, const float* pb, float* dgamma, float* dbeta, int grid, int d, int accumulate,
                       cudaStream_t stream) {
  const bool both = !rms && dbeta;
  st::chained(reduce_partials_kernel, dim3((d + 31) / 32, both ? 2 : 1), 1024, 0, stream)(pg, dgamma, pb, dbeta, grid, d, accumulate);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

}  // namespace

namespace st {
int norm_bwd_grid(int rows) {
  int g = sm_count() * 2;
  return rows < g ? rows : g;
}
// CTAs for the regular entry: as many as stay resident (register footprint grows with d)
int norm_bwd_grid_for(int rows, int d) {
  if (d <= kWarpRowFeatures) {
    // Two rows per CTA are one step; four as soon as the chip is full, because the sum over the partials grows with the CTAs:
    // 4000 rows of 264, RMSNorm, 12.9 us with two, 10.3 with four, 11.4 with eight; 600 rows 5.5, 6.9, 9.1.
    if (rows <= 2 * sm_count()) return rows;
    const int resident = kRowsThreads / bwd_threads(d);
    const int need = rows <= 6 * sm_count() ? (rows + 1) / 2 : (rows + 3) / 4, most = sm_count() * (resident < 16 ? resident : 16);
    return need < most ? need : most;
  }
  const int per_sm = d <= 2048 ? 4 : 2;
  int g = sm_count() * per_sm;
  return rows < g ? rows : g;
}
}  // namespace st

static int check_dims(int rows, int d) {
  if (rows <= 0 || d <= 0) return st::fail(ST_ERR_INVALID, "norm: non-positive dimension");
  if (d & 7) return st::fail(ST_ERR_INVALID, "norm: feature dimension must be a multiple of 8");
  if (d > NT * MAXV * 8) return st::fail(ST_ERR_TOO_LARGE, "norm: feature dimension above 8192");
  return ST_OK;
}

ST_API int st_norm_fwd(int rms, const void* x, const void* residual, const void* gamma,
                       const void* beta, void* y, void* sum_out, float* mean, float* rstd, int rows,
                       int d, float eps, void* stream_v) {
  if (int e = check_dims(rows, d)) return e;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto R = static_cast<const __nv_bfloat16*>(residual);
  auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto B = static_cast<const __nv_bfloat16*>(beta);
  auto Y = static_cast<__nv_bfloat16*>(y);
  auto S = static_cast<__nv_bfloat16*>(sum_out);
  // A warp per row, or a block while that leaves SMs without enough warps: 600 rows of 1024, LayerNorm 4.2 us in warps and 3.0 in
  // blocks (RMSNorm 3.2, 2.4), of 512 both 2.9; 1500 rows 4.7 and 4.5, 3000 4.8 and 6.2.  Up to 256 features the warp has one
  // vector per lane and never loses.
  const bool few = rows <= (d > 512 ? 8 : 4) * st::sm_count() && d > 256;
  if (d <= kWarpRowFeatures && !few) return fwd_warp<__nv_bfloat16>(rms, X, R, G, B, Y, S, mean, rstd, rows, d, eps, s);
#define ST_NORM_FWD(RMSV, MVV) st::chained(norm_fwd_kernel<RMSV, MVV>, rows, NT, 0, s)(X, R, G, B, Y, S, mean, rstd, rows, d, eps)
  const int mv = d <= NT * 8 ? 1 : (d <= NT * 16 ? 2 : 4);
  if (rms) {
    if (mv == 1) ST_NORM_FWD(true, 1); else if (mv == 2) ST_NORM_FWD(true, 2); else ST_NORM_FWD(true, 4);
  } else {
    if (mv == 1) ST_NORM_FWD(false, 1); else if (mv == 2) ST_NORM_FWD(false, 2); else ST_NORM_FWD(false, 4);
  }
#undef ST_NORM_FWD
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// Number of fp32 scratch elements st_norm_bwd needs for `rows` x `d`.
ST_API long long st_norm_bwd_scratch_elems(int rows, int d) {
  return 2ll * st::norm_bwd_grid_for(rows, d) * d;
}

int st::norm_bwd_launch(int rms, const void* dy, const void* x, const void* gamma,
                        const float* mean, const float* rstd, const void* dres, void* dx,
                        float* dgamma, float* dbeta, int accumulate, float* scratch, int rows,
                        int d, int grid, cudaStream_t s) {
  if (int e = check_dims(rows, d)) return e;
  if (grid < 1) return st::fail(ST_ERR_INVALID, "norm_bwd: grid must be positive");
  float* pg = scratch;
  float* pb = scratch + (size_t)grid * d;      // (a smaller grid below leaves the space between unused)
  auto DY = static_cast<const __nv_bfloat16*>(dy);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto DR = static_cast<const __nv_bfloat16*>(dres);
  auto DX = static_cast<__nv_bfloat16*>(dx);
  // few rows: a block per row is one step without a second row's share (64 x 264 4.0 us, in pairs 4.9; 600 x 264 7.4 and 5.5)
  if (rms && rows <= 2 * st::sm_count() && d <= NT * 8) {
    grid = grid < rows ? grid : rows;
    st::chained(rms_bwd_ahead_kernel, grid, NT, 0, s)(DY, X, G, rstd, DR, DX, pg, rows, d);
    ST_CUDA_CHECK(cudaGetLastError());
    return reduce_param_grads(rms, pg, pb, dgamma, dbeta, grid, d, accumulate, s);
  }
  if (rows_kernel(rms, d)) {
    grid = step_grid(grid, rows);
    if (d > kWarpRowFeatures && grid > st::sm_count() * 3) grid = st::sm_count() * 3;      // 768 of 256 threads
    if (int e = bwd_rows<__nv_bfloat16>(rms, DY, X, G, mean, rstd, DR, DX, pg, rms ? nullptr : pb, rows, d, grid, s)) return e;
    return reduce_param_grads(rms, pg, pb, dgamma, dbeta, grid, d, accumulate, s);
  }
#define ST_NORM_BWD(RMSV, MVV, PB) st::chained(norm_bwd_kernel<RMSV, MVV>, grid, NT, 0, s)(DY, X, G, mean, rstd, DR, DX, pg, PB, rows, d)
  const int mv = d <= NT * 8 ? 1 : (d <= NT * 16 ? 2 : 4);
  if (rms) {
    if (mv == 1) st::chained(rms_bwd_ahead_kernel, grid, NT, 0, s)(DY, X, G, rstd, DR, DX, pg, rows, d);
    else if (mv == 2) ST_NORM_BWD(true, 2, nullptr); else ST_NORM_BWD(true, 4, nullptr);
  } else {
    if (mv == 2) ST_NORM_BWD(false, 2, pb); else ST_NORM_BWD(false, 4, pb);
  }
#undef ST_NORM_BWD
  ST_CUDA_CHECK(cudaGetLastError());
  return reduce_param_grads(rms, pg, pb, dgamma, dbeta, grid, d, accumulate, s);
}

// out[i] (+)= sum over p of partial[p * n + i], in a fixed order.
ST_API int st_reduce_partials(const float* partial, float* out, int parts, int n, int accumulate, void* stream_v) {
  if (!partial || !out || parts <= 0 || n <= 0) return st::fail(ST_ERR_INVALID, "reduce_partials: bad arguments");
  st::chained(reduce_partials_kernel, (n + 31) / 32, 1024, 0, reinterpret_cast<cudaStream_t>(stream_v))(partial, out, nullptr, nullptr, parts, n, accumulate);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// LayerNorm followed by GELU (tanh form), bf16, rows of at most 2048 features: y = gelu(round(LayerNorm(x))), and its
// backward from x and the row statistics.  scratch: st_norm_bwd_scratch_elems floats.
ST_API int st_norm_gelu_max_features() { return NT * 8; }
ST_API int st_norm_gelu_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows, int d,
                            float eps, void* stream_v) {
  if (int e = check_dims(rows, d)) return e;
  if (d > NT * 8) return st::fail(ST_ERR_TOO_LARGE, "norm_gelu: feature dimension above 2048");
  if (!beta) return st::fail(ST_ERR_INVALID, "norm_gelu: LayerNorm with offset only");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto B = static_cast<const __nv_bfloat16*>(beta);
  auto Y = static_cast<__nv_bfloat16*>(y);
  const __nv_bfloat16* none = nullptr;
  __nv_bfloat16* no_sum = nullptr;
  const int grid = (rows + WARP_ROWS - 1) / WARP_ROWS;
#define ST_NORM_GELU(MVV) st::chained(norm_fwd_warp_kernel<__nv_bfloat16, false, MVV, true>, grid, NT, 0, s)(X, none, G, B, Y, no_sum, mean, rstd, rows, d, eps)
  if (d > kWarpRowFeatures) st::chained(norm_fwd_kernel<false, 1, true>, rows, NT, 0, s)(X, none, G, B, Y, no_sum, mean, rstd, rows, d, eps);
  else if (d > 768) ST_NORM_GELU(4);
  else if (d > 512) ST_NORM_GELU(3);
  else if (d > 256) ST_NORM_GELU(2);
  else ST_NORM_GELU(1);
#undef ST_NORM_GELU
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
ST_API int st_norm_gelu_bwd(const void* dy, const void* x, const void* gamma, const void* beta, const float* mean, const float* rstd,
                            void* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v) {
  if (int e = check_dims(rows, d)) return e;
  if (d > NT * 8) return st::fail(ST_ERR_TOO_LARGE, "norm_gelu: feature dimension above 2048");
  if (!beta || !dbeta || !scratch) return st::fail(ST_ERR_INVALID, "norm_gelu: offset, its gradient and scratch are required");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  int grid = step_grid(st::norm_bwd_grid_for(rows, d), rows);
  if (d > kWarpRowFeatures && grid > st::sm_count() * 3) grid = st::sm_count() * 3;
  float* pb = scratch + (size_t)grid * d;
  const __nv_bfloat16* none = nullptr;
  st::chained(norm_bwd_rows_kernel<__nv_bfloat16, false, 2, true>, grid, bwd_threads(d), 0, s)(
      static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), mean, rstd,
      none, static_cast<__nv_bfloat16*>(dx), scratch, pb, rows, d, static_cast<const __nv_bfloat16*>(beta));
  ST_CUDA_CHECK(cudaGetLastError());
  return reduce_param_grads(0, scratch, pb, dgamma, dbeta, grid, d, accumulate, s);
}

// fp32 tensors, rows of at most 1024 features, 16-byte aligned: the layer protocol's LayerNorm without conversion passes.
// scratch: st_norm_bwd_scratch_elems floats.
namespace {
template <typename T>
int fwd_f32(int rms, const float* x, const float* residual, const float* gamma, const float* beta, float* y, float* sum_out,
            float* mean, float* rstd, int rows, int d, float eps, void* stream_v) {
  if (int e = check_dims(rows, d)) return e;
  if (d > kWarpRowFeatures) return st::fail(ST_ERR_TOO_LARGE, "norm_f32: feature dimension above 1024");
  auto in = [](const float* p) { return reinterpret_cast<const T*>(p); };
  return fwd_warp<T>(rms, in(x), in(residual), in(gamma), in(beta), reinterpret_cast<T*>(y), reinterpret_cast<T*>(sum_out), mean, rstd,
                     rows, d, eps, reinterpret_cast<cudaStream_t>(stream_v));
}
template <typename T>
int bwd_f32(int rms, const float* dy, const float* x, const float* gamma, const float* mean, const float* rstd, const float* dres,
            float* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows, int d, void* stream_v) {
  if (int e = check_dims(rows, d)) return e;
  if (d > kWarpRowFeatures) return st::fail(ST_ERR_TOO_LARGE, "norm_f32: feature dimension above 1024");
  if (!scratch) return st::fail(ST_ERR_INVALID, "norm_f32: scratch buffer is required");
  const int grid = step_grid(st::norm_bwd_grid_for(rows, d), rows);
  float* pb = scratch + (size_t)grid * d;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  auto in = [](const float* p) { return reinterpret_cast<const T*>(p); };
  if (int e = bwd_rows<T>(rms, in(dy), in(x), in(gamma), mean, rstd, in(dres), reinterpret_cast<T*>(dx), scratch, rms ? nullptr : pb,
                          rows, d, grid, s))
    return e;
  return reduce_param_grads(rms, scratch, pb, dgamma, dbeta, grid, d, accumulate, s);
}
}  // namespace

ST_API int st_norm_f32_max_features() { return kWarpRowFeatures; }
ST_API int st_norm_fwd_f32(int rms, const float* x, const float* residual, const float* gamma, const float* beta, float* y,
                           float* sum_out, float* mean, float* rstd, int rows, int d, float eps, void* stream_v) {
  return fwd_f32<float>(rms, x, residual, gamma, beta, y, sum_out, mean, rstd, rows, d, eps, stream_v);
}
ST_API int st_norm_bwd_f32(int rms, const float* dy, const float* x, const float* gamma, const float* mean, const float* rstd,
                           const float* dres, float* dx, float* dgamma, float* dbeta, int accumulate, float* scratch, int rows,
                           int d, void* stream_v) {
  return bwd_f32<float>(rms, dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, accumulate, scratch, rows, d, stream_v);
}
// The same with every operand and result rounded to bf16 (F32AsBf16).
ST_API int st_norm_fwd_f32_rounded(int rms, const float* x, const float* residual, const float* gamma, const float* beta, float* y,
                                   float* sum_out, float* mean, float* rstd, int rows, int d, float eps, void* stream_v) {
  return fwd_f32<F32AsBf16>(rms, x, residual, gamma, beta, y, sum_out, mean, rstd, rows, d, eps, stream_v);
}
ST_API int st_norm_bwd_f32_rounded(int rms, const float* dy, const float* x, const float* gamma, const float* mean, const float* rstd,
                                   const float* dres, float* dx, float* dgamma, float* dbeta, int accumulate, float* scratch,
                                   int rows, int d, void* stream_v) {
  return bwd_f32<F32AsBf16>(rms, dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, accumulate, scratch, rows, d, stream_v);
}

// dgamma / dbeta are fp32 [d]; with accumulate != 0 the kernel adds to them.
ST_API int st_norm_bwd(int rms, const void* dy, const void* x, const void* gamma,
                       const float* mean, const float* rstd, const void* dres, void* dx,
                       float* dgamma, float* dbeta, int accumulate, float* scratch, int rows,
                       int d, void* stream_v) {
  if (!scratch) return st::fail(ST_ERR_INVALID, "norm_bwd: scratch buffer is required");
  return st::norm_bwd_launch(rms, dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, accumulate,
                             scratch, rows, d, st::norm_bwd_grid_for(rows, d), reinterpret_cast<cudaStream_t>(stream_v));
}

// ------------------------------------------------------------------------------------------
// Entry point that allocates nothing (see norm_noalloc.h).
// ------------------------------------------------------------------------------------------
#include "norm_noalloc.h"
#include <cstdio>

// Scratch for the per-CTA dgamma / dbeta partials.  In host code this name is only a handle
// for cudaGetSymbolAddress; the kernels get the real device address as an argument.
static __device__ __align__(256) float g_norm_bwd_static_scratch[ST_NORM_BWD_NOALLOC_MAX_ELEMS];

namespace {
constexpr int kNoallocMaxDevices = 16;
float* g_noalloc_ptr[kNoallocMaxDevices] = {nullptr};
}  // namespace

ST_API int st_norm_bwd_noalloc(int rms, const void* dy, const void* x, const void* gamma,
                               const float* mean, const float* rstd, const void* dres, void* dx,
                               float* dgamma, float* dbeta, int accumulate, int rows, int d,
                               void* stream_v) {
  if (rows <= 0 || d <= 0) return st::fail(ST_ERR_INVALID, "norm_bwd_noalloc: non-positive dimension");
  const long long need = 2ll * st::norm_bwd_grid(rows) * d;
  if (need > (long long)ST_NORM_BWD_NOALLOC_MAX_ELEMS) {
    char buf[200];
    snprintf(buf, sizeof(buf),
             "norm_bwd_noalloc: rows=%d d=%d needs %lld scratch floats, the built-in buffer holds %d; "
             "use st_norm_bwd with a caller-provided scratch buffer",
             rows, d, need, (int)ST_NORM_BWD_NOALLOC_MAX_ELEMS);
    return st::fail(ST_ERR_TOO_LARGE, buf);
  }
  int dev = 0;
  ST_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoallocMaxDevices) return st::fail(ST_ERR_INVALID, "norm_bwd_noalloc: device index out of range");
  if (g_noalloc_ptr[dev] == nullptr) {
    // once per device, with that device current: resolve the array's device address
    float* p = nullptr;
    ST_CUDA_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_norm_bwd_static_scratch));
    if (p == nullptr) return st::fail(ST_ERR_CUDA, "norm_bwd_noalloc: cudaGetSymbolAddress returned null");
    g_noalloc_ptr[dev] = p;
  }
  // Up to 1024 features a CTA has 32 to 128 threads, and two of them leave an SM idle: as many as the regular entry takes, if the
  // array holds their partials.  RMSNorm over 16384 rows of 256 / 768 / 1024 features, with two per SM and now: 38 / 47 / 61 and
  // 18 / 28 / 40 us (a block per row 39 / 45 / 66).
  const int least = st::norm_bwd_grid(rows), room = ST_NORM_BWD_NOALLOC_MAX_ELEMS / (2 * d);
  int grid = st::norm_bwd_grid_for(rows, d);
  grid = grid < room ? grid : room;
  return st::norm_bwd_launch(rms, dy, x, gamma, mean, rstd, dres, dx, dgamma, dbeta, accumulate, g_noalloc_ptr[dev], rows, d,
                             grid > least ? grid : least, reinterpret_cast<cudaStream_t>(stream_v));
}
