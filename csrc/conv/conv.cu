// 3x3 convolution (stride 1, padding 1) as implicit GEMM on the tcgen05 kernel, plus pooling.
//
// Activations are NHWC bf16, so a block of output pixels x 64 input channels at one filter tap
// is a rectangular box of the input tensor: the TMA unit fetches it directly (zero-filling the
// halo), no im2col matrix is ever materialised.  Weights are stored [OC][tap][IC] (tap-major K).
//
//   forward        Y[p, oc]  = act(Σ_tap Σ_ic X[p + tap, ic] · W[oc, tap, ic] + bias[oc])
//   data gradient  dX[p, ic] = (Σ_tap Σ_oc dY[p + tap, oc] · Wt[ic, tap, oc]) ⊙ [X[p, ic] > 0]
//                  — the same kernel on dY with the flipped/transposed weights Wt and the ReLU mask of
//                  the layer input fused in the epilogue
//   weight gradient dW[oc, tap, ic] += Σ_p dY[p, oc] · X[p + tap, ic]
//                  — K runs over pixels and N over (tap, ic), one K split per batch index, fp32 atomics into dW
// The first layer (3 input channels) uses a small explicit im2col (K padded to 32).
//
// Pooling: 2x2 max pool forward/backward and global average pool forward/backward on NHWC bf16.
//
// Reference parity: fused_im2col_matmul.wgsl, fused_grad_input_col2im.wgsl (crates/st-tensor/src/
// wgpu_shaders), CPU im2col path of crates/st-nn/src/layers/conv.rs:607-1017, pooling entry points
// of tensor_utils.wgsl.
#include "conv_halo.cuh"
#include <cstring>

namespace {
using namespace st;
using namespace st::gemm;

template <int BN, int STAGES, bool A_MN, bool B_MN>
int launch_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const OutMaps& tmC, const GemmParams& p,
                cudaStream_t stream) {
  using L = SmemLayout<BN, STAGES>;
  auto kern = gemm_bf16_kernel<BN, STAGES, A_MN, B_MN, COMM_NONE>;
  static bool configured[st::kMaxDevices] = {false};   // the attribute is per device
  const int dev = st::current_device();
  if (!configured[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    configured[dev] = true;
  }
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.batch;
  const int grid = tiles < st::sm_count() ? tiles : st::sm_count();
  GemmComm none{};
  st::chained(kern, grid, NUM_THREADS, L::TOTAL, stream)(tmA, tmB, tmC, tmA, p, none);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// pixel block of `pixels` (128 or 64) output positions: W columns x Hb rows x Nb images
bool block_geometry(int N, int H, int W, int pixels, int* Hb, int* Nb) {
  if (W <= 0 || W > pixels || pixels % W != 0) return false;
  int hb = pixels / W;
  int nb = 1;
  if (hb > H) {
    if (hb % H != 0) return false;
    nb = hb / H;
    hb = H;
  }
  if (H % hb != 0 || N % nb != 0) return false;
  *Hb = hb;
  *Nb = nb;
  return true;
}

bool nhwc_map(CUtensorMap* out, const void* base, int N, int H, int W, int C, int Wb, int Hb, int Nb) {
  uint64_t dims[4] = {(uint64_t)C, (uint64_t)W, (uint64_t)H, (uint64_t)N};
  uint64_t strides[3] = {(uint64_t)C * 2, (uint64_t)W * C * 2, (uint64_t)H * W * C * 2};
  uint32_t box[4] = {64, (uint32_t)Wb, (uint32_t)Hb, (uint32_t)Nb};
  return encode_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// One thread writes eight neighbouring entries of a pixel's row of the column matrix with one 16-byte store: the bound is
// that store (67 MB and 230 us before for 256 images of 64 x 64 x 3, one 2-byte store and four divisions per entry).
// The index is 32-bit where the matrix allows it: 64-bit divisions took 61 us here.
template <typename Index>
__global__ void __launch_bounds__(256)
im2col3x3_small_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col,
                       int N, int H, int W, int C, int Kpad, int aligned) {
  chain_begin(x);
  const int K8 = Kpad / 8;
  const Index total = (Index)N * H * W * K8;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (Index)gridDim.x * blockDim.x) {
    const int k0 = (int)(i % K8) * 8;
    const Index pix = i / K8;
    const int w = (int)(pix % W);
    const int h = (int)((pix / W) % H);
    int tap = k0 / C, c = k0 - tap * C;
    __nv_bfloat16 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = __float2bfloat16(0.0f);
      const int dh = tap / 3 - 1, dw = tap % 3 - 1;
      if (tap < 9 && h + dh >= 0 && h + dh < H && w + dw >= 0 && w + dw < W) v[j] = x[((long long)pix + dh * W + dw) * C + c];
      if (++c == C) { c = 0; ++tap; }
    }
    if (aligned) {
      uint4 u;
      u.x = __bfloat16_as_ushort(v[0]) | (uint32_t)__bfloat16_as_ushort(v[1]) << 16;
      u.y = __bfloat16_as_ushort(v[2]) | (uint32_t)__bfloat16_as_ushort(v[3]) << 16;
      u.z = __bfloat16_as_ushort(v[4]) | (uint32_t)__bfloat16_as_ushort(v[5]) << 16;
      u.w = __bfloat16_as_ushort(v[6]) | (uint32_t)__bfloat16_as_ushort(v[7]) << 16;
      *reinterpret_cast<uint4*>(col + (long long)i * 8) = u;
    } else {
      for (int j = 0; j < 8; ++j) col[(long long)i * 8 + j] = v[j];
    }
  }
}

// Image channel counts (1 to 4), rows of the usual width (9 C rounded up to 32) and a 16-byte aligned matrix: a thread per
// pixel and no division per entry, which bounded the kernel above (55 us for 256 images of 64 x 64 x 3).  The row goes
// through shared memory, as 16-byte units in an order without bank conflicts, so that neighbouring threads store
// neighbouring units; what is left is the store of 67 MB.
// PLANES: the images are [N][C][H][W] instead of [N][H][W][C] (a pass that only reorders them takes 7 us for the same batch), and
// the weights [OC][9 C], if given, are padded to the matrix's width in the same launch.
template <int C, bool PLANES>
__global__ void __launch_bounds__(256)
im2col3x3_image_kernel(const __nv_bfloat16* __restrict__ x, uint4* __restrict__ col, long long pixels, int H, int W,
                       const __nv_bfloat16* __restrict__ weights, __nv_bfloat16* __restrict__ padded, int OC) {
  chain_begin(x, weights);
  constexpr int K8 = (9 * C + 31) / 32 * 4;
  __shared__ uint4 rows[256 * K8];
  const __nv_bfloat16 zero = __float2bfloat16(0.0f);
  if (PLANES && weights) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < OC * K8 * 8; i += gridDim.x * 256) {
      const int oc = i / (K8 * 8), k = i - oc * (K8 * 8);
      padded[i] = k < 9 * C ? weights[oc * (9 * C) + k] : zero;
    }
  }
  const long long plane = (long long)H * W;
  for (long long base = (long long)blockIdx.x * 256; base < pixels; base += (long long)gridDim.x * 256) {
    const long long pix = base + threadIdx.x;
    uint32_t v[K8 * 4];
#pragma unroll
    for (int j = 0; j < K8 * 4; ++j) v[j] = 0;
    if (pix < pixels) {
      const int w = (int)(pix % W), h = (int)((pix / W) % H);
#pragma unroll
      for (int dh = -1; dh <= 1; ++dh) {
        const bool row_in = h + dh >= 0 && h + dh < H;
        const __nv_bfloat16* src = PLANES ? x + pix + pix / plane * (C - 1) * plane + (long long)dh * W - 1
                                          : x + (pix + (long long)dh * W - 1) * C;
#pragma unroll
        for (int e = 0; e < 3 * C; ++e) {
          const int dw = e / C - 1, k = (dh + 1) * 3 * C + e;
          const bool in = row_in && (dw < 0 ? w > 0 : dw > 0 ? w + 1 < W : true);
          const uint32_t u = __bfloat16_as_ushort(in ? src[PLANES ? e % C * plane + e / C : e] : zero);
          v[k / 2] |= (k & 1) ? u << 16 : u;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < K8; ++q)
      rows[threadIdx.x * K8 + (q ^ ((threadIdx.x >> (K8 == 4 ? 1 : 0)) & (K8 - 1)))] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    __syncthreads();
    const long long units = (pixels - base < 256 ? pixels - base : 256) * K8;
#pragma unroll
    for (int i = 0; i < K8; ++i) {
      const int unit = i * 256 + threadIdx.x, p = unit / K8, q = unit % K8;
      if (unit < units) col[base * K8 + unit] = rows[p * K8 + (q ^ ((p >> (K8 == 4 ? 1 : 0)) & (K8 - 1)))];
    }
    __syncthreads();
  }
}

// The same with C % 8 == 0 and 16-byte aligned input: eight channels of one tap are one load and one store.
template <typename Index>
__global__ void __launch_bounds__(256)
im2col3x3_c8_kernel(const uint4* __restrict__ x, uint4* __restrict__ col, int N, int H, int W, int C8, int K8) {
  chain_begin(x);
  const Index total = (Index)N * H * W * K8;
  for (Index i = (Index)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (Index)gridDim.x * blockDim.x) {
    const int k = (int)(i % K8);
    const Index pix = i / K8;
    const int w = (int)(pix % W);
    const int h = (int)((pix / W) % H);
    const int tap = k / C8, c = k - tap * C8;
    const int dh = tap / 3 - 1, dw = tap % 3 - 1;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (tap < 9 && h + dh >= 0 && h + dh < H && w + dw >= 0 && w + dw < W) v = x[((long long)pix + dh * W + dw) * C8 + c];
    col[i] = v;
  }
}

// Weights of the data-gradient convolution: out[ic][8 - tap][oc] = in[oc][tap][ic], 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256)
dgrad_weights_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, int OC, int IC) {
  chain_begin(in);
  __shared__ __nv_bfloat16 tile[32][33];
  const int tap = blockIdx.z, ic0 = blockIdx.x * 32, oc0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (oc0 + r < OC && ic0 + threadIdx.x < IC) tile[r][threadIdx.x] = in[((long long)(oc0 + r) * 9 + tap) * IC + ic0 + threadIdx.x];
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8)
    if (ic0 + r < IC && oc0 + threadIdx.x < OC) out[((long long)(ic0 + r) * 9 + 8 - tap) * OC + oc0 + threadIdx.x] = tile[threadIdx.x][r];
}

// Eight channels per thread (16-byte loads, one 16-byte store of y and one 8-byte store of idx); C % 8 == 0.
__global__ void __launch_bounds__(256)
maxpool2_fwd8_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                     unsigned char* __restrict__ idx, int N, int H, int W, int C) {
  chain_begin(x);
  const int OH = H / 2, OW = W / 2, C8 = C / 8;
  const long long total = (long long)N * OH * OW * C8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c8 = i % C8;
    const long long p = i / C8;
    const int ow = p % OW;
    const int oh = (p / OW) % OH;
    const int n = p / ((long long)OW * OH);
    uint4 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
      v[t] = *reinterpret_cast<const uint4*>(
          x + ((((long long)n * H + oh * 2 + (t >> 1)) * W + ow * 2 + (t & 1)) * C + c8 * 8));
    float best[8];
    unsigned arg[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { best[j] = -INFINITY; arg[j] = 0; }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint32_t w[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = unpack_bf16x2(w[q]);
        if (f.x > best[2 * q]) { best[2 * q] = f.x; arg[2 * q] = t; }
        if (f.y > best[2 * q + 1]) { best[2 * q + 1] = f.y; arg[2 * q + 1] = t; }
      }
    }
    uint4 o;
    o.x = pack_bf16x2(best[0], best[1]); o.y = pack_bf16x2(best[2], best[3]);
    o.z = pack_bf16x2(best[4], best[5]); o.w = pack_bf16x2(best[6], best[7]);
    *reinterpret_cast<uint4*>(y + (p * C + c8 * 8)) = o;
    uint2 a;
    a.x = arg[0] | (arg[1] << 8) | (arg[2] << 16) | (arg[3] << 24);
    a.y = arg[4] | (arg[5] << 8) | (arg[6] << 16) | (arg[7] << 24);
    if (idx) *reinterpret_cast<uint2*>(idx + (p * C + c8 * 8)) = a;
  }
}

// y[n, h/2, w/2, c] = max over the 2x2 window; idx (uint8) records the arg-max for the backward pass
__global__ void maxpool2_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                    unsigned char* __restrict__ idx, int N, int H, int W, int C) {
  chain_begin(x);
  const int OH = H / 2, OW = W / 2;
  const long long total = (long long)N * OH * OW * (C / 2);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c2 = i % (C / 2);
    const long long p = i / (C / 2);
    const int ow = p % OW;
    const int oh = (p / OW) % OH;
    const int n = p / ((long long)OW * OH);
    float2 best = make_float2(-INFINITY, -INFINITY);
    int ix = 0, iy = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(
          x + ((((long long)n * H + oh * 2 + (t >> 1)) * W + ow * 2 + (t & 1)) * C + c2 * 2));
      const float2 f = __bfloat1622float2(v);
      if (f.x > best.x) { best.x = f.x; ix = t; }
      if (f.y > best.y) { best.y = f.y; iy = t; }
    }
    *reinterpret_cast<__nv_bfloat162*>(y + (p * C + c2 * 2)) = __floats2bfloat162_rn(best.x, best.y);
    if (idx) {
      idx[p * C + c2 * 2] = (unsigned char)ix;
      idx[p * C + c2 * 2 + 1] = (unsigned char)iy;
    }
  }
}

// Eight channels per thread; C % 8 == 0 and 16-byte aligned tensors.  With `pooled` (the forward's output) the gradient
// is also masked where the pooled value is not positive, which is the ReLU in front of the pool: only the arg-max of a
// window receives a gradient, and its value is the pooled one.  With `dbias` the masked gradient's channel sums are added
// to it: each thread keeps to one group of eight channels (C / 8 divides the block), so the sums stay in registers.
// Bound by its bytes: 134 MB written and 84 MB read for 256 x 64 x 64 x 64; the scalar kernel, the mask and the column
// sums took 318 us in five launches.
__global__ void __launch_bounds__(256)
maxpool2_bwd8_kernel(const uint4* __restrict__ dy, const uint2* __restrict__ idx, const uint4* __restrict__ pooled,
                     uint4* __restrict__ dx, float* __restrict__ dbias, int N, int H, int W, int C8) {
  chain_begin(dy, idx, pooled);
  const int OH = H / 2, OW = W / 2;
  const long long total = (long long)N * OH * OW * C8;
  float sum[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sum[j] = 0.0f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C8);
    const long long p = i / C8;
    const int ow = (int)(p % OW);
    const long long nh = p / OW;                     // image * OH + row: the window's first row is 2 nh of N * H
    const uint4 gv = dy[i];
    const uint2 av = idx[i];
    uint32_t g[4] = {gv.x, gv.y, gv.z, gv.w};
    if (pooled) {
      const uint4 yv = pooled[i];
      const uint32_t y[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = unpack_bf16x2(y[q]);
        g[q] &= (f.x > 0.0f ? 0x0000FFFFu : 0u) | (f.y > 0.0f ? 0xFFFF0000u : 0u);
      }
    }
    if (dbias) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = unpack_bf16x2(g[q]);
        sum[2 * q] += f.x;
        sum[2 * q + 1] += f.y;
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t a = (q < 2 ? av.x : av.y) >> ((q & 1) * 16);     // arg-max of channels 2 q and 2 q + 1
        o[q] = g[q] & (((a & 0xFFu) == t ? 0x0000FFFFu : 0u) | (((a >> 8) & 0xFFu) == t ? 0xFFFF0000u : 0u));
      }
      dx[((2 * nh + (t >> 1)) * W + 2 * ow + (t & 1)) * C8 + c] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (!dbias) return;
  __shared__ float sh[256 * 8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sh[threadIdx.x * 8 + j] = sum[j];
  __syncthreads();
  for (int ch = threadIdx.x; ch < C8 * 8; ch += 256) {                  // thread t owns channels of group t % C8
    float s = 0.0f;
    for (int t = ch >> 3; t < 256; t += C8) s += sh[t * 8 + (ch & 7)];
    atomicAdd(dbias + ch, s);
  }
}

__global__ void maxpool2_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const unsigned char* __restrict__ idx,
                                    __nv_bfloat16* __restrict__ dx, int N, int H, int W, int C) {
  chain_begin(dy, idx);
  const int OH = H / 2, OW = W / 2;
  const long long total = (long long)N * OH * OW * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = i % C;
    const long long p = i / C;
    const int ow = p % OW;
    const int oh = (p / OW) % OH;
    const int n = p / ((long long)OW * OH);
    const int t = idx[i];
    const __nv_bfloat16 g = dy[i];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      dx[(((long long)n * H + oh * 2 + (q >> 1)) * W + ow * 2 + (q & 1)) * C + c] =
          q == t ? g : __float2bfloat16(0.0f);
  }
}

// y[n, c] = mean over H*W
__global__ void avgpool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int N,
                                   int HW, int C) {
  chain_begin(x);
  const int n = blockIdx.x;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float s = 0.0f;
    for (int p = 0; p < HW; ++p) s += __bfloat162float(x[((long long)n * HW + p) * C + c]);
    y[(long long)n * C + c] = __float2bfloat16(s / HW);
  }
}
__global__ void avgpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, int N,
                                   int HW, int C) {
  chain_begin(dy);
  const long long total = (long long)N * HW * C;
  const float inv = 1.0f / HW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = i % C;
    const long long n = i / ((long long)HW * C);
    dx[i] = __float2bfloat16(__bfloat162float(dy[n * C + c]) * inv);
  }
}

inline int grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  const long long cap = (long long)st::sm_count() * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

struct StConvArgs {
  const void* x;       // bf16 NHWC [N, H, W, C]
  const void* w;       // bf16 [OC, 9*C] (tap-major)
  const void* bias;    // bf16 [OC] or null
  void* y;             // bf16 NHWC [N, H, W, OC]
  const void* aux_in;  // bf16 [N*H*W, OC]: ReLU mask source for act == 4, or null
  int N, H, W, C, OC;
  int act;             // 0 none, 1 relu, 4 relu_bwd(aux_in)
};

// Plan of the shared-row form (conv_halo.cuh): false where the geometry or the shared memory does not allow it.  `us` is its
// modelled time, about 4.2 (64 channels) or 5.5 us plus 1.0 us for every box of rows that an SM walks.  It loses where tiles
// of 256 pixels leave most SMs without one: 1 x 32 x 32, 64 to 128 channels, takes 8.6 us and 7.2 in 16 tiles of 128 x 64;
// 24 x 32 x 32, 128 to 128: 12.2 and 15.8; 256 x 32 x 32: 58 and 80; 256 x 64 x 64, 64 to 64: 88 and 141 (data gradient 95
// and 153).
struct HaloPlan {
  int bn, resident, smem;
  double us;
  st::conv::HaloParams p;
};
static bool halo_plan(const StConvArgs* a, HaloPlan* out) {
  using namespace st::conv;
  if (a->OC > 128 || (reinterpret_cast<uintptr_t>(a->aux_in) & 15) != 0 || a->W < 8 || kHaloPixels % a->W != 0) return false;
  const int rows = kHaloPixels / a->W;
  if (a->H % rows != 0) return false;
  HaloPlan& h = *out;
  h.bn = a->OC <= 64 ? 64 : 128;
  const int b_tile = h.bn * BK * 2, a_bytes = (rows + 2) * a->W * BK * 2, fixed = kHaloCStage + kHaloTail;
  h.resident = a->C == 64 && h.bn == 64 && 9 * b_tile + 2 * a_bytes + fixed <= kSmemLimit;
  const int base = fixed + (h.resident ? 9 * b_tile : 0), stage = a_bytes + (h.resident ? 0 : 3 * b_tile);
  int stages = (kSmemLimit - base) / stage;
  if (stages < 2) return false;
  if (stages > kHaloMaxStages) stages = kHaloMaxStages;
  h.smem = base + stages * stage;
  h.p = HaloParams{};
  h.p.hblocks = a->H / rows;
  h.p.tiles = a->N * h.p.hblocks;
  h.p.rows = rows; h.p.W = a->W;
  h.p.chunks = a->C / 64; h.p.C = a->C; h.p.OC = a->OC;
  h.p.act = a->act; h.p.stages = stages;
  h.p.bias = static_cast<const __nv_bfloat16*>(a->bias);
  h.p.aux_in = static_cast<const __nv_bfloat16*>(a->aux_in);
  h.p.err = st::error_word();
  h.us = (h.bn == 64 ? 4.2 : 5.5) + 3.0 * h.p.chunks * ((h.p.tiles + st::sm_count() - 1) / st::sm_count());
  return true;
}

ST_API int st_conv3x3_fwd(const StConvArgs* a, void* stream_v) {
  if (!a || !a->x || !a->w || !a->y) return st::fail(ST_ERR_INVALID, "conv3x3: null pointer");
  if (a->C % 64 != 0) return st::fail(ST_ERR_INVALID, "conv3x3: input channels must be a multiple of 64");
  if (a->OC % 8 != 0) return st::fail(ST_ERR_INVALID, "conv3x3: output channels must be a multiple of 8");
  int Hb, Nb;
  if (!block_geometry(a->N, a->H, a->W, BM, &Hb, &Nb))
    return st::fail(ST_ERR_INVALID, "conv3x3: image width must divide 128 and the batch must fill whole pixel blocks");
  const int P = a->N * a->H * a->W;
  CUtensorMap tmA, tmB;
  const TileChoice tile = choose_tile(P, a->OC, 9ll * a->C, 1, st::sm_count(), a->act == ACT_RELU_BWD ? EPI_OPERAND : EPI_PLAIN, true);
  HaloPlan halo;
  const bool use_halo = halo_plan(a, &halo) && halo.us <= tile.us;
  const int BN = use_halo ? halo.bn : tile.bn;
  const bool pair = tile.pair && !use_halo;
  if (!nhwc_map(&tmA, a->x, a->N, a->H, a->W, a->C, a->W, use_halo ? halo.p.rows + 2 : Hb, use_halo ? 1 : Nb)) return ST_ERR_CUDA;
  {
    uint64_t dims[3] = {(uint64_t)9 * a->C, (uint64_t)a->OC, 1};
    uint64_t strides[2] = {(uint64_t)9 * a->C * 2, (uint64_t)9 * a->C * 2 * a->OC};
    uint32_t box[3] = {BK, (uint32_t)(pair ? BN / 2 : BN), 1};
    if (!encode_tmap(&tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a->w, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return ST_ERR_CUDA;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  if (use_halo) {
    CUtensorMap tmY;
    uint64_t dims[3] = {(uint64_t)a->OC, (uint64_t)P, 1};
    uint64_t strides[2] = {(uint64_t)a->OC * 2, (uint64_t)a->OC * 2 * P};
    uint32_t box[3] = {64, 32, 1};
    if (!encode_tmap(&tmY, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a->y, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return ST_ERR_CUDA;
    if (halo.resident) return st::conv::launch_halo<64, true>(tmA, tmB, tmY, halo.p, halo.smem, s);
    if (BN == 64) return st::conv::launch_halo<64, false>(tmA, tmB, tmY, halo.p, halo.smem, s);
    return st::conv::launch_halo<128, false>(tmA, tmB, tmY, halo.p, halo.smem, s);
  }
  GemmParams p{};
  p.conv.mode = 1;
  p.conv.H = a->H; p.conv.W = a->W; p.conv.Hb = Hb; p.conv.Nb = Nb;
  p.conv.c_chunks = a->C / 64;
  p.C = a->y; p.ldc = a->OC;
  p.bias = static_cast<const __nv_bfloat16*>(a->bias);
  p.aux_in = static_cast<const __nv_bfloat16*>(a->aux_in);
  p.ld_aux_in = a->OC;
  p.M = P; p.N = a->OC; p.K = 9 * a->C;
  p.alpha = 1.0f; p.act = a->act; p.batch = 1;
  p.err = st::error_word();
  OutMaps tmC;
  if (!plan_epilogue(p, tmC)) return ST_ERR_CUDA;
  if (pair) return launch_pair<false, false>(tmA, tmB, tmC, p, s);
  if (tile.parts > 1) return launch_parts<false, false>(BN, tile.parts, tmA, tmB, tmC, p, s);
  if (BN == 64) return launch_gemm<64, 8, false, false>(tmA, tmB, tmC, p, s);
  if (BN == 128)
    return staged_epilogue(p) ? launch_gemm<128, 5, false, false>(tmA, tmB, tmC, p, s) : launch_gemm<128, 6, false, false>(tmA, tmB, tmC, p, s);
  return launch_gemm<256, 4, false, false>(tmA, tmB, tmC, p, s);
}

struct StConvWgradArgs {
  const void* dy;   // bf16 [N*H*W, OC]
  const void* x;    // bf16 NHWC [N, H, W, C]
  float* dw;        // fp32 [OC, 9*C]; the kernel ADDS into it
  int N, H, W, C, OC;
  int splits;       // K splits over pixels (0 = choose)
};

ST_API int st_conv3x3_wgrad(const StConvWgradArgs* a, void* stream_v) {
  if (!a || !a->dy || !a->x || !a->dw) return st::fail(ST_ERR_INVALID, "conv3x3_wgrad: null pointer");
  if (a->C % 64 != 0 || a->OC % 8 != 0) return st::fail(ST_ERR_INVALID, "conv3x3_wgrad: C % 64 and OC % 8 must be 0");
  int Hb, Nb;
  if (!block_geometry(a->N, a->H, a->W, BK, &Hb, &Nb))
    return st::fail(ST_ERR_INVALID, "conv3x3_wgrad: image width must divide 64 and the batch must fill whole pixel blocks");
  const int P = a->N * a->H * a->W;
  const int kblocks_total = P / BK;
  // One product over N = 9 C columns: a wide tile of them reads dY once where a tile per tap read it nine times (C = 64 in
  // tiles of 192: 96 KB of loads per 64 pixels instead of 144).  The form (tile width, or pairs over 256 output channels) and
  // the splits by the cost of a K block as in choose_tile, plus about 6 us of atomics for each tile of an SM.  A caller's own
  // split count fixes the summation order with one CTA per tile and split; narrow tiles then keep more SMs at work.
  // Measured, with a tile per tap and in this form: 256 x 64 x 64 pixels, C = OC = 64: 240 and 118 us (655 TFLOP/s; half of the
  // 128 rows of a tile are padding); 256 x 32 x 32, 128 to 128: 134 and 66; 256 x 16 x 16, 256 to 256: 86 and 55 (1399 TFLOP/s).
  struct Form { int bn, rows, sms; double c; };
  static const Form forms[4] = {{192, BM, 1, 0.33}, {256, BM, 1, 0.40}, {256, 2 * BM, 2, 0.33}, {64, BM, 1, 0.228}};
  const long long N9 = 9ll * a->C;
  int splits = a->splits, form = 0;
  if (splits > 0) {
    if (kblocks_total % splits != 0) return st::fail(ST_ERR_INVALID, "conv3x3_wgrad: splits must divide the pixel blocks");
    form = a->C <= 192 ? 3 : 1;
  } else {
    double best = 1e30;
    const long long most = kblocks_total / 8 > 0 ? kblocks_total / 8 : 1;      // at least eight K blocks per split
    for (int f = 0; f < 4; ++f) {
      if (forms[f].rows > BM && a->OC <= BM) continue;
      const long long tiles = (a->OC + forms[f].rows - 1) / forms[f].rows * ((N9 + forms[f].bn - 1) / forms[f].bn);
      const int at_once = st::sm_count() / forms[f].sms;
      for (int r = 1; r <= 3; ++r) {
        long long n = (long long)r * at_once / tiles;
        n = n < 1 ? 1 : (n > most ? most : n);
        const double rounds = (double)((tiles * n + at_once - 1) / at_once);
        const double t = rounds * ((double)((kblocks_total + n - 1) / n) * forms[f].c + 6.0);
        if (t < best) { best = t; splits = (int)n; form = f; }
      }
    }
  }
  CUtensorMap tmA, tmB;
  {
    uint64_t dims[3] = {(uint64_t)a->OC, (uint64_t)P, 1};
    uint64_t strides[2] = {(uint64_t)a->OC * 2, (uint64_t)a->OC * 2 * P};
    uint32_t box[3] = {64, BK, 1};
    if (!encode_tmap(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a->dy, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
      return ST_ERR_CUDA;
  }
  if (!nhwc_map(&tmB, a->x, a->N, a->H, a->W, a->C, a->W, Hb, Nb)) return ST_ERR_CUDA;
  GemmParams p{};
  p.conv.mode = 2;
  p.conv.H = a->H; p.conv.W = a->W; p.conv.Hb = Hb; p.conv.Nb = Nb;
  p.conv.c_chunks = a->C / 64; p.conv.blocks = kblocks_total;
  p.C = a->dw; p.ldc = N9;
  p.M = a->OC; p.N = (int)N9; p.K = P;
  p.alpha = 1.0f; p.batch = splits; p.batch_stride_c = 0;
  p.out_fp32 = 1; p.accumulate = 2;
  p.err = st::error_word();
  OutMaps tmC;
  if (!plan_epilogue(p, tmC)) return ST_ERR_CUDA;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  if (form == 0) return launch_gemm<192, 4, true, true>(tmA, tmB, tmC, p, s);
  if (form == 2) return launch_pair<true, true>(tmA, tmB, tmC, p, s);
  if (form == 3) return launch_gemm<64, 8, true, true>(tmA, tmB, tmC, p, s);
  return launch_gemm<256, 4, true, true>(tmA, tmB, tmC, p, s);
}

ST_API int st_im2col3x3_small(const void* x, void* col, int N, int H, int W, int C, int Kpad, void* stream_v) {
  if (9 * C > Kpad || (Kpad & 7)) return st::fail(ST_ERR_INVALID, "im2col: Kpad must be a multiple of 8 and >= 9*C");
  const bool aligned = (reinterpret_cast<uintptr_t>(col) & 15) == 0;
  const long long total = (long long)N * H * W * (Kpad / 8);
  const int grid = grid_for(total, 256);
  const bool narrow = total + (long long)grid * 256 < (1ll << 31);     // the last step's index must not wrap either
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  if (aligned && C >= 1 && C <= 4 && Kpad == (9 * C + 31) / 32 * 32) {
    const long long pixels = (long long)N * H * W;
    auto kern = C == 1 ? im2col3x3_image_kernel<1, false> : C == 2 ? im2col3x3_image_kernel<2, false>
                : C == 3 ? im2col3x3_image_kernel<3, false> : im2col3x3_image_kernel<4, false>;
    st::chained(kern, grid_for(pixels, 256), 256, 0, s)(static_cast<const __nv_bfloat16*>(x), static_cast<uint4*>(col), pixels, H, W, nullptr, nullptr, 0);
  } else if (aligned && (C & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    auto kern = narrow ? im2col3x3_c8_kernel<unsigned> : im2col3x3_c8_kernel<long long>;
    st::chained(kern, grid, 256, 0, s)(static_cast<const uint4*>(x), static_cast<uint4*>(col), N, H, W, C / 8, Kpad / 8);
  } else {
    auto kern = narrow ? im2col3x3_small_kernel<unsigned> : im2col3x3_small_kernel<long long>;
    st::chained(kern, grid, 256, 0, s)(static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(col), N, H, W, C, Kpad, aligned);
  }
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// Columns of 3x3 patches straight from images [N][C][H][W] of 1 to 4 channels, rows of K = 9 C rounded up to 32, and the weights
// [OC][9 C] padded to K (padded: [OC][K]).
ST_API int st_im2col3x3_planes(const void* x, void* col, const void* weights, void* padded, int N, int H, int W, int C, int OC, void* stream_v) {
  if (!x || !col || !weights || !padded || N <= 0 || H <= 0 || W <= 0 || OC <= 0) return st::fail(ST_ERR_INVALID, "im2col planes: bad arguments");
  if (C < 1 || C > 4 || (reinterpret_cast<uintptr_t>(col) & 15) != 0)
    return st::fail(ST_ERR_INVALID, "im2col planes: 1 to 4 channels and a 16-byte aligned matrix");
  const long long pixels = (long long)N * H * W;
  auto kern = C == 1 ? im2col3x3_image_kernel<1, true> : C == 2 ? im2col3x3_image_kernel<2, true>
              : C == 3 ? im2col3x3_image_kernel<3, true> : im2col3x3_image_kernel<4, true>;
  ST_CUDA_CHECK(st::chained(kern, grid_for(pixels, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(x), static_cast<uint4*>(col), pixels, H, W, static_cast<const __nv_bfloat16*>(weights),
      static_cast<__nv_bfloat16*>(padded), OC));
  return ST_OK;
}

// idx may be null: no backward pass follows.
ST_API int st_maxpool2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, void* stream_v) {
  if ((H & 1) || (W & 1) || (C & 1)) return st::fail(ST_ERR_INVALID, "maxpool2: H, W and C must be even");
  if ((C & 7) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(idx) & 7) == 0) {
    st::chained(maxpool2_fwd8_kernel, grid_for((long long)N * (H / 2) * (W / 2) * (C / 8), 256), 256, 0,
                           reinterpret_cast<cudaStream_t>(stream_v))(
        static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), static_cast<unsigned char*>(idx), N, H, W, C);
    ST_CUDA_CHECK(cudaGetLastError());
    return ST_OK;
  }
  st::chained(maxpool2_fwd_kernel, grid_for((long long)N * (H / 2) * (W / 2) * (C / 2), 256), 256, 0,
                        reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), static_cast<unsigned char*>(idx), N, H, W, C);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
// Weights [OC][9][IC] (tap-major) to those of the data gradient, [IC][9][OC] with the taps reversed.
ST_API int st_conv3x3_dgrad_weights(const void* w, void* wt, int OC, int IC, void* stream_v) {
  if (!w || !wt || OC <= 0 || IC <= 0) return st::fail(ST_ERR_INVALID, "conv3x3_dgrad_weights: bad arguments");
  st::chained(dgrad_weights_kernel, dim3((IC + 31) / 32, (OC + 31) / 32, 9), dim3(32, 8), 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(wt), OC, IC);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// Backward of ReLU followed by the pool: dx, and the channel sums of dx added to dbias (fp32 [C], may be null).  Needs
// C / 8 to divide 256 and 16-byte aligned tensors.
ST_API int st_maxpool2_relu_bwd(const void* dy, const void* idx, const void* pooled, void* dx, float* dbias, int N, int H,
                                int W, int C, void* stream_v) {
  if (!dy || !idx || !pooled || !dx || N <= 0) return st::fail(ST_ERR_INVALID, "maxpool2_relu_bwd: bad arguments");
  if ((H & 1) || (W & 1) || (C & 7) || C <= 0 || 256 % (C / 8) != 0)
    return st::fail(ST_ERR_INVALID, "maxpool2_relu_bwd: H and W must be even and C / 8 must divide 256");
  if (((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(pooled) | reinterpret_cast<uintptr_t>(dx)) & 15) ||
      (reinterpret_cast<uintptr_t>(idx) & 7))
    return st::fail(ST_ERR_INVALID, "maxpool2_relu_bwd: tensors must be 16-byte aligned");
  st::chained(maxpool2_bwd8_kernel, grid_for((long long)N * (H / 2) * (W / 2) * (C / 8), 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const uint4*>(dy), static_cast<const uint2*>(idx), static_cast<const uint4*>(pooled),
      static_cast<uint4*>(dx), dbias, N, H, W, C / 8);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_maxpool2_bwd(const void* dy, const void* idx, void* dx, int N, int H, int W, int C, void* stream_v) {
  if ((H & 1) == 0 && (W & 1) == 0 && (C & 7) == 0 &&
      ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 15) == 0 && (reinterpret_cast<uintptr_t>(idx) & 7) == 0) {
    st::chained(maxpool2_bwd8_kernel, grid_for((long long)N * (H / 2) * (W / 2) * (C / 8), 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_v))(
        static_cast<const uint4*>(dy), static_cast<const uint2*>(idx), nullptr, static_cast<uint4*>(dx), nullptr, N, H, W, C / 8);
    ST_CUDA_CHECK(cudaGetLastError());
    return ST_OK;
  }
  st::chained(maxpool2_bwd_kernel, grid_for((long long)N * (H / 2) * (W / 2) * C, 256), 256, 0,
                        reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(dy), static_cast<const unsigned char*>(idx), static_cast<__nv_bfloat16*>(dx),
      N, H, W, C);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
ST_API int st_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream_v) {
  st::chained(avgpool_fwd_kernel, N, 256, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), N, HW, C);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
ST_API int st_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream_v) {
  st::chained(avgpool_bwd_kernel, grid_for((long long)N * HW * C, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_v))(
      static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dx), N, HW, C);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
