// Spectral kernels: batched 1-D FFT in shared memory (any stride, real or complex input, optional window,
// power-of-two lengths by Stockham radix-8 passes with the butterflies in registers and other lengths by a direct
// DFT against a shared twiddle table), spectral multipliers for the fractional operators, and the temporal volume
// renderer.
//
// All of them are bandwidth-bound elementwise / small-transform work: one pass over the data, fp32 math,
// no tensor cores.  A transform lives entirely in one CTA's shared memory (two ping-pong buffers), so a batch
// of transforms costs one read and one write of the data whatever the length.
#include <cuda_runtime.h>
#include <cstdint>
#include <math_constants.h>

#include "../common/host.h"
#include "../common/ptx.cuh"

namespace {

constexpr int kMaxFftLen = 8192;        // 2 x 8192 complex fp32 = 128 KB of shared memory
constexpr int kMaxDftLen = 4096;        // direct DFT: input + twiddle table
constexpr float kTau = 6.283185307179586f;
constexpr int kMaxRenderTableFrames = 4096;   // 32 KB of (sin, cos) per CTA
constexpr int kRenderRegChannels = 8;         // harmonic amplitudes kept in registers across the frame loop

struct FftLayout {
  // element (b0, b1, i) of the input lives at in[b0 * in_b0 + b1 * in_b1 + i * in_i] (in floats; complex input
  // has its imaginary part at +1); the output, always interleaved complex, at out[b0 * out_b0 + b1 * out_b1 + i * out_i]
  long long in_b0, in_b1, in_i;
  long long out_b0, out_b1, out_i;
  int batch1;                           // batches are numbered b = b0 * batch1 + b1
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ---- in-register DFTs of 2, 4 and 8 points (forward sign, natural output order) -------------------------------
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul_neg_i(float2 a) { return make_float2(a.y, -a.x); }          // a * (-i)

__device__ __forceinline__ void dft4(float2& x0, float2& x1, float2& x2, float2& x3) {
  const float2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = mul_neg_i(csub(x1, x3));
  x0 = cadd(a, c); x1 = cadd(b, d); x2 = csub(a, c); x3 = csub(b, d);
}

template <int R>
__device__ __forceinline__ void dft_regs(float2 (&v)[8]) {
  if constexpr (R == 2) {
    const float2 a = v[0];
    v[0] = cadd(a, v[1]); v[1] = csub(a, v[1]);
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3]);
  } else {
    float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4(e0, e1, e2, e3);
    dft4(o0, o1, o2, o3);
    constexpr float h = 0.70710678118654752f;
    o1 = make_float2(h * (o1.x + o1.y), h * (o1.y - o1.x));            // * exp(-i pi / 4)
    o2 = mul_neg_i(o2);                                                 // * exp(-i pi / 2)
    o3 = make_float2(h * (o3.y - o3.x), -h * (o3.x + o3.y));           // * exp(-3 i pi / 4)
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  }
}

// Shared-memory slot of point i: 8 slots of padding per 64 points (the second pass writes groups of 8 consecutive
// points that are 64 points apart) and the low three bits XOR-ed with bits 4..6 of i (the first pass writes 8
// consecutive points per thread, so 16 threads of a half-warp would land on two bank pairs without it).  With both,
// every 64-bit shared-memory access of every pass touches 16 distinct bank pairs per half-warp.
__device__ __forceinline__ int slot(int i) { return (i + ((i >> 6) << 3)) ^ ((i >> 4) & 7); }

// One Stockham pass of radix R over a transform of n points whose sub-transforms already have length ns:
//   v[r] = src[j + r n/R] * w^r (w = exp(-2 pi i (j mod ns) / (ns R))), DFT_R(v), dst[(j / ns) ns R + (j mod ns) + r ns] = v[r]
// FIRST reads the (strided, possibly real, windowed) input from global memory, LAST writes the output there, so a
// transform of three passes crosses shared memory twice.  The inverse transform is conj(FFT(conj(x))) / n.
// NSC is ns when it is 1, 8 or 64 and 0 for a run-time ns that is a multiple of 512: each case has a closed form of
// slot() for its eight outputs (one XOR and one add per output instead of the shifts of the general formula).
// VEC: input and output are interleaved complex with unit stride, moved as float2.
template <int R, bool FIRST, bool LAST, int NSC, bool VEC>
__device__ __forceinline__ void stockham_pass(const float2* __restrict__ src, float2* __restrict__ dst, const float* __restrict__ gin,
                                              float* __restrict__ gout, const float* __restrict__ window, long long in_i,
                                              long long out_i, int n, int ns_rt, int complex_in, int inverse, float scale) {
  const int ns = NSC ? NSC : ns_rt;
  const int m = n / R;
  const bool stride_reads = (m & 127) == 0;          // slot(j + r m) = slot(j) + r (m + m / 8)
  const int m_slots = m + (m >> 3);
  const float angle_scale = -2.0f / (float)(ns * R);  // a power of two: exact
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    float2 v[8];
    if constexpr (FIRST) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = j + r * m;
        const float w = window ? window[i] : 1.0f;
        float re, im;
        if constexpr (VEC) {
          const float2 x = reinterpret_cast<const float2*>(gin)[i];
          re = x.x; im = x.y;
        } else {
          re = gin[i * in_i];
          im = complex_in ? gin[i * in_i + 1] : 0.0f;
        }
        v[r] = make_float2(re * w, inverse ? -im * w : im * w);
      }
    } else {
      const int s0 = slot(j);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = src[stride_reads ? s0 + r * m_slots : slot(j + r * m)];
    }
    const int k = j & (ns - 1);
    if constexpr (!FIRST) {
      float sn, cs;
      sincospif((float)k * angle_scale, &sn, &cs);
      const float2 w1 = make_float2(cs, sn);
      v[1] = cmul(v[1], w1);
      if constexpr (R >= 4) {
        const float2 w2 = cmul(w1, w1), w3 = cmul(w2, w1);
        v[2] = cmul(v[2], w2); v[3] = cmul(v[3], w3);
        if constexpr (R == 8) {
          const float2 w4 = cmul(w2, w2);
          v[4] = cmul(v[4], w4); v[5] = cmul(v[5], cmul(w4, w1)); v[6] = cmul(v[6], cmul(w4, w2)); v[7] = cmul(v[7], cmul(w4, w3));
        }
      }
    }
    dft_regs<R>(v);
    if constexpr (LAST) {
      const int j0 = (j - k) * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int o = j0 + r * ns;
        const float2 y = make_float2(v[r].x * scale, (inverse ? -v[r].y : v[r].y) * scale);
        if constexpr (VEC) {
          reinterpret_cast<float2*>(gout)[o] = y;
        } else {
          gout[o * out_i] = y.x;
          gout[o * out_i + 1] = y.y;
        }
      }
    } else {
      static_assert(LAST || R == 8, "only radix-8 passes write shared memory");
      if constexpr (NSC == 1) {
        const int base = j * 8 + ((j >> 3) << 3), x = (j >> 1) & 7;
#pragma unroll
        for (int r = 0; r < 8; ++r) dst[base + (r ^ x)] = v[r];
      } else if constexpr (NSC == 8) {
        const int g = j >> 3, base = g * 72, x = k ^ ((g & 1) << 2);
#pragma unroll
        for (int r = 0; r < 8; ++r) dst[base + r * 8 + (x ^ (r >> 1))] = v[r];
      } else if constexpr (NSC == 64) {
        const int base = (j >> 6) * 576, x = k ^ (k >> 4);
#pragma unroll
        for (int r = 0; r < 8; ++r) dst[base + r * 72 + (x ^ ((r & 1) << 2))] = v[r];
      } else {
        const int ns_slots = ns + (ns >> 3);
        const int base = ((j - k) / ns) * 8 * ns_slots + slot(k);
#pragma unroll
        for (int r = 0; r < 8; ++r) dst[base + r * ns_slots] = v[r];
      }
    }
  }
}

// One transform per CTA: n = 8^a * tail with tail in {1, 2, 4}; `a` radix-8 passes, then the tail pass.
template <bool VEC>
__global__ void __launch_bounds__(512, 2)
fft_pow2_kernel(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ window,
                FftLayout L, int n, int log2n, int complex_in, int inverse) {
  extern __shared__ float2 smem[];
  const int padded = n + (((n - 1) >> 6) << 3);
  float2* a = smem;
  float2* b = smem + padded;
  const int batch = blockIdx.x;
  const int b0 = batch / L.batch1, b1 = batch % L.batch1;
  const float* gin = in + b0 * L.in_b0 + b1 * L.in_b1;
  float* gout = out + b0 * L.out_b0 + b1 * L.out_b1;
  const float scale = inverse ? 1.0f / (float)n : 1.0f;
  const int eights = log2n / 3, tail = 1 << (log2n - 3 * eights);
#define ST_FFT_PASS(R, FIRST, LAST, NSC, SRC, DST, NS) \
  stockham_pass<R, FIRST, LAST, NSC, VEC>(SRC, DST, gin, gout, window, L.in_i, L.out_i, n, NS, complex_in, inverse, scale)
  if (n == 1) {
    if (threadIdx.x == 0) {
      const float w = window ? window[0] : 1.0f;
      gout[0] = gin[0] * w;
      gout[1] = complex_in ? gin[1] * w : 0.0f;
    }
    return;
  }
  if (eights == 0) {               // n = 2 or 4: a single pass from global to global
    if (tail == 2) ST_FFT_PASS(2, true, true, 1, nullptr, nullptr, 1);
    else ST_FFT_PASS(4, true, true, 1, nullptr, nullptr, 1);
    return;
  }
  if (eights == 1 && tail == 1) {  // n = 8
    ST_FFT_PASS(8, true, true, 1, nullptr, nullptr, 1);
    return;
  }
  ST_FFT_PASS(8, true, false, 1, nullptr, a, 1);
  __syncthreads();
  float2* src = a;
  float2* dst = b;
  int ns = 8;
  for (int p = 1; p < eights; ++p) {
    if (p == eights - 1 && tail == 1) {
      if (p == 1) ST_FFT_PASS(8, false, true, 8, src, nullptr, 8);
      else if (p == 2) ST_FFT_PASS(8, false, true, 64, src, nullptr, 64);
      else ST_FFT_PASS(8, false, true, 0, src, nullptr, ns);
      return;
    }
    if (p == 1) ST_FFT_PASS(8, false, false, 8, src, dst, 8);
    else if (p == 2) ST_FFT_PASS(8, false, false, 64, src, dst, 64);
    else ST_FFT_PASS(8, false, false, 0, src, dst, ns);
    __syncthreads();
    float2* t = src; src = dst; dst = t;
    ns *= 8;
  }
  if (tail == 2) ST_FFT_PASS(2, false, true, 0, src, nullptr, ns);
  else ST_FFT_PASS(4, false, true, 0, src, nullptr, ns);
#undef ST_FFT_PASS
}

// ---- long batches of complex rows: radix-16 passes, twiddles in shared memory, next rows prefetched ----------------------
// A persistent CTA of 256 threads works on 4096 points at a time: one row of 4096 or 4096 / n shorter ones.  Every thread
// holds 16 points, so a transform is log16(n) passes and a tail of 2, 4 or 8, with one exchange buffer between them; while
// the passes of one group run, bulk asynchronous copies bring the next group into a staging buffer.  The radix-8 kernel
// above with such copies was bound by instruction issue (883 per 8 points at n = 4096: four passes, a sincospi and a chain
// of products for each butterfly's twiddles): 134 us for 8192 rows of 4096, where this one takes 103 and the bytes 82.
constexpr int F16_POINTS = 4096, F16_THREADS = F16_POINTS / 16;

__device__ __forceinline__ float2 add_c(float2 a, float2 b) { return st::add2(a, b); }                       // one packed add
__device__ __forceinline__ float2 sub_c(float2 a, float2 b) { return st::fma2(b, make_float2(-1.0f, -1.0f), a); }

__device__ __forceinline__ void dft4_c(float2& x0, float2& x1, float2& x2, float2& x3) {
  const float2 a = add_c(x0, x2), b = sub_c(x0, x2), c = add_c(x1, x3), d = mul_neg_i(sub_c(x1, x3));
  x0 = add_c(a, c); x1 = add_c(b, d); x2 = sub_c(a, c); x3 = sub_c(b, d);
}

// 16-point DFT as 4 x 4: input b + 4 a, output c + 4 d in v[4 c + d]
__device__ __forceinline__ void dft16(float2 (&v)[16]) {
#pragma unroll
  for (int b = 0; b < 4; ++b) dft4_c(v[b], v[b + 4], v[b + 8], v[b + 12]);
  constexpr float h = 0.70710678118654752f, c1 = 0.92387953251128674f, s1 = 0.38268343236508977f;
  auto rot45 = [](float2 x) { return make_float2(h * (x.x + x.y), h * (x.y - x.x)); };                 // * exp(-i pi / 4)
  v[5] = cmul(v[5], make_float2(c1, -s1));
  v[6] = rot45(v[6]);
  v[7] = cmul(v[7], make_float2(s1, -c1));
  v[9] = rot45(v[9]);
  v[10] = mul_neg_i(v[10]);
  v[11] = mul_neg_i(rot45(v[11]));
  v[13] = cmul(v[13], make_float2(s1, -c1));
  v[14] = mul_neg_i(rot45(v[14]));
  v[15] = cmul(v[15], make_float2(-c1, s1));
#pragma unroll
  for (int c = 0; c < 4; ++c) dft4_c(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}
__device__ __forceinline__ constexpr int dft16_at(int k) { return 4 * (k & 3) + (k >> 2); }

template <int LOGN>
struct Fft16 {
  static constexpr int N = 1 << LOGN, TPR = N / 16, ROWS = F16_POINTS / N;
  static constexpr int PASSES = LOGN / 4, TAIL = 1 << (LOGN % 4);
  // twiddle tables, entry (r - 1) ns + k = exp(-2 pi i r k / (radix ns)): pass 1 (ns 16), pass 2 (ns 256), tail (ns N / TAIL)
  static constexpr int TW1 = PASSES > 1 ? 15 * 16 : 0, TW2 = PASSES > 2 ? 15 * 256 : 0;
  static constexpr int TWT = TAIL > 1 ? (TAIL - 1) * (N / TAIL) : 0;
  // one slot of padding per 16: the first pass writes 16 neighbours per thread, every other access is contiguous
  static constexpr int BUF = F16_POINTS + F16_POINTS / 16;
  static constexpr int SMEM = (BUF + F16_POINTS + TW1 + TW2 + TWT) * 8 + 32;
};

template <int LOGN>
__global__ void __launch_bounds__(F16_THREADS, 3)
fft16_stream_kernel(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ window, FftLayout L,
                    int inverse, int batches, unsigned* err) {
  using F = Fft16<LOGN>;
  constexpr int N = F::N, TPR = F::TPR;
  extern __shared__ __align__(16) float2 smem[];
  float2* buf = smem;
  float2* stage = buf + F::BUF;                                       // 16-byte aligned: BUF is even
  float2* tw1 = stage + F16_POINTS;
  float2* tw2 = tw1 + F::TW1;
  float2* twt = tw2 + F::TW2;
  uint64_t* bar = reinterpret_cast<uint64_t*>(twt + F::TWT + ((F::TW1 + F::TW2 + F::TWT) & 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bar + 1);
  const int t = threadIdx.x, g = t / TPR, j = t % TPR;
  const int groups = (batches + F::ROWS - 1) / F::ROWS;
  const bool packed = F::ROWS == 1 || (L.batch1 == 1 && L.in_b0 == 2 * N);      // a group's rows are one piece of memory
  auto table = [&](float2* w, int entries, int ns, int radix) {
    for (int e = t; e < entries; e += F16_THREADS) {
      float sn, cs;
      sincospif(-2.0f * (float)((e / ns + 1) * (e % ns)) / (float)(radix * ns), &sn, &cs);      // exact quotient
      w[e] = make_float2(cs, sn);
    }
  };
  if (F::TW1) table(tw1, F::TW1, 16, 16);
  if (F::TW2) table(tw2, F::TW2, 256, 16);
  if (F::TWT) table(twt, F::TWT, N / F::TAIL, F::TAIL);
  if (t == 0) {
    st::mbar_init(st::smem_u32(bar), 1);
    *abort_flag = 0;
    st::fence_barrier_init();
  }
  __syncthreads();
  auto fetch = [&](int group) {      // by one thread
    const int first = group * F::ROWS, rows = min(F::ROWS, batches - first);
    st::mbar_arrive_expect_tx(st::smem_u32(bar), rows * N * 8);
    for (int r = 0; r < (packed ? 1 : rows); ++r) {
      const int b = first + r;
      st::bulk_load_g2s(st::smem_u32(stage + r * N), in + (b / L.batch1) * L.in_b0 + (b % L.batch1) * L.in_b1,
                        (packed ? rows : 1) * N * 8, st::smem_u32(bar));
    }
  };
  if (t == 0 && static_cast<int>(blockIdx.x) < groups) fetch(blockIdx.x);
  const float scale = inverse ? 1.0f / (float)N : 1.0f;
  // slots of this thread's 16 points g N + j + q TPR (the second term of a slot does not depend on j where TPR < 16)
  float2* const mine = buf + g * (N + N / 16) + j + (TPR >= 16 ? j / 16 : 0);
  auto at = [](int q) { return q * TPR + q * TPR / 16; };
  uint32_t phase = 0;
  for (int group = blockIdx.x; group < groups; group += gridDim.x) {
    const int batch = group * F::ROWS + g;
    const bool live = batch < batches;
    // bounded wait; the CTA decides together, so nobody is left at a barrier by a thread that gave up
    if (!__syncthreads_and(st::mbar_wait(st::smem_u32(bar), phase, abort_flag) ? 1 : 0)) break;
    phase ^= 1u;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      float2 x = stage[g * N + j + q * TPR];       // rows past the batch hold an earlier group's points: not stored
      if (window) {
        const float w = window[j + q * TPR];
        x.x *= w; x.y *= w;
      }
      v[q] = make_float2(x.x, inverse ? -x.y : x.y);
    }
    dft16(v);
    __syncthreads();                               // the staging buffer and the exchange buffer have been read by everyone
    if (t == 0 && group + static_cast<int>(gridDim.x) < groups) fetch(group + gridDim.x);
    {
      float2* o = buf + g * (N + N / 16) + 17 * j;
#pragma unroll
      for (int k = 0; k < 16; ++k) o[k] = v[dft16_at(k)];
    }
    __syncthreads();
    if constexpr (F::PASSES == 3 || (F::PASSES == 2 && F::TAIL > 1)) {
      const int k = j & 15;
      v[0] = mine[0];
#pragma unroll
      for (int q = 1; q < 16; ++q) v[q] = cmul(mine[at(q)], tw1[(q - 1) * 16 + k]);
      dft16(v);
      __syncthreads();
      float2* o = buf + g * (N + N / 16) + (j / 16) * 272 + k;
#pragma unroll
      for (int r = 0; r < 16; ++r) o[17 * r] = v[dft16_at(r)];
      __syncthreads();
    }
    float2* gout = reinterpret_cast<float2*>(out + (live ? (batch / L.batch1) * L.out_b0 + (batch % L.batch1) * L.out_b1 : 0)) + j;
    auto put = [&](int q, float2 y) {
      if (live) gout[q * TPR] = make_float2(y.x * scale, (inverse ? -y.y : y.y) * scale);
    };
    if constexpr (F::TAIL == 1) {
      const float2* w = F::PASSES == 3 ? tw2 : tw1;
      v[0] = mine[0];
#pragma unroll
      for (int q = 1; q < 16; ++q) v[q] = cmul(mine[at(q)], w[(q - 1) * TPR + j]);
      dft16(v);
#pragma unroll
      for (int q = 0; q < 16; ++q) put(q, v[dft16_at(q)]);
    } else {
      constexpr int R = F::TAIL, B = 16 / R, NS = N / R;      // B butterflies of radix R: points b + r B of the thread's 16
#pragma unroll
      for (int b = 0; b < B; ++b) {
        float2 x[8];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          x[r] = mine[at(b + r * B)];
          if (r > 0) x[r] = cmul(x[r], twt[(r - 1) * NS + j + b * TPR]);
        }
        dft_regs<R>(x);
#pragma unroll
        for (int r = 0; r < R; ++r) put(b + r * B, x[r]);
      }
    }
  }
  if (*abort_flag && t == 0) st::report_error(err, st::ERR_MBAR_TIMEOUT, 0xF7F1u);
}

template <int LOGN>
int launch_fft16(const float* in, float* out, const float* window, const FftLayout& L, int inverse, int batches, cudaStream_t stream) {
  using F = Fft16<LOGN>;
  static int resident[st::kMaxDevices] = {};      // CTAs per SM: 2 or 3, by the size of the twiddle tables
  const int dev = st::current_device();
  if (!resident[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(fft16_stream_kernel<LOGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, F::SMEM));
    int n = 0;
    ST_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fft16_stream_kernel<LOGN>, F16_THREADS, F::SMEM));
    resident[dev] = n > 0 ? n : 1;
  }
  const int groups = (batches + F::ROWS - 1) / F::ROWS, most = resident[dev] * st::sm_count();
  fft16_stream_kernel<LOGN><<<groups < most ? groups : most, F16_THREADS, F::SMEM, stream>>>(in, out, window, L, inverse, batches,
                                                                                           st::error_word());
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// Direct DFT for lengths that are not powers of two: out[k] = sum_i x[i] * w^(k*i mod n), twiddles from a table.
__global__ void dft_kernel(const float* __restrict__ in, float* __restrict__ out, const float* __restrict__ window,
                           FftLayout L, int n, int complex_in, int inverse) {
  extern __shared__ float2 smem[];
  float2* x = smem;
  float2* tw = smem + n;
  const int batch = blockIdx.x;
  const int b0 = batch / L.batch1, b1 = batch % L.batch1;
  const float* src_ptr = in + b0 * L.in_b0 + b1 * L.in_b1;
  const float sign = inverse ? 1.0f : -1.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float w = window ? window[i] : 1.0f;
    x[i] = make_float2(src_ptr[i * L.in_i] * w, complex_in ? src_ptr[i * L.in_i + 1] * w : 0.0f);
    float sn, cs;
    sincospif(sign * 2.0f * (float)i / (float)n, &sn, &cs);
    tw[i] = make_float2(cs, sn);
  }
  __syncthreads();
  const float scale = inverse ? 1.0f / (float)n : 1.0f;
  float* dst_ptr = out + b0 * L.out_b0 + b1 * L.out_b1;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    float2 acc = make_float2(0.0f, 0.0f);
    int idx = 0;                                    // k * i mod n, advanced incrementally
    for (int i = 0; i < n; ++i) {
      const float2 p = cmul(x[i], tw[idx]);
      acc.x += p.x; acc.y += p.y;
      idx += k;
      if (idx >= n) idx -= n;
    }
    dst_ptr[k * L.out_i] = acc.x * scale;
    dst_ptr[k * L.out_i + 1] = acc.y * scale;
  }
}

// mode 0: fractional-Laplacian envelope, scale = min(col, cols - 1 - col)^power (real multiplier)
// mode 1: fractional derivative, multiplier = (i * omega_col)^alpha with omega = 2 pi * fftfreq(cols, h);
//         the zero frequency is set to 0 for alpha > 0
// One thread owns a column: the multiplier (a pow and, for the derivative, a sincos) is computed once and applied to
// that column of `rows_per_block` consecutive rows, so the kernel is a streaming multiply.
__global__ void specmul_kernel(const float* __restrict__ x, float* __restrict__ y, long long rows, int cols, float power,
                               float inv_h, int mode, int rows_per_block) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= cols) return;
  float2 mult;
  bool passthrough = false, infinite = false;
  if (mode == 0) {
    const int mirror = cols - 1 - col;
    mult = make_float2(powf(fmaxf((float)(col < mirror ? col : mirror), 0.0f), power), 0.0f);
  } else {
    const int k = col < (cols + 1) / 2 ? col : col - cols;      // fftfreq ordering
    const float omega = kTau * (float)k * inv_h / (float)cols;
    if (k == 0) {
      mult = make_float2(0.0f, 0.0f);
      passthrough = power == 0.0f;
      infinite = power < 0.0f;
    } else {
      // (i omega)^a = |omega|^a * exp(i * a * sign(omega) * pi / 2)
      const float mag = powf(fabsf(omega), power);
      float sn, cs;
      sincosf(power * (omega > 0.0f ? 1.0f : -1.0f) * 1.5707963267948966f, &sn, &cs);
      mult = make_float2(mag * cs, mag * sn);
    }
  }
  const long long r0 = (long long)blockIdx.y * rows_per_block;
  const long long r1 = r0 + rows_per_block < rows ? r0 + rows_per_block : rows;
  const float2* xp = reinterpret_cast<const float2*>(x);
  float2* yp = reinterpret_cast<float2*>(y);
#pragma unroll 4
  for (long long r = r0; r < r1; ++r) {
    const float2 v = xp[r * cols + col];
    yp[r * cols + col] = passthrough ? v : (infinite ? make_float2(CUDART_INF_F, CUDART_INF_F) : cmul(v, mult));
  }
}

// out[f, v] = (voxel[v] + sum_c harm[v, c] * sin((c + 1) * tau * t_f)) * exp(-decay[v] * t_f), t_f = f / rate.
// decay: non-finite -> 1, negative -> 0; decay <= eps gives 0.  sin((c+1) theta) advances by the Chebyshev
// recurrence s_{c+1} = 2 cos(theta) s_c - s_{c-1}, so a frame costs one sincos per voxel however many channels.
__global__ void temporal_render_kernel(const float* __restrict__ voxels, const float* __restrict__ harmonics,
                                       const float* __restrict__ decay, float* __restrict__ out, long long n_voxels,
                                       int channels, int frames, float dt) {
  // sin / cos of the base angle of every frame are the same for all voxels: one table per CTA
  extern __shared__ float2 frame_sc[];
  const bool table = channels > 0 && frames <= kMaxRenderTableFrames;
  if (table) {
    for (int f = threadIdx.x; f < frames; f += blockDim.x) {
      float sn, cs;
      sincosf(kTau * ((float)f * dt), &sn, &cs);
      frame_sc[f] = make_float2(sn, cs);
    }
    __syncthreads();
  }
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n_voxels;
       v += (long long)gridDim.x * blockDim.x) {
    const float base0 = voxels[v];
    float d = decay[v];
    d = isfinite(d) ? fmaxf(d, 0.0f) : 1.0f;
    const float* h = harmonics + v * channels;
    float amp[kRenderRegChannels];
    const bool in_regs = channels <= kRenderRegChannels;
    if (in_regs) {
#pragma unroll
      for (int c = 0; c < kRenderRegChannels; ++c) amp[c] = c < channels ? h[c] : 0.0f;
    }
    for (int f = 0; f < frames; ++f) {
      const float t = (float)f * dt;
      float base = base0;
      if (channels > 0) {
        float sn, cs;
        if (table) { sn = frame_sc[f].x; cs = frame_sc[f].y; } else { sincosf(kTau * t, &sn, &cs); }
        float s_prev = 0.0f, s_cur = sn;                 // sin(0 * theta), sin(1 * theta)
        const float two_c = 2.0f * cs;
        if (in_regs) {
#pragma unroll
          for (int c = 0; c < kRenderRegChannels; ++c) {
            if (fabsf(amp[c]) > 1.1920929e-07f) base += amp[c] * s_cur;
            const float s_next = two_c * s_cur - s_prev;
            s_prev = s_cur; s_cur = s_next;
          }
        } else {
          for (int c = 0; c < channels; ++c) {
            const float a = h[c];
            if (fabsf(a) > 1.1920929e-07f) base += a * s_cur;
            const float s_next = two_c * s_cur - s_prev;
            s_prev = s_cur; s_cur = s_next;
          }
        }
      }
      out[(long long)f * n_voxels + v] = d <= 1.1920929e-07f ? 0.0f : base * __expf(-d * t);
    }
  }
}

}  // namespace

struct StFftArgs {
  const float* in;
  float* out;
  const float* window;     // n coefficients or null
  long long in_b0, in_b1, in_i, out_b0, out_b1, out_i;
  int n, batch0, batch1, complex_in, inverse;
};

ST_API int st_fft_max_len() { return kMaxFftLen; }
ST_API int st_dft_max_len() { return kMaxDftLen; }

ST_API int st_fft_1d(const StFftArgs* a, void* stream_v) {
  if (!a || !a->in || !a->out) return st::fail(ST_ERR_INVALID, "fft_1d: null argument");
  if (a->n <= 0 || a->batch0 <= 0 || a->batch1 <= 0) return st::fail(ST_ERR_INVALID, "fft_1d: empty problem");
  if ((long long)a->batch0 * a->batch1 > 2147483647LL) return st::fail(ST_ERR_TOO_LARGE, "fft_1d: too many transforms");
  const bool pow2 = (a->n & (a->n - 1)) == 0;
  if (pow2 ? a->n > kMaxFftLen : a->n > kMaxDftLen)
    return st::fail(ST_ERR_TOO_LARGE, "fft_1d: length above the shared-memory capacity (8192 power-of-two, 4096 other)");
  FftLayout L{a->in_b0, a->in_b1, a->in_i, a->out_b0, a->out_b1, a->out_i, a->batch1};
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  const int grid = a->batch0 * a->batch1;
  const size_t padded = (size_t)a->n + (((size_t)a->n - 1) >> 6 << 3);          // 8 slots of padding per 64 points, as slot() in the kernel
  const size_t smem = pow2 ? 2 * padded * sizeof(float2) : 2 * (size_t)a->n * sizeof(float2);
  static bool configured[st::kMaxDevices][2] = {};
  const int dev = st::current_device();
  if (pow2) {
    if (smem > 48 * 1024 && !configured[dev][0]) {
      const int max_smem = 2 * (kMaxFftLen + kMaxFftLen / 8) * (int)sizeof(float2);
      ST_CUDA_CHECK(cudaFuncSetAttribute(fft_pow2_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
      ST_CUDA_CHECK(cudaFuncSetAttribute(fft_pow2_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
      configured[dev][0] = true;
    }
    int log2n = 0;
    while ((1 << log2n) < a->n) ++log2n;
    int threads = a->n / 8;                    // one radix-8 butterfly per thread and pass
    threads = threads < 32 ? 32 : (threads > 512 ? 512 : threads);
    // interleaved complex on both sides with unit stride and 8-byte aligned transforms: float2 loads and stores
    const bool vec = a->complex_in && a->in_i == 2 && a->out_i == 2 && a->n > 1 &&
                     ((a->in_b0 | a->in_b1 | a->out_b0 | a->out_b1) & 1) == 0 &&
                     ((reinterpret_cast<uintptr_t>(a->in) | reinterpret_cast<uintptr_t>(a->out)) & 7) == 0;
    // 16-byte aligned rows, and at least one group of 4096 points per SM (below that, a CTA per row spreads the work wider).  Long
    // rows fill the chip as well in CTAs of their own, two at once per SM: 296 of 4096 6.6 us and 6.9 streamed, 303 9.1 and 8.3;
    // 385 of 2048 5.1 and 5.6, 473 6.1 and 5.6.
    const long long least = a->n == 4096 ? 2ll * st::sm_count() + 1 : (a->n == 2048 ? 3ll * st::sm_count() : (long long)F16_POINTS * st::sm_count() / a->n);
    if (vec && log2n >= 6 && log2n <= 12 && grid >= least &&
        ((a->in_b0 | a->in_b1) & 3) == 0 && (reinterpret_cast<uintptr_t>(a->in) & 15) == 0) {
      switch (log2n) {
        case 6: return launch_fft16<6>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        case 7: return launch_fft16<7>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        case 8: return launch_fft16<8>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        case 9: return launch_fft16<9>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        case 10: return launch_fft16<10>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        case 11: return launch_fft16<11>(a->in, a->out, a->window, L, a->inverse, grid, stream);
        default: return launch_fft16<12>(a->in, a->out, a->window, L, a->inverse, grid, stream);
      }
    }
    if (vec) fft_pow2_kernel<true><<<grid, threads, smem, stream>>>(a->in, a->out, a->window, L, a->n, log2n, a->complex_in, a->inverse);
    else fft_pow2_kernel<false><<<grid, threads, smem, stream>>>(a->in, a->out, a->window, L, a->n, log2n, a->complex_in, a->inverse);
  } else {
    if (smem > 48 * 1024 && !configured[dev][1]) {
      ST_CUDA_CHECK(cudaFuncSetAttribute(dft_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kMaxDftLen * (int)sizeof(float2)));
      configured[dev][1] = true;
    }
    const int threads = a->n >= 512 ? 256 : 64;
    dft_kernel<<<grid, threads, smem, stream>>>(a->in, a->out, a->window, L, a->n, a->complex_in, a->inverse);
  }
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_specmul(const float* x_reim, float* y_reim, long long rows, int cols, float power, float h, int mode,
                      void* stream_v) {
  if (rows <= 0 || cols <= 0) return st::fail(ST_ERR_INVALID, "specmul: empty problem");
  if (mode != 0 && mode != 1) return st::fail(ST_ERR_INVALID, "specmul: mode is 0 (Laplace envelope) or 1 (derivative)");
  if (!isfinite(power)) return st::fail(ST_ERR_INVALID, "specmul: power must be finite");
  if (mode == 1 && !(h > 0.0f)) return st::fail(ST_ERR_INVALID, "specmul: sample spacing must be positive");
  const int threads = cols >= 128 ? 128 : 32;
  const int col_blocks = (cols + threads - 1) / threads;
  // enough row chunks to fill the machine a few times over, each long enough to amortise the multiplier
  long long chunks = ((long long)st::sm_count() * 16 + col_blocks - 1) / col_blocks;
  if (chunks > rows) chunks = rows;
  if (chunks > 65535) chunks = 65535;
  if (chunks < 1) chunks = 1;
  const long long rows_per_block = (rows + chunks - 1) / chunks;
  if (rows_per_block > 2147483647LL) return st::fail(ST_ERR_TOO_LARGE, "specmul: too many rows");
  chunks = (rows + rows_per_block - 1) / rows_per_block;
  specmul_kernel<<<dim3(col_blocks, (unsigned)chunks), threads, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(
      x_reim, y_reim, rows, cols, power, mode == 1 ? 1.0f / h : 0.0f, mode, (int)rows_per_block);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

ST_API int st_temporal_render(const float* voxels, const float* harmonics, const float* decay, float* out,
                              long long n_voxels, int channels, int frames, float sample_rate_hz, void* stream_v) {
  if (n_voxels <= 0) return st::fail(ST_ERR_INVALID, "temporal_render: empty volume");
  if (frames <= 0) return st::fail(ST_ERR_INVALID, "temporal_render: needs at least one frame");
  if (!(sample_rate_hz > 0.0f) || !isfinite(sample_rate_hz)) return st::fail(ST_ERR_INVALID, "temporal_render: sample rate must be positive and finite");
  if (channels < 0 || (channels > 0 && !harmonics)) return st::fail(ST_ERR_INVALID, "temporal_render: harmonic buffer missing");
  long long blocks = (n_voxels + 255) / 256;
  const long long cap = (long long)st::sm_count() * 8;
  if (blocks > cap) blocks = cap;
  const size_t table = (channels > 0 && frames <= kMaxRenderTableFrames) ? (size_t)frames * sizeof(float2) : 0;
  temporal_render_kernel<<<(int)blocks, 256, table, reinterpret_cast<cudaStream_t>(stream_v)>>>(
      voxels, harmonics, decay, out, n_voxels, channels, frames, 1.0f / sample_rate_hz);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
