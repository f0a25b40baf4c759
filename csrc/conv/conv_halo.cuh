// 3x3 convolution for up to 128 output channels, each input row block fetched three times instead of nine.
//
// A tile is 256 output pixels (R = 256 / W whole rows of one image) by all output channels, as two accumulators of 128 rows.
// For a channel chunk and a horizontal tap dw, the box of R + 2 input rows shifted by dw - 1 serves all three vertical taps: the
// tap dh reads the same shared memory from row dh on, which is a descriptor offset of dh * W * 128 bytes (W is a multiple of 8,
// so the offset keeps the 1024-byte period of the swizzle).  With 64 input channels and at most 64 output channels the nine
// weight tiles (72 KB) stay in shared memory for the life of the CTA.
//
// The general GEMM fetches a box per tap, and with few output channels those fetches bound it: 24 KB per K block of 128 x 64 at
// the 64 bytes per cycle that an SM takes from L2 is 384 cycles, the MMAs need 128.  Here 256 pixels of a 64-wide image with 64
// channels cost 144 KB instead of 432, two epilogue warps per 32 lanes keep up with the shorter tiles, and the ReLU mask of
// the data gradient is fetched before the accumulator is awaited.
#pragma once
#include "../gemm/gemm_kernel.cuh"

namespace st {
namespace conv {
using namespace st::gemm;

constexpr int kHaloPixels = 256;
constexpr int kHaloThreads = 320;      // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-9: epilogue
constexpr int kHaloMaxStages = 4;
constexpr int kHaloCStage = 8 * 4096;  // one 32 x 64 block per epilogue warp
constexpr int kSmemLimit = 232448;     // 227 KB per CTA
constexpr int kHaloTail = 256 + 512 + 1024;      // barriers, bias, alignment slack

struct HaloParams {
  int tiles, hblocks, rows, W;        // tiles of `rows` image rows, `hblocks` per image
  int chunks, C, OC, act, stages;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* aux_in;        // [pixels, OC]: ReLU mask source for ACT_RELU_BWD
  unsigned* err;
};

template <int BN, bool RESIDENT>
__global__ void __launch_bounds__(kHaloThreads, 1)
conv3x3_halo_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                    const __grid_constant__ CUtensorMap tmY, const HaloParams p) {
  constexpr int B_TILE = BN * BK * 2;
  constexpr int RES_BYTES = RESIDENT ? 9 * B_TILE : 0;
  constexpr uint32_t TMEM_COLS = 4 * BN;      // two accumulators of two halves
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a_bytes = (p.rows + 2) * p.W * BK * 2;
  const int stage_bytes = a_bytes + (RESIDENT ? 0 : 3 * B_TILE);
  uint8_t* cstage = smem + RES_BYTES + p.stages * stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(cstage + kHaloCStage);
  uint64_t *full_bar = bars, *empty_bar = bars + kHaloMaxStages, *tfull_bar = bars + 2 * kHaloMaxStages;
  uint64_t *tempty_bar = tfull_bar + 2, *w_bar = tfull_bar + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_bias = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tfull_bar[a]), 1);
      mbar_init(smem_u32(&tempty_bar[a]), 8);
    }
    mbar_init(smem_u32(w_bar), 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_begin();      // set up beside the previous kernel's end; global memory is touched from here on

  if (warp == 0) {
    // ------------------------------- TMA producer (converged warp, one lane issues) -------------------------------
    const bool leader = elect_one();
    const uint32_t smem0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t full0 = __shfl_sync(0xffffffffu, smem_u32(full_bar), 0), empty0 = full0 + kHaloMaxStages * 8;
    if (RESIDENT && leader) {
      const uint32_t wb = smem_u32(w_bar);
      mbar_arrive_expect_tx(wb, 9 * B_TILE);
      for (int tap = 0; tap < 9; ++tap) tma_load_3d(smem0 + tap * B_TILE, &tmW, wb, tap * p.C, 0, 0);
    }
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      const int img = t / p.hblocks, h0 = (t - img * p.hblocks) * p.rows;
      for (int chunk = 0; chunk < p.chunks && ok; ++chunk)
        for (int dw = 0; dw < 3; ++dw) {
          if (!mbar_wait_warp(empty0 + stage * 8, phase ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t fb = full0 + stage * 8, sa = smem0 + RES_BYTES + stage * stage_bytes;
          if (leader) {
            mbar_arrive_expect_tx(fb, stage_bytes);
            tma_load_4d(sa, &tmX, fb, chunk * 64, dw - 1, h0 - 1, img);
            if constexpr (!RESIDENT) {
#pragma unroll
              for (int dh = 0; dh < 3; ++dh) tma_load_3d(sa + a_bytes + dh * B_TILE, &tmW, fb, (dh * 3 + dw) * p.C + chunk * 64, 0, 0);
            }
          }
          __syncwarp();
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(BM, BN, false, false);
    constexpr uint32_t desc_hi = smem_desc_hi(1024);
    const uint32_t smem0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t tmem0 = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t full0 = __shfl_sync(0xffffffffu, smem_u32(full_bar), 0), empty0 = full0 + kHaloMaxStages * 8;
    const uint32_t tfull0 = full0 + 2 * kHaloMaxStages * 8, tempty0 = tfull0 + 16;
    const uint32_t a0 = smem_desc_lo(smem0 + RES_BYTES, 16), b0 = smem_desc_lo(RESIDENT ? smem0 : smem0 + a_bytes, 16);
    const uint32_t dh_step = (p.W * BK * 2) >> 4;
    int stage = 0, iter = 0;
    uint32_t phase = 0;
    bool ok = !RESIDENT || mbar_wait_warp(smem_u32(w_bar), 0, abort_flag);
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++iter) {
      const int acc = iter & 1;
      if (!mbar_wait_warp(tempty0 + acc * 8, ((iter >> 1) & 1) ^ 1u, abort_flag)) break;
      tc_fence_after();
      const uint32_t tmem_d = tmem0 + acc * 2 * BN;
      for (int chunk = 0; chunk < p.chunks && ok; ++chunk)
        for (int dw = 0; dw < 3; ++dw) {
          if (!mbar_wait_warp(full0 + stage * 8, phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_lo = a0 + stage * (stage_bytes >> 4);
          const uint32_t b_lo = RESIDENT ? b0 + dw * (B_TILE >> 4) : b0 + stage * (stage_bytes >> 4);
          if (leader) {
#pragma unroll
            for (int dh = 0; dh < 3; ++dh)
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                  umma_bf16_ss_split(tmem_d + half * BN, a_lo + dh * dh_step + half * (BM * BK * 2 >> 4) + k * (UMMA_K * 2 >> 4), desc_hi,
                                     b_lo + dh * (RESIDENT ? 3 : 1) * (B_TILE >> 4) + k * (UMMA_K * 2 >> 4), desc_hi, idesc,
                                     (chunk | dw | dh | k) != 0 ? 1u : 0u);
            umma_commit(empty0 + stage * 8);
            if (chunk + 1 == p.chunks && dw == 2) umma_commit(tfull0 + acc * 8);
          }
          __syncwarp();
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
    }
  } else {
    // ------------------------------- epilogue: one warp per 32 lanes and half -------------------------------
    const int quad = warp & 3, half = (warp - 2) >> 2;
    uint8_t* cs = cstage + (warp - 2) * 4096;
    // only these warps read the bias; it is fetched behind chain_begin(), as the kernel before this one may have written it
    const int oc = threadIdx.x - 64;
    if (oc < BN) s_bias[oc] = p.bias && oc < p.OC ? __bfloat162float(p.bias[oc]) : 0.0f;
    asm volatile("bar.sync 1, %0;" ::"n"(kHaloThreads - 64) : "memory");
    int iter = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++iter) {
      const int acc = iter & 1;
      const int row0 = t * kHaloPixels + half * BM + quad * 32;
      const __nv_bfloat16* aux = p.aux_in + (long long)(row0 + lane) * p.OC;
#pragma unroll
      for (int g = 0; g < BN / 64; ++g) {
        if (g > 0 && g * 64 >= p.OC) break;
        uint4 m[8];
        if (p.act == ACT_RELU_BWD) {
#pragma unroll
          for (int q = 0; q < 8; ++q)
            m[q] = g * 64 + q * 8 < p.OC ? *reinterpret_cast<const uint4*>(aux + g * 64 + q * 8) : make_uint4(0, 0, 0, 0);
        }
        if (g == 0) {
          if (!mbar_wait_warp(smem_u32(&tfull_bar[acc]), (iter >> 1) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after();
        }
        uint32_t r[2][32];
        const uint32_t src = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (acc * 2 + half) * BN + g * 64;
        tmem_ld_32x32(src, r[0]);
        tmem_ld_32x32(src + 32, r[1]);
        if (lane == 0) tma_store_wait_read<0>();      // the previous block has left the staging area
        tmem_ld_wait();
        if ((g + 1) * 64 >= BN || (g + 1) * 64 >= p.OC) tc_fence_before();
        __syncwarp();
        if (((g + 1) * 64 >= BN || (g + 1) * 64 >= p.OC) && lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float v[8];
          const float4 b0 = *reinterpret_cast<const float4*>(s_bias + g * 64 + q * 8), b1 = *reinterpret_cast<const float4*>(s_bias + g * 64 + q * 8 + 4);
          const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[q >> 2][(q & 3) * 8 + j]) + b[j];
          if (p.act == ACT_RELU) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.0f);
          } else if (p.act == ACT_RELU_BWD) {
            const uint32_t u[4] = {m[q].x, m[q].y, m[q].z, m[q].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = unpack_bf16x2(u[j]);
              v[2 * j] = f.x > 0.0f ? v[2 * j] : 0.0f;
              v[2 * j + 1] = f.y > 0.0f ? v[2 * j + 1] : 0.0f;
            }
          }
          *reinterpret_cast<uint4*>(cs + sw128_offset(lane, q)) =
              make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&tmY, smem_u32(cs), g * 64, row0, 0);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) report_error(p.err, ERR_MBAR_TIMEOUT, 0x6E01u);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);      // copies still in flight land before the memory is released
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int BN, bool RESIDENT>
int launch_halo(const CUtensorMap& tmX, const CUtensorMap& tmW, const CUtensorMap& tmY, const HaloParams& p, int smem, cudaStream_t stream) {
  auto kern = conv3x3_halo_kernel<BN, RESIDENT>;
  static bool configured[st::kMaxDevices] = {false};   // the attribute is per device
  const int dev = st::current_device();
  if (!configured[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    configured[dev] = true;
  }
  st::chained(kern, p.tiles < st::sm_count() ? p.tiles : st::sm_count(), kHaloThreads, smem, stream)(tmX, tmW, tmY, p);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

}  // namespace conv
}  // namespace st
