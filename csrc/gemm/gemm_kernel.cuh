// The persistent tcgen05 GEMM kernel, shared by the plain launcher (gemm_sm100.cu) and the
// tensor-parallel launchers (csrc/comm/tp_gemm.cu).
//
// COMM selects what else the launch does:
//   COMM_NONE  C = epilogue(alpha * A·Bᵀ)
//   COMM_AG    all-gather → GEMM.  A is the gathered activation [T, K].  Every CTA of the launch
//              has two extra warps that push a 1/gridDim slice of this rank's shard into every
//              rank's gather buffer (bulk copies through a small shared-memory ring, plain peer
//              writes over NVLink, destinations in ring order) and count per-sub-chunk arrivals,
//              while its other warps run GEMM tiles.  The TMA producer waits (bounded) for the
//              counter of the rows it is about to load; the local rows are read from the shard
//              itself; tiles are ordered local chunk first, then in ring order.
//   COMM_RS    GEMM → reduce-scatter.  Tiles are ordered so that the chunk this rank owns comes last (or, with
//              row-block groups, so that each group of the own chunk comes one group after the remote tiles of
//              the same group: see map_tile).
//              For the other chunks the epilogue TMA-stores each partial tile straight into the
//              owner's staging slot (peer writes over NVLink) and counts the tile on the owner's
//              per-row-block counter.  For its own chunk the epilogue waits (bounded) until every
//              peer's partial of the row block has landed, adds them and the optional residual to
//              the accumulator in fp32, and writes the final bf16 rows — there is no separate
//              reduction pass and the local partial is never staged.
#pragma once
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "../comm/comm.cuh"
#include <cstring>

namespace st {
namespace gemm {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int num_threads(int sets) { return 64 + 128 * sets; }      // warp 0: TMA, warp 1: MMA + TMEM owner, then the epilogue's warps
constexpr int NUM_THREADS = num_threads(2);
constexpr int NUM_THREADS_RS = 192;  // reduce-scatter variant: one epilogue warp per 32 lanes
constexpr int NUM_THREADS_AG = 256;  // all-gather variant: + warp 6 (shard push) and warp 7 (arrival publisher)
constexpr int AG_RING_CHUNK = 16384;  // bytes per bulk copy of the push ring
constexpr int AG_RING_SLOTS = 3;      // the ring sits behind the barriers of the 3-stage GEMM layout

enum Act : int { ACT_NONE = 0, ACT_RELU = 1, ACT_GELU = 2, ACT_GELU_BWD = 3, ACT_RELU_BWD = 4 };
enum Comm : int { COMM_NONE = 0, COMM_AG = 1, COMM_RS = 2 };
constexpr int kMaxSubChunks = 16;   // arrival counters reserved per source rank (AG)

struct GemmComm {
  PeerGroup g;
  int rows_per_chunk;   // rows owned by each rank (T / world), multiple of BM
  int sub_per_chunk;    // arrival-flag granularity (AG): sub-chunks per rank shard
  int gemm_ctas;        // CTAs that run GEMM tiles; CTAs beyond them only push (AG)
  int slot_enter;       // entry rendezvous slot (world words)
  // ---- AG ----
  const __nv_bfloat16* src_shard;          // [rows_per_chunk, K] contiguous
  __nv_bfloat16* gather_peers[kMaxRanks];  // [T, K] contiguous on every rank
  __nv_bfloat16* gather_mc;                // multicast alias or null
  int slot_arrive;      // arrival words: slot_arrive + src * kMaxSubChunks + sub
  unsigned arrive_target;  // value an arrival word must reach: the epoch (peer-store path, one
                           // writer per word) or a cumulative count (multicast path, n_comm writers)
  unsigned long long* trace;  // optional [gridDim.x][4] globaltimer stamps (start, entry, tiles/push done, end)
  int sub_major;        // tile order of the remote chunks: 0 chunk by chunk (ring), 1 sub-chunk by sub-chunk
  int local_in_place;   // AG: the shard already lives in this rank's slot of its own gather buffer (no local copy)
  int rs_groups;        // RS: row-block groups per chunk; remote and local tiles are interleaved group by group
  int rs_lag;           // RS: groups a local group trails the remote group of the same index (>= 1)
  // ---- RS ----
  __nv_bfloat16* stage_peers[kMaxRanks];   // on each owner: [world][rows_per_chunk, N]
  int slot_done;        // counters: slot_done + row block within the chunk
  unsigned done_target; // counter value meaning "every rank's tiles of this row block landed"
  __nv_bfloat16* rs_out;                   // [rows_per_chunk, N] reduced local shard
  const __nv_bfloat16* rs_residual;        // optional, added during the reduction
};

// Implicit-GEMM convolution (3x3, stride 1, padding 1, NHWC activations).
//   mode 1 (forward / data gradient): the A tile of 128 output pixels is a 4-D TMA box
//          {64 channels, W, Hb, Nb} taken at the tap's (kh-1, kw-1) offset; pixels outside the image
//          are zero-filled by TMA.  K = 9 * C runs tap-major, matching weights stored [OC][tap][C].
//   mode 2 (weight gradient): K runs over pixels, N over (tap, channel); the B tile is a row of 4-D boxes, one per
//          64 columns (64 pixels x 64 channels of the input shifted by the column's tap), A is dYᵀ; the batch index
//          is the K split, whose share of the pixel blocks need not be the same for all.
struct ConvGeom {
  int mode;
  int H, W;          // image size
  int Hb, Nb;        // rows / images per pixel block (mode 1: 128 pixels, mode 2: 64 pixels)
  int c_chunks;      // input channels / 64
  int blocks;        // pixel blocks over all splits (mode 2)
};

struct GemmParams {
  ConvGeom conv;
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  __nv_bfloat16* aux_out;
  long long ld_aux_out;
  const __nv_bfloat16* aux_in;
  long long ld_aux_in;
  int M, N, K;
  float alpha;
  int act;
  int out_fp32;
  int accumulate;
  int batch;
  long long batch_stride_c;
  int use_tma_store;   // OutputMode: the output goes through shared memory and the copy engine
  int operand_tma;     // the epilogue's operand (aux_in of a derivative, else the residual) arrives by TMA, OutMaps.m[1]
  int aux_tma;         // aux_out leaves by TMA, OutMaps.m[2]
  unsigned* err;
};
enum OutputMode : int { STORE_DIRECT = 0, STORE_BF16 = 1, STORE_FP32 = 2, STORE_FP32_ADD = 3 };

// Tensor maps of the output, one per owner rank for GEMM → reduce-scatter.  Plain product: [0] the output, [1] the epilogue's
// operand, [2] the saved pre-activation.
struct OutMaps {
  CUtensorMap m[kMaxRanks];
};

// CBUF: 4 KiB staging blocks per epilogue warp of the plain product (four times SETS warps), as many as fit beside the operand
// ring; the tensor-parallel variants have four warps with two blocks each, which is the room of CBUF = 1 of eight.
constexpr int kSmemMax = 232448;      // 227 KiB
template <int BN, int STAGES, int CB = 0, int SETS = 2>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BAR_BYTES = 512;                            // barriers
  static constexpr int SLACK = BAR_BYTES + 1024;                   // and alignment
  static constexpr int ROOM = (kSmemMax - SLACK - STAGES * STAGE_BYTES) / (4 * SETS * 4096);
  static constexpr int CBUF = CB ? CB : ROOM < 4 ? ROOM : 4;
  static_assert(CBUF >= 1, "no room for the staged output");
  static constexpr int CSTAGE_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int CSTAGE_BYTES = 4 * SETS * CBUF * 4096;
  static constexpr int BAR_OFFSET = CSTAGE_OFFSET + CSTAGE_BYTES;
  static constexpr int OPBAR_OFFSET = BAR_OFFSET + 256;            // one barrier per epilogue warp and staging block (at most 32)
  static constexpr int TOTAL = BAR_OFFSET + SLACK;
};

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
  // groups of 8 M-tiles share the same B tiles while they are L2-resident
  constexpr int GM = 8;
  const int group_size = GM * tiles_n;
  const int g = t / group_size;
  const int first_m = g * GM;
  const int gm = min(GM, tiles_m - first_m);
  const int r = t - g * group_size;
  tm = first_m + r % gm;
  tn = r / gm;
}

// Tile index → (batch, tm, tn); with a communication plan the M dimension is walked chunk by
// chunk in ring order (`chunk_shift` = 0 starts at the local chunk, 1 ends with it).
template <int COMM>
__device__ __forceinline__ void map_tile(int t, int tiles_m, int tiles_n, int tiles_per_batch,
                                         const GemmComm& c, int& b, int& tm, int& tn) {
  if constexpr (COMM == COMM_NONE) {
    b = t / tiles_per_batch;
    tile_coords(t - b * tiles_per_batch, tiles_m, tiles_n, tm, tn);
  } else {
    b = 0;
    const int tiles_m_chunk = c.rows_per_chunk / BM;
    const int per_chunk = tiles_m_chunk * tiles_n;
    if (COMM == COMM_AG && c.sub_major && t >= per_chunk) {
      // remote rows: for every sub-chunk index, the W-1 remote chunks in ring order
      const int msub = tiles_m_chunk / c.sub_per_chunk;       // M tiles per sub-chunk
      const int per_sub = msub * tiles_n;
      const int r = t - per_chunk;
      const int blk = r / per_sub;
      const int s = blk / (c.g.world - 1);
      const int ci = 1 + blk % (c.g.world - 1);
      const int rr = r - blk * per_sub;
      tn = rr / msub;
      tm = ((c.g.rank + ci) % c.g.world) * tiles_m_chunk + s * msub + rr % msub;
      return;
    }
    if (COMM == COMM_RS && c.rs_groups > 1) {
      // Row blocks of every chunk are split into G groups.  Order (lag 1): R(0), R(1), L(0), R(2), L(1), ...,
      // R(G-1), L(G-2), L(G-1), where R(g) are the tiles of group g of the W-1 remote chunks (ring order) and
      // L(g) the tiles of group g of this rank's own chunk.  A local tile needs every peer's partial of its row
      // block; peers deliver those in their R(g), so running L(g) `lag` groups late lets the final reduction of
      // group g ride behind later transfers instead of after all of them.  lag >= G is "all remote, then local".
      const int W = c.g.world, G = c.rs_groups;
      const int lag = min(max(c.rs_lag, 1), G);          // local group g runs after remote group g + lag
      const int msub = tiles_m_chunk / G;
      const int per_l = msub * tiles_n;
      const int per_r = (W - 1) * per_l;
      int g, r;
      bool local;
      if (t < lag * per_r) {                             // R(0) .. R(lag-1)
        g = per_r > 0 ? t / per_r : 0; local = false; r = t - g * per_r;
      } else {
        const int u = t - lag * per_r;
        const int pairs = G - lag;                       // (R(lag + i), L(i)) for i < pairs
        if (u < pairs * (per_r + per_l)) {
          const int pair = u / (per_r + per_l);
          const int v = u - pair * (per_r + per_l);
          if (v < per_r) { g = lag + pair; local = false; r = v; }
          else { g = pair; local = true; r = v - per_r; }
        } else {                                         // L(pairs) .. L(G-1)
          const int w = u - pairs * (per_r + per_l);
          g = pairs + w / per_l; local = true; r = w - (w / per_l) * per_l;
        }
      }
      int lm;
      if (local) {
        tile_coords(r, msub, tiles_n, lm, tn);
        tm = c.g.rank * tiles_m_chunk + g * msub + lm;
      } else {
        const int ci = r / per_l;
        tile_coords(r - ci * per_l, msub, tiles_n, lm, tn);
        tm = ((c.g.rank + 1 + ci) % W) * tiles_m_chunk + g * msub + lm;
      }
      return;
    }
    const int ci = t / per_chunk;
    int lm;
    tile_coords(t - ci * per_chunk, tiles_m_chunk, tiles_n, lm, tn);
    const int shift = (COMM == COMM_AG) ? 0 : 1;
    const int chunk = (c.g.rank + shift + ci) % c.g.world;
    tm = chunk * tiles_m_chunk + lm;
  }
}

// ---- reduce-scatter: sources added to a tile of the rows this rank owns ----------------------
constexpr int kRsBatch = 4;   // sources whose loads are in flight together (4 x 64 B per lane each)

__device__ __forceinline__ void prefetch_l2(const void* ptr) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
}

// Source s of the local reduction: the staged partials of the other ranks in rank order (this
// rank's own slot is skipped), then the residual.
__device__ __forceinline__ const __nv_bfloat16* rs_src(const GemmComm& cm, int s, long long slot_stride) {
  const int q = s + (s >= cm.g.rank ? 1 : 0);
  return q < cm.g.world ? cm.stage_peers[cm.g.rank] + q * slot_stride
                        : cm.rs_residual;
}

__device__ __forceinline__ void rs_load_batch(const GemmComm& cm, long long slot_stride, int s0, int n_srcs, long long off,
                                              uint4 (&buf)[kRsBatch][4]) {
#pragma unroll
  for (int i = 0; i < kRsBatch; ++i) {
    if (s0 + i < n_srcs) {
      const uint4* sp = reinterpret_cast<const uint4*>(rs_src(cm, s0 + i, slot_stride) + off);
#pragma unroll
      for (int k = 0; k < 4; ++k) buf[i][k] = sp[k];
    }
  }
}

__device__ __forceinline__ void rs_add_batch(int s0, int n_srcs, const uint4 (&buf)[kRsBatch][4], float* v) {
#pragma unroll
  for (int i = 0; i < kRsBatch; ++i) {
    if (s0 + i < n_srcs) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 f0 = unpack_bf16x2(buf[i][k].x), f1 = unpack_bf16x2(buf[i][k].y), f2 = unpack_bf16x2(buf[i][k].z),
               f3 = unpack_bf16x2(buf[i][k].w);
        v[k * 8 + 0] += f0.x; v[k * 8 + 1] += f0.y; v[k * 8 + 2] += f1.x; v[k * 8 + 3] += f1.y;
        v[k * 8 + 4] += f2.x; v[k * 8 + 5] += f2.y; v[k * 8 + 6] += f3.x; v[k * 8 + 7] += f3.y;
      }
    }
  }
}

// Pixel blocks of split b of a convolution's weight gradient
__device__ __forceinline__ int split_begin(const GemmParams& p, int b) {
  return static_cast<int>((long long)p.conv.blocks * b / p.batch);
}
__device__ __forceinline__ int split_blocks(const GemmParams& p, int b) { return split_begin(p, b + 1) - split_begin(p, b); }

// ---- epilogue of the plain product -----------------------------------------------------------
__device__ __forceinline__ uint4 pack8_bf16(const float* v) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ void add8_bf16(float* v, const uint4& u) {
  const float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z), f3 = unpack_bf16x2(u.w);
  v[0] += f0.x; v[1] += f0.y; v[2] += f1.x; v[3] += f1.y;
  v[4] += f2.x; v[5] += f2.y; v[6] += f3.x; v[7] += f3.y;
}
// Whether a row segment starting at `p`, on a 32-column boundary of its matrix, may be accessed 16 bytes at a time
__device__ __forceinline__ bool vec8(const __nv_bfloat16* p, long long ld) {
  return (ld & 7) == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}
// 32 values of a row, of which `n` exist (the rest is zero)
__device__ __forceinline__ void load32_bf16(uint4 (&x)[4], const __nv_bfloat16* a, long long ld, bool full, int n) {
  if (full && n > 0 && vec8(a, ld)) {
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = reinterpret_cast<const uint4*>(a)[q];
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = q * 8 + i * 2;
      const uint32_t lo = j < n ? __bfloat16_as_ushort(a[j]) : 0u, hi = j + 1 < n ? __bfloat16_as_ushort(a[j + 1]) : 0u;
      w[i] = lo | (hi << 16);
    }
    x[q] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// KS > 1 (COMM_NONE only): a cluster of KS CTAs shares one tile, each with a KS-th of its K blocks; they add their fp32 sums through
// shared memory in a fixed order, and each finishes a KS-th of the rows.  One tile per cluster.
// CG = 2 (COMM_NONE only): a cluster of two CTAs works on one tile of 256 x BN.  Each CTA brings its 128 rows of A and its half
// of B into its own shared memory, the even CTA's MMA warp issues for both, and each CTA's epilogue stores its own 128 rows.
// A K block then costs an SM 32 KB of loads instead of 48 (BN = 256), and the ring holds six stages instead of four.
template <int BN, int STAGES, bool A_MN, bool B_MN, int COMM, int CG = 1, int KS = 1, int SETS_ = 2>
__global__ void __launch_bounds__(COMM == COMM_AG ? NUM_THREADS_AG : COMM == COMM_RS ? NUM_THREADS_RS : num_threads(SETS_), 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ OutMaps tmC, const __grid_constant__ CUtensorMap tmA_local,
                 const GemmParams p, const GemmComm cm) {
  static_assert((CG == 1 && KS == 1) || (COMM == COMM_NONE && (CG == 1 || KS == 1)), "CTA pairs and K parts run the plain product only");
  using L = SmemLayout<BN / CG, STAGES, COMM == COMM_NONE ? 0 : 1, SETS_>;
  // Epilogue warps per 32 lanes of the accumulator.  Two or three of them take 64-column groups in turn, or, where a tile has only
  // one group, whole tiles in turn: one warp's loads, arithmetic and stores for a tile are longer than the main loop of a short K.
  constexpr int SETS = COMM == COMM_NONE ? SETS_ : 1, GROUPS = BN / 64;
  constexpr bool SPLIT = SETS >= 2 && BN > 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  const int cta = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int kpart = KS > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int gemm_bid = blockIdx.x / (CG * KS);

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tiles_m = (p.M + BM * CG - 1) / (BM * CG);
  const int tiles_n = (p.N + BN - 1) / BN;
  const int tiles_per_batch = tiles_m * tiles_n;
  const int total_tiles = tiles_per_batch * p.batch;
  const int k_blocks = (p.K + BK - 1) / BK;
  const int grid_stride = gridDim.x / (CG * KS);
  const int k_first = KS > 1 ? k_blocks * kpart / KS : 0;
  const int k_own = KS > 1 ? k_blocks * (kpart + 1) / KS - k_first : k_blocks;       // K blocks of this CTA
  constexpr uint32_t TMEM_COLS = (2 * BN <= 32) ? 32 : (2 * BN <= 64) ? 64 : (2 * BN <= 128) ? 128
                                 : (2 * BN <= 256) ? 256 : 512;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tfull_bar[a]), 1);
      mbar_init(smem_u32(&tempty_bar[a]), (SPLIT ? 4 * SETS : 4) * CG);
    }
    if constexpr (COMM == COMM_NONE)
      for (int i = 0; i < 4 * SETS * L::CBUF; ++i) mbar_init(smem_u32(smem + L::OPBAR_OFFSET) + i * 8, 1);
    *abort_flag = 0;
    if constexpr (COMM == COMM_AG) {
      tmem_slot[2] = 0;   // items whose stores are complete (push warp → publisher warp)
      tmem_slot[3] = 0;   // push warp has finished
    }
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if constexpr (COMM == COMM_RS) {
      // tell every peer that this rank has left the previous launch that used the staging area
      if (blockIdx.x == 0) {
        fence_sys();
        for (int q = 0; q < cm.g.world; ++q)
          st_relaxed_sys(cm.g.signals[q] + cm.slot_enter + cm.g.rank, cm.g.epoch);
      }
    }
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_pair(smem_u32(tmem_slot), TMEM_COLS);
    } else {
      tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncwarp();
  if constexpr (CG == 2) cluster_sync(); else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // barriers, tensor memory and descriptors are set up beside the previous kernel's end; global memory is touched from here on
  if constexpr (COMM == COMM_NONE) chain_begin();

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------------
    // The whole warp walks the schedule and one lane issues.  With warp-uniform control flow the loop's addresses and
    // coordinates sit in uniform registers, which TMA and tcgen05 instructions read; issued from inside a one-lane
    // branch, with descriptors rebuilt per instruction, the producer's and the issuer's loops set the pace of short or narrow
    // K blocks: the weight gradient of a 64-channel 3x3 convolution over a million pixels, in tiles of 64 columns, takes 240 us
    // this way and 315 in the other.  Wide products do not change.
    const bool leader = COMM == COMM_AG ? lane == 0 : elect_one();
    const uint32_t smem0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t full0 = __shfl_sync(0xffffffffu, smem_u32(full_bar), 0);
    const uint32_t empty0 = full0 + STAGES * 8;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = gemm_bid; t < total_tiles && ok; t += grid_stride) {
      int b, tm, tn;
      map_tile<COMM>(t, tiles_m, tiles_n, tiles_per_batch, cm, b, tm, tn);
      const int m0 = tm * BM * CG + cta * BM, n0 = tn * BN + cta * (BN / CG);      // this CTA's rows of A and of B
      const CUtensorMap* mapA = &tmA;
      int m_coord = m0;
      if constexpr (COMM == COMM_AG) {
        const int src = m0 / cm.rows_per_chunk;
        const int sub = (m0 - src * cm.rows_per_chunk) / (cm.rows_per_chunk / cm.sub_per_chunk);
        if (src == cm.g.rank) {
          // the local rows are read from the shard itself; nothing to wait for
          mapA = &tmA_local;
          m_coord = m0 - src * cm.rows_per_chunk;
        } else {
          bool landed = true;
          if (leader) {
            landed = wait_flag_ge(cm.g.signals[cm.g.rank] + cm.slot_arrive + src * kMaxSubChunks + sub, cm.arrive_target);
            if (!landed) {
              *abort_flag = 1;
              report_error(p.err, ERR_FLAG_TIMEOUT, 0xA601u);
            }
          }
          if (!__all_sync(0xffffffffu, landed)) break;
        }
        if (leader) fence_proxy_async_global();
      }
      const int k_count = A_MN && B_MN && p.conv.mode == 2 ? split_blocks(p, b) : k_own;
      // one K block per ring stage: wait until its MMAs have read it, then hand the copies to the TMA unit
      auto k_loop = [&](uint32_t bytes, auto&& copies) {
        for (int kb = 0; kb < k_count; ++kb) {
          if (!mbar_wait_warp(empty0 + stage * 8, phase ^ 1u, abort_flag)) return false;
          const uint32_t fb = CG == 2 ? (full0 + stage * 8) & kPairLeaderMask : full0 + stage * 8;
          const uint32_t sa = smem0 + stage * L::STAGE_BYTES;
          if (leader && cta == 0) mbar_arrive_expect_tx(fb, bytes * CG);       // the even CTA's barrier counts both CTAs' bytes
          copies(kb, fb, sa, sa + L::A_BYTES);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        return true;
      };
      // MN-major operands arrive as 64-wide boxes: a box wholly outside the matrix is not fetched (what the shared
      // memory holds in its place only reaches rows or columns of the accumulator that are never stored)
      constexpr int BNC = BN / CG;         // rows of B per CTA
      const int boxes_a = (A_MN && COMM == COMM_NONE && CG == 1) ? min(BM / 64, (p.M - m0 + 63) / 64) : BM / 64;
      const int boxes_b = (B_MN && COMM == COMM_NONE && CG == 1) ? min(BN / 64, (p.N - n0 + 63) / 64) : BNC / 64;
      const bool whole = boxes_a == BM / 64 && boxes_b == BNC / 64;
      const uint32_t stage_bytes = (boxes_a + boxes_b) * (64 * BK * 2);
      auto load3 = [](uint32_t dst, const CUtensorMap* map, uint32_t fb, int c0, int c1, int c2) {
        if constexpr (CG == 2) tma_load_3d_pair(dst, map, fb, c0, c1, c2); else tma_load_3d(dst, map, fb, c0, c1, c2);
      };
      auto load4 = [](uint32_t dst, const CUtensorMap* map, uint32_t fb, int c0, int c1, int c2, int c3) {
        if constexpr (CG == 2) tma_load_4d_pair(dst, map, fb, c0, c1, c2, c3); else tma_load_4d(dst, map, fb, c0, c1, c2, c3);
      };
      // Convolution coordinates advance by additions: six divisions per K block took about 950 SM cycles, twice the
      // tensor work of the largest tile.
      if (!A_MN && !B_MN && p.conv.mode == 1) {
        // A: 128 output pixels (Nb images x Hb rows x W) shifted by the tap, 64 channels
        const int hblocks = p.conv.H / p.conv.Hb;
        const int block = tm * CG + cta;
        const int img = (block / hblocks) * p.conv.Nb, h0 = (block % hblocks) * p.conv.Hb;
        int tap_w = -1, tap_h = -1, chunk = 0;
        if constexpr (KS > 1) {
          const int tap = k_first / p.conv.c_chunks;
          chunk = k_first - tap * p.conv.c_chunks;
          tap_w = tap % 3 - 1;
          tap_h = tap / 3 - 1;
        }
        ok = k_loop(stage_bytes, [&](int kb, uint32_t fb, uint32_t sa, uint32_t sb) {
          if (leader) {
            load4(sa, mapA, fb, chunk * 64, tap_w, h0 + tap_h, img);
            load3(sb, &tmB, fb, (k_first + kb) * BK, n0, 0);
          }
          if (++chunk == p.conv.c_chunks) {
            chunk = 0;
            if (++tap_w == 2) { tap_w = -1; ++tap_h; }
          }
        });
      } else if (A_MN && B_MN && p.conv.mode == 2) {
        // K block = 64 consecutive pixels; each 64 columns of B are one tap and channel block
        const int hblocks = p.conv.H / p.conv.Hb;
        int tap_w[BNC / 64], tap_h[BNC / 64], chan[BNC / 64];
#pragma unroll
        for (int j = 0; j < BNC / 64; ++j) {
          const int col = n0 / 64 + j, tap = col / p.conv.c_chunks;
          chan[j] = (col - tap * p.conv.c_chunks) * 64;
          tap_w[j] = tap % 3 - 1;
          tap_h[j] = tap / 3 - 1;
        }
        int pix_block = split_begin(p, b);
        int img = (pix_block / hblocks) * p.conv.Nb, h0 = (pix_block % hblocks) * p.conv.Hb;
        ok = k_loop(stage_bytes, [&](int, uint32_t fb, uint32_t sa, uint32_t sb) {
          if (leader) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              if (j < boxes_a) load3(sa + j * (64 * BK * 2), mapA, fb, m_coord + 64 * j, pix_block * BK, 0);
#pragma unroll
            for (int j = 0; j < BNC / 64; ++j)
              if (j < boxes_b) load4(sb + j * (64 * BK * 2), &tmB, fb, chan[j], tap_w[j], h0 + tap_h[j], img);
          }
          ++pix_block;
          h0 += p.conv.Hb;
          if (h0 == p.conv.H) { h0 = 0; img += p.conv.Nb; }
        });
      } else if (whole) {
        ok = k_loop(L::STAGE_BYTES, [&](int kb, uint32_t fb, uint32_t sa, uint32_t sb) {
          if (!leader) return;
          kb += k_first;
          if constexpr (!A_MN) {
            load3(sa, mapA, fb, kb * BK, m_coord, b);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              load3(sa + j * (64 * BK * 2), mapA, fb, m_coord + 64 * j, kb * BK, b);
          }
          if constexpr (!B_MN) {
            load3(sb, &tmB, fb, kb * BK, n0, b);
          } else {
#pragma unroll
            for (int j = 0; j < BNC / 64; ++j)
              load3(sb + j * (64 * BK * 2), &tmB, fb, n0 + 64 * j, kb * BK, b);
          }
        });
      } else {
        ok = k_loop(stage_bytes, [&](int kb, uint32_t fb, uint32_t sa, uint32_t sb) {
          if (!leader) return;
          kb += k_first;
          if constexpr (!A_MN) {
            load3(sa, mapA, fb, kb * BK, m_coord, b);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              if (j < boxes_a) load3(sa + j * (64 * BK * 2), mapA, fb, m_coord + 64 * j, kb * BK, b);
          }
          if constexpr (!B_MN) {
            load3(sb, &tmB, fb, kb * BK, n0, b);
          } else {
#pragma unroll
            for (int j = 0; j < BNC / 64; ++j)
              if (j < boxes_b) load3(sb + j * (64 * BK * 2), &tmB, fb, n0 + 64 * j, kb * BK, b);
          }
        });
      }
    }
    if constexpr (KS > 1) {       // the epilogue warps' two meetings
      __syncwarp();
      cluster_sync();
      cluster_sync();
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer ---------------------------------------
    const bool leader = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(BM * CG, BN, A_MN, B_MN);
    // descriptor words are formed once: the high word is common, the low word advances by constants
    constexpr uint32_t desc_hi = smem_desc_hi(1024);
    constexpr uint32_t a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4, b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    const uint32_t smem0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t tmem0 = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t full0 = __shfl_sync(0xffffffffu, smem_u32(full_bar), 0);
    const uint32_t empty0 = full0 + STAGES * 8, tfull0 = full0 + 2 * STAGES * 8, tempty0 = tfull0 + 16;
    const uint32_t a_lo0 = smem_desc_lo(smem0, A_MN ? 64 * BK * 2 : 16);
    const uint32_t b_lo0 = smem_desc_lo(smem0 + L::A_BYTES, B_MN ? 64 * BK * 2 : 16);
    int stage = 0;
    uint32_t phase = 0;
    int iter = 0;
    bool ok = true;
    for (int t = cta == 0 ? gemm_bid : total_tiles; t < total_tiles && ok; t += grid_stride, ++iter) {      // the even CTA issues
      const int acc = iter & 1;
      const uint32_t acc_phase = (iter >> 1) & 1;
      if (!mbar_wait_warp(tempty0 + acc * 8, acc_phase ^ 1u, abort_flag)) break;
      tc_fence_after();
      const uint32_t tmem_d = tmem0 + acc * BN;
      const int k_count = A_MN && B_MN && p.conv.mode == 2 ? split_blocks(p, t / tiles_per_batch) : k_own;
      for (int kb = 0; kb < k_count; ++kb) {
        if (!mbar_wait_warp(full0 + stage * 8, phase, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_lo = a_lo0 + stage * (L::STAGE_BYTES >> 4), b_lo = b_lo0 + stage * (L::STAGE_BYTES >> 4);
        if (leader) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            if constexpr (CG == 2)
              umma_bf16_ss_split_pair(tmem_d, a_lo + k * a_step, desc_hi, b_lo + k * b_step, desc_hi, idesc, (kb | k) != 0 ? 1u : 0u);
            else
              umma_bf16_ss_split(tmem_d, a_lo + k * a_step, desc_hi, b_lo + k * b_step, desc_hi, idesc, (kb | k) != 0 ? 1u : 0u);
          // frees the smem stage (of both CTAs) when the MMAs finish
          if constexpr (CG == 2) umma_commit_pair(empty0 + stage * 8); else umma_commit(empty0 + stage * 8);
          if (kb + 1 == k_count) {
            if constexpr (CG == 2) umma_commit_pair(tfull0 + acc * 8); else umma_commit(tfull0 + acc * 8);
          }
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if constexpr (KS > 1) {
      __syncwarp();
      cluster_sync();
      cluster_sync();
    }
  } else if (COMM == COMM_NONE) {
    // ------------------------------- epilogue warps, plain product ----------------------------------------
    // A warp takes 32 rows and 64 columns at a time.  Everything that is wide leaves and arrives through the copy engine and
    // this warp's staging blocks: a lane that reads or writes its own row of global memory touches a 16-byte piece of 32
    // lines per instruction.
    //   operand (saved pre-activation or residual): the warp's blocks land in its staging blocks in turn, asked for ahead of the
    //     arithmetic, and are replaced there by the result, which is stored from the same place;
    //   saved pre-activation out: a staging block beside the result's;
    //   fp32: 32 x 32 blocks, stored, or added by the copy engine (one adder per element unless K is split).
    // Outputs, operands and leading dimensions that TMA cannot take keep the element-wise accesses.
    constexpr int CBUF = L::CBUF;
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    const int set = (warp - 2) >> 2;
    uint8_t* const bufs = smem + L::CSTAGE_OFFSET + (set * 4 + quad) * (CBUF * 4096);
    const uint32_t op_bar = smem_u32(smem + L::OPBAR_OFFSET) + (set * 4 + quad) * (CBUF * 8);
    const bool tma_op = CBUF >= 2 && p.operand_tma, tma_aux = CBUF >= 2 && p.aux_tma;
    const bool bwd = p.act == ACT_GELU_BWD || p.act == ACT_RELU_BWD;
    int iter = 0, blocks = 0;       // blocks staged by this warp
    // the warp's 64-column groups: every SETS-th, counted over its CTA's tiles (SPLIT), or the only one of every SETS-th tile
    auto first_group = [&](int iter) { return SPLIT ? (set + SETS * GROUPS - iter * GROUPS % SETS) % SETS : 0; };
    auto groups_of = [&](int t, int& m0, int& n0, int& b) {
      int tm, tn;
      map_tile<COMM>(t, tiles_m, tiles_n, tiles_per_batch, cm, b, tm, tn);
      m0 = tm * BM * CG + cta * BM + quad * 32;
      n0 = tn * BN;
      if (KS > 1 && quad / (4 / KS) != kpart) return 0;
      return m0 < p.M ? min(GROUPS, (p.N - n0 + 63) >> 6) : 0;
    };
    // K parts: CTA i of the cluster finishes rows [i, i + 1) * 128 / KS of the tile.  Once every CTA's products are complete the
    // operand ring is idle and takes the others' partial sums of those rows, [source][column / 4][row] in 16-byte pieces.
    constexpr int OWN_ROWS = BM / KS, PART_ELEMS = OWN_ROWS * BN;
    static_assert(KS == 1 || (KS - 1) * PART_ELEMS * 4 <= STAGES * L::STAGE_BYTES, "the ring is too small for the partial sums");
    if constexpr (KS > 1) {
      const bool done = mbar_wait_warp(smem_u32(&tfull_bar[0]), 0, abort_flag);
      tc_fence_after();
      cluster_sync();
      const int owner = quad / (4 / KS);
      if (done && owner != kpart) {
        int b, tm, tn;
        map_tile<COMM>(gemm_bid, tiles_m, tiles_n, tiles_per_batch, cm, b, tm, tn);
        const int slot = kpart < owner ? kpart : kpart - 1;
        const uint32_t dst = cluster_map(smem_u32(smem), owner) + (slot * PART_ELEMS + ((quad % (4 / KS)) * 32 + lane) * 4) * 4;
        for (int c = set; c < BN / 32 && tn * BN + c * 32 < p.N; c += SETS) {
          uint32_t r[32];
          tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) cluster_store_16(dst + (c * 8 + q) * (OWN_ROWS * 16), r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
        }
      }
      cluster_sync();
    }
    // operand requests run up to CBUF - 1 blocks ahead of the arithmetic
    int req_t = SPLIT ? gemm_bid : gemm_bid + set * grid_stride, req_iter = 0, req_g = first_group(0), requested = 0;
    auto request = [&]() {
      int m0, n0, b;
      while (req_t < total_tiles && req_g >= groups_of(req_t, m0, n0, b)) {
        req_t += SPLIT ? grid_stride : SETS * grid_stride;
        req_g = first_group(++req_iter);
      }
      if (req_t >= total_tiles) return;
      if (lane == 0) {
        const uint32_t bar = op_bar + (requested % CBUF) * 8;
        mbar_arrive_expect_tx(bar, 4096);
        tma_load_3d(smem_u32(bufs + (requested % CBUF) * 4096), &tmC.m[1], bar, n0 + req_g * 64, m0, 0);
      }
      ++requested;
      req_g += SPLIT ? SETS : GROUPS;
    };
    if (tma_op)
      for (int i = 1; i < CBUF; ++i) request();
    for (int t = gemm_bid; t < total_tiles; t += grid_stride, ++iter) {
      if (!SPLIT && iter % SETS != set) continue;
      int m0, n0, b;
      const int groups = groups_of(t, m0, n0, b);
      const int acc = iter & 1;
      if (!mbar_wait_warp(smem_u32(&tfull_bar[acc]), (iter >> 1) & 1, abort_flag)) break;
      tc_fence_after();
      const int row = m0 + lane;
      const bool row_ok = row < p.M;
      bool held = true, alive = true;
      auto release = [&]() {       // hands the accumulator back to the MMA warp
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (CG == 2) mbar_arrive_cluster(smem_u32(&tempty_bar[acc]) & kPairLeaderMask);
          else mbar_arrive(smem_u32(&tempty_bar[acc]));
        }
        held = false;
      };
#pragma unroll 1
      for (int g = first_group(iter); g < groups; g += SPLIT ? SETS : 1) {
        // saved pre-activation and result take turns
        const int at = tma_aux ? (2 * blocks) % (CBUF & ~1) : blocks % CBUF;
        uint8_t* const cs = bufs + (tma_aux ? at + 1 : at) * 4096;
        uint8_t* const aux_block = bufs + at * 4096;
        if (tma_op && !mbar_wait_warp(op_bar + (blocks % CBUF) * 8, (blocks / CBUF) & 1, abort_flag)) {
          alive = false;
          break;
        }
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          const int col0 = n0 + g * 64 + half * 32;
          if (col0 >= p.N) {
            if (held && g + (SPLIT ? SETS : 1) >= groups) release();
            break;  // uniform across the warp
          }
          uint32_t r[32];
          tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN + g * 64 + half * 32, r);
          tmem_ld_wait();
          if (half == 1 && g + (SPLIT ? SETS : 1) >= groups) release();
          if constexpr (KS > 1) {
            const float4* part = reinterpret_cast<const float4*>(smem) + (g * 64 + half * 32) / 4 * OWN_ROWS + (quad % (4 / KS)) * 32 + lane;
#pragma unroll
            for (int i = 0; i < KS - 1; ++i)
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const float4 u = part[i * (PART_ELEMS / 4) + q * OWN_ROWS];
                r[q * 4] = __float_as_uint(__uint_as_float(r[q * 4]) + u.x);
                r[q * 4 + 1] = __float_as_uint(__uint_as_float(r[q * 4 + 1]) + u.y);
                r[q * 4 + 2] = __float_as_uint(__uint_as_float(r[q * 4 + 2]) + u.z);
                r[q * 4 + 3] = __float_as_uint(__uint_as_float(r[q * 4 + 3]) + u.w);
              }
          }
          const bool full = col0 + 32 <= p.N;
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
          if (p.bias) {
            if (full && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
#pragma unroll
              for (int q = 0; q < 4; ++q) add8_bf16(v + q * 8, __ldg(reinterpret_cast<const uint4*>(p.bias + col0) + q));
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (full || col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
            }
          }
          // the staging blocks written below were handed to the copy engine a block or more ago
          if (half == 0 && p.use_tma_store == STORE_BF16 && !tma_op) {
            if (lane == 0) {
              if (tma_aux) tma_store_wait_read<(CBUF >= 4 ? 1 : 0)>(); else tma_store_wait_read<CBUF - 1>();
            }
            __syncwarp();
          }
          if (p.aux_out) {
            if (tma_aux) {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(aux_block + sw128_offset(lane, half * 4 + q)) = pack8_bf16(v + q * 8);
            } else if (row_ok) {
              __nv_bfloat16* a = p.aux_out + (long long)row * p.ld_aux_out + col0;
              if (full && vec8(a, p.ld_aux_out)) {
#pragma unroll
                for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(a)[q] = pack8_bf16(v + q * 8);
              } else {
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.N) a[j] = __float2bfloat16(v[j]);
              }
            }
          }
          if (p.act == ACT_RELU) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
          } else if (p.act == ACT_GELU) {
#pragma unroll
            for (int j = 0; j < 32; j += 2) gelu_tanh_pair(v[j], v[j + 1]);
          } else if (bwd) {
            uint4 x[4];
            if (tma_op) {
#pragma unroll
              for (int q = 0; q < 4; ++q) x[q] = *reinterpret_cast<const uint4*>(cs + sw128_offset(lane, half * 4 + q));
            } else {
              load32_bf16(x, p.aux_in + (long long)row * p.ld_aux_in + col0, p.ld_aux_in, full, row_ok ? p.N - col0 : 0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t w[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 f = unpack_bf16x2(w[i]);
                float* const d = v + q * 8 + i * 2;
                if (p.act == ACT_GELU_BWD) {
                  const float2 s = gelu_tanh_grad_pair(f);
                  d[0] *= s.x;
                  d[1] *= s.y;
                } else {
                  d[0] = f.x > 0.0f ? d[0] : 0.0f;
                  d[1] = f.y > 0.0f ? d[1] : 0.0f;
                }
              }
            }
          }
          if (p.residual) {
            if (tma_op && !bwd) {
#pragma unroll
              for (int q = 0; q < 4; ++q) add8_bf16(v + q * 8, *reinterpret_cast<const uint4*>(cs + sw128_offset(lane, half * 4 + q)));
            } else {
              uint4 x[4];
              load32_bf16(x, p.residual + (long long)row * p.ldr + col0, p.ldr, full, row_ok ? p.N - col0 : 0);
#pragma unroll
              for (int q = 0; q < 4; ++q) add8_bf16(v + q * 8, x[q]);
            }
          }
          if (p.use_tma_store == STORE_BF16) {
            // 32 rows x 64 columns (128-byte swizzle)
#pragma unroll
            for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(cs + sw128_offset(lane, half * 4 + q)) = pack8_bf16(v + q * 8);
          } else if (p.use_tma_store) {
            uint8_t* const fs = bufs + (blocks % CBUF) * 4096;
            if (lane == 0) tma_store_wait_read<CBUF - 1>();
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              *reinterpret_cast<float4*>(fs + sw128_offset(lane, q)) = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              const int bc = p.batch_stride_c ? b : 0;       // the parts of a split sum meet in the same place
              if (p.use_tma_store == STORE_FP32_ADD) tma_reduce_add_3d(&tmC.m[0], smem_u32(fs), col0, m0, bc);
              else tma_store_3d(&tmC.m[0], smem_u32(fs), col0, m0, bc);
              tma_store_commit();
            }
            ++blocks;
          } else if (row_ok) {
            const long long at0 = (long long)b * p.batch_stride_c + (long long)row * p.ldc + col0;
            if (p.out_fp32) {
              float* cp = reinterpret_cast<float*>(p.C) + at0;
              if (full && (p.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(cp) & 15) == 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  float4 o = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                  if (p.accumulate == 2) {  // split-K: several CTAs add into the same tile
                    atomicAdd(reinterpret_cast<float4*>(cp) + q, o);
                    continue;
                  }
                  if (p.accumulate) {
                    float4 old = reinterpret_cast<float4*>(cp)[q];
                    o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
                  }
                  reinterpret_cast<float4*>(cp)[q] = o;
                }
              } else {
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.N) {
                    if (p.accumulate == 2) atomicAdd(cp + j, v[j]); else cp[j] = p.accumulate ? cp[j] + v[j] : v[j];
                  }
              }
            } else {
              __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + at0;
              if (full && vec8(cp, p.ldc)) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  if (p.accumulate) add8_bf16(v + q * 8, reinterpret_cast<const uint4*>(cp)[q]);
                  reinterpret_cast<uint4*>(cp)[q] = pack8_bf16(v + q * 8);
                }
              } else {
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.N) {
                    float o = v[j];
                    if (p.accumulate) o += __bfloat162float(cp[j]);
                    cp[j] = __float2bfloat16(o);
                  }
              }
            }
          }
          if (half == 0 && tma_op) {
            // the block before this one has been handed over half a block's time ago: its place takes another operand
            if (lane == 0) tma_store_wait_read<0>();
            request();
          }
        }
        if (p.use_tma_store == STORE_BF16) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (tma_aux) tma_store_3d(&tmC.m[2], smem_u32(aux_block), n0 + g * 64, m0, 0);
            tma_store_3d(&tmC.m[0], smem_u32(cs), n0 + g * 64, m0, b);
            tma_store_commit();
          }
          ++blocks;
        }
      }
      if (!alive) break;
      if (held) release();
    }
    if (p.use_tma_store && lane == 0) tma_store_wait<0>();
  } else if (warp < 6) {
    // ------------------------------- epilogue warps, tensor-parallel variants ------------------------------
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    int iter = 0;
    // staging buffers per warp: two, and one in the 4-stage all-gather variant, whose push ring takes the upper half of the
    // staging area
    constexpr int CSB = (COMM == COMM_AG && STAGES == 4) ? 1 : 2;
    uint8_t* const cs_warp = smem + L::CSTAGE_OFFSET + quad * CSB * 4096;
    int store_seq = 0;          // TMA stores issued by this warp (selects the staging buffer)
    int tile_seq0 = 0;          // value of store_seq when the current tile started
    constexpr int kPubBatch = 3;
    int pend_owner[kPubBatch], pend_block[kPubBatch], n_pend = 0;   // RS: tiles stored, not yet published
    bool alive = true;
    bool saw_local = false;     // RS tracing: the first local tile has been stamped
    const bool tracer = (COMM != COMM_NONE) && cm.trace && quad == 2 && lane == 0;   // warp 2
    if (tracer) cm.trace[blockIdx.x * 4 + 0] = globaltimer_ns();
    if constexpr (COMM == COMM_RS) {
      // peers' staging areas are free once every peer has entered this launch
      bool ok = true;
      if (lane == 0)
        for (int q = 0; q < cm.g.world && ok; ++q)
          ok = wait_flag_ge(cm.g.signals[cm.g.rank] + cm.slot_enter + q, cm.g.epoch);
      alive = __all_sync(0xffffffffu, ok);
      if (!alive) {
        *abort_flag = 1;
        if (lane == 0) report_error(p.err, ERR_FLAG_TIMEOUT, 0xA602u);
      }
    }
    if (tracer) cm.trace[blockIdx.x * 4 + 1] = globaltimer_ns();
    for (int t = gemm_bid; t < total_tiles && alive; t += grid_stride, ++iter) {
      int b, tm, tn;
      map_tile<COMM>(t, tiles_m, tiles_n, tiles_per_batch, cm, b, tm, tn);
      const int m0 = tm * BM, n0 = tn * BN;
      const int acc = iter & 1;
      const uint32_t acc_phase = (iter >> 1) & 1;
      if (!mbar_wait_warp(smem_u32(&tfull_bar[acc]), acc_phase, abort_flag)) break;
      tc_fence_after();
      tile_seq0 = store_seq;
      const int row = m0 + quad * 32 + lane;
      const bool row_ok = row < p.M;
      void* c_ptr = p.C;
      long long c_base = (long long)b * p.batch_stride_c + (long long)row * p.ldc;
      int owner = 0;
      bool local_tile = false;
      int n_srcs = 0;             // RS local tile: staged partials + residual to add
      long long red_off = 0;      // element offset of this lane's row segment inside a source
      bool pf_valid = false;      // pf holds the first batch of the next column group
      uint4 pf[kRsBatch][4];
      const long long slot_stride = (long long)cm.rows_per_chunk * p.ldc;
      if constexpr (COMM == COMM_RS) {
        owner = m0 / cm.rows_per_chunk;
        local_tile = owner == cm.g.rank;
        if (local_tile) {
          if (tracer && !saw_local) cm.trace[(gridDim.x + blockIdx.x) * 4 + 0] = globaltimer_ns();
          // Everything this warp still owes its peers is published first: they wait for it before
          // they can finish, exactly as this rank is about to wait for them.
          if (lane == 0 && n_pend > 0) {
            if (p.use_tma_store) tma_store_wait<0>();
            fence_proxy_async_global();
            fence_sys();
            for (int i = 0; i < n_pend; ++i)
              red_relaxed_sys_add(cm.g.signals[pend_owner[i]] + cm.slot_done + pend_block[i], 1u);
            n_pend = 0;
          }
          // this rank owns these rows: wait until every peer's partial of the row block has landed,
          // then the column loop adds them (and the residual) and writes the final rows
          bool okc = true;
          if (lane == 0)
            okc = wait_flag_ge(cm.g.signals[cm.g.rank] + cm.slot_done + (m0 - owner * cm.rows_per_chunk) / BM,
                               cm.done_target);
          okc = __all_sync(0xffffffffu, okc);
          if (!okc) {
            *abort_flag = 1;
            if (lane == 0) report_error(p.err, ERR_FLAG_TIMEOUT, 0xA603u);
            break;
          }
          c_ptr = cm.rs_out;
          c_base = (long long)(row - owner * cm.rows_per_chunk) * p.ldc;
          if (tracer && !saw_local) {
            saw_local = true;
            cm.trace[(gridDim.x + blockIdx.x) * 4 + 1] = globaltimer_ns();
          }
          // Sources to add: the other ranks' staged partials (slot q of this rank's staging area), then
          // the residual.  The whole row segment goes to L2 now; the first batch of the first column
          // group is loaded before the accumulator is read, and every later group's first batch is
          // loaded while the previous group is converted and stored.
          n_srcs = cm.g.world - 1 + (cm.rs_residual ? 1 : 0);
          red_off = c_base + n0;
          if (row_ok) {
            const int lines = (min(BN, p.N - n0) * 2 + 127) / 128;
            for (int s_ = 0; s_ < n_srcs; ++s_)
              for (int l_ = 0; l_ < lines; ++l_) prefetch_l2(rs_src(cm, s_, slot_stride) + red_off + l_ * 64);
            pf_valid = n0 + 32 <= p.N;
            if (pf_valid) rs_load_batch(cm, slot_stride, 0, n_srcs, red_off, pf);
          }
        } else {
          c_ptr = cm.stage_peers[owner];
          c_base = ((long long)cm.g.rank * cm.rows_per_chunk + (row - owner * cm.rows_per_chunk)) * p.ldc;
        }
      }
      // TMA mode: after the second half of a 64-column chunk (or the last valid half) one lane
      // hands the warp's staged 32 x 64 block to the copy engine
      auto issue_store = [&](int c, int col0) {
        if ((c & 1) == 0 && col0 + 32 < p.N) return;
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const CUtensorMap* om = &tmC.m[COMM == COMM_RS ? owner : 0];
          const int r0 = (COMM == COMM_RS ? m0 - owner * cm.rows_per_chunk : m0) + quad * 32;
          tma_store_3d(om, smem_u32(cs_warp + (store_seq % CSB) * 4096),
                       n0 + (c >> 1) * 64, r0, b);
          tma_store_commit();
        }
        ++store_seq;
      };
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        const int col0 = n0 + c * 32;
        if (col0 >= p.N) break;  // uniform across the warp
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN + c * 32, r);
        tmem_ld_wait();
        if (p.use_tma_store && (c & 1) == 0 && store_seq >= CSB) {
          // the staging buffer about to be rewritten was handed to TMA CSB stores ago
          if (lane == 0) tma_store_wait_read<CSB - 1>();
          __syncwarp();
        }
        if (!row_ok) {
          // rows past M: nothing to compute; in TMA mode the warp still issues its store
          // (the copy clips rows and columns that fall outside the tensor)
          if (p.use_tma_store) issue_store(c, col0);
          continue;
        }
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
        const bool full = (col0 + 32 <= p.N);
        if constexpr (COMM == COMM_RS) {
          if (local_tile) {
            const long long off = red_off + c * 32;
            if (full) {
              if (!pf_valid) rs_load_batch(cm, slot_stride, 0, n_srcs, off, pf);
              rs_add_batch(0, n_srcs, pf, v);
              for (int s0 = kRsBatch; s0 < n_srcs; s0 += kRsBatch) {
                uint4 more[kRsBatch][4];
                rs_load_batch(cm, slot_stride, s0, n_srcs, off, more);
                rs_add_batch(s0, n_srcs, more, v);
              }
              pf_valid = (c + 1 < BN / 32) && (col0 + 64 <= p.N);
              if (pf_valid) rs_load_batch(cm, slot_stride, 0, n_srcs, off + 32, pf);
            } else {
              pf_valid = false;
              for (int s_ = 0; s_ < n_srcs; ++s_) {
                const __nv_bfloat16* src = rs_src(cm, s_, slot_stride) + off;
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.N) v[j] += __bfloat162float(src[j]);
              }
            }
          }
        }
        if (p.bias) {
          if (full && (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 u = __ldg(reinterpret_cast<const uint4*>(p.bias + col0) + q);
              const float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z), f3 = unpack_bf16x2(u.w);
              v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
              v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (full || col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
          }
        }
        if (p.aux_out) {
          __nv_bfloat16* a = p.aux_out + (long long)row * p.ld_aux_out + col0;
          if (full && (p.ld_aux_out & 7) == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 u;
              u.x = pack_bf16x2(v[q * 8 + 0], v[q * 8 + 1]);
              u.y = pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]);
              u.z = pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]);
              u.w = pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]);
              reinterpret_cast<uint4*>(a)[q] = u;
            }
          } else {
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) a[j] = __float2bfloat16(v[j]);
          }
        }
        if (p.act == ACT_RELU) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
        } else if (p.act == ACT_GELU) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
        } else if (p.act == ACT_GELU_BWD || p.act == ACT_RELU_BWD) {
          const __nv_bfloat16* a = p.aux_in + (long long)row * p.ld_aux_in + col0;
          float x[32];
          if (full && (p.ld_aux_in & 7) == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 u = reinterpret_cast<const uint4*>(a)[q];
              float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z),
                     f3 = unpack_bf16x2(u.w);
              x[q * 8 + 0] = f0.x; x[q * 8 + 1] = f0.y; x[q * 8 + 2] = f1.x; x[q * 8 + 3] = f1.y;
              x[q * 8 + 4] = f2.x; x[q * 8 + 5] = f2.y; x[q * 8 + 6] = f3.x; x[q * 8 + 7] = f3.y;
            }
          } else {
            for (int j = 0; j < 32; ++j) x[j] = (col0 + j < p.N) ? __bfloat162float(a[j]) : 0.0f;
          }
          if (p.act == ACT_GELU_BWD) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= gelu_tanh_grad(x[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = x[j] > 0.0f ? v[j] : 0.0f;
          }
        }
        if (p.residual) {
          const __nv_bfloat16* rs = p.residual + (long long)row * p.ldr + col0;
          if (full && (p.ldr & 7) == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 u = reinterpret_cast<const uint4*>(rs)[q];
              float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z),
                     f3 = unpack_bf16x2(u.w);
              v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
              v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
            }
          } else {
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) v[j] += __bfloat162float(rs[j]);
          }
        }
        if (p.use_tma_store) {
          // stage this warp's 32 rows x 64 columns (128-byte swizzle) and store them by TMA
          const int half = c & 1;
          uint8_t* cs = cs_warp + (store_seq % CSB) * 4096;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = pack_bf16x2(v[q * 8 + 0], v[q * 8 + 1]);
            o.y = pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]);
            o.z = pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]);
            o.w = pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]);
            *reinterpret_cast<uint4*>(cs + sw128_offset(lane, half * 4 + q)) = o;
          }
        } else if (p.out_fp32) {
          float* cp = reinterpret_cast<float*>(c_ptr) + c_base + col0;
          if (full && (p.ldc & 3) == 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              float4 o = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
              if (p.accumulate == 2) {  // split-K: several CTAs add into the same tile
                atomicAdd(reinterpret_cast<float4*>(cp) + q, o);
                continue;
              }
              if (p.accumulate) {
                float4 old = reinterpret_cast<float4*>(cp)[q];
                o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
              }
              reinterpret_cast<float4*>(cp)[q] = o;
            }
          } else {
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) cp[j] = p.accumulate ? cp[j] + v[j] : v[j];
          }
        } else {
          __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(c_ptr) + c_base + col0;
          if (full && (p.ldc & 7) == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (p.accumulate) {
                uint4 u = reinterpret_cast<const uint4*>(cp)[q];
                float2 f0 = unpack_bf16x2(u.x), f1 = unpack_bf16x2(u.y), f2 = unpack_bf16x2(u.z),
                       f3 = unpack_bf16x2(u.w);
                v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
                v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
              }
              uint4 o;
              o.x = pack_bf16x2(v[q * 8 + 0], v[q * 8 + 1]);
              o.y = pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]);
              o.z = pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]);
              o.w = pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]);
              reinterpret_cast<uint4*>(cp)[q] = o;
            }
          } else {
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) {
                float o = v[j];
                if (p.accumulate) o += __bfloat162float(cp[j]);
                cp[j] = __float2bfloat16(o);
              }
          }
        }
        if (p.use_tma_store) issue_store(c, col0);
      }
      // hand the accumulator back to the MMA warp
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      if constexpr (COMM == COMM_RS) {
        // Publish this warp's 32 rows to the owner (the counter counts warp arrivals, so no
        // CTA-wide barrier is needed).  Waiting for the stores of the tile just issued would put
        // an NVLink round trip into every tile, and so would a system-scope release per tile:
        // finished tiles are queued and published kPubBatch at a time behind one fence, after
        // the wait that leaves only the newest tile's store groups outstanding.
        if (lane == 0 && !local_tile) {
          if (p.use_tma_store) {
            if (n_pend == kPubBatch) {
              const int groups = store_seq - tile_seq0;      // bulk groups committed for this tile
              switch (groups) {
                case 0: tma_store_wait<0>(); break;
                case 1: tma_store_wait<1>(); break;
                case 2: tma_store_wait<2>(); break;
                case 3: tma_store_wait<3>(); break;
                default: tma_store_wait<4>(); break;
              }
              fence_proxy_async_global();
              fence_sys();
              for (int i = 0; i < n_pend; ++i)
                red_relaxed_sys_add(cm.g.signals[pend_owner[i]] + cm.slot_done + pend_block[i], 1u);
              n_pend = 0;
            }
            pend_owner[n_pend] = owner;
            pend_block[n_pend] = (m0 - owner * cm.rows_per_chunk) / BM;
            ++n_pend;
          } else {
            red_release_sys_add(cm.g.signals[owner] + cm.slot_done + (m0 - owner * cm.rows_per_chunk) / BM, 1u);
          }
        }
      }
    }
    if (p.use_tma_store && lane == 0) tma_store_wait<0>();
    if (tracer) cm.trace[blockIdx.x * 4 + 2] = globaltimer_ns();
    if constexpr (COMM == COMM_RS) {
      if (lane == 0 && n_pend > 0) {
        fence_proxy_async_global();
        fence_sys();
        for (int i = 0; i < n_pend; ++i)
          red_relaxed_sys_add(cm.g.signals[pend_owner[i]] + cm.slot_done + pend_block[i], 1u);
      }
    }

  } else if constexpr (COMM == COMM_AG) {
    // ---------------------------------------------------------------------------------------
    // All-gather: EVERY CTA pushes its 1/gridDim slice of this rank's shard while its other warps
    // run GEMM tiles (one SM sustains only ~20 GB/s of peer writes, so the push is spread over
    // all of them instead of a few dedicated CTAs).  A work item is one sub-chunk for one
    // destination; items go destination-major in ring order (rank-1, rank-2, ..., own buffer
    // last), so in every phase the W senders address W different receivers and a receiver gets
    // the chunks in the order its GEMM tiles consume them.  Warp 6 lane 0 drives bulk copies
    // local HBM → shared-memory ring → destination; warp 7 lane 0 adds one arrival per finished
    // item to the destination's counter, so the system-scope release never stalls the copies.
    // ---------------------------------------------------------------------------------------
    volatile int* s_done_items = reinterpret_cast<volatile int*>(tmem_slot + 2);
    volatile int* s_finished = reinterpret_cast<volatile int*>(tmem_slot + 3);
    const int W = cm.g.world, R = cm.g.rank;
    const int SUBS = cm.sub_per_chunk;
    // the copy into this rank's own gather buffer comes last and is skipped when the shard already lives there
    const int items = (cm.local_in_place ? W - 1 : W) * SUBS;
    auto dest_of = [&](int item) {
      const int q = item / SUBS;
      return q < W - 1 ? (R - 1 - q + W) % W : R;
    };
    if (warp == 7 && lane == 0) {
      int sent = 0;
      const uint64_t t0 = globaltimer_ns();
      for (;;) {
        const int fin = *s_finished;
        const int d = *s_done_items;
        if (sent < d) {
          // one fence for everything that completed since the last look, then plain atomics
          __threadfence_block();
          fence_proxy_async_global();
          fence_sys();
          for (; sent < d; ++sent)
            red_relaxed_sys_add(cm.g.signals[dest_of(sent)] + cm.slot_arrive + R * kMaxSubChunks + sent % SUBS, 1u);
        }
        if (sent >= items || (fin && sent >= *s_done_items)) break;
        if (globaltimer_ns() - t0 > (uint64_t)(W + 2) * wait_limit_ns()) break;   // the copy thread reports the cause
        __nanosleep(64);
      }
    } else if (warp == 6 && lane == 0) {
      bool ok = true;
      if (cm.trace) cm.trace[(gridDim.x + blockIdx.x) * 4 + 0] = globaltimer_ns();
      if (blockIdx.x == 0) {
        fence_sys();
        for (int q = 0; q < W; ++q) st_relaxed_sys(cm.g.signals[q] + cm.slot_enter + R, cm.g.epoch);
      }
      // peers must have left the previous launch that read this gather buffer
      for (int q = 0; q < W && ok; ++q) ok = wait_flag_ge(cm.g.signals[R] + cm.slot_enter + q, cm.g.epoch);
      if (cm.trace) cm.trace[(gridDim.x + blockIdx.x) * 4 + 1] = globaltimer_ns();
      if (!ok) {
        report_error(p.err, ERR_FLAG_TIMEOUT, 0xA600u);
      } else {
        // 3-stage variant (communication-bound shapes): 3 x 16 KB behind the barriers; 4-stage variant
        // (compute-bound shapes): 2 x 8 KB in the upper half of the output staging area
        constexpr int NB = (STAGES == 4) ? 2 : AG_RING_SLOTS;
        constexpr uint32_t CH = (STAGES == 4) ? 8192 : AG_RING_CHUNK;
        uint8_t* ring = (STAGES == 4) ? smem + L::CSTAGE_OFFSET + 16384 : smem + L::BAR_OFFSET + 256;
        uint64_t* cbar = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET + 128);
        const long long sub_bytes = (long long)(cm.rows_per_chunk / SUBS) * p.K * 2;
        long long slice = (sub_bytes + gridDim.x - 1) / gridDim.x;
        slice = (slice + 127) & ~127ll;
        const long long lo = min(sub_bytes, (long long)blockIdx.x * slice);
        const long long hi = min(sub_bytes, lo + slice);
        const int n_ch = (int)((hi - lo + CH - 1) / CH);     // chunks per item for this CTA (may be 0)
        if (n_ch == 0 || items == 0) {
          *s_done_items = items;                              // nothing to copy: the arrivals still count
        } else {
          volatile int local_abort = 0;
          for (int i = 0; i < NB; ++i) mbar_init(smem_u32(&cbar[i]), 1);
          fence_barrier_init();
          const char* src_base = reinterpret_cast<const char*>(cm.src_shard);
          const long long dst_base = (long long)R * cm.rows_per_chunk * p.K * 2;
          const int total = items * n_ch;
          auto chunk_of = [&](int c, int& item, uint32_t& sz) {
            item = c / n_ch;
            const long long o = lo + (long long)(c - item * n_ch) * CH;
            sz = (uint32_t)min((long long)CH, hi - o);
            return (long long)(item % SUBS) * sub_bytes + o;
          };
          auto issue_load = [&](int c) {
            int item;
            uint32_t sz;
            const long long off = chunk_of(c, item, sz);
            const int b = c % NB;
            mbar_arrive_expect_tx(smem_u32(&cbar[b]), sz);
            bulk_load_g2s(smem_u32(ring + b * CH), src_base + off, sz, smem_u32(&cbar[b]));
          };
          // one load ahead of the store being issued; a buffer is reloaded once the store that
          // used it has finished reading shared memory (NB - 1 stores may be in flight)
          issue_load(0);
          uint32_t phase_bits = 0;
          for (int c = 0; c < total; ++c) {
            const int b = c % NB;
            if (c + 1 < total) {
              if (c + 1 >= NB) tma_store_wait_read<NB - 2>();   // store c + 1 - NB has released its buffer
              issue_load(c + 1);
            }
            if (!mbar_wait(smem_u32(&cbar[b]), (phase_bits >> b) & 1u, &local_abort)) { ok = false; break; }
            phase_bits ^= (1u << b);
            int item;
            uint32_t sz;
            const long long off = chunk_of(c, item, sz);
            bulk_store_s2g(reinterpret_cast<char*>(cm.gather_peers[dest_of(item)]) + dst_base + off,
                           smem_u32(ring + b * CH), sz);
            tma_store_commit();
            if (c >= NB - 1) {
              tma_store_wait<NB - 1>();                       // every store up to chunk c - (NB - 1) is complete
              const int cc = c - (NB - 1);
              if (cc % n_ch == n_ch - 1) {
                fence_proxy_async_global();
                __threadfence_block();
                *s_done_items = cc / n_ch + 1;
                if (cm.trace && cc / n_ch + 1 == (W - 1) * SUBS)     // every remote store of this CTA has completed
                  cm.trace[(2 * gridDim.x + blockIdx.x) * 4 + 0] = globaltimer_ns();
              }
            }
          }
          tma_store_wait<0>();
          if (!ok) {
            report_error(p.err, ERR_MBAR_TIMEOUT, 0xA604u);
          } else {
            fence_proxy_async_global();
            __threadfence_block();
            *s_done_items = items;
          }
        }
      }
      if (cm.trace) cm.trace[(gridDim.x + blockIdx.x) * 4 + 2] = globaltimer_ns();
      __threadfence_block();
      *s_finished = 1;
    }
  }

  // ------------------------------- teardown -------------------------------------------
  if constexpr (COMM != COMM_NONE) {
    if (cm.trace && threadIdx.x == 64) cm.trace[blockIdx.x * 4 + 3] = globaltimer_ns();
  }
  tc_fence_before();
  __syncwarp();
  if constexpr (CG == 2) cluster_sync(); else __syncthreads();      // the pair's barriers and tensor memory outlive both CTAs' use
  if (*abort_flag) {
    if (threadIdx.x == 0) report_error(p.err, ERR_MBAR_TIMEOUT, 0x6E00u);
    // give copies that are still in flight a bounded time to land before smem is released
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, TMEM_COLS); else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// How the output leaves and the epilogue's operands arrive: tensor maps where leading dimensions and addresses allow them.
// Returns false after recording an error.
inline bool plan_epilogue(GemmParams& p, OutMaps& maps) {
  memset(&maps, 0, sizeof(maps));
  p.use_tma_store = STORE_DIRECT;
  p.operand_tma = p.aux_tma = 0;
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  auto bf16_map = [&](CUtensorMap* m, const void* base, long long ld, long long batch, long long stride) {
    const uint64_t dims[3] = {(uint64_t)p.N, (uint64_t)p.M, (uint64_t)batch};
    const uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)(batch > 1 ? stride : ld * p.M) * 2};
    const uint32_t box[3] = {64, 32, 1};
    return st::encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  const int per16 = p.out_fp32 ? 4 : 8;
  const long long batch = p.batch_stride_c ? p.batch : 1;      // without a stride every part of the batch has the same output
  if (p.ldc % per16 != 0 || !aligned(p.C) || p.batch_stride_c % per16 != 0 || p.batch_stride_c < 0) return true;
  if (p.out_fp32) {
    if (p.batch > 1 && batch == 1 && p.accumulate != 2) return true;
    const uint64_t dims[3] = {(uint64_t)p.N, (uint64_t)p.M, (uint64_t)batch};
    const uint64_t strides[2] = {(uint64_t)p.ldc * 4, (uint64_t)(batch > 1 ? p.batch_stride_c : p.ldc * p.M) * 4};
    const uint32_t box[3] = {32, 32, 1};
    p.use_tma_store = p.accumulate ? STORE_FP32_ADD : STORE_FP32;
    return st::encode_tmap(&maps.m[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, p.C, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  }
  if (p.accumulate || (p.batch > 1 && batch == 1)) return true;
  p.use_tma_store = STORE_BF16;
  if (!bf16_map(&maps.m[0], p.C, p.ldc, batch, p.batch_stride_c)) return false;
  const bool bwd = p.act == ACT_GELU_BWD || p.act == ACT_RELU_BWD;
  const __nv_bfloat16* operand = bwd ? p.aux_in : p.residual;
  const long long ld = bwd ? p.ld_aux_in : p.ldr;
  if (operand && (ld & 7) == 0 && ld >= p.N && aligned(operand)) {
    p.operand_tma = 1;
    if (!bf16_map(&maps.m[1], operand, ld, 1, 0)) return false;
  } else if (p.aux_out && (p.ld_aux_out & 7) == 0 && p.ld_aux_out >= p.N && aligned(p.aux_out)) {
    p.aux_tma = 1;
    if (!bf16_map(&maps.m[2], p.aux_out, p.ld_aux_out, 1, 0)) return false;
  }
  return true;
}
// Whether an operand of the epilogue arrives by TMA: it deserves more staging blocks per warp at the price of a stage of the
// operand ring (16384 x 3072 x 768 plus residual 82 us and 93).  Elsewhere the deeper ring is worth 2 to 4 %, most where large
// weights come from HBM.
inline bool staged_epilogue(const GemmParams& p) { return p.operand_tma != 0; }

// Tile width of a product.  A tile's main loop takes about c per K block (c2 from the 33rd on, where the start-up of the ring no
// longer counts) and its epilogue e, which runs beside the next tile's main loop; what does not overlap is the first main loop and
// the last epilogue:
//   time = a + (rounds - 1) max(main, e) + main + e
// in microseconds, fitted to 551 products of 64 to 16384 rows, 64 to 50304 columns and K of 64 to 16384 with every epilogue
// (large weights not in L2).  Narrow tiles lose throughput but fill the chip where wide ones leave SMs without a tile: 777 x 2048 x
// 8192 takes 38 us with 112 tiles of 128 x 128 and 50 with 56 of 128 x 256.
// Where the tiles are so few that two or four CTAs can share each, their K loops are split (launch_parts): the same product takes
// 31 us with two CTAs on each of 56 tiles; 128 x 2048 x 8192 20 and 39; 777 x 512 x 4608 13 in four parts and 20 in tiles of 64
// columns; 128 x 768 x 3072 9.8 and 13.8.  The exchange costs about 4 us, so a K of 768 stays whole (777 x 768 x 768: 8.6 and
// 7.2).  A cluster of four needs four SMs of one graphics processing cluster, and 33 such clusters are resident at once (a query of the
// occupancy; 74 of two): the rule takes 32 of 148 SMs / 4 = 37, as 36 took two rounds (128 x 4608 x 1536: 19 us against 11).  Parts
// are taken when they promise 4 % or more.  Their sums are added in a fixed order, and shorter chains are no further from 64 bits
// (relative error of fp32 outputs, whole and in parts: 128 x 2048 x 8192 9.1e-6 and 2.1e-6, 777 x 2048 x 8192 9.1e-6 and 4.4e-6, 128 x
// 768 x 3072 3.2e-6 and 0.7e-6).
// 128 x 256 and the pair come out within a few percent of one another over much of the range, timed alone; inside a training
// step, under the power limit, the pair is the faster one (the products of the 85 M byte model's step, K = 768 and 3072: 7.87 ms
// against 8.10), so it is taken where the model has it up to 11 % above.  Timed alone that preference changes little (plain outputs
// 0.3 % above the fastest form of each product on average with it and 0.5 without, GELU with its saved input 0.9 and 0.8).
// Over 528 products, captured and with K-major operands, the rule is above the fastest form by 0.3 % on average with plain outputs, 0.6
// with a residual, 0.9 with GELU and its saved input, nothing with GELU' and 0.1 with fp32 outputs, and by 4 % where fp32 outputs are
// added to; for single products by up to 29 % (306 x 1024 x 512, added: 8.6 us against 6.7).
enum TileEpilogue : int { EPI_PLAIN, EPI_OPERAND, EPI_GELU, EPI_GELU_BWD, EPI_FP32, EPI_FP32_ADD };
struct TileCost {
  double a, c, c2, e[6];
};
constexpr TileCost kTileCost[8] = {
    //  a    c      c2     plain operand gelu gelu'  fp32  added
    {2.86, 0.249, 0.224, {1.32, 2.20, 2.39, 3.38, 1.55, 4.13}},      // 128 x 64
    {1.67, 0.288, 0.248, {2.73, 3.79, 4.43, 5.53, 3.30, 5.98}},      // 128 x 128
    {0.00, 0.398, 0.327, {4.62, 7.10, 7.93, 10.70, 5.35, 7.66}},     // 128 x 256
    {1.00, 0.368, 0.282, {5.07, 6.67, 8.29, 10.52, 6.08, 9.23}},     // 256 x 256 on a pair
    {5.43, 0.258, 0.263, {1.79, 2.68, 3.30, 4.63, 2.03, 2.03}},      // 128 x 128, two K parts (c, c2 per block of a part)
    {5.26, 0.287, 1.179, {2.38, 3.27, 3.83, 5.23, 2.75, 2.75}},      // 128 x 128, four
    {7.34, 0.298, 0.415, {1.60, 3.51, 4.16, 7.52, 2.25, 2.25}},      // 128 x 256, two
    {7.13, 0.360, 0.402, {2.85, 4.79, 5.46, 8.90, 3.58, 3.58}}};     // 128 x 256, four
struct TileChoice {
  int bn;
  bool pair;
  int parts;      // CTAs that share the K blocks of a tile
  double us;      // modelled time
};
inline TileChoice choose_tile(long long M, long long N, long long K, long long batch, int ctas, TileEpilogue epi, bool may_split) {
  const double kb = (double)((K + BK - 1) / BK);
  auto tiles = [&](int bm, int bn) { return ((M + bm - 1) / bm) * ((N + bn - 1) / bn) * batch; };
  auto cost = [&](const TileCost& t, int bm, int bn, long long at_once, double blocks) {
    const double main = t.c * (blocks < 32 ? blocks : 32) + t.c2 * (blocks > 32 ? blocks - 32 : 0), e = t.e[epi];
    return t.a + (double)((tiles(bm, bn) + at_once - 1) / at_once - 1) * (main > e ? main : e) + main + e;
  };
  TileChoice best{64, false, 1, cost(kTileCost[0], BM, 64, ctas, kb)};
  auto take = [&](int bn, bool pair, int parts, double us) {
    if (us <= best.us) best = {bn, pair, parts, us};
  };
  if (N > 64) take(128, false, 1, cost(kTileCost[1], BM, 128, ctas, kb));
  if (N > 128) take(256, false, 1, cost(kTileCost[2], BM, 256, ctas, kb));
  if (N > 128 && M > BM && ctas >= 2) take(256, true, 1, 0.9 * cost(kTileCost[3], 2 * BM, 256, ctas / 2, kb));
  if (may_split && N > 64)
    for (int f = 0; f < 4; ++f) {
      const int bn = f < 2 ? 128 : 256, parts = f & 1 ? 4 : 2, at_once = parts == 2 ? ctas / 2 : ctas * 7 / 32;
      if (N > bn / 2 && kb >= 4 * parts && tiles(BM, bn) <= at_once) take(bn, false, parts, 1.04 * cost(kTileCost[4 + f], BM, bn, at_once, kb / parts));
    }
  return best;
}

// Launch of the CTA-pair form: an even grid of at most one CTA per SM, in clusters of two.
template <bool A_MN, bool B_MN, int STAGES, int SETS = 2>
int launch_pair_ring(const CUtensorMap& tmA, const CUtensorMap& tmB, const OutMaps& tmC, const GemmParams& p, cudaStream_t stream) {
  constexpr int BN = 256;
  using L = SmemLayout<BN / 2, STAGES, 0, SETS>;
  auto kern = gemm_bf16_kernel<BN, STAGES, A_MN, B_MN, COMM_NONE, 2, 1, SETS>;
  static bool configured[st::kMaxDevices] = {false};   // the attribute is per device
  const int dev = st::current_device();
  if (!configured[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    configured[dev] = true;
  }
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN) * p.batch;
  const int pairs = st::sm_count() / 2;
  GemmComm none{};
  ST_CUDA_CHECK(st::chained(kern, 2 * (tiles < pairs ? tiles : pairs), num_threads(SETS), L::TOTAL, stream, 2)(tmA, tmB, tmC, tmA, p, none));
  return ST_OK;
}

template <bool A_MN, bool B_MN>
int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const OutMaps& tmC, const GemmParams& p, cudaStream_t stream) {
  // With operands, a saved pre-activation or GELU the epilogue of a tile is longer than the main loop of a short K.  A third set of
  // warps shares it then, with four ring stages and two staging blocks per warp where anything is staged beside the output.  us, two
  // sets and three (captured): 16384 x 3072 x 768 with GELU' 135 and 111, GELU and its saved input 123 and 101, GELU alone 83 and 76,
  // plus residual 80 and 78.  Where the longer main loop makes the ring matter more depends on the epilogue: GELU' 141 and 135 at K =
  // 1536, 164 and 164 at 2048, 226 and 231 at 3072; GELU and its saved input 132 and 130, 158 and 163; GELU alone equal from 1280 on;
  // a residual 92 and 90 at 1024, but 103 and 106 at 1280 and 118 and 122 at 1536.  One line for all of them lies where GELU', the
  // longest, still gains.  A bare output gains nothing (58.2 and 58.2).
  if constexpr (!A_MN) {
    const bool staged = p.operand_tma || p.aux_tma;
    if (p.K <= 1536 && staged) return launch_pair_ring<false, B_MN, 4, 3>(tmA, tmB, tmC, p, stream);
    if (p.K <= 1536 && p.act == ACT_GELU) return launch_pair_ring<false, B_MN, 5, 3>(tmA, tmB, tmC, p, stream);
    if (staged_epilogue(p)) return launch_pair_ring<false, B_MN, 5>(tmA, tmB, tmC, p, stream);
  }
  return launch_pair_ring<A_MN, B_MN, 6>(tmA, tmB, tmC, p, stream);
}

// Launch of the K-part form: a cluster of KS CTAs per tile.
template <int BN, int STAGES, int KS, bool A_MN, bool B_MN>
int launch_parts_of(const CUtensorMap& tmA, const CUtensorMap& tmB, const OutMaps& tmC, const GemmParams& p, cudaStream_t stream) {
  using L = SmemLayout<BN, STAGES>;
  auto kern = gemm_bf16_kernel<BN, STAGES, A_MN, B_MN, COMM_NONE, 1, KS>;
  static bool configured[st::kMaxDevices] = {false};   // the attribute is per device
  const int dev = st::current_device();
  if (!configured[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
    configured[dev] = true;
  }
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.batch;
  GemmComm none{};
  ST_CUDA_CHECK(st::chained(kern, KS * tiles, NUM_THREADS, L::TOTAL, stream, KS)(tmA, tmB, tmC, tmA, p, none));
  return ST_OK;
}
template <bool A_MN, bool B_MN>
int launch_parts(int bn, int parts, const CUtensorMap& tmA, const CUtensorMap& tmB, const OutMaps& tmC, const GemmParams& p, cudaStream_t stream) {
  if (bn == 128) return parts == 2 ? launch_parts_of<128, 5, 2, A_MN, B_MN>(tmA, tmB, tmC, p, stream) : launch_parts_of<128, 5, 4, A_MN, B_MN>(tmA, tmB, tmC, p, stream);
  return parts == 2 ? launch_parts_of<256, 4, 2, A_MN, B_MN>(tmA, tmB, tmC, p, stream) : launch_parts_of<256, 4, 4, A_MN, B_MN>(tmA, tmB, tmC, p, stream);
}

}  // namespace gemm
}  // namespace st
