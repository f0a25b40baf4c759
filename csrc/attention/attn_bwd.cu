// Attention backward (dQ, dK, dV) on sm_100a tensor cores.
//
// Three launches:
//   1. delta[b,h,s] = sum_d O·dO                          (one warp per row)
//   2. dK/dV pass (MODE_KV): one CTA owns a 128-row KV tile of one (batch, head) and walks the
//      query tiles that attend to it.  Per query tile, four tcgen05 GEMMs:
//          S  = Q·Kᵀ, dP = dO·Vᵀ                          (TMEM, fp32)
//          P  = exp2(S·c − lse), dS = P∘(dP − delta)      (registers → bf16 in shared memory)
//          dK += dSᵀ·Q, dV += Pᵀ·dO                       (TMEM accumulators that live across tiles)
//      Pᵀ and dSᵀ need no transposition pass: the bytes written for the K-major operand
//      (rows = queries) are read again through an MN-major descriptor.
//   3. dQ pass (MODE_Q): one CTA owns a 128-row query tile and walks the KV tiles it attends to:
//          S, dP as above; dS → shared memory; dQ += dS·K  (TMEM accumulator across KV tiles)
//      and writes dQ once, scaled, as bf16.
// Recomputing S and dP in the dQ pass costs two extra GEMMs per tile pair, but no pass needs more than 512 TMEM columns minus
// one operand, which lets both software-pipeline: the element-wise phase is split in two (P from S, then dS from dP), S of the
// next tile is issued as soon as this tile's S has been read, and dP of the next tile right after this tile's accumulate GEMMs,
// so the tensor pipe works while the element-wise warps do.  At head_dim 128 S, dP, dV and dK take all 512 columns; dQ of a pair could
// only have dP's between the read of dP and dP of the next tile, with its drain between two tiles and eight fp32 sums for sixteen
// KV tiles.  That form has not been built, so how it compares is not known.
// At head_dim 64 with up to eight KV tiles, one pass does it all (MODE_ONE, launches 2 and 3 in one): dV, dK and two tiles of
// dQ fit the tensor memory, dQ[q, d] = dS·K of a pair is drained while the next pair's GEMMs run and added by TMA to fp32 sums in
// memory, and a last pass rounds them.  A sum receives the parts of two KV tiles only, in whatever order they come, so that the
// result does not depend on it: an order kept by counters made every CTA wait for the one before it (170 us where the
// unordered form takes 120).  us for everything after the forward, two passes and one: 96 contexts of 500 to 1000 keys 197 and
// 160; 384 heads of 512, causal, 165 and 140.
// Gradients leave by TMA: with a row per lane a store instruction touched 32 lines, 4 us per work item.
// Warp 16 is the TMA producer (two stationary tiles once; the streamed pair through a ring),
// warp 17 issues the MMAs and owns TMEM, warps 0-15 do the element-wise work with four threads
// per row (with two, the element-wise phase was latency-bound: 2 warps per scheduler cannot hide
// the TMEM-load and MUFU latencies).
//
// The reference has no attention backward; the oracle is PyTorch autograd of the fp32 math.
#include "../common/host.h"
#include "../common/ptx.cuh"

namespace st {
bool encode_bshd_tmap(CUtensorMap* out, const void* base, int B, int S, int H, int D,
                      long long sb, long long ss, long long sh, int box_rows);
bool encode_out_tmap(CUtensorMap* out, const void* base, bool f32, int B, int S, int H, int D, long long sb, long long ss, long long sh);
int attn_key_bias(const float* kb, long long kb_sb, long long kb_sh, const int* lengths, float* ws, int B, int H, int Sk,
                  long long* out_sb, long long* out_sh, cudaStream_t stream);
}

namespace {
using namespace st;

constexpr int BLK = 128;
constexpr int EW_WARPS = 16;                       // element-wise warps: four threads per row, 32 key columns each
constexpr int EW_THREADS = EW_WARPS * 32;
constexpr int NUM_THREADS = EW_THREADS + 64;       // + TMA producer warp + MMA warp
constexpr int MODE_KV = 0, MODE_Q = 1, MODE_ONE = 2;
// KV tiles up to which the one-pass form is taken: its sums of dQ take half as many times the size of dQ in fp32.
constexpr int kOnePassTiles = 8;
constexpr int kQueueFloats = 4;      // the work queue, behind the sums: before them it would move them off their 512-byte blocks (1 % slower)
// Biases: none; a bias per (query, key) among them, read and compared per element; key bias and length only, as padded rows
// in the log2 domain (minus infinity where masked): 16-byte loads, no comparisons.
constexpr int BIAS_NONE = 0, BIAS_FULL = 1, BIAS_KEYS = 2;

struct AttnBwdParams {
  const float* lse;
  const float* delta;
  int B, H, Sq, Sk;
  float scale, scale_log2;
  int causal;
  unsigned* err;
  // optional additive biases and valid lengths, as in the forward kernel (null = absent)
  const float* key_bias;
  const float* attn_bias;
  const int* lengths;
  long long kb_sb, kb_sh, ab_sb, ab_sh, ab_sq;
  const float* kb_pad;          // BIAS_KEYS
  long long kp_sb, kp_sh;
  int grad_f32;                 // dQ, dK and dV are fp32
  struct Grad {
    void* p;
    long long sb, ss, sh;       // in elements
  } dq, dk, dv;                 // where the lanes store their own rows
  unsigned* queue;              // items drawn beyond the first of every CTA, or null
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// dQ, dK and dV in boxes of 32 rows and 64 bytes
struct GradMaps {
  CUtensorMap dq, dk, dv;
};

template <int D, int MODE, int BIAS>
struct BwdSmem {
  static_assert(MODE != MODE_ONE || D == 64, "dV, dK and two dQ tiles fit the tensor memory at head_dim 64 only");
  static constexpr int TILE = BLK * D * 2;
  static constexpr int P_TILE = BLK * BLK * 2;
  // streamed tiles: stream A is Q (dK/dV pass) or K (dQ pass), stream B is dO or V.  The A tile is read by
  // the first GEMM of an iteration (S) and by the last one (dK or dQ), so it lives for more than a whole
  // iteration; the B tile is released early (after dV, or right after dP in the dQ pass).  The dK/dV pass
  // has room for three streamed tiles next to K, V, P and dS: two A, one B.  The dQ pass has no P buffer:
  // three A (with two, the issuer measured 0.47 us per iteration waiting for K), one B.
  // One pass: K is read until the item's last GEMM, so the stationary pair is double-buffered.
  static constexpr int NA = MODE == MODE_Q ? 3 : 2;
  static constexpr int NB = 1;
  static constexpr int NS = MODE == MODE_ONE ? 2 : 1;
  static constexpr int STAT0_OFF = 0;                  // K, or Q (MODE_Q)
  static constexpr int STAT1_OFF = STAT0_OFF + TILE;   // V, or dO (MODE_Q)
  static constexpr int A_OFF = 2 * NS * TILE;
  static constexpr int B_OFF = A_OFF + NA * TILE;
  static constexpr int DS_OFF = B_OFF + NB * TILE;
  static constexpr int P_OFF = DS_OFF + P_TILE;        // not in MODE_Q
  // Gradients leave by TMA, 2 KB per warp at a time; at head_dim 128 they are staged in the dS tile, which is idle then.  With a bias per
  // (query, key) at head_dim 64 the lanes store their own rows: 32 KB for staging would leave half as much L1, through which they read
  // the bias (us, 22 contexts of 504, 16 heads, causal: 450 staged, 344 from the lanes; 2 of 1738, 8 heads, 353 and 262), and staged in
  // the dS tile contexts of up to 32 queries wait for it, 13 % of their time.
  static constexpr int STG = 2048;
  static constexpr bool LANES = D == 64 && BIAS == BIAS_FULL;
  static constexpr bool OWN_STG = D == 64 && !LANES;
  static constexpr int STG_OFF = OWN_STG ? P_OFF + (MODE == MODE_Q ? 0 : P_TILE) : DS_OFF;
  static constexpr int BAR_OFF = P_OFF + (MODE == MODE_Q ? 0 : P_TILE) + (OWN_STG ? EW_WARPS * STG : 0);
  static constexpr int TOTAL = BAR_OFF + 320;
  static_assert(TOTAL <= 232448 && EW_WARPS * STG <= P_TILE, "shared memory");
};

// 16 bytes of eight values → bf16, written at the swizzled position of (row r, 16-byte chunk c16)
__device__ __forceinline__ void store8_bf16(uint8_t* tile, int r, int c16, const float* v) {
  uint4 u;
  u.x = pack_bf16x2(v[0], v[1]); u.y = pack_bf16x2(v[2], v[3]);
  u.z = pack_bf16x2(v[4], v[5]); u.w = pack_bf16x2(v[6], v[7]);
  *reinterpret_cast<uint4*>(tile + sw128_offset(r, c16)) = u;
}

template <int D, int MODE, int BIAS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ GradMaps tmG, const AttnBwdParams p) {
  using L = BwdSmem<D, MODE, BIAS>;
  constexpr int KB = D / 64;
  constexpr int NA = L::NA, NB = L::NB;
  // TMEM columns.  MODE_KV: S, dP, dV, dK.  MODE_Q: S, dP (even tiles), dQ, dP (odd tiles).
  // MODE_ONE: S, dP, dV, dK, dQ of even and of odd tiles.
  constexpr bool KV = MODE != MODE_Q;            // the CTA owns keys
  constexpr uint32_t S_COL = 0, DP_COL = 128, ACC0_COL = 256, ACC1_COL = MODE == MODE_ONE ? 320 : 384, DQ_COL = 384;
  constexpr uint32_t TMEM_COLS = 512;

  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) report_error(p.err, ERR_BOUNDS, 0xA7B1u);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* stat_full = bars;          // 1
  uint64_t* a_full = bars + 1;         // 3
  uint64_t* a_empty = bars + 4;        // 3
  uint64_t* b_full = bars + 7;         // 1
  uint64_t* b_empty = bars + 8;        // 1
  uint64_t* s_full = bars + 9;         // S of tile n is in TMEM
  uint64_t* dp_full = bars + 10;       // 2: dP of tile n is in TMEM (barrier n & 1)
  uint64_t* s_free = bars + 12;        // one arrival per element-wise warp: S of tile n has been read (MODE_KV: and P is in shared memory)
  uint64_t* pds_full = bars + 13;      // one arrival per element-wise warp: dS of tile n is in shared memory, dP has been read
  uint64_t* ds_free = bars + 14;       // MODE_Q: the dQ GEMM of tile n has finished reading dS
  uint64_t* acc_done = bars + 15;      // every GEMM of the current work item has completed
  uint64_t* stat_empty = bars + 16;    // the last S / dP GEMM of the work item has read the stationary tiles
  uint64_t* acc_free = bars + 17;
  uint64_t* p_ready = bars + 18;       // MODE_KV, one arrival per warp: P of tile n is in shared memory
  uint64_t* p_free = bars + 19;        // MODE_KV: the dV GEMM of tile n has finished reading P
  // acc_free: one arrival per warp: the accumulators of the work item have been read out
  uint64_t* stg_free = bars + 20;      // one arrival per warp: the dS tile no longer holds gradients on their way out
  uint64_t* dq_full = bars + 21;       // 2, MODE_ONE: dQ of tile n is in TMEM (barrier n & 1)
  uint64_t* dq_free = bars + 23;       // 2, MODE_ONE, one arrival per warp: it has been read
  uint64_t* stat_full1 = bars + 25;    // stat_full and stat_empty of the second stationary pair (MODE_ONE)
  uint64_t* stat_empty1 = bars + 26;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* item_full = bars + 29;     // 2: the next work item's index has been drawn
  uint64_t* item_empty = bars + 31;    // 2, one arrival per element-wise warp and the issuer: it has been read
  volatile int* item_slot = reinterpret_cast<volatile int*>(bars + 33);      // 2

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_q = (p.Sq + BLK - 1) / BLK;
  const int n_kv = (p.Sk + BLK - 1) / BLK;
  // Persistent CTAs: work item w = (owned tile, head, batch), tile-major so that under a causal mask
  // the long items come first; CTA c takes items c, c + gridDim.x, ..., or item c and then, one at a time, those that nobody has
  // taken yet (p.queue): with valid lengths the items differ by a factor of two, and 96 contexts of 500 to 1000 keys leave the
  // longest CTA of a fixed distribution 50 % behind the mean, of a drawn one 18 %.  Barrier phases run on over
  // the items (g counts streamed tiles, it counts items), so TMEM, the barriers and the pipelines
  // are set up once and the loads of the next item overlap the tail of the current one.
  const int hb = p.H * p.B;
  const int total_items = (KV ? n_kv : n_q) * hb;
  struct Item { int own, h, b, t_begin, n_iter; };
  auto item_at = [&](int w) {
    Item I;
    const int idx = w / hb, rem = w - idx * hb;
    I.own = KV ? idx : n_q - 1 - idx;
    I.h = rem % p.H;
    I.b = rem / p.H;
    I.t_begin = KV ? (p.causal ? I.own : 0) : 0;
    int t_end = KV ? n_q : (p.causal ? min(I.own + 1, n_kv) : n_kv);
    if (BIAS != BIAS_NONE && p.lengths) {      // keys and queries from the valid length on contribute nothing
      const int live = (max(0, min(p.Sk, p.lengths[I.b])) + BLK - 1) / BLK;
      t_end = I.own < live ? min(t_end, live) : 0;
    }
    I.n_iter = max(t_end - I.t_begin, 0);
    return I;
  };

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(stat_full), 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(smem_u32(&a_full[s]), 1);
      mbar_init(smem_u32(&a_empty[s]), 1);
    }
    mbar_init(smem_u32(b_full), 1);
    mbar_init(smem_u32(b_empty), 1);
    mbar_init(smem_u32(&dp_full[0]), 1);
    mbar_init(smem_u32(&dp_full[1]), 1);
    mbar_init(smem_u32(p_ready), EW_WARPS);
    mbar_init(smem_u32(p_free), 1);
    mbar_init(smem_u32(s_full), 1);
    mbar_init(smem_u32(s_free), EW_WARPS);        // one arrival per warp: 512 arrivals on one word cost ~0.5 us
    mbar_init(smem_u32(pds_full), EW_WARPS);
    mbar_init(smem_u32(ds_free), 1);
    mbar_init(smem_u32(acc_done), 1);
    mbar_init(smem_u32(stat_empty), 1);
    mbar_init(smem_u32(acc_free), EW_WARPS);
    mbar_init(smem_u32(stg_free), EW_WARPS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&dq_full[i]), 1);
      mbar_init(smem_u32(&dq_free[i]), EW_WARPS);
    }
    mbar_init(smem_u32(stat_full1), 1);
    mbar_init(smem_u32(stat_empty1), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&item_full[i]), 1);
      mbar_init(smem_u32(&item_empty[i]), EW_WARPS + 1);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == EW_WARPS + 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_begin();      // set up beside the previous kernel's end; global memory is touched from here on

  if (warp == EW_WARPS) {
    // ---------------------------- TMA producer -----------------------------------------
    if (lane == 0) {
      const CUtensorMap* st0 = KV ? &tmK : &tmQ;
      const CUtensorMap* st1 = KV ? &tmV : &tmdO;
      const CUtensorMap* ma = KV ? &tmQ : &tmK;
      const CUtensorMap* mb = KV ? &tmdO : &tmV;
      int g = 0, it = 0;
      bool ok = true;
      auto next = [&](int w, int k) {      // draws the item after the k-th one and hands its index to the other warps
        if (!p.queue) return w + (int)gridDim.x;
        if (!mbar_wait(smem_u32(&item_empty[k & 1]), ((k >> 1) & 1) ^ 1u, abort_flag)) return total_items;
        const int n = (int)(gridDim.x + atomicAdd(p.queue, 1u));
        item_slot[k & 1] = n;
        mbar_arrive(smem_u32(&item_full[k & 1]));
        return n;
      };
      for (int w = blockIdx.x, k = 0; w < total_items && ok; w = next(w, k++)) {
        const Item I = item_at(w);
        if (I.n_iter == 0) continue;
        const int pair = it % L::NS;
        if (!(ok = mbar_wait(smem_u32(pair ? stat_empty1 : stat_empty), ((it / L::NS) & 1) ^ 1u, abort_flag))) break;
        const uint32_t sb = smem_u32(pair ? stat_full1 : stat_full);
        uint8_t* const stat = smem + pair * 2 * L::TILE;
        mbar_arrive_expect_tx(sb, 2 * L::TILE);
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
          tma_load_4d(smem_u32(stat + L::STAT0_OFF + kb * (BLK * 128)), st0, sb, kb * 64, I.h, I.own * BLK, I.b);
          tma_load_4d(smem_u32(stat + L::STAT1_OFF + kb * (BLK * 128)), st1, sb, kb * 64, I.h, I.own * BLK, I.b);
        }
        for (int n = 0; n < I.n_iter && ok; ++n, ++g) {
          const int row0 = (I.t_begin + n) * BLK;
          {
            const int slot = g % NA;
            if (!(ok = mbar_wait(smem_u32(&a_empty[slot]), ((g / NA) & 1) ^ 1u, abort_flag))) break;
            const uint32_t fb = smem_u32(&a_full[slot]);
            mbar_arrive_expect_tx(fb, L::TILE);
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
              tma_load_4d(smem_u32(smem + L::A_OFF + slot * L::TILE + kb * (BLK * 128)), ma, fb, kb * 64, I.h, row0, I.b);
          }
          {
            const int slot = g % NB;
            if (!(ok = mbar_wait(smem_u32(&b_empty[slot]), ((g / NB) & 1) ^ 1u, abort_flag))) break;
            const uint32_t fb = smem_u32(&b_full[slot]);
            mbar_arrive_expect_tx(fb, L::TILE);
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
              tma_load_4d(smem_u32(smem + L::B_OFF + slot * L::TILE + kb * (BLK * 128)), mb, fb, kb * 64, I.h, row0, I.b);
          }
        }
        ++it;
      }
    }
  } else if (warp == EW_WARPS + 1) {
    // ---------------------------- MMA issuer -------------------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BLK, BLK, false, false);   // S, dP
      constexpr uint32_t idesc_t = make_idesc_bf16(BLK, D, true, true);       // dV, dK
      constexpr uint32_t idesc_q = make_idesc_bf16(BLK, D, false, true);      // dQ
      constexpr uint32_t HI = smem_desc_hi(1024);
      // descriptor low words of every tile: K-major view (16-byte leading offset) and MN-major view
      // (64-column blocks BLK*128 bytes apart); a K step adds a constant
      const uint32_t st0_first = smem_desc_lo(smem_u32(smem + L::STAT0_OFF), 16);
      const uint32_t st1_first = smem_desc_lo(smem_u32(smem + L::STAT1_OFF), 16);
      uint32_t st0_k = st0_first, st1_k = st1_first;
      const uint32_t k_mn_first = smem_desc_lo(smem_u32(smem + L::STAT0_OFF), BLK * 128);
      const uint32_t ds_k = smem_desc_lo(smem_u32(smem + L::DS_OFF), 16);
      const uint32_t ds_mn = smem_desc_lo(smem_u32(smem + L::DS_OFF), BLK * 128);
      const uint32_t p_mn = smem_desc_lo(smem_u32(smem + L::P_OFF), BLK * 128);
      auto a_k = [&](int n) { return smem_desc_lo(smem_u32(smem + L::A_OFF + (n % NA) * L::TILE), 16); };
      auto a_mn = [&](int n) { return smem_desc_lo(smem_u32(smem + L::A_OFF + (n % NA) * L::TILE), BLK * 128); };
      auto b_k = [&](int n) { return smem_desc_lo(smem_u32(smem + L::B_OFF + (n % NB) * L::TILE), 16); };
      auto b_mn = [&](int n) { return smem_desc_lo(smem_u32(smem + L::B_OFF + (n % NB) * L::TILE), BLK * 128); };
      auto wait_a = [&](int n) { return mbar_wait(smem_u32(&a_full[n % NA]), (n / NA) & 1, abort_flag); };
      auto wait_b = [&](int n) { return mbar_wait(smem_u32(&b_full[n % NB]), (n / NB) & 1, abort_flag); };
      // S = Q·Kᵀ and dP = dO·Vᵀ: both operands K-major, D/16 K steps
      auto issue_sdp = [&](uint32_t col, uint32_t a_lo, uint32_t b_lo) {
#pragma unroll
        for (int kb = 0; kb < KB; ++kb)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t off = (kb * (BLK * 128) + k * 32) >> 4;
            umma_bf16_ss_split(tmem_base + col, a_lo + off, HI, b_lo + off, HI, idesc_s, (kb | k) != 0 ? 1u : 0u);
          }
      };
      // accumulate GEMMs over the 128 rows of the streamed tile: A and B read through MN-major views
      auto issue_acc_mn = [&](uint32_t col, uint32_t a_lo, uint32_t b_lo, bool acc_first) {
#pragma unroll
        for (int kk = 0; kk < BLK / 16; ++kk) {
          const uint32_t off = (kk * (16 * 128)) >> 4;
          umma_bf16_ss_split(tmem_base + col, a_lo + off, HI, b_lo + off, HI, idesc_t, (acc_first || kk != 0) ? 1u : 0u);
        }
      };
      auto issue_s = [&](int n) {
        if (KV) issue_sdp(S_COL, a_k(n), st0_k); else issue_sdp(S_COL, st0_k, a_k(n));
        umma_commit(smem_u32(s_full));
      };
      auto issue_dp = [&](int n) {
        const uint32_t col = (MODE == MODE_Q && (n & 1)) ? ACC1_COL : DP_COL;
        if (KV) issue_sdp(col, b_k(n), st1_k); else issue_sdp(col, st1_k, b_k(n));
        umma_commit(smem_u32(&dp_full[n & 1]));
        if (MODE == MODE_Q) umma_commit(smem_u32(&b_empty[n % NB]));   // V is only needed by dP
      };
      int g = 0, it = 0;
      bool ok = true;
      auto next = [&](int w, int k) {
        if (!p.queue) return w + (int)gridDim.x;
        if (!mbar_wait(smem_u32(&item_full[k & 1]), (k >> 1) & 1, abort_flag)) return total_items;
        const int n = item_slot[k & 1];
        mbar_arrive(smem_u32(&item_empty[k & 1]));
        return n;
      };
      for (int w = blockIdx.x, k = 0; w < total_items && ok; w = next(w, k++)) {
        const Item I = item_at(w);
        if (I.n_iter == 0) continue;
        // prologue: S and dP of the item's first tile.  Their TMEM columns are free: every iteration,
        // the previous item's last one included, waits for s_free and pds_full.
        const int stat = it % L::NS;
        const uint32_t stat_off = (stat * 2 * L::TILE) >> 4;
        st0_k = st0_first + stat_off;
        st1_k = st1_first + stat_off;
        if (!(ok = mbar_wait(smem_u32(stat ? stat_full1 : stat_full), (it / L::NS) & 1, abort_flag))) break;
        if (!(ok = wait_a(g))) break;
        tc_fence_after();
        issue_s(g);
        if (!(ok = wait_b(g))) break;
        tc_fence_after();
        issue_dp(g);
        for (int n = 0; n < I.n_iter && ok; ++n, ++g) {
          const bool more = n + 1 < I.n_iter;
          // every S / dP GEMM of the item has been issued: the stationary tiles can be replaced
          // as soon as those complete
          if (MODE != MODE_ONE && !more) umma_commit(smem_u32(stat_empty));
          if (!(ok = mbar_wait(smem_u32(s_free), g & 1, abort_flag))) break;
          // the first accumulate GEMM of an item overwrites accumulators that the element-wise warps
          // may still be reading out for the previous item
          if (n == 0 && it > 0 && !(ok = mbar_wait(smem_u32(acc_free), (it - 1) & 1, abort_flag))) break;
          tc_fence_after();
          if (more) {
            // S of the next tile, as soon as this tile's S has been read
            if (!(ok = wait_a(g + 1))) break;
            tc_fence_after();
            issue_s(g + 1);
            if (MODE == MODE_Q) {
              // dP of the next tile goes to the other dP buffer, read last by tile g-1
              if (!(ok = wait_b(g + 1))) break;
              tc_fence_after();
              issue_dp(g + 1);
            }
          }
          if (KV) {
            // dV[kv, d] += sum_q P[q, kv] dO[q, d], once P has been stored (S of the next tile is already
            // running: the element-wise warps release S before they convert and store P)
            if (!(ok = mbar_wait(smem_u32(p_ready), g & 1, abort_flag))) break;
            tc_fence_after();
            issue_acc_mn(ACC0_COL, p_mn, b_mn(g), n != 0);
            umma_commit(smem_u32(&b_empty[g % NB]));
            umma_commit(smem_u32(p_free));
          }
          if (!(ok = mbar_wait(smem_u32(pds_full), g & 1, abort_flag))) break;
          tc_fence_after();
          if (KV) {
            // dK[kv, d] += sum_q dS[q, kv] Q[q, d]
            issue_acc_mn(ACC1_COL, ds_mn, a_mn(g), n != 0);
            umma_commit(smem_u32(&a_empty[g % NA]));
            if constexpr (MODE == MODE_ONE) {
              // dQ[q, d] of this tile pair, into the buffer that the pair before the last one has left
              if (!(ok = mbar_wait(smem_u32(&dq_free[g & 1]), ((g >> 1) & 1) ^ 1u, abort_flag))) break;
              tc_fence_after();
#pragma unroll
              for (int kk = 0; kk < BLK / 16; ++kk)
                umma_bf16_ss_split(tmem_base + DQ_COL + (g & 1) * 64, ds_k + (((kk >> 2) * (BLK * 128) + (kk & 3) * 32) >> 4), HI,
                                   k_mn_first + stat_off + ((kk * (16 * 128)) >> 4), HI, idesc_q, kk != 0 ? 1u : 0u);
              umma_commit(smem_u32(&dq_full[g & 1]));
              if (!more) umma_commit(smem_u32(stat ? stat_empty1 : stat_empty));
            }
          } else {
            // dQ[q, d] += sum_kv dS[q, kv] K[kv, d]: dS K-major, K through its MN-major view
            const uint32_t k_lo = a_mn(g);
#pragma unroll
            for (int kk = 0; kk < BLK / 16; ++kk)
              umma_bf16_ss_split(tmem_base + ACC0_COL, ds_k + (((kk >> 2) * (BLK * 128) + (kk & 3) * 32) >> 4), HI,
                                 k_lo + ((kk * (16 * 128)) >> 4), HI, idesc_q, (n | kk) != 0 ? 1u : 0u);
            umma_commit(smem_u32(&a_empty[g % NA]));
            umma_commit(smem_u32(ds_free));
          }
          if (!more) {
            umma_commit(smem_u32(acc_done));
          } else if (KV) {
            // dP of the next tile: its columns were read before pds_full(g) completed
            if (!(ok = wait_b(g + 1))) break;
            tc_fence_after();
            issue_dp(g + 1);
          }
        }
        ++it;
      }
    }
  } else {
    // ---------------------------- element-wise warps -----------------------------------
    const int quad = warp & 3;
    const int part = warp >> 2;                 // which 32 key columns of the tile this thread handles
    const int r = quad * 32 + lane;             // query row inside the tile
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const float LOG2E = 1.4426950408889634f;
    bool ok = true;
    int g = 0, it = 0, handed = 0;
    uint8_t* const stg = smem + L::STG_OFF + warp * L::STG;
    // 32 rows and 64 bytes (16 fp32 or 32 bf16 columns from `col`) of a gradient through this warp's staging block
    auto hand_over = [&](const CUtensorMap* map, bool add, int col, int row0, int h, int b) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (add) tma_reduce_add_4d(map, smem_u32(stg), col, h, row0, b); else tma_store_4d(map, smem_u32(stg), col, h, row0, b);
        tma_store_commit();
      }
    };
    auto stage_16 = [&](const uint32_t* t, float scale) {
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(stg + sw64_offset(lane, q)) =
            make_float4(__uint_as_float(t[4 * q]) * scale, __uint_as_float(t[4 * q + 1]) * scale,
                        __uint_as_float(t[4 * q + 2]) * scale, __uint_as_float(t[4 * q + 3]) * scale);
    };
    // 32 columns of an accumulator, by the lane whose row it is
    auto store_row = [&](const AttnBwdParams::Grad& to, int rows, const uint32_t (&t)[32], float scale, int col, int row0, int h, int b) {
      if (row0 + lane >= rows) return;
      const long long at = b * to.sb + (row0 + lane) * to.ss + h * to.sh + col;
      auto v = [&](int i) { return __uint_as_float(t[i]) * scale; };
      if (p.grad_f32) {
        float4* const o = reinterpret_cast<float4*>(static_cast<float*>(to.p) + at);
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = make_float4(v(4 * q), v(4 * q + 1), v(4 * q + 2), v(4 * q + 3));
      } else {
        uint4* const o = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(to.p) + at);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          o[q] = make_uint4(pack_bf16x2(v(8 * q), v(8 * q + 1)), pack_bf16x2(v(8 * q + 2), v(8 * q + 3)),
                            pack_bf16x2(v(8 * q + 4), v(8 * q + 5)), pack_bf16x2(v(8 * q + 6), v(8 * q + 7)));
      }
    };
    // 32 columns of an accumulator
    auto store_grad = [&](const CUtensorMap* map, const uint32_t (&t)[32], float scale, int col, int row0, int h, int b) {
      if (p.grad_f32) {
        stage_16(t, scale);
        hand_over(map, false, col, row0, h, b);
        stage_16(t + 16, scale);
        hand_over(map, false, col + 16, row0, h, b);
        return;
      }
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 u;
        u.x = pack_bf16x2(__uint_as_float(t[q * 8 + 0]) * scale, __uint_as_float(t[q * 8 + 1]) * scale);
        u.y = pack_bf16x2(__uint_as_float(t[q * 8 + 2]) * scale, __uint_as_float(t[q * 8 + 3]) * scale);
        u.z = pack_bf16x2(__uint_as_float(t[q * 8 + 4]) * scale, __uint_as_float(t[q * 8 + 5]) * scale);
        u.w = pack_bf16x2(__uint_as_float(t[q * 8 + 6]) * scale, __uint_as_float(t[q * 8 + 7]) * scale);
        *reinterpret_cast<uint4*>(stg + sw64_offset(lane, q)) = u;
      }
      hand_over(map, false, col, row0, h, b);
    };
    // MODE_ONE: this warp's 16 columns of dQ of the g-th streamed tile, query tile t, are added to an fp32 result.  Every two KV
    // tiles have one of their own: a sum of two does not depend on their order, so neither does dQ.
    auto drain_dq = [&](int g, int t, int own, int h, int b) {
      if (!mbar_wait_warp(smem_u32(&dq_full[g & 1]), (g >> 1) & 1, abort_flag)) return false;
      tc_fence_after();
      uint32_t q_r[16];
      tmem_ld_32x16(tmem_base + lane_off + DQ_COL + (g & 1) * 64 + part * 16, q_r);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&dq_free[g & 1]));
      stage_16(q_r, p.scale);
      hand_over(&tmG.dq, true, part * 16, t * BLK + quad * 32, h, (own >> 1) * p.B + b);
      return true;
    };
    auto next = [&](int w, int k) {
      if (!p.queue) return w + (int)gridDim.x;
      if (!mbar_wait_warp(smem_u32(&item_full[k & 1]), (k >> 1) & 1, abort_flag)) return total_items;
      const int n = item_slot[k & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&item_empty[k & 1]));
      return n;
    };
    for (int w = blockIdx.x, k = 0; w < total_items && ok; w = next(w, k++)) {
    const Item I = item_at(w);
    const int own = I.own, h = I.h, b = I.b, t_begin = I.t_begin, n_iter = I.n_iter;
    float lse2 = 0.0f, dlt = 0.0f;
    int row_g = own * BLK + r;
    bool row_ok = row_g < p.Sq;
    int q_live = p.Sq, kv_live = p.Sk;          // queries and keys from here on are masked
    if (BIAS == BIAS_KEYS && p.lengths) {
      kv_live = max(0, min(p.Sk, p.lengths[b]));
      q_live = min(p.Sq, kv_live);
    }
    if (MODE == MODE_Q && row_ok) {
      const long long stat_idx = ((long long)b * p.H + h) * p.Sq + row_g;
      lse2 = p.lse[stat_idx] * LOG2E;
      dlt = p.delta[stat_idx];
    }
    float lse_next = 0.0f, dlt_next = 0.0f;      // MODE_KV: statistics of the next query tile's row
    if (KV && n_iter > 0 && t_begin * BLK + r < p.Sq) {
      const long long stat_idx = ((long long)b * p.H + h) * p.Sq + t_begin * BLK + r;
      lse_next = p.lse[stat_idx];
      dlt_next = p.delta[stat_idx];
    }
    for (int n = 0; n < n_iter; ++n, ++g) {
      const int t = t_begin + n;                               // streamed tile index
      const int q_tile = KV ? t : own;
      const int kv_tile = KV ? own : t;
      if (KV) {
        // this tile's row statistics were loaded one iteration ago; start the loads for the next tile
        // now so that their latency hides behind this iteration
        row_g = q_tile * BLK + r;
        row_ok = row_g < p.Sq;
        lse2 = lse_next * LOG2E;
        dlt = dlt_next;
        const int row_n = row_g + BLK;
        if (n + 1 < n_iter && row_n < p.Sq) {
          const long long stat_idx = ((long long)b * p.H + h) * p.Sq + row_n;
          lse_next = p.lse[stat_idx];
          dlt_next = p.delta[stat_idx];
        } else {
          lse_next = 0.0f;
          dlt_next = 0.0f;
        }
      }
      const int kv0 = kv_tile * BLK;
      // tiles that need no masking: every row and column valid and strictly below the diagonal
      constexpr bool biased = BIAS != BIAS_NONE;   // additive biases / valid lengths: instantiations of their own
      const bool plain = (q_tile + 1) * BLK <= p.Sq && (kv_tile + 1) * BLK <= p.Sk &&
                         !(p.causal && kv_tile >= q_tile) && !biased;
      float pv[32];
      uint8_t* const p_tile = smem + L::P_OFF + (part >> 1) * (BLK * 128);    // 64-column block of the P / dS tile
      uint8_t* const ds_tile = smem + L::DS_OFF + (part >> 1) * (BLK * 128);
      const int c16_0 = (part & 1) * 4;                                        // first 16-byte chunk inside the 128-byte row
      // ---- phase A: P = exp2(S·c − lse) --------------------------------------------------
      // s_full(n) was committed after the dV GEMM of tile n-1: the P buffer is free
      if (!mbar_wait_warp(smem_u32(s_full), g & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t s_r[32];
        tmem_ld_32x32(tmem_base + lane_off + S_COL + part * 32, s_r);
        tmem_ld_wait();
        if constexpr (BIAS == BIAS_KEYS) {
          // exp2(S c + bias - lse): masked keys carry -inf in the bias; a fully masked row has lse = -inf and contributes
          // nothing.  Padded queries and keys may hold values that are not finite: their rows, and their columns in the
          // tile that holds the length, are set to zero by comparison.
          const bool row_live = row_g < q_live && lse2 > -INFINITY;
          const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), ns2 = make_float2(-lse2, -lse2);
          const float4* bias = reinterpret_cast<const float4*>(p.kb_pad + b * p.kp_sb + h * p.kp_sh + kv0 + part * 32);
#pragma unroll
          for (int q = 0; q < 32; q += 4) {
            const float4 v = __ldg(bias + q / 4);
            const float2 x = fma2(make_float2(__uint_as_float(s_r[q]), __uint_as_float(s_r[q + 1])), sc2, add2(make_float2(v.x, v.y), ns2));
            const float2 y = fma2(make_float2(__uint_as_float(s_r[q + 2]), __uint_as_float(s_r[q + 3])), sc2, add2(make_float2(v.z, v.w), ns2));
            pv[q] = fast_exp2(x.x); pv[q + 1] = fast_exp2(x.y);
            pv[q + 2] = fast_exp2(y.x); pv[q + 3] = fast_exp2(y.y);
          }
          if ((p.causal && kv_tile >= q_tile) || kv0 + BLK > kv_live) {
#pragma unroll
            for (int q = 0; q < 32; ++q) {
              const int colg = kv0 + part * 32 + q;
              if (colg >= kv_live || (p.causal && colg > row_g)) pv[q] = 0.0f;
            }
          }
          if (!row_live) {
#pragma unroll
            for (int q = 0; q < 32; ++q) pv[q] = 0.0f;
          }
        } else if (plain) {
#pragma unroll
          for (int q = 0; q < 32; ++q) pv[q] = fast_exp2(__uint_as_float(s_r[q]) * p.scale_log2 - lse2);
        } else if constexpr (!biased) {
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            const int colg = kv0 + part * 32 + q;
            const bool dead = !row_ok || colg >= p.Sk || (p.causal && colg > row_g);
            pv[q] = dead ? 0.0f : fast_exp2(__uint_as_float(s_r[q]) * p.scale_log2 - lse2);
          }
        } else {
          // the forward's logits were scale * q·k + key_bias + attn_bias with keys (and queries) beyond the
          // valid length masked; a fully masked row has lse = -inf and contributes nothing
          int kv_len = p.Sk;
          if (p.lengths) kv_len = max(0, min(p.Sk, p.lengths[b]));
          const bool row_live = row_ok && (!p.lengths || row_g < kv_len) && lse2 > -INFINITY;
          const float* kb = p.key_bias ? p.key_bias + (long long)b * p.kb_sb + (long long)h * p.kb_sh : nullptr;
          const float* ab = (p.attn_bias && row_ok)
                                ? p.attn_bias + (long long)b * p.ab_sb + (long long)h * p.ab_sh + (long long)row_g * p.ab_sq
                                : nullptr;
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            const int colg = kv0 + part * 32 + q;
            const bool dead = !row_live || colg >= kv_len || (p.causal && colg > row_g);
            float e = 0.0f;
            if (!dead) {
              float bias = kb ? kb[colg] : 0.0f;
              if (ab) bias += ab[colg];
              e = fast_exp2(fmaf(__uint_as_float(s_r[q]), p.scale_log2, bias * LOG2E) - lse2);
            }
            pv[q] = e;
          }
        }
      }
      // S has been read: the next S GEMM may overwrite it while P is converted and stored
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(s_free));
      if (KV) {
        // the dV GEMM of the previous tile must have finished reading the P buffer
        if (g > 0 && !mbar_wait_warp(smem_u32(p_free), (g - 1) & 1, abort_flag)) { ok = false; break; }
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) store8_bf16(p_tile, r, c16_0 + c8, &pv[c8 * 8]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(p_ready));
      }
      // ---- phase B: dS = P∘(dP − delta) → shared memory ---------------------------------------
      if (!mbar_wait_warp(smem_u32(&dp_full[g & 1]), (g >> 1) & 1, abort_flag)) { ok = false; break; }
      // the previous tile's GEMM that reads the dS buffer must be done: in the dK/dV pass dP(n) was
      // issued after it; the dQ pass issues dP early and signals the buffer separately
      if (MODE == MODE_Q && g > 0 && !mbar_wait_warp(smem_u32(ds_free), (g - 1) & 1, abort_flag)) { ok = false; break; }
      if (!L::OWN_STG && !L::LANES && n == 0 && w != blockIdx.x) {
        // the dS tile still held gradients of the items before: every warp's have been read
        if (lane == 0) {
          tma_store_wait_read<0>();
          mbar_arrive(smem_u32(stg_free));
        }
        if (!mbar_wait_warp(smem_u32(stg_free), handed & 1, abort_flag)) { ok = false; break; }
        ++handed;
      }
      tc_fence_after();
      const uint32_t dp_col = (MODE == MODE_Q && (g & 1)) ? ACC1_COL : DP_COL;
      {
        uint32_t dp_r[32];
        tmem_ld_32x32(tmem_base + lane_off + dp_col + part * 32, dp_r);
        tmem_ld_wait();
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) {
          float dsv[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) dsv[q] = pv[c8 * 8 + q] * (__uint_as_float(dp_r[c8 * 8 + q]) - dlt);
          store8_bf16(ds_tile, r, c16_0 + c8, dsv);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(pds_full));
      // dQ of the previous tile, while this tile's GEMMs run
      if (MODE == MODE_ONE && n > 0 && !drain_dq(g - 1, t - 1, own, h, b)) { ok = false; break; }
    }
    if (ok && n_iter > 0 && !mbar_wait_warp(smem_u32(acc_done), it & 1, abort_flag)) ok = false;
    if (MODE == MODE_ONE && ok && n_iter > 0) ok = drain_dq(g - 1, t_begin + n_iter - 1, own, h, b);
    if (ok) {
      // 32 accumulator columns per warp and accumulator.  TMEM loads are warp-collective: every lane issues them; rows that do
      // not exist are clipped by the copy.  An item to which nothing attends has zero gradients.
      const int row0 = own * BLK + quad * 32;
      uint32_t acc_r[32];
      constexpr bool BOTH = KV && D == 128;         // a warp has a chunk of both accumulators, or of one of them
      const int ch = D == 128 ? part : part & 1;
      const bool first = D == 128 || part < 2;      // dV (or dQ); else dK
      auto read = [&](uint32_t col, bool last) {
        if (n_iter > 0) {
          tc_fence_after();
          tmem_ld_32x32(tmem_base + lane_off + col + ch * 32, acc_r);
          tmem_ld_wait();
          if (last) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(acc_free));
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; ++q) acc_r[q] = 0;
        }
      };
      read(KV && !first ? ACC1_COL : ACC0_COL, !BOTH);
      if constexpr (L::LANES) {
        if (!KV) {
          if (first) store_row(p.dq, p.Sq, acc_r, p.scale, ch * 32, row0, h, b);
        } else {
          store_row(first ? p.dv : p.dk, p.Sk, acc_r, first ? 1.0f : p.scale, ch * 32, row0, h, b);
        }
      } else if (!KV) {
        if (first) store_grad(&tmG.dq, acc_r, p.scale, ch * 32, row0, h, b);
      } else {
        store_grad(first ? &tmG.dv : &tmG.dk, acc_r, first ? 1.0f : p.scale, ch * 32, row0, h, b);
        if (BOTH) {
          read(ACC1_COL, true);
          store_grad(&tmG.dk, acc_r, p.scale, ch * 32, row0, h, b);
        }
      }
      if (n_iter > 0) ++it;
    }
    }   // work items
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) report_error(p.err, ERR_MBAR_TIMEOUT, 0xA7B0u + MODE);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  if (warp == EW_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Sums of dQ (MODE_ONE) that query s belongs to: one for every two KV tiles that its tile attends to
__device__ __forceinline__ int dq_buffers(int s, int n_kv, int causal, const int* lengths, int b) {
  const int tile = s / BLK;
  if (lengths) {
    n_kv = (max(0, min(n_kv * BLK, lengths[b])) + BLK - 1) / BLK;      // clamped first: a length may be the largest int
    if (tile >= n_kv) return 0;
  }
  return ((causal ? min(n_kv, tile + 1) : n_kv) + 1) >> 1;
}

// delta[b,h,s] = sum_d O[b,s,h,d] * dO[b,s,h,d].  D / 8 lanes share one (b,s,h) row, each with one
// 16-byte load of O and of dO (a warp covers 2 rows at D = 128, 4 at D = 64): one row per warp with 4-byte
// loads left this bandwidth-bound pass at a quarter of the copy rate.
// With F32 the gradient arrives in fp32: this pass also writes the bf16 form that the tensor cores read (strides do_*) and
// takes the products with it.  dq (or null): the fp32 sums of dQ that the one-pass form adds to, zeroed here.
// Index is 32-bit wherever the row count allows it: with 64-bit divisions 8 x 2048 x 16 rows of 128 took 38.5 us,
// with 32-bit ones 35.1 (20.5 of bytes).
template <int D, bool F32, typename Index>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ O, __nv_bfloat16* __restrict__ dO, const float* __restrict__ dO32,
                  float* __restrict__ delta, int B, int S, int H, long long o_sb, long long o_ss, long long o_sh,
                  long long do_sb, long long do_ss, long long do_sh, float* __restrict__ dq, long long dq_sb, long long dq_ss,
                  long long dq_sh, long long dq_buffer, int n_kv, int causal, const int* __restrict__ lengths,
                  unsigned* __restrict__ queue) {
  chain_begin(O, dO32, lengths);
  if (queue && blockIdx.x == 0 && threadIdx.x == 0) *queue = 0;
  constexpr int LPR = D / 8;                       // lanes per row
  const Index total = (Index)B * S * H;
  const int sub = threadIdx.x % LPR;
  const Index stride = (Index)gridDim.x * (blockDim.x / LPR);
  for (Index w = blockIdx.x * (Index)(blockDim.x / LPR) + threadIdx.x / LPR; ; w += stride) {
    // every lane of a warp takes the same number of trips: the shuffles below need the full warp
    const bool live = w < total;
    if (!__any_sync(0xffffffffu, live)) break;
    float acc = 0.0f;
    int hh = 0, s = 0, bb = 0;
    if (live) {
      hh = (int)(w % H);
      const Index bs = w / H;
      s = (int)(bs % S);
      bb = (int)(bs / S);
      const uint4 a = *reinterpret_cast<const uint4*>(O + bb * o_sb + s * o_ss + hh * o_sh + sub * 8);
      __nv_bfloat16* gp = dO + bb * do_sb + s * do_ss + hh * do_sh + sub * 8;
      uint4 g;
      if constexpr (F32) {
        const float4* src = reinterpret_cast<const float4*>(dO32 + (long long)w * D + sub * 8);
        const float4 u = src[0], v = src[1];
        g = make_uint4(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
        *reinterpret_cast<uint4*>(gp) = g;
      } else {
        g = *reinterpret_cast<const uint4*>(gp);
      }
      if (dq) {
        float* z = dq + bb * dq_sb + s * dq_ss + hh * dq_sh + sub * 8;
        for (int i = dq_buffers(s, n_kv, causal, lengths, bb); i > 0; --i, z += dq_buffer)
          reinterpret_cast<float4*>(z)[0] = reinterpret_cast<float4*>(z)[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      const uint32_t av[4] = {a.x, a.y, a.z, a.w}, gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = unpack_bf16x2(av[i]), y = unpack_bf16x2(gv[i]);
        acc += x.x * y.x + x.y * y.y;
      }
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (live && sub == 0) delta[((long long)bb * H + hh) * S + s] = acc;
  }
}

// dQ from its fp32 sums, [buffer][B, S, H, 64] contiguous, in the order of the KV tiles; eight lanes per row
template <typename T>
__global__ void __launch_bounds__(256)
attn_dq_sum_kernel(const float* __restrict__ sums, T* __restrict__ dq, long long rows, int S, int H, int n_kv, int causal,
                   const int* __restrict__ lengths, long long sb, long long ss, long long sh) {
  chain_begin(sums, lengths);
  const int sub = threadIdx.x & 7;
  for (long long w = blockIdx.x * 32ll + (threadIdx.x >> 3); w < rows; w += gridDim.x * 32ll) {
    const int h = (int)(w % H);
    const long long bs = w / H, b = bs / S, i = bs - b * S;
    const float4* src = reinterpret_cast<const float4*>(sums + w * 64 + sub * 8);
    float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = u;
#pragma unroll 4
    for (int n = dq_buffers((int)i, n_kv, causal, lengths, (int)b); n > 0; --n, src += rows * 16) {
      const float4 x = src[0], y = src[1];
      u.x += x.x; u.y += x.y; u.z += x.z; u.w += x.w;
      v.x += y.x; v.y += y.y; v.z += y.z; v.w += y.w;
    }
    T* out = dq + b * sb + i * ss + h * sh + sub * 8;
    if constexpr (sizeof(T) == 4) {
      reinterpret_cast<float4*>(out)[0] = u;
      reinterpret_cast<float4*>(out)[1] = v;
    } else {
      *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    }
  }
}

}  // namespace

struct StAttnBwdArgs {
  const void* Q; const void* K; const void* V; const void* O; const void* dO;
  const float* lse; float* delta; float* dQ_acc;
  void* dQ; void* dK; void* dV;
  long long q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, o_sb, o_ss, o_sh;
  long long do_sb, do_ss, do_sh, dq_sb, dq_ss, dq_sh, dk_sb, dk_ss, dk_sh, dv_sb, dv_ss, dv_sh;
  int B, H, Sq, Sk, D;
  float scale;
  int causal;
  // optional additive biases (fp32) and valid lengths (int32 [B]) of the forward pass; null = absent
  const float* key_bias;  long long kb_sb, kb_sh;
  const float* attn_bias; long long ab_sb, ab_sh, ab_sq;
  const int* lengths;
};

namespace {
int attn_bwd_run(const StAttnBwdArgs* a, const float* dO32, int grad_f32, float* bias_ws, float* dq_sums, void* stream_v) {
  if (!a || !a->Q || !a->K || !a->V || !a->O || !a->dO || !a->lse || !a->delta ||
      !a->dQ || !a->dK || !a->dV)
    return st::fail(ST_ERR_INVALID, "attn_bwd: null pointer");
  if (a->D != 64 && a->D != 128) return st::fail(ST_ERR_INVALID, "attn_bwd: head_dim must be 64 or 128");
  if (a->causal && a->Sq != a->Sk) return st::fail(ST_ERR_INVALID, "attn_bwd: causal needs seq_q == seq_k");
  const long long strides[] = {a->q_sb, a->q_ss, a->q_sh, a->k_sb, a->k_ss, a->k_sh, a->v_sb, a->v_ss,
                               a->v_sh, a->o_sb, a->o_ss, a->o_sh, a->do_sb, a->do_ss, a->do_sh,
                               a->dq_sb, a->dq_ss, a->dq_sh, a->dk_sb, a->dk_ss, a->dk_sh,
                               a->dv_sb, a->dv_ss, a->dv_sh};
  for (long long s : strides)
    if (s & 7) return st::fail(ST_ERR_INVALID, "attn_bwd: strides must be multiples of 8 elements");
  const void* ptrs[] = {a->Q, a->K, a->V, a->O, a->dO, a->dQ, a->dK, a->dV};
  for (const void* q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15) return st::fail(ST_ERR_INVALID, "attn_bwd: pointers must be 16-byte aligned");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  // One pass where the caller gives the workspace: the fp32 sums of dQ (with one of them and fp32 gradients: dQ itself)
  const bool biased = a->key_bias || a->attn_bias || a->lengths;
  const bool keyb = biased && !a->attn_bias && bias_ws;
  const int n_kv = (a->Sk + BLK - 1) / BLK;
  const bool one = dq_sums && a->D == 64 && n_kv <= kOnePassTiles && (!biased || keyb);
  if (one && (reinterpret_cast<uintptr_t>(dq_sums) & 15)) return st::fail(ST_ERR_INVALID, "attn_bwd: the dQ workspace must be 16-byte aligned");
  const bool in_place = one && grad_f32 && n_kv <= 2;
  float* const acc = !one ? nullptr : in_place ? static_cast<float*>(a->dQ) : dq_sums;
  const long long acc_sb = in_place ? a->dq_sb : (long long)a->Sq * a->H * a->D, acc_ss = in_place ? a->dq_ss : (long long)a->H * a->D,
                  acc_sh = in_place ? a->dq_sh : a->D, acc_buffer = (long long)a->B * a->Sq * a->H * a->D;
  unsigned* const queue = one ? reinterpret_cast<unsigned*>(dq_sums + (in_place ? 0 : acc_buffer * ((n_kv + 1) / 2))) : nullptr;

  {
    const long long rows = (long long)a->B * a->Sq * a->H;
    const int rows_per_block = 256 / (a->D / 8);
    long long blocks = (rows + rows_per_block - 1) / rows_per_block;
    if (blocks > 148 * 16) blocks = 148 * 16;
    auto Op = static_cast<const __nv_bfloat16*>(a->O);
    auto dOp = static_cast<__nv_bfloat16*>(const_cast<void*>(a->dO));        // written only from dO32
    auto delta = [&](auto kernel) {
      st::chained(kernel, (unsigned)blocks, 256, 0, s)(Op, dOp, dO32, a->delta, a->B, a->Sq, a->H, a->o_sb, a->o_ss, a->o_sh, a->do_sb,
                                              a->do_ss, a->do_sh, acc, acc_sb, acc_ss, acc_sh, acc_buffer, n_kv, a->causal,
                                              in_place ? nullptr : a->lengths, queue);
    };
    const bool narrow = rows + blocks * rows_per_block < (1ll << 31);      // the last step's index must not wrap either
    auto pick = [&](auto d) {
      constexpr int D = decltype(d)::value;
      if (narrow) { if (dO32) delta(attn_delta_kernel<D, true, unsigned>); else delta(attn_delta_kernel<D, false, unsigned>); }
      else { if (dO32) delta(attn_delta_kernel<D, true, long long>); else delta(attn_delta_kernel<D, false, long long>); }
    };
    if (a->D == 128) pick(std::integral_constant<int, 128>{}); else pick(std::integral_constant<int, 64>{});
    ST_CUDA_CHECK(cudaGetLastError());
  }

  CUtensorMap tq, tk, tv, tdo;
  if (!st::encode_bshd_tmap(&tq, a->Q, a->B, a->Sq, a->H, a->D, a->q_sb, a->q_ss, a->q_sh, BLK) ||
      !st::encode_bshd_tmap(&tk, a->K, a->B, a->Sk, a->H, a->D, a->k_sb, a->k_ss, a->k_sh, BLK) ||
      !st::encode_bshd_tmap(&tv, a->V, a->B, a->Sk, a->H, a->D, a->v_sb, a->v_ss, a->v_sh, BLK) ||
      !st::encode_bshd_tmap(&tdo, a->dO, a->B, a->Sq, a->H, a->D, a->do_sb, a->do_ss, a->do_sh, BLK))
    return ST_ERR_CUDA;
  GradMaps tg;
  if (!st::encode_out_tmap(&tg.dk, a->dK, grad_f32, a->B, a->Sk, a->H, a->D, a->dk_sb, a->dk_ss, a->dk_sh) ||
      !st::encode_out_tmap(&tg.dv, a->dV, grad_f32, a->B, a->Sk, a->H, a->D, a->dv_sb, a->dv_ss, a->dv_sh) ||
      !(one ? st::encode_out_tmap(&tg.dq, acc, true, in_place ? a->B : a->B * ((n_kv + 1) / 2), a->Sq, a->H, a->D, acc_sb, acc_ss, acc_sh)
            : st::encode_out_tmap(&tg.dq, a->dQ, grad_f32, a->B, a->Sq, a->H, a->D, a->dq_sb, a->dq_ss, a->dq_sh)))
    return ST_ERR_CUDA;
  AttnBwdParams p;
  p.lse = a->lse; p.delta = a->delta;
  p.B = a->B; p.H = a->H; p.Sq = a->Sq; p.Sk = a->Sk;
  p.scale = a->scale;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.causal = a->causal;
  p.err = st::error_word();
  p.key_bias = a->key_bias; p.kb_sb = a->kb_sb; p.kb_sh = a->kb_sh;
  p.attn_bias = a->attn_bias; p.ab_sb = a->ab_sb; p.ab_sh = a->ab_sh; p.ab_sq = a->ab_sq;
  p.lengths = a->lengths;
  p.grad_f32 = grad_f32;
  p.dq = {a->dQ, a->dq_sb, a->dq_ss, a->dq_sh};
  p.dk = {a->dK, a->dk_sb, a->dk_ss, a->dk_sh};
  p.dv = {a->dV, a->dv_sb, a->dv_ss, a->dv_sh};
  p.queue = queue;
  p.kb_pad = nullptr; p.kp_sb = p.kp_sh = 0;
  if (keyb) {
    if (int e = st::attn_key_bias(a->key_bias, a->kb_sb, a->kb_sh, a->lengths, bias_ws, a->B, a->H, a->Sk, &p.kp_sb, &p.kp_sh, s)) return e;
    p.kb_pad = bias_ws;
  }
  static int num_sms = 0;
  if (num_sms == 0) {
    int dev = 0;
    ST_CUDA_CHECK(cudaGetDevice(&dev));
    ST_CUDA_CHECK(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
  }
  const int items_kv = ((a->Sk + BLK - 1) / BLK) * a->H * a->B;
  const int items_q = ((a->Sq + BLK - 1) / BLK) * a->H * a->B;
  const dim3 grid_kv(items_kv < num_sms ? items_kv : num_sms);
  const dim3 grid_q(items_q < num_sms ? items_q : num_sms);
  auto launch = [&](auto kernel, int smem_bytes, dim3 grid) -> int {
    ST_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    // A kernel that starts early finds the L1 that the one before it left: 28 KB behind a product.  The bias per (query, key) needs more:
    // us with a product of 2048 x 4096 x 1024 before it, early and in order: 13 contexts of 602, 12 heads, causal, 645 and 358; 13 of
    // 212 200 and 108.
    const bool own_l1 = a->attn_bias && a->D == 64;
    (own_l1 ? st::in_order(kernel, grid, NUM_THREADS, smem_bytes, s) : st::chained(kernel, grid, NUM_THREADS, smem_bytes, s))(tq, tk, tv, tdo, tg, p);
    ST_CUDA_CHECK(cudaGetLastError());
    return ST_OK;
  };
  // both passes of a bias form: dK / dV per KV tile, then dQ per query tile
  auto both = [&](auto kv, int kv_smem, auto q, int q_smem) -> int {
    if (int e = launch(kv, kv_smem, grid_kv)) return e;
    return launch(q, q_smem, grid_q);
  };
  if (one) {
    const int e = keyb ? launch(attn_bwd_kernel<64, MODE_ONE, BIAS_KEYS>, BwdSmem<64, MODE_ONE, BIAS_KEYS>::TOTAL, grid_kv)
                       : launch(attn_bwd_kernel<64, MODE_ONE, BIAS_NONE>, BwdSmem<64, MODE_ONE, BIAS_NONE>::TOTAL, grid_kv);
    if (e || in_place) return e;
    const long long rows = (long long)a->B * a->Sq * a->H;
    const long long blocks = (rows + 31) / 32, most = 16ll * st::sm_count();
    auto sum = [&](auto* dq) {
      return st::chained(attn_dq_sum_kernel<std::remove_pointer_t<decltype(dq)>>, (unsigned)(blocks < most ? blocks : most), 256, 0, s)(
          acc, dq, rows, a->Sq, a->H, n_kv, a->causal, a->lengths, a->dq_sb, a->dq_ss, a->dq_sh);
    };
    ST_CUDA_CHECK(grad_f32 ? sum(static_cast<float*>(a->dQ)) : sum(static_cast<__nv_bfloat16*>(a->dQ)));
    return ST_OK;
  }
#define ST_BWD_BOTH(DV, BV) \
  both(attn_bwd_kernel<DV, MODE_KV, BV>, BwdSmem<DV, MODE_KV, BV>::TOTAL, attn_bwd_kernel<DV, MODE_Q, BV>, BwdSmem<DV, MODE_Q, BV>::TOTAL)
  if (a->D == 128) return keyb ? ST_BWD_BOTH(128, BIAS_KEYS) : biased ? ST_BWD_BOTH(128, BIAS_FULL) : ST_BWD_BOTH(128, BIAS_NONE);
  return keyb ? ST_BWD_BOTH(64, BIAS_KEYS) : biased ? ST_BWD_BOTH(64, BIAS_FULL) : ST_BWD_BOTH(64, BIAS_NONE);
#undef ST_BWD_BOTH
}
}  // namespace

// delta: fp32 [B,H,Sq] workspace.  dQ_acc is unused (kept in the argument block for ABI stability).
ST_API int st_attn_bwd(const StAttnBwdArgs* a, void* stream_v) { return attn_bwd_run(a, nullptr, 0, nullptr, nullptr, stream_v); }

// The same with, all optional: the output's gradient in fp32 (dO32, contiguous [B, Sq, H, D]; a->dO then receives its bf16
// form), gradients in fp32 (grad_f32: dQ, dK, dV are float*, strides in elements), and a workspace of
// st_attn_bias_workspace floats for a key bias or lengths.
ST_API int st_attn_bwd_f32(const StAttnBwdArgs* a, const float* dO32, int grad_f32, float* bias_workspace, void* stream_v) {
  return attn_bwd_run(a, dO32, grad_f32, bias_workspace, nullptr, stream_v);
}

// Floats of workspace (16-byte aligned) of the one-pass form, whatever the gradients' type; 0 where it does not apply.
ST_API long long st_attn_bwd_workspace(int B, int H, int Sq, int Sk, int D) {
  const int n_kv = (Sk + BLK - 1) / BLK;
  return D == 64 && n_kv <= kOnePassTiles ? (long long)B * Sq * H * D * ((n_kv + 1) / 2) + kQueueFloats : 0;
}

// What fp32 gradients need of it: with one sum, which is dQ itself, only the work queue.
ST_API long long st_attn_bwd_workspace_f32(int B, int H, int Sq, int Sk, int D) {
  return D == 64 && Sk <= 2 * BLK ? kQueueFloats : st_attn_bwd_workspace(B, H, Sq, Sk, D);
}

// st_attn_bwd_f32 in one pass over the tile pairs where dq_workspace (as above) is given; in two with null, with
// a bias per query and key, and with a key bias or lengths without their workspace.
ST_API int st_attn_bwd_one_pass(const StAttnBwdArgs* a, const float* dO32, int grad_f32, float* bias_workspace, float* dq_workspace,
                                void* stream_v) {
  return attn_bwd_run(a, dO32, grad_f32, bias_workspace, dq_workspace, stream_v);
}
