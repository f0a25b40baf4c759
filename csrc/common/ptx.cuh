// Blackwell (sm_100a) PTX building blocks shared by every kernel in this library:
// mbarrier with bounded waits, TMA tiled loads (never cluster-multicast), tcgen05 MMA /
// TMEM allocation / TMEM loads, shared-memory matrix descriptors and the instruction
// descriptor for kind::f16.
//
// Every wait in this file is bounded: after wait_limit_ns() (2 s unless the host changed it with
// st_set_wait_timeout_ns) the waiter raises the CTA-wide abort flag and returns false, and callers
// unwind to their teardown (TMEM is released, the error word is written) instead of spinning for ever.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda.h>
#include <stdint.h>
#include "chain.cuh"

#ifndef ST_WAIT_TIMEOUT_NS
#define ST_WAIT_TIMEOUT_NS 2000000000ull  // 2 s
#endif

namespace st {

// ---------------------------------------------------------------------------------------
// Wait limit.  Every translation unit that includes this header owns one copy of the device
// word (no relocatable device code is used) and registers a setter for it at load time, so
// st_set_wait_timeout_ns() on the host reaches all of them.  Kernels read the word only on
// the slow path of a wait (once every few hundred polls).
// ---------------------------------------------------------------------------------------
typedef cudaError_t (*WaitLimitSetter)(unsigned long long);
void register_wait_limit_setter(WaitLimitSetter fn);   // defined in runtime/runtime.cu

static __device__ unsigned long long g_wait_limit_ns = ST_WAIT_TIMEOUT_NS;
static cudaError_t set_wait_limit_here(unsigned long long ns) {
  return cudaMemcpyToSymbol(g_wait_limit_ns, &ns, sizeof(ns));
}
struct WaitLimitRegistration {
  WaitLimitRegistration() { register_wait_limit_setter(&set_wait_limit_here); }
};
static WaitLimitRegistration g_wait_limit_registration;

__device__ __forceinline__ uint64_t wait_limit_ns() {
  return *reinterpret_cast<volatile unsigned long long*>(&g_wait_limit_ns);
}

// ---------------------------------------------------------------------------------------
// error word: [0] = code, [1] = detail, [2] = block, [3] = count.  Lives in mapped pinned
// host memory so the host can read it without a device synchronisation.
// ---------------------------------------------------------------------------------------
enum ErrCode : unsigned {
  ERR_NONE = 0,
  ERR_MBAR_TIMEOUT = 1,
  ERR_FLAG_TIMEOUT = 2,
  ERR_BOUNDS = 3,
};

__device__ __forceinline__ void report_error(unsigned* err, unsigned code, unsigned detail) {
  if (err == nullptr) return;
  if (atomicCAS(err, 0u, code) == 0u) {
    err[1] = detail;
    err[2] = blockIdx.x;
  }
  atomicAdd(err + 3, 1u);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.b32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  `abort_flag` is a CTA-shared int: a waiter that runs out of time sets it,
// and every other waiter of the CTA leaves as soon as it sees it.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t it = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++it) & 0x3F) == 0) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > wait_limit_ns()) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}

// Whole-warp variant: every lane waits and the warp agrees on the outcome, so that the
// warp-collective tcgen05 instructions that follow are never issued by a partial warp.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const bool ok = mbar_wait(bar, parity, abort_flag);
  return __all_sync(0xffffffffu, ok);
}

// ---------------------------------------------------------------------------------------
// proxies / fences
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---------------------------------------------------------------------------------------
// TMA tiled loads into this CTA's shared memory (no cluster multicast anywhere).
// Coordinates are innermost first; c0 * element size must be a multiple of 16 bytes.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
// TMA tiled store shared -> global (bulk group completion).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
// TMA tiled addition shared -> global (the element type is the map's).
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}
// Untiled bulk copies (both addresses 16-byte aligned, size a multiple of 16 bytes).
__device__ __forceinline__ void bulk_load_g2s(uint32_t dst_smem, const void* src_gmem, uint32_t bytes,
                                              uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst_smem), "l"(src_gmem), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_store_s2g(void* dst_gmem, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(dst_gmem), "r"(src_smem), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------------------------------
// CTA pairs (clusters of two): one thread of the even CTA issues MMAs over both CTAs' shared and tensor memory.
// A shared-memory address with the rank bits cleared names the even CTA's copy of the object.
// ---------------------------------------------------------------------------------------
constexpr uint32_t kPairLeaderMask = 0xFEFFFFFFu;
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Every thread of both CTAs; orders shared-memory accesses across the pair.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// Address of this CTA's shared-memory address `addr` in CTA `rank` of the cluster, and a 16-byte store to one.
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store_16(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Loads into this CTA's shared memory whose bytes count on the even CTA's barrier (`bar` with the rank bits cleared).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {      // one warp of each CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_ss_split_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "mov.b64 da, {%1, %2};\n"
      "mov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3))
               : "memory");
}

// ---------------------------------------------------------------------------------------
// TMEM allocation (one full warp executes these)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

// ---------------------------------------------------------------------------------------
// Descriptors
// ---------------------------------------------------------------------------------------
// Shared-memory matrix descriptor for a tile written by TMA with the 128-byte swizzle.
//  K-major operand (rows of 64 bf16 = 128 B, 8-row groups 1024 B apart):
//      lbo_bytes is ignored by the hardware for swizzled K-major tiles (set to 16),
//      sbo_bytes = 1024.
//  MN-major operand (each K row holds 64 contiguous MN elements = 128 B; 8 K rows form a
//  1024 B group; 64-element MN blocks are separate TMA boxes):
//      lbo_bytes = distance between MN blocks, sbo_bytes = 1024.
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes,
                                                         uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version for sm_100
  d |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::f16, bf16 x bf16 -> fp32 accumulate.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool a_mn_major,
                                                       bool b_mn_major) {
  return (1u << 4)                                  // D format: f32
         | (1u << 7)                                // A format: bf16
         | (1u << 10)                               // B format: bf16
         | (static_cast<uint32_t>(a_mn_major) << 15)
         | (static_cast<uint32_t>(b_mn_major) << 16)
         | (static_cast<uint32_t>(N >> 3) << 17)
         | (static_cast<uint32_t>(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void umma_bf16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same instruction with the descriptors given as (low word, high word): the high word of a
// descriptor is the same for every K step of a tile and the low word advances by a constant, so an
// issue loop needs one 32-bit add per operand instead of rebuilding 64-bit descriptors.
__device__ __forceinline__ void umma_bf16_ss_split(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi,
                                                   uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                   uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "mov.b64 da, {%1, %2};\n"
      "mov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: the A operand (M = 128 rows in lanes 0..127, K-major) is read from tensor
// memory, where each 32-bit column holds two consecutive bf16 K elements of the lane's row, so one K = 16 step
// reads 8 columns starting at tmem_a.  Issued by ONE thread.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with the B descriptor given as (low word, high word), as in umma_bf16_ss_split.
__device__ __forceinline__ void umma_bf16_ts_split(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
                                                   uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b64 db;\n"
      "setp.ne.b32 p, %5, 0;\n"
      "mov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Low / high words of make_smem_desc_sw128(addr, lbo, sbo); a byte offset `off` (multiple of 16) inside
// the tile is applied as `lo + (off >> 4)`.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFF) >> 4) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
}
__device__ __forceinline__ constexpr uint32_t smem_desc_hi(uint32_t sbo_bytes) {
  return ((sbo_bytes >> 4) & 0x3FFF) | (1u << 14) | (2u << 29);   // version 1 at bit 46, SWIZZLE_128B at bit 61
}
// Make `bar` complete once every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               ::"r"(bar)
               : "memory");
}

// TMEM -> registers: 32 lanes x 32 consecutive fp32 columns; thread i of the warp receives
// lane (lane_base + i).  taddr = (lane << 16) | column.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Registers -> TMEM: thread i of the warp writes 32 consecutive 32-bit columns of lane (lane_base + i).
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Byte offset of 16-byte chunk `chunk16` (0..7) of row `row` inside a 128-byte-swizzled
// tile whose rows are 128 bytes and whose base is 1024-byte aligned.
__device__ __forceinline__ uint32_t sw128_offset(uint32_t row, uint32_t chunk16) {
  return row * 128u + (((chunk16 ^ (row & 7u)) & 7u) << 4);
}

// The same for rows of 64 bytes with the 64-byte swizzle, chunk 0..3 and a 512-byte aligned base.
__device__ __forceinline__ uint32_t sw64_offset(uint32_t row, uint32_t chunk16) {
  return row * 64u + (((chunk16 ^ (row >> 1)) & 3u) << 4);
}

// ---------------------------------------------------------------------------------------
// small math helpers
// ---------------------------------------------------------------------------------------
// GELU in its tanh form, 0.5 x (1 + tanh u) = x / (1 + exp(-2u)) with u = k0 (x + k1 x^3), k0 = sqrt(2 / pi), k1 = 0.044715.
// Written over E = exp(-2 |u|) <= 1 and q = E / (1 + E), the smaller of the two probabilities, so that nothing cancels:
// max(x, 0) - |x| q, and for the derivative s + 2 x q (1 - q) u' with s = q or 1 - q.  For |x| < 1 the derivative takes
// s = 1/2 + h instead, where h = tanh(u) / 2 is an odd polynomial (least squares over [0, 1], 1.3e-9 off): q has an error of its
// own before it meets the 1, that of h fades with x.  tanhf's two branches, both taken by a warp of mixed magnitudes, set the pace
// of fused epilogues.
// Error against 64 bits for normally distributed x (root mean square, maximum), with tanhf and now: standard deviation 0.3
// 7.3e-9, 1.1e-7 and 7.0e-9, 8e-8; 1.0 2.5e-8, 4.1e-7 and 1.9e-8, 2.4e-7; 0.1 2.0e-9 and 2.6e-9.  Derivative: 0.3 2.2e-8, 1.4e-7 and 2.0e-8, 1.2e-7; 1.0
// 3.0e-8, 4.8e-7 and 2.6e-8, 1.5e-7.  Uniform over |x| < 4: 5.4e-8 and 3.7e-8, derivative 7.4e-8 and 2.8e-8.
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void gelu_parts(float x, float z, float& q, float& p) {      // z = x^2; q <= 1/2, p = 1 - q
  constexpr double c = 2.0 * 0.7978845608028654 * 1.4426950408889634;                   // 2 k0 log2(e)
  constexpr float c0 = static_cast<float>(c), c1 = static_cast<float>(c * 0.044715);
  const float e = exp2_ftz(-fabsf(x) * fmaf(c1, z, c0));
  p = __fdividef(1.0f, 1.0f + e);
  q = e * p;
}
__device__ __forceinline__ float gelu_half_tanh(float x, float z) {                      // |x| < 1
  const float t = fmaf(fmaf(fmaf(fmaf(-7.50559184e-06f, z, 1.18915079e-04f), z, -1.24431029e-03f), z, 1.02022300e-02f), z, -6.68196306e-02f);
  return fmaf(3.98942292e-01f, x, x * z * t);
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float z = x * x;
  float q, p;
  gelu_parts(x, z, q, p);
  return x > 0.0f ? x - fminf(x, 3.402823466e38f) * q : x * q;                           // the bound keeps inf * 0 out of gelu(inf)
}
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  constexpr float d0 = static_cast<float>(2.0 * 0.7978845608028654), d1 = static_cast<float>(6.0 * 0.7978845608028654 * 0.044715);
  const float z = x * x;
  float q, p;
  gelu_parts(x, z, q, p);
  const float h = gelu_half_tanh(x, z);
  const bool narrow = fabsf(x) < 1.0f;
  const float s = narrow ? 0.5f + h : (x > 0.0f ? 1.0f - q : q);
  return fmaf(x * fmaf(d1, z, d0), narrow ? fmaf(-h, h, 0.25f) : q * p, s);               // 2 x u' s (1 - s) + s
}
// Packed fp32 pairs (one issue slot for two lanes of arithmetic) and the three-input maximum.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2,%3};\n mov.b64 rb, {%4,%5};\n mov.b64 rc, {%6,%7};\n"
      " fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2,%3};\n mov.b64 rb, {%4,%5};\n"
      " add.rn.f32x2 rd, ra, rb;\n mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2,%3};\n mov.b64 rb, {%4,%5};\n"
      " mul.rn.f32x2 rd, ra, rb;\n mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// gelu_tanh and gelu_tanh_grad of two values with packed arithmetic: the same operations in the same order, so the same bits.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 splat2(float x) { return make_float2(x, x); }
__device__ __forceinline__ void gelu_parts_pair(float2 x, float2 z, float2& q, float2& p) {
  constexpr double c = 2.0 * 0.7978845608028654 * 1.4426950408889634;
  constexpr float c0 = static_cast<float>(c), c1 = static_cast<float>(c * 0.044715);
  const float2 a = mul2(make_float2(-fabsf(x.x), -fabsf(x.y)), fma2(splat2(c1), z, splat2(c0)));
  const float2 e = make_float2(exp2_ftz(a.x), exp2_ftz(a.y));
  const float2 d = add2(splat2(1.0f), e);
  p = make_float2(rcp_approx(d.x), rcp_approx(d.y));
  q = mul2(e, p);
}
__device__ __forceinline__ void gelu_tanh_pair(float& x0, float& x1) {
  const float2 x = make_float2(x0, x1), z = mul2(x, x);
  float2 q, p;
  gelu_parts_pair(x, z, q, p);
  x0 = x.x > 0.0f ? x.x - fminf(x.x, 3.402823466e38f) * q.x : x.x * q.x;
  x1 = x.y > 0.0f ? x.y - fminf(x.y, 3.402823466e38f) * q.y : x.y * q.y;
}
__device__ __forceinline__ float2 gelu_tanh_grad_pair(float2 x) {
  constexpr float d0 = static_cast<float>(2.0 * 0.7978845608028654), d1 = static_cast<float>(6.0 * 0.7978845608028654 * 0.044715);
  const float2 z = mul2(x, x);
  float2 q, p;
  gelu_parts_pair(x, z, q, p);
  const float2 t = fma2(fma2(fma2(fma2(splat2(-7.50559184e-06f), z, splat2(1.18915079e-04f)), z, splat2(-1.24431029e-03f)), z,
                             splat2(1.02022300e-02f)), z, splat2(-6.68196306e-02f));
  const float2 h = fma2(splat2(3.98942292e-01f), x, mul2(mul2(x, z), t));
  const float2 w = fma2(make_float2(-h.x, -h.y), h, splat2(0.25f)), qp = mul2(q, p), g = mul2(x, fma2(splat2(d1), z, splat2(d0)));
  const bool n0 = fabsf(x.x) < 1.0f, n1 = fabsf(x.y) < 1.0f;
  const float s0 = n0 ? 0.5f + h.x : (x.x > 0.0f ? 1.0f - q.x : q.x), s1 = n1 ? 0.5f + h.y : (x.y > 0.0f ? 1.0f - q.y : q.y);
  return fma2(g, make_float2(n0 ? w.x : qp.x, n1 ? w.y : qp.y), make_float2(s0, s1));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace st
