// Row-wise rank selection (top-k / bottom-k / mid-k) and row compaction.
//
// Selection semantics (crates/st-core/src/backend/rankk_software.rs:38-110, the CPU mirror of
// cuda_topk_rankk.cu): non-finite entries are ignored; candidates are ordered by value
// (descending for top, ascending for bottom and mid) with the LOWER column index winning ties;
// top/bottom take the first k, mid takes the k entries centred in the ascending order
// (start = (finite - take) / 2); unused output slots hold NaN / -1.
//
// Keys are 64 bit: order-preserving float bits in the high word (inverted for top), column index in the low word, so
// the smallest key is the best and the order is total and deterministic.  Four forms:
//   * top / bottom, k = 1: block arg-max over a row of up to 4096 columns (rank_k1_kernel);
//   * top / bottom, k <= 128: a sorted list of the best 32, 64 or 128 keys per warp, kept in registers while the warp
//     streams its share of the row; up to 16 warps of a CTA share a row, and eight in each of up to 64 CTAs a wide one
//     (rank_topk_kernel);
//   * mid, and larger k: a radix select over the row in shared memory finds the two boundary values of the wanted
//     range of ranks, and only the keys inside it are sorted (rank_range_kernel);
//   * k so large that the range's sort would be as wide as the row's: one bitonic sort (rank_select_kernel).
// (The reference keeps 8 candidates per thread and lets thread 0 select serially.)
//
// Compaction (crates/st-kernel-contracts/src/compaction.rs:369-400): per row, keep the entries
// with low <= v <= high in their original order, write values and column indices densely,
// zero the padding and return the per-row counts.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include <cfloat>

namespace {
using namespace st;

enum Mode : int { TOP = 0, BOTTOM = 1, MID = 2 };

__device__ __forceinline__ unsigned orderable(float v) {
  unsigned u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // ascending order of floats
}
__device__ __forceinline__ float from_orderable(unsigned o) {
  unsigned u = (o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o;
  return __uint_as_float(u);
}

constexpr unsigned long long KEY_INVALID = 0xFFFFFFFFFFFFFFFFull;

__global__ void rank_select_kernel(const float* __restrict__ in, float* __restrict__ out_v,
                                   int* __restrict__ out_i, int rows, int cols, int k, int mode,
                                   int padded) {
  extern __shared__ unsigned long long keys[];
  __shared__ int s_finite;
  const int row = blockIdx.x;
  const float* x = in + (size_t)row * cols;
  if (threadIdx.x == 0) s_finite = 0;
  __syncthreads();
  int local = 0;
  for (int c = threadIdx.x; c < padded; c += blockDim.x) {
    unsigned long long key = KEY_INVALID;
    if (c < cols) {
      const float v = x[c];
      if (isfinite(v)) {
        unsigned o = orderable(v);
        if (mode == TOP) o = ~o;  // descending value == ascending key
        key = (static_cast<unsigned long long>(o) << 32) | static_cast<unsigned>(c);
        ++local;
      }
    }
    keys[c] = key;
  }
  atomicAdd(&s_finite, local);
  __syncthreads();
  for (int size = 2; size <= padded; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < padded / 2; t += blockDim.x) {
        const int lo = (t / stride) * (stride << 1) + (t % stride);
        const int hi = lo + stride;
        const bool up = ((lo & size) == 0);
        const unsigned long long a = keys[lo], b = keys[hi];
        if ((a > b) == up) {
          keys[lo] = b;
          keys[hi] = a;
        }
      }
      __syncthreads();
    }
  }
  const int finite = s_finite;
  const int take = min(k, finite);
  const int start = (mode == MID) ? (finite - take) / 2 : 0;
  for (int s = threadIdx.x; s < k; s += blockDim.x) {
    float v = __int_as_float(0x7FC00000);
    int idx = -1;
    if (s < take) {
      const unsigned long long key = keys[start + s];
      unsigned o = static_cast<unsigned>(key >> 32);
      if (mode == TOP) o = ~o;
      v = from_orderable(o);
      idx = static_cast<int>(key & 0xFFFFFFFFu);
    }
    out_v[(size_t)row * k + s] = v;
    out_i[(size_t)row * k + s] = idx;
  }
}

// k == 1: block arg-max (mode TOP) / arg-min (BOTTOM); lower index wins ties.
__global__ void rank_k1_kernel(const float* __restrict__ in, float* __restrict__ out_v,
                               int* __restrict__ out_i, int rows, int cols, int mode) {
  __shared__ unsigned long long sh[32];
  const int row = blockIdx.x;
  const float* x = in + (size_t)row * cols;
  unsigned long long best = KEY_INVALID;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const float v = x[c];
    if (!isfinite(v)) continue;
    unsigned o = orderable(v);
    if (mode == TOP) o = ~o;
    const unsigned long long key = (static_cast<unsigned long long>(o) << 32) | static_cast<unsigned>(c);
    best = key < best ? key : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other < best ? other : best;
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = best;
  __syncthreads();
  if (w == 0) {
    best = l < (blockDim.x >> 5) ? sh[l] : KEY_INVALID;
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other < best ? other : best;
    }
    if (l == 0) {
      if (best == KEY_INVALID) {
        out_v[row] = __int_as_float(0x7FC00000);
        out_i[row] = -1;
      } else {
        unsigned o = static_cast<unsigned>(best >> 32);
        if (mode == TOP) o = ~o;
        out_v[row] = from_orderable(o);
        out_i[row] = static_cast<int>(best & 0xFFFFFFFFu);
      }
    }
  }
}

// ---- top / bottom with k <= 128: warp-resident candidate lists ------------------------------------------------------
// A row is read once, so the bound is its bytes.  What made the full sort slow was shared memory: 78 exchange stages
// over 4096 keys per row.  Here an element costs one comparison with a bound on the k-th best value; the few that pass
// go to a small queue, and a full queue is sorted in registers and merged into the list.  4096 x 4096, k = 32: 19.4 us
// (the bytes take 10), bound by the latency of two passes over a row; two sorts of row halves and the merge of
// their lists took 669.
using u64 = unsigned long long;
constexpr int TOPK_MAX_K = 128;
constexpr int TOPK_GROUP = 128;             // columns of a warp-wide load: four per lane
constexpr int TOPK_STEP = 4 * TOPK_GROUP;   // columns per step of a warp: 2 KB of loads in flight
constexpr int topk_capacity(int R) { return 32 * R + TOPK_STEP; }
constexpr int TOPK_MAX_WARPS = 16;          // warps of one CTA on one row
constexpr int TOPK_BOUND_SHARE = 512;       // columns of a share per list register from which a bound is looked for first
__host__ __device__ inline int topk_share(int cols, int split) {
  return ((cols + split - 1) / split + TOPK_GROUP - 1) / TOPK_GROUP * TOPK_GROUP;
}

__device__ __forceinline__ u64 min64(u64 a, u64 b) { return a < b ? a : b; }
__device__ __forceinline__ u64 max64(u64 a, u64 b) { return a < b ? b : a; }

// Bitonic stages over 32 R keys, key i = 32 r + lane.  DESC sorts descending, otherwise ascending.
template <int R, bool DESC>
__device__ __forceinline__ void bitonic_stage(u64 (&v)[R], int size, int stride, int lane) {
  if (stride >= 32) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int rs = stride >> 5;
      if ((r & rs) == 0 && (r | rs) < R) {
        const bool up = (((r * 32) & size) == 0) != DESC;
        const u64 a = v[r], b = v[r | rs];
        v[r] = up ? min64(a, b) : max64(a, b);
        v[r | rs] = up ? max64(a, b) : min64(a, b);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const u64 other = __shfl_xor_sync(0xffffffffu, v[r], stride);
      const bool up = (((r * 32 + lane) & size) == 0) != DESC;
      v[r] = (((lane & stride) == 0) == up) ? min64(v[r], other) : max64(v[r], other);
    }
  }
}

template <int R>
__device__ __forceinline__ void sort_descending(u64 (&v)[R], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * R; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) bitonic_stage<R, true>(v, size, stride, lane);
}

// best (ascending) := the 32 R smallest of best and q (descending), ascending
template <int R>
__device__ __forceinline__ void keep_best(u64 (&best)[R], const u64 (&q)[R], int lane) {
#pragma unroll
  for (int r = 0; r < R; ++r) best[r] = min64(best[r], q[r]);
#pragma unroll
  for (int stride = 16 * R; stride > 0; stride >>= 1) bitonic_stage<R, false>(best, 64 * R, stride, lane);
}

// Pairwise merge of the lists of `warps` neighbouring warps, through their queues; the first of them ends with the result.
template <int R>
__device__ __forceinline__ void merge_warps(u64 (&best)[R], u64* queue, int wr, int warps, int lane) {
  constexpr int N = 32 * R, CAP = topk_capacity(R);
  for (int s = 1; s < warps; s <<= 1) {
    __syncthreads();
    if (wr & s) {
#pragma unroll
      for (int r = 0; r < R; ++r) queue[r * 32 + lane] = best[r];
    }
    __syncthreads();
    if ((wr & (2 * s - 1)) == 0) {
      const u64* other = queue + s * CAP;
      u64 q[R];
#pragma unroll
      for (int r = 0; r < R; ++r) q[r] = other[N - 1 - (r * 32 + lane)];
      keep_best<R>(best, q, lane);
    }
  }
}

template <int R>
__device__ __forceinline__ void write_best(const u64 (&best)[R], float* out_v, int* out_i, int k, bool top, int lane) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = r * 32 + lane;
    if (i >= k) continue;
    float val = __int_as_float(0x7FC00000);
    int idx = -1;
    if (best[r] != KEY_INVALID) {
      const unsigned o = static_cast<unsigned>(best[r] >> 32);
      val = from_orderable(top ? ~o : o);
      idx = static_cast<int>(best[r] & 0xFFFFFFFFu);
    }
    out_v[i] = val;
    out_i[i] = idx;
  }
}

// `warps` warps (a power of two) share a row, each with a contiguous share of its columns; a CTA holds
// blockDim / (32 warps) rows.  With parts > 1 a row is also split over `parts` CTAs, whose lists go to `lists`
// [rows][parts][N].  VEC: rows start at 16-byte boundaries and are read as float4.  BOUNDED: shares are long enough for a bound.
template <int R, bool VEC, bool TOP_MODE, bool BOUNDED>
__global__ void __launch_bounds__(TOPK_MAX_WARPS * 32)
rank_topk_kernel(const float* __restrict__ in, float* __restrict__ out_v, int* __restrict__ out_i, int rows, int cols,
                 int k, int warps, int parts, u64* __restrict__ lists) {
  chain_begin(in);
  constexpr int N = 32 * R, CAP = topk_capacity(R);
  extern __shared__ u64 queues[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wr = warp & (warps - 1);
  const long long row = (long long)(blockIdx.x / parts) * ((blockDim.x >> 5) / warps) + warp / warps;
  const int part = blockIdx.x % parts;
  u64* queue = queues + warp * CAP;
  u64 best[R];
#pragma unroll
  for (int r = 0; r < R; ++r) best[r] = KEY_INVALID;
  u64 thr = KEY_INVALID;                               // k-th best key so far
  float thr_v = TOP_MODE ? -FLT_MAX : FLT_MAX;         // a bound: an element beyond it cannot be among the k best, nor can infinities
  int qn = 0;
  if (row < rows) {
    const float* x = in + row * cols;
    const int share = topk_share(cols, warps * parts);
    const int c_begin = (int)min((long long)cols, (long long)(part * warps + wr) * share), c_end = min(cols, c_begin + share);
    // element j of a group sits at column 4 lane + j (VEC) or lane + 32 j; columns past the share read as NaN, which
    // fails every comparison
    auto load = [&](int c0) {
      float4 f = make_float4(NAN, NAN, NAN, NAN);
      if constexpr (VEC) {
        if (c0 + lane * 4 < c_end) f = *reinterpret_cast<const float4*>(x + c0 + lane * 4);
      } else {
        const int c = c0 + lane;
        if (c < c_end) f.x = x[c];
        if (c + 32 < c_end) f.y = x[c + 32];
        if (c + 64 < c_end) f.z = x[c + 64];
        if (c + 96 < c_end) f.w = x[c + 96];
      }
      return f;
    };
    // A bound on the k-th best before the lists start: every lane keeps 2 R maxima (minima), each over its own part of
    // the share; k of the warp's 64 R parts hold a value at least as good as the k-th best of these, so the k-th best of
    // the row does too.  With 64 parts and k = 32 about 45 of 4096 elements then pass, instead of some 300 with a list
    // that starts empty, whose sorts were most of the time.  The second read of the share comes from L2.
    bool infinities = true;                         // whether the share may hold the infinity on the better side
    if (BOUNDED && c_end - c_begin >= TOPK_BOUND_SHARE * R) {
      constexpr int PARTS = 2 * R;
      float ext[PARTS];
#pragma unroll
      for (int g = 0; g < PARTS; ++g) ext[g] = TOP_MODE ? -INFINITY : INFINITY;
      constexpr int AHEAD = 8;                      // loads in flight per lane
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += TOPK_GROUP * AHEAD) {
        float4 f[AHEAD];
#pragma unroll
        for (int g = 0; g < AHEAD; ++g) f[g] = load(c0 + g * TOPK_GROUP);
#pragma unroll
        for (int g = 0; g < AHEAD; ++g) {
          float& e = ext[g % PARTS];
          e = TOP_MODE ? fmaxf(fmaxf(fmaxf(e, f[g].x), fmaxf(f[g].y, f[g].z)), f[g].w)
                       : fminf(fminf(fminf(e, f[g].x), fminf(f[g].y, f[g].z)), f[g].w);
        }
      }
      bool infinite = false;
#pragma unroll
      for (int g = 0; g < PARTS; ++g) infinite |= ext[g] == (TOP_MODE ? INFINITY : -INFINITY);
      infinities = __any_sync(0xffffffffu, infinite);
      unsigned better[PARTS];                       // larger is better; 0 for a part whose extreme is not finite
#pragma unroll
      for (int g = 0; g < PARTS; ++g) better[g] = !isfinite(ext[g]) ? 0u : (TOP_MODE ? orderable(ext[g]) : ~orderable(ext[g]));
      unsigned bound = 0;                           // the upper 16 bits of the k-th best, found bit by bit
#pragma unroll 1
      for (unsigned bit = 0x80000000u; bit >= 0x10000u; bit >>= 1) {
        int n = 0;
#pragma unroll
        for (int g = 0; g < PARTS; ++g) n += __popc(__ballot_sync(0xffffffffu, better[g] >= (bound | bit)));
        if (n >= k) bound |= bit;
      }
      // the smallest finite values share their upper bits with infinities and NaNs: no bound then
      if (bound >= 0x00800000u) thr_v = from_orderable(TOP_MODE ? bound : ~bound);
    }
    // The queue and merge code sits once in a rolled loop: unrolled per element it outgrew the instruction cache.
    // With a bound few elements pass: a step's loads are under way while the step before it is examined, and a lane marks its
    // elements that pass and hands over one mark at a time, so that a step takes as many rounds as the lane with the most marks
    // has.  Without one most of the first steps pass, and the sixteen elements are voted on in turn.
    // us, votes and marks: 4096 x 4096, k = 32, 24.0 and 20.6 (from DRAM 31 and 27); 335 x 50000 35.3 and 26.4; 3000 x 4100, k = 128,
    // 43.3 and 38.9; without a bound 16 x 50000 23.4 and 25.7, 8192 x 512, k = 64, 61 and 67.
    float4 next[4];
    if constexpr (BOUNDED) {
#pragma unroll
      for (int g = 0; g < 4; ++g) next[g] = load(c_begin + g * TOPK_GROUP);
    }
#pragma unroll 1
    for (int c0 = c_begin; c0 < c_end; c0 += TOPK_STEP) {
      float v[16];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float4 f = BOUNDED ? next[g] : load(c0 + g * TOPK_GROUP);
        v[4 * g] = f.x; v[4 * g + 1] = f.y; v[4 * g + 2] = f.z; v[4 * g + 3] = f.w;
        if constexpr (BOUNDED) next[g] = load(c0 + TOPK_STEP + g * TOPK_GROUP);
      }
      // equal values are decided by the whole key: the lower column wins
      auto enqueue = [&](float e, int j, bool near) {
        const int c = c0 + (j >> 2) * TOPK_GROUP + (VEC ? lane * 4 + (j & 3) : lane + 32 * (j & 3));
        unsigned o = orderable(e);
        if (TOP_MODE) o = ~o;
        const u64 key = (static_cast<u64>(o) << 32) | static_cast<unsigned>(c);
        const bool pass = near && isfinite(e) && key < thr;
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (pass) queue[qn + __popc(m & ((1u << lane) - 1u))] = key;
        qn += __popc(m);
      };
      auto near = [&](float e) { return TOP_MODE ? e >= thr_v : e <= thr_v; };
      if constexpr (BOUNDED) {
        unsigned marks = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) marks |= near(v[j]) ? 1u << j : 0u;
        // The infinity on the better side passes every bound, and every element that passes takes a round: 1257 x 26588, seven of ten -inf,
        // bottom 4, 155 us so and 57 without their marks.  Only where there is one: 4096 x 4096, k = 32, 27 us with a comparison each.
        if (infinities) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (isinf(v[j])) marks &= ~(1u << j);
        }
        while (__any_sync(0xffffffffu, marks != 0)) {
          const int j = marks ? __ffs(marks) - 1 : 0;
          float e8[8], e4[4], e2[2];                      // v[j]
#pragma unroll
          for (int i = 0; i < 8; ++i) e8[i] = j & 1 ? v[2 * i + 1] : v[2 * i];
#pragma unroll
          for (int i = 0; i < 4; ++i) e4[i] = j & 2 ? e8[2 * i + 1] : e8[2 * i];
#pragma unroll
          for (int i = 0; i < 2; ++i) e2[i] = j & 4 ? e4[2 * i + 1] : e4[2 * i];
          enqueue(j & 8 ? e2[1] : e2[0], j, marks != 0);
          marks &= marks - 1;
        }
      } else {
        bool any = false;
#pragma unroll
        for (int j = 0; j < 16; ++j) any |= near(v[j]);
        if (__any_sync(0xffffffffu, any)) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (__any_sync(0xffffffffu, near(v[j]))) enqueue(v[j], j, near(v[j]));
        }
      }
      // full queue, or the end of the share: sort it and merge it into the list
      while (qn >= N || (qn > 0 && c0 + TOPK_STEP >= c_end)) {
        __syncwarp();
        const int n = min(qn, N);
        qn -= n;
        u64 q[R];                                    // the newest keys; the order in the queue does not matter
#pragma unroll
        for (int r = 0; r < R; ++r) q[r] = r * 32 + lane < n ? queue[qn + r * 32 + lane] : KEY_INVALID;
        __syncwarp();
        sort_descending<R>(q, lane);
        keep_best<R>(best, q, lane);
        u64 t = best[0];
#pragma unroll
        for (int r = 1; r < R; ++r)
          if (r == (k - 1) >> 5) t = best[r];
        thr = __shfl_sync(0xffffffffu, t, (k - 1) & 31);
        if (thr != KEY_INVALID) {
          // the next better value: in the columns to come an equal one loses against the k-th best, which stands further left.
          // With the value itself rows of few values passed whole: 859 x 17693 equal ones, k = 1, 71 us and 44.
          const unsigned o = static_cast<unsigned>(thr >> 32);
          thr_v = from_orderable(TOP_MODE ? ~o + 1u : o - 1u);
        }
      }
    }
  }
  merge_warps<R>(best, queue, wr, warps, lane);
  if (wr != 0 || row >= rows) return;
  if (parts > 1) {
#pragma unroll
    for (int r = 0; r < R; ++r) lists[(row * parts + part) * N + r * 32 + lane] = best[r];
    return;
  }
  write_best<R>(best, out_v + row * k, out_i + row * k, k, TOP_MODE, lane);
}

// Merges the `parts` lists of every row; one CTA per row.
constexpr int MERGE_WARPS = 8;
template <int R>
__global__ void __launch_bounds__(MERGE_WARPS * 32)
rank_merge_kernel(const u64* __restrict__ lists, float* __restrict__ out_v, int* __restrict__ out_i, int k, int parts, int top) {
  chain_begin(lists);
  constexpr int N = 32 * R, CAP = topk_capacity(R);
  __shared__ u64 queues[MERGE_WARPS * CAP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row = blockIdx.x;
  u64 best[R];
#pragma unroll
  for (int r = 0; r < R; ++r) best[r] = KEY_INVALID;
  for (int part = warp; part < parts; part += MERGE_WARPS) {
    u64 q[R];
#pragma unroll
    for (int r = 0; r < R; ++r) q[r] = lists[(row * parts + part) * N + N - 1 - (r * 32 + lane)];
    keep_best<R>(best, q, lane);
  }
  merge_warps<R>(best, queues + warp * CAP, warp, MERGE_WARPS, lane);
  if (warp == 0) write_best<R>(best, out_v + row * k, out_i + row * k, k, top != 0, lane);
}

// CTAs that share a row: fewer than 16 warps per SM over all rows leaves loads unissued, so a wide row (above the
// 8192 columns that one CTA of 16 warps reads in a few microseconds) is split until there are enough, but not below 256 columns
// per warp of an 8-warp CTA.
int topk_parts(int rows, int cols) {
  if (cols <= 8192 || (long long)rows * 32 >= 16ll * st::sm_count()) return 1;
  const long long want = (2ll * st::sm_count() + rows - 1) / rows, most = cols / (8 * 256);
  const long long parts = want < most ? want : most;
  return (int)(parts < 64 ? parts : 64);
}
int topk_list(int k) { return k <= 32 ? 1 : (k <= 64 ? 2 : 4); }

template <int R, bool VEC>
int launch_topk(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, u64* lists, cudaStream_t s) {
  // Enough warps to keep every SM's loads in flight (16 warps x 2 KB per SM), as long as a warp's share of the row is
  // at least 256 columns: below that the warp spends its time filling and merging lists instead of reading.
  const int parts = lists ? topk_parts(rows, cols) : 1;
  int warps = parts > 1 ? 8 : 1;
  while (parts == 1 && warps < TOPK_MAX_WARPS && (long long)rows * warps < 16ll * st::sm_count() && cols / (2 * warps) >= 256)
    warps <<= 1;
  // four warps per CTA where they suffice: 4096 rows are 6.9 such CTAs per SM, but 3.5 of eight, a last wave half empty
  const int threads = (warps <= 4 ? 4 : warps) * 32;
  const int per_cta = (threads / 32) / warps;
  const int grid = ((rows + per_cta - 1) / per_cta) * parts;
  const size_t smem = (size_t)(threads / 32) * topk_capacity(R) * sizeof(u64);
  auto run = [&](auto kernel, bool* cfg) -> int {
    const int dev = st::current_device();      // the attribute is per device
    if (!cfg[dev]) {
      const int most = TOPK_MAX_WARPS * topk_capacity(R) * (int)sizeof(u64);       // at most 80 KB
      ST_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
      cfg[dev] = true;
    }
    // Up to six blocks per SM in order: blocks that start while the kernel before them drains pile up on the SMs that fall free first, and
    // nothing evens them out.  us with a product of 2048 x 4096 x 1024 before it (included), early and in order: 29 x 1002, k = 47, 52
    // and 28; 2995 x 13521, k = 59, 126 and 95.  With more blocks the earlier start gains: 4096 x 4096, k = 32, one after the other,
    // 25.3 early and 28.7 in order.
    const bool early = grid > 6 * st::sm_count();
    ST_CUDA_CHECK((early ? st::chained(kernel, grid, threads, smem, s) : st::in_order(kernel, grid, threads, smem, s))(
        in, out_v, out_i, rows, cols, k, warps, parts, lists));
    return ST_OK;
  };
  static bool cfg[4][st::kMaxDevices] = {{false}};
  const bool bounded = topk_share(cols, warps * parts) >= TOPK_BOUND_SHARE * R;
  const int rc = mode == TOP ? (bounded ? run(rank_topk_kernel<R, VEC, true, true>, cfg[0]) : run(rank_topk_kernel<R, VEC, true, false>, cfg[1]))
                             : (bounded ? run(rank_topk_kernel<R, VEC, false, true>, cfg[2]) : run(rank_topk_kernel<R, VEC, false, false>, cfg[3]));
  if (rc != ST_OK) return rc;
  if (parts > 1) {
    ST_CUDA_CHECK(st::chained(rank_merge_kernel<R>, rows, MERGE_WARPS * 32, 0, s)(lists, out_v, out_i, k, parts, mode == TOP));
  }
  return ST_OK;
}

template <bool VEC>
int launch_topk_list(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, u64* lists, cudaStream_t s) {
  // the list is the smallest that holds k: a longer one only makes the merges dearer
  switch (topk_list(k)) {
    case 1: return launch_topk<1, VEC>(in, out_v, out_i, rows, cols, k, mode, lists, s);
    case 2: return launch_topk<2, VEC>(in, out_v, out_i, rows, cols, k, mode, lists, s);
    default: return launch_topk<4, VEC>(in, out_v, out_i, rows, cols, k, mode, lists, s);
  }
}

int dispatch_topk(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, u64* lists, cudaStream_t s) {
  const bool vec = (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  return vec ? launch_topk_list<true>(in, out_v, out_i, rows, cols, k, mode, lists, s)
             : launch_topk_list<false>(in, out_v, out_i, rows, cols, k, mode, lists, s);
}

// ---- any range of ranks: radix select, then a sort of the range only --------------------------------------------------
// The keys of ranks [start, start + take) of the ascending order: top / bottom have start = 0, mid the centred range.
// Three digits (11, 11, 10 bits) of a histogram in shared memory give the value at a rank; elements strictly between
// the two boundary values are taken in any order, elements equal to one of them by their column order when not all of
// them belong to the range.
constexpr int RANGE_THREADS = 512;
constexpr int RANGE_BINS = 2048;
constexpr unsigned ORD_INVALID = 0xFFFFFFFFu;     // no finite value maps to it

__global__ void __launch_bounds__(RANGE_THREADS)
rank_range_kernel(const float* __restrict__ in, float* __restrict__ out_v, int* __restrict__ out_i, int cols, int k,
                  int mode, int key_slots) {
  extern __shared__ u64 range_keys[];              // key_slots keys, then the row's ordered bits
  unsigned* ord = reinterpret_cast<unsigned*>(range_keys + key_slots);
  __shared__ int hist[RANGE_BINS];
  __shared__ int s_finite, s_bin, s_before, s_equal, s_taken;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row = blockIdx.x;
  const float* x = in + row * cols;
  if (threadIdx.x == 0) { s_finite = 0; s_taken = 0; }
  __syncthreads();
  int local = 0;
  for (int c = threadIdx.x; c < cols; c += RANGE_THREADS) {
    const float v = x[c];
    unsigned o = ORD_INVALID;
    if (isfinite(v)) {
      o = orderable(v);
      if (mode == TOP) o = ~o;
      ++local;
    }
    ord[c] = o;
  }
  local = __reduce_add_sync(0xffffffffu, local);
  if (lane == 0) atomicAdd(&s_finite, local);
  __syncthreads();
  const int finite = s_finite, take = min(k, finite);
  const int start = mode == MID ? (finite - take) / 2 : 0;

  // value at `rank` of the ascending order, how many are smaller and how many equal it
  auto value_at = [&](int rank, unsigned& value, int& less, int& equal) {
    unsigned prefix = 0, mask = 0;
    less = 0;
    equal = 0;
#pragma unroll 1
    for (int digit = 0; digit < 3; ++digit) {
      const int shift = digit == 0 ? 21 : (digit == 1 ? 10 : 0);
      const unsigned bins = digit == 2 ? 1024u : 2048u;
      for (int i = threadIdx.x; i < RANGE_BINS; i += RANGE_THREADS) hist[i] = 0;
      __syncthreads();
      for (int c = threadIdx.x; c < cols; c += RANGE_THREADS) {
        const unsigned o = ord[c];
        if (o != ORD_INVALID && (o & mask) == prefix) atomicAdd(&hist[(o >> shift) & (bins - 1)], 1);
      }
      __syncthreads();
      if (warp == 0) {
        const int per = RANGE_BINS / 32;
        int sum = 0;
        for (int i = 0; i < per; ++i) sum += hist[lane * per + i];
        int upto = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, upto, d);
          if (lane >= d) upto += t;
        }
        int before = upto - sum;
        if (rank >= before && rank < upto) {
          int b = lane * per;
          while (rank >= before + hist[b]) before += hist[b++];
          s_bin = b; s_before = before; s_equal = hist[b];
        }
      }
      __syncthreads();
      prefix |= static_cast<unsigned>(s_bin) << shift;
      mask |= (bins - 1) << shift;
      rank -= s_before;
      less += s_before;
      equal = s_equal;
      __syncthreads();
    }
    value = prefix;
  };

  if (take > 0) {
    unsigned v_lo = 0, v_hi = 0;
    int less_lo = 0, equal_lo = 0, less_hi = 0, equal_hi = 0;
    value_at(start + take - 1, v_hi, less_hi, equal_hi);
    if (start > 0) value_at(start, v_lo, less_lo, equal_lo);
    // not every element of a boundary value is in the range: those are picked in column order
    const bool cut_lo = start > less_lo, cut_hi = less_hi + equal_hi > start + take;
    for (int c = threadIdx.x; c < cols; c += RANGE_THREADS) {
      const unsigned o = ord[c];
      if (o == ORD_INVALID || o < v_lo || o > v_hi) continue;
      if ((cut_lo && o == v_lo) || (cut_hi && o == v_hi)) continue;
      range_keys[atomicAdd(&s_taken, 1)] = (static_cast<u64>(o) << 32) | static_cast<unsigned>(c);
    }
    __syncthreads();
    if (warp == 0 && (cut_lo || cut_hi)) {
      int n = s_taken, seen_lo = 0, seen_hi = 0;
      for (int c0 = 0; c0 < cols; c0 += 32) {
        const int c = c0 + lane;
        const unsigned o = c < cols ? ord[c] : ORD_INVALID;
        const bool lo = cut_lo && o == v_lo && c < cols, hi = cut_hi && o == v_hi && c < cols;
        const unsigned m_lo = __ballot_sync(0xffffffffu, lo), m_hi = __ballot_sync(0xffffffffu, hi);
        const unsigned below = (1u << lane) - 1u;
        const int rank = lo ? less_lo + seen_lo + __popc(m_lo & below) : less_hi + seen_hi + __popc(m_hi & below);
        const bool in_range = (lo || hi) && rank >= start && rank < start + take;
        const unsigned m = __ballot_sync(0xffffffffu, in_range);
        if (in_range) range_keys[n + __popc(m & below)] = (static_cast<u64>(o) << 32) | static_cast<unsigned>(c);
        n += __popc(m);
        seen_lo += __popc(m_lo);
        seen_hi += __popc(m_hi);
      }
    }
  }
  __syncthreads();
  for (int i = take + threadIdx.x; i < key_slots; i += RANGE_THREADS) range_keys[i] = KEY_INVALID;
  __syncthreads();
  for (int size = 2; size <= key_slots; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < key_slots / 2; t += RANGE_THREADS) {
        const int lo = (t / stride) * (stride << 1) + (t % stride);
        const u64 a = range_keys[lo], b = range_keys[lo + stride];
        if ((a > b) == ((lo & size) == 0)) {
          range_keys[lo] = b;
          range_keys[lo + stride] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < k; i += RANGE_THREADS) {
    float v = __int_as_float(0x7FC00000);
    int idx = -1;
    if (i < take) {
      const u64 key = range_keys[i];
      const unsigned o = static_cast<unsigned>(key >> 32);
      v = from_orderable(mode == TOP ? ~o : o);
      idx = static_cast<int>(key & 0xFFFFFFFFu);
    }
    out_v[row * k + i] = v;
    out_i[row * k + i] = idx;
  }
}

__global__ void __launch_bounds__(256)
compact_rows_kernel(const float* __restrict__ in, float* __restrict__ out_v, int* __restrict__ out_i,
                    int* __restrict__ counts, int rows, int cols, float low, float high) {
  __shared__ int warp_tot[8];
  __shared__ int base;
  const int row = blockIdx.x;
  const float* x = in + (size_t)row * cols;
  float* ov = out_v + (size_t)row * cols;
  int* oi = out_i + (size_t)row * cols;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int c0 = 0; c0 < cols; c0 += 256) {
    const int c = c0 + threadIdx.x;
    const float v = c < cols ? x[c] : 0.0f;
    const bool keep = c < cols && v >= low && v <= high;  // NaN fails both comparisons
    const unsigned ballot = __ballot_sync(0xffffffffu, keep);
    const int in_warp = __popc(ballot & ((1u << l) - 1u));
    if (l == 0) warp_tot[w] = __popc(ballot);
    __syncthreads();
    int before = base;
    for (int i = 0; i < w; ++i) before += warp_tot[i];
    if (keep) {
      ov[before + in_warp] = v;
      oi[before + in_warp] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int i = 0; i < 8; ++i) t += warp_tot[i];
      base += t;
    }
    __syncthreads();
  }
  const int n = base;
  for (int c = n + threadIdx.x; c < cols; c += 256) {
    ov[c] = 0.0f;
    oi[c] = 0;
  }
  if (threadIdx.x == 0) counts[row] = n;
}

// dst[r, p*k + s] = src_p[r, s] for every peer p: gathers the candidate lists of all ranks.
__global__ void gather_candidates_kernel(const float* const* __restrict__ vals, const int* const* __restrict__ idxs,
                                         float* __restrict__ dst_v, int* __restrict__ dst_i, int world,
                                         int rows, int k) {
  const long long total = (long long)world * rows * k;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int s = i % k;
    const long long t = i / k;
    const int r = t % rows;
    const int p = t / rows;
    dst_v[((long long)r * world + p) * k + s] = vals[p][(long long)r * k + s];
    dst_i[((long long)r * world + p) * k + s] = idxs[p][(long long)r * k + s];
  }
}

}  // namespace

// Whether the radix select and the sort of its range (key_slots) beat the sort of the whole row (padded columns).  The select is
// a chain of histograms, about 17 us for one row and 150 to 200 for 4096, whatever the row's length; the sort grows with it.
// Sort against select, in us: 4096 rows of 64: 9.6 and 160, of 256: 39 and 178, of 512: 90 and 182 (k = 32 and less), of 606:
// 217 and 189; k = 128 217 and 214; k = 250 218 and 235.  600 rows of 1000: k = 32 45 and 41, k = 250 45 and 49; one row 16 and
// 18.  Top and bottom have one boundary to find: 1000 rows of 606, k = 200 59 and 47, k = 500 59 and 63.  From 2048 columns on the
// sort loses (1 x 1500 30 and 15, 4096 x 4096 1108 and 215), except for a few rows with a range of half the row (1 x 2000,
// k = 1000: 30 and 34).
static bool range_pays(int rows, int padded, int key_slots, int mode) {
  const int sms = st::sm_count();
  if (2 * key_slots > padded || padded <= 512) return false;
  if (padded > 1024) return padded > 2048 || mode != MID || 2 * key_slots < padded || rows >= sms / 2;
  if (mode != MID) return rows >= 4 * sms && (key_slots <= 256 || rows >= 16 * sms);
  return rows >= (key_slots <= 32 ? 2 : 16) * sms && key_slots <= 128;
}

// mode: 0 top, 1 bottom, 2 mid.  in: fp32 [rows, cols]; out_v fp32 [rows, k]; out_i int32 [rows, k].
ST_API int st_rank_select(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode,
                          void* stream_v) {
  if (rows < 0 || cols < 0 || k < 0) return st::fail(ST_ERR_INVALID, "rank_select: negative dimension");
  if (rows == 0 || k == 0) return ST_OK;
  if (mode < 0 || mode > 2) return st::fail(ST_ERR_INVALID, "rank_select: mode must be 0 (top), 1 (bottom) or 2 (mid)");
  if (cols > 8192) return st::fail(ST_ERR_TOO_LARGE, "rank_select: rows of more than 8192 columns are not supported");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_v);
  // One value needs no list: rows of 64 / 1000 / 4096 columns, up to 600 of them, take 2.0 / 5.3 / 5.5 us (1.8 to 2.4 times that
  // with a list, which fills and merges before it knows anything).  Many long rows are bound by their bytes, which warps with
  // lists keep in flight better: 2400 x 1500 7.4 us against 7.0, 4096 x 4096 21.9 against 12.9; one row of 8192 8.4 against 6.1.
  if (mode != MID && k == 1 && cols <= 4096 && (cols <= 1024 || rows <= 8 * st::sm_count())) {
    rank_k1_kernel<<<rows, cols >= 1024 ? 256 : 64, 0, s>>>(in, out_v, out_i, rows, cols, mode);
    ST_CUDA_CHECK(cudaGetLastError());
    return ST_OK;
  }
  if (mode != MID && k <= TOPK_MAX_K) return dispatch_topk(in, out_v, out_i, rows, cols, k, mode, nullptr, s);
  int padded = 2;
  while (padded < cols) padded <<= 1;
  int key_slots = 2;
  while (key_slots < k) key_slots <<= 1;
  static bool cfg[st::kMaxDevices] = {false};      // the attribute is per device
  const int dev = st::current_device();
  if (!cfg[dev]) {
    ST_CUDA_CHECK(cudaFuncSetAttribute(rank_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * 8));
    ST_CUDA_CHECK(cudaFuncSetAttribute(rank_range_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4096 * 8 + 8192 * 4));
    cfg[dev] = true;
  }
  if (range_pays(rows, padded, key_slots, mode)) {
    const size_t range_smem = (size_t)key_slots * sizeof(unsigned long long) + (size_t)cols * sizeof(unsigned);
    rank_range_kernel<<<rows, RANGE_THREADS, range_smem, s>>>(in, out_v, out_i, cols, k, mode, key_slots);
    ST_CUDA_CHECK(cudaGetLastError());
    return ST_OK;
  }
  const size_t smem = (size_t)padded * sizeof(unsigned long long);
  int threads = padded / 2;
  threads = threads < 32 ? 32 : (threads > 1024 ? 1024 : threads);
  rank_select_kernel<<<rows, threads, smem, s>>>(in, out_v, out_i, rows, cols, k, mode, padded);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// 64-bit words of workspace that st_rank_topk wants for few wide rows (0: none; the rows are not split).
ST_API long long st_rank_topk_workspace(int rows, int cols, int k) {
  if (rows <= 0 || cols <= 0 || k <= 0 || k > TOPK_MAX_K) return 0;
  const int parts = topk_parts(rows, cols);
  return parts > 1 ? (long long)rows * parts * 32 * topk_list(k) : 0;
}

// Top (mode 0) or bottom (mode 1) with k <= 128 over rows of any length, e.g. a vocabulary: same outputs as st_rank_select.
// workspace: st_rank_topk_workspace words, or null (then one CTA reads a row).
ST_API int st_rank_topk(const float* in, float* out_v, int* out_i, int rows, int cols, int k, int mode, void* workspace,
                        void* stream_v) {
  if (rows < 0 || cols < 0 || k < 0) return st::fail(ST_ERR_INVALID, "rank_topk: negative dimension");
  if (rows == 0 || k == 0) return ST_OK;
  if (mode != TOP && mode != BOTTOM) return st::fail(ST_ERR_INVALID, "rank_topk: mode must be 0 (top) or 1 (bottom)");
  if (k > TOPK_MAX_K) return st::fail(ST_ERR_TOO_LARGE, "rank_topk: at most 128 candidates");
  return dispatch_topk(in, out_v, out_i, rows, cols, k, mode, static_cast<u64*>(workspace), reinterpret_cast<cudaStream_t>(stream_v));
}

ST_API int st_compact_rows(const float* in, float* out_v, int* out_i, int* counts, int rows, int cols,
                           float low, float high, void* stream_v) {
  if (rows < 0 || cols < 0) return st::fail(ST_ERR_INVALID, "compaction dimensions must be non-negative");
  if (!(low <= high) || isinf(low) || isinf(high))
    return st::fail(ST_ERR_INVALID, "compaction bounds must be finite and ordered");
  if (rows == 0) return ST_OK;
  compact_rows_kernel<<<rows, 256, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(in, out_v, out_i, counts,
                                                                                 rows, cols, low, high);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}

// vals / idxs: device arrays of `world` pointers (peer memory allowed) to [rows, k] candidate lists.
ST_API int st_gather_candidates(const void* vals, const void* idxs, float* dst_v, int* dst_i, int world,
                                int rows, int k, void* stream_v) {
  const long long total = (long long)world * rows * k;
  if (total <= 0) return ST_OK;
  long long blocks = (total + 255) / 256;
  if (blocks > 1024) blocks = 1024;
  gather_candidates_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream_v)>>>(
      static_cast<const float* const*>(vals), static_cast<const int* const*>(idxs), dst_v, dst_i, world, rows, k);
  ST_CUDA_CHECK(cudaGetLastError());
  return ST_OK;
}
