// Batched k-means that reproduces the reference's CPU k-means bit for bit
// (kodama_matrix.cpp:664-799 kmeans_labels, CPU branch): a batch is P
// independent problems of n rows each (rows picked from one device matrix),
// k clusters, at most max_iter Lloyd iterations with early exit, then a final
// assignment.
//
// Float order contract (the reference is built for x86-64 without FMA):
//   dot(a,b): 16 partial sums p[l] over i = l mod 16 on the leading multiple of
//     16, lanes ((p[l]+p[l+4]) + (p[l+8]+p[l+12])), then ((l0+l1)+l2)+l3, then
//     the tail added one product at a time (dot_float32 :91-122, SSE branch);
//   distance = (|x|^2 + |c|^2) - 2*dot, ties to the lower cluster;
//   centroid sums in ascending row order (:778-791), scaled by 1/size;
//   empty clusters split from a donor picked by a float Fenwick tree over
//   max(0, size-1) with mt19937(1234) uniforms (:566-662).
// Every product and sum uses explicit round-to-nearest intrinsics.
#include "bf16_split.cuh"
#include "kmeans.cuh"
#include "knn.cuh"
#include "launch_count.cuh"
#include "smem_limit.cuh"
#include "tcgen05.cuh"

#include <cuda_runtime.h>
#include <math.h>

#include <cmath>

namespace kgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
// std::max(0.0f, v)
__device__ __forceinline__ float pos_part(float v) { return (0.0f < v) ? v : 0.0f; }

// dot in the x86 SSE order; a from registers/global, b from shared/global.
template <class A, class B>
__device__ __forceinline__ float dot_x86(A a, B b, int d) {
  float p[16];
#pragma unroll
  for (int l = 0; l < 16; ++l) p[l] = 0.0f;
  int i = 0;
  for (; i + 15 < d; i += 16) {
#pragma unroll
    for (int l = 0; l < 16; ++l) p[l] = fadd(p[l], fmul(a(i + l), b(i + l)));
  }
  float lane[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) lane[l] = fadd(fadd(p[l], p[4 + l]), fadd(p[8 + l], p[12 + l]));
  float sum = fadd(fadd(fadd(lane[0], lane[1]), lane[2]), lane[3]);
  for (; i < d; ++i) sum = fadd(sum, fmul(a(i), b(i)));
  return sum;
}

__global__ void row_norms_kernel(const float* __restrict__ x, int n, int d, float* __restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const float* xr = x + static_cast<size_t>(r) * d;
  out[r] = dot_x86([&](int j) { return xr[j]; }, [&](int j) { return xr[j]; }, d);
}

__global__ void init_centroids_kernel(KMeansBatch B) {
  const int p = blockIdx.y;
  const int c = blockIdx.x;
  const int orow = B.init_rows[static_cast<size_t>(p) * B.k + c];
  const int grow = B.rows ? B.rows[static_cast<size_t>(p) * B.n + orow] : orow;
  float* cent = B.cent + (static_cast<size_t>(p) * B.k + c) * B.d;
  for (int j = threadIdx.x; j < B.d; j += blockDim.x) cent[j] = B.x[static_cast<size_t>(grow) * B.d + j];
  if (threadIdx.x == 0 && c == 0) {
    B.active[p] = 1;
    B.changed[p] = 0;
  }
}

__global__ void centroid_norms_kernel(KMeansBatch B, int final_pass) {
  const int p = blockIdx.y;
  if (!final_pass && !B.active[p]) return;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= B.k) return;
  const float* cent = B.cent + (static_cast<size_t>(p) * B.k + c) * B.d;
  B.cnorm[static_cast<size_t>(p) * B.k + c] =
      dot_x86([&](int j) { return cent[j]; }, [&](int j) { return cent[j]; }, B.d);
}

// Two rows per thread; centroids of the problem staged in shared memory with
// rows padded to a multiple of 4 floats so they are read with 128-bit loads.
constexpr int kAssignRows = 2;

template <int NB>
__device__ __forceinline__ void dot2_x86(const float (&a)[kAssignRows][16 * NB], const float (&at)[kAssignRows][16],
                                         const float* b, int d, int nfull, float (&out)[kAssignRows]) {
  float p[kAssignRows][16];
#pragma unroll
  for (int q = 0; q < kAssignRows; ++q)
#pragma unroll
    for (int l = 0; l < 16; ++l) p[q][l] = 0.0f;
#pragma unroll
  for (int blk = 0; blk < NB; ++blk) {
    if (blk < nfull) {
#pragma unroll
      for (int l4 = 0; l4 < 4; ++l4) {
        const float4 c = *reinterpret_cast<const float4*>(b + 16 * blk + 4 * l4);
        const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
          for (int q = 0; q < kAssignRows; ++q)
            p[q][4 * l4 + e] = fadd(p[q][4 * l4 + e], fmul(a[q][16 * blk + 4 * l4 + e], cv[e]));
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kAssignRows; ++q) {
    float lane[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) lane[l] = fadd(fadd(p[q][l], p[q][4 + l]), fadd(p[q][8 + l], p[q][12 + l]));
    out[q] = fadd(fadd(fadd(lane[0], lane[1]), lane[2]), lane[3]);
  }
  // tail d - 16*nfull < 16 elements, held separately so indices stay static
  const int tn = d - 16 * nfull;
  const float* bt = b + 16 * nfull;
#pragma unroll
  for (int t = 0; t < 16; ++t) {
    if (t < tn) {
      const float bv = bt[t];
#pragma unroll
      for (int q = 0; q < kAssignRows; ++q) out[q] = fadd(out[q], fmul(at[q][t], bv));
    }
  }
}

template <int NB>
__global__ void assign_kernel(KMeansBatch B, int final_pass) {
  extern __shared__ float cs[];
  const int p = blockIdx.y;
  if (!final_pass && !B.active[p]) return;
  const int k = B.k, d = B.d;
  const int dp = (d + 3) & ~3;
  const float* cent = B.cent + static_cast<size_t>(p) * k * d;
  float* cn = cs + static_cast<size_t>(k) * dp;  // centroid norms, staged after the centroids
  for (int i = threadIdx.x; i < k * dp; i += blockDim.x) {
    const int c = i / dp, j = i % dp;
    cs[i] = j < d ? cent[static_cast<size_t>(c) * d + j] : 0.0f;
  }
  for (int c = threadIdx.x; c < k; c += blockDim.x) cn[c] = B.cnorm[static_cast<size_t>(p) * k + c];
  __syncthreads();
  const int r0 = (blockIdx.x * blockDim.x + threadIdx.x) * kAssignRows;
  if (r0 >= B.n) return;
  int grow[kAssignRows];
  bool live[kAssignRows];
#pragma unroll
  for (int q = 0; q < kAssignRows; ++q) {
    live[q] = r0 + q < B.n;
    const int r = live[q] ? r0 + q : r0;
    grow[q] = B.rows ? B.rows[static_cast<size_t>(p) * B.n + r] : r;
  }
  int best[kAssignRows];
  float bestd[kAssignRows];
  float pn[kAssignRows];
#pragma unroll
  for (int q = 0; q < kAssignRows; ++q) {
    best[q] = 0;
    bestd[q] = INFINITY;
    pn[q] = B.pnorm[grow[q]];
  }
  if constexpr (NB > 0) {
    const int nfull = d >> 4;
    float pt[kAssignRows][16 * NB];
    float ptail[kAssignRows][16];
#pragma unroll
    for (int q = 0; q < kAssignRows; ++q) {
#pragma unroll
      for (int j = 0; j < 16 * NB; ++j) pt[q][j] = j < 16 * nfull ? B.x[static_cast<size_t>(grow[q]) * d + j] : 0.0f;
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        const int j = 16 * nfull + t;
        ptail[q][t] = j < d ? B.x[static_cast<size_t>(grow[q]) * d + j] : 0.0f;
      }
    }
    for (int c = 0; c < k; ++c) {
      float dt[kAssignRows];
      dot2_x86<NB>(pt, ptail, cs + static_cast<size_t>(c) * dp, d, nfull, dt);
#pragma unroll
      for (int q = 0; q < kAssignRows; ++q) {
        const float dist = __fsub_rn(fadd(pn[q], cn[c]), fmul(2.0f, dt[q]));
        if (dist < bestd[q] || (dist == bestd[q] && c < best[q])) {
          bestd[q] = dist;
          best[q] = c;
        }
      }
    }
  } else {
    for (int c = 0; c < k; ++c) {
      const float* cc = cs + static_cast<size_t>(c) * dp;
#pragma unroll
      for (int q = 0; q < kAssignRows; ++q) {
        const float* xr = B.x + static_cast<size_t>(grow[q]) * d;
        const float dt = dot_x86([&](int j) { return xr[j]; }, [&](int j) { return cc[j]; }, d);
        const float dist = __fsub_rn(fadd(pn[q], cn[c]), fmul(2.0f, dt));
        if (dist < bestd[q] || (dist == bestd[q] && c < best[q])) {
          bestd[q] = dist;
          best[q] = c;
        }
      }
    }
  }
  int* as = B.assign + static_cast<size_t>(p) * B.n;
  bool moved = false;
#pragma unroll
  for (int q = 0; q < kAssignRows; ++q) {
    if (!live[q]) continue;
    const int r = r0 + q;
    if (final_pass) {
      B.labels[static_cast<size_t>(p) * B.n + r] = best[q] + 1;
    } else if (as[r] != best[q]) {
      as[r] = best[q];
      moved = true;
    }
  }
  // the reference only tests whether any assignment changed: one plain store
  // per warp instead of an atomic per row (per-row atomics on one counter
  // serialise in L2)
  const unsigned any = __ballot_sync(__activemask(), moved);
  if (any != 0u && (threadIdx.x & 31) == __ffs(__activemask()) - 1) B.changed[p] = 1;
}

// ---------------------------------------------------------------------------
// Tensor-core assignment.  Approximate distances a_c = |c|^2 - 2 dot_tc(x, c)
// (the canonical distance less |x|^2), where dot_tc is the bf16 hi + lo product
// (hi.hi + hi.lo + lo.hi) accumulated in f32 by tcgen05.mma and the norms are
// the exact ones of the canonical formula.  |a_c + |x|^2 - dist_c| <= delta
// (tc_error_factor), so the exact nearest centroid has a_c <= min a + 2 delta:
// a row with one such centroid takes it without an exact dot (an exact tie
// would make both tied centroids candidates); the others get the canonical
// x86-order distance for their candidates, ties to the lower cluster.  Rows or
// centroids with norms that are not finite or above 1e37 send every centroid
// to the exact distance.
//
// A CTA multiplies tiles of 128 rows with all k centroids (padded to 16) of a
// problem.  Warps 8-11 gather the rows' bf16 halves into a ring of 32-coordinate
// stages with cp.async (a row list scatters them, so no bulk copy), one thread
// issues the products into TMEM, and two groups of four warps (warps 0-7) take
// the tiles in turn: a thread owns one row of the accumulator, so minimum and
// candidate masks need no exchange between lanes.  Masks are formed in one pass
// against the running minimum, 32 centroids at a time; a chunk whose own
// minimum lies above the final threshold is dropped at the end.  Up to 256
// centroids there are two accumulators; above, one of up to 512 columns.
// The rows with several candidates are listed and get their exact distances from
// all warps after the tiles.
//
// The mma.sync form this replaces spent about 1400 warp instructions per 16
// rows on fragments, minima over quads and masks, and above 128 centroids the
// exact form had to take every x86-order dot.  Whole landmark k-means, device
// time before and now: 100 problems x 10000 rows x 50 coordinates, 50 clusters
// 3.55 -> 1.66 ms; with 300 clusters 41 -> 5.2 ms; 50 problems x 7500 rows x
// 200, 100 clusters 16.5 -> 3.5 ms.  What bounds it now: the products (92 cycles
// each at 64 centroids), the epilogue above 256 centroids (one accumulator),
// and in the sums the row gather from L2.
// ---------------------------------------------------------------------------
constexpr int kRows = 128;       // rows per tile (mma M = TMEM lanes)
constexpr int kThreads5 = 512;
constexpr int kWarps5 = kThreads5 / 32;
constexpr int kStageChunks = 8;  // 16-byte chunks of 8 coordinates per stage and row
constexpr int kMaxStages = 6;
constexpr int kMaxK = 512;       // accumulator columns
constexpr size_t kStageBytes = 2 * static_cast<size_t>(kStageChunks) * kRows * 16;  // hi and lo
constexpr size_t kSmemLimit = 227 * 1024;
constexpr size_t kShared5Room = 256;  // static shared memory of the kernels

struct Layout5 {
  int kpad, nch, stages;  // centroids padded to 16; 32-column chunks of the accumulator; row ring
  size_t o_b, o_a, o_cn, o_as, o_wh, o_off, o_fs, o_di, o_or, total;
};

__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~static_cast<size_t>(15); }

// persistent: also the problem's assignments and the grouping's tables.  The
// row ring takes the room that is left, two to six stages of 32 KB: about 1000
// cycles of L2 latency at the SM's 64 bytes a cycle are two stages in flight.
__host__ __device__ inline Layout5 layout5(int n, int k, int dp, bool persistent) {
  Layout5 L{};
  L.kpad = (k + 15) / 16 * 16;
  L.nch = (L.kpad + 31) / 32;
  size_t o = 0;
  L.o_b = o; o = align16(o + 2 * static_cast<size_t>(L.kpad) * dp * 2);
  L.o_cn = o; o = align16(o + sizeof(float) * L.nch * 32);
  if (persistent) {
    L.o_as = o; o = align16(o + sizeof(uint16_t) * static_cast<size_t>(n));
    L.o_wh = o; o = align16(o + sizeof(int) * kWarps5 * k);
    L.o_off = o; o = align16(o + sizeof(int) * (k + 1));
    L.o_fs = o; o = align16(o + sizeof(float) * (3 * k + 1));
    L.o_di = o; o = align16(o + k);
    L.o_or = o; o = align16(o + sizeof(uint16_t) * k);
  }
  L.o_a = o = (o + 1023) & ~static_cast<size_t>(1023);
  L.stages = kMaxStages;
  while (L.stages > 2 && o + L.stages * kStageBytes + kShared5Room > kSmemLimit) --L.stages;
  L.total = o + L.stages * kStageBytes;
  // one CTA per SM: it allocates all of the SM's TMEM
  if (L.total < 116 * 1024) L.total = 116 * 1024;
  return L;
}

struct Shared5 {
  uint64_t full[kMaxStages], ready[kMaxStages], empty[kMaxStages], afull[2], aempty[2], drain;
  uint32_t tmem;
  int stop;
  int changed, queue, multi, many;
  float cmax;
};
static_assert(sizeof(Shared5) <= kShared5Room, "static shared memory");

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait_groups() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// arrives at a barrier once this thread's copies issued so far have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// shared-memory writes this thread has made, or has seen through a barrier,
// become visible to the tensor core's reads
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// The x86-order dot by half a warp (all 16 lanes get it): lane l holds the
// partial sum over coordinates l + 16 b, the sixteen are combined in the
// reference's order and the tail is added one product at a time.
__device__ __forceinline__ float half_warp_dot(const float* a, const float* b, int d) {
  const int hl = threadIdx.x & 15, hb = threadIdx.x & 16, nfull = d >> 4, tn = d - 16 * nfull;
  const unsigned hm = 0xffffu << hb;
  float p = 0.0f;
#pragma unroll 4
  for (int i = 0; i < nfull; ++i) p = fadd(p, fmul(a[hl + 16 * i], b[hl + 16 * i]));
  const float tp = hl < tn ? fmul(a[16 * nfull + hl], b[16 * nfull + hl]) : 0.0f;
  const float q4 = __shfl_sync(hm, p, hb + ((hl + 4) & 15));
  const float q8 = __shfl_sync(hm, p, hb + ((hl + 8) & 15));
  const float q12 = __shfl_sync(hm, p, hb + ((hl + 12) & 15));
  const float lv = fadd(fadd(p, q4), fadd(q8, q12));
  float sum = fadd(fadd(fadd(__shfl_sync(hm, lv, hb), __shfl_sync(hm, lv, hb + 1)), __shfl_sync(hm, lv, hb + 2)),
                   __shfl_sync(hm, lv, hb + 3));
  for (int q = 0; q < tn; ++q) sum = fadd(sum, __shfl_sync(hm, tp, hb + q));
  return sum;
}

// The problem's centroid operand (bf16 halves), exact norms and their largest.
__device__ void stage_centroids(const KMeansBatch& B, const Layout5& L, unsigned char* sm, Shared5& sh,
                                const float* cent) {
  const int k = B.k, d = B.d, dp = B.dp, kpad = L.kpad;
  uint4* bh = reinterpret_cast<uint4*>(sm + L.o_b);
  uint4* bl = bh + static_cast<size_t>(kpad) * dp / 8;
  float* cn = reinterpret_cast<float*>(sm + L.o_cn);
  const int chunks = dp / 8;
  for (int e = threadIdx.x; e < kpad * chunks; e += kThreads5) {
    const int c = e / chunks, ch = e % chunks;
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t hb[2], lb[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int j = ch * 8 + 2 * q + s;
        const float v = c < k && j < d ? cent[static_cast<size_t>(c) * d + j] : 0.0f;
        hb[s] = bf16_bits(v);
        lb[s] = bf16_bits(__fsub_rn(v, __uint_as_float(hb[s] << 16)));
      }
      h[q] = hb[0] | (hb[1] << 16);
      l[q] = lb[0] | (lb[1] << 16);
    }
    bh[static_cast<size_t>(ch) * kpad + c] = make_uint4(h[0], h[1], h[2], h[3]);
    bl[static_cast<size_t>(ch) * kpad + c] = make_uint4(l[0], l[1], l[2], l[3]);
  }
  for (int c = threadIdx.x >> 4; c < L.nch * 32; c += kThreads5 / 16) {
    const float* cc = cent + static_cast<size_t>(c) * d;
    const float v = c < k ? half_warp_dot(cc, cc, d) : INFINITY;
    if ((threadIdx.x & 15) == 0) cn[c] = v;
  }
  fence_async_proxy();
  __syncthreads();
  if (threadIdx.x < 32) {
    // a NaN norm counts as +inf
    float mx = 0.0f;
    for (int c = threadIdx.x; c < k; c += 32) mx = fmaxf(mx, cn[c] >= 0.0f ? cn[c] : INFINITY);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
    if (threadIdx.x == 0) {
      sh.cmax = mx;
      sh.multi = 0;
      sh.many = 0;
    }
  }
  __syncthreads();
}

// Tiles and ring stages handled so far by this CTA (the same in every thread),
// from which every role takes its barrier phases.
struct Progress {
  int tiles = 0, stages = 0;
};

// Assigns the rows of tiles [t0, t1) of problem p.  put(row, cluster) stores a
// result.  Ends with a block barrier.
template <int NCH, class Put>
__device__ __forceinline__ void assign_tiles(const KMeansBatch& B, const Layout5& L, unsigned char* sm, Shared5& sh,
                                             uint32_t tmem, int p, int t0, int t1, const float* cent, Progress& pg,
                                             Put&& put) {
  const int n = B.n, k = B.k, d = B.d, dp = B.dp, kpad = L.kpad, chunks = dp / 8;
  const int warp = tc5::warp_index(), lane = threadIdx.x & 31;
  const int* rows = B.rows != nullptr ? B.rows + static_cast<size_t>(p) * n : nullptr;
  const int groups = (chunks + kStageChunks - 1) / kStageChunks;  // stages per tile
  const int nbuf = kpad <= 256 ? 2 : 1, S = L.stages;
  const float* cn = reinterpret_cast<const float*>(sm + L.o_cn);
  volatile int* stop = &sh.stop;
  // rows with two to four candidates from the front of the list, (row, id,
  // candidates), those with more from its back, (row, id, norm) and masks
  const int cap = min(n, t1 * kRows) - t0 * kRows;
  int4* list = B.multi + static_cast<size_t>(p) * n + static_cast<size_t>(t0) * kRows;
  uint32_t* lmask = B.multi_mask + (static_cast<size_t>(p) * n + static_cast<size_t>(t0) * kRows) * L.nch;
  const float cmax = sh.cmax;

  if (warp >= 8 && warp < 12) {
    // ---- row gather: warp w of the four takes rows 32 w .. 32 w + 31 of the
    // tile, four rows per copy instruction, the eight lanes of a row its 128
    // bytes (with 16-byte pieces of 16 rows per instruction the scattered
    // sectors held a tile to 3000 cycles)
    const uint32_t abase = tc5::smem_u32(sm + L.o_a);
    int s = pg.stages;
    bool ok = true;
    // the ids of the next tile's rows (a lane each) are fetched while this tile
    // is copied
    auto row_id = [&](int t) {
      const int r = min(t * kRows + (warp - 8) * 32 + lane, n - 1);
      return rows != nullptr ? rows[r] : r;
    };
    int next = row_id(t0);
    for (int t = t0; ok && t < t1; ++t) {
      const int id = next;
      if (t + 1 < t1) next = row_id(t + 1);
      for (int g = 0; g < groups; ++g, ++s) {
        ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.empty[s % S]), ((s / S) & 1) ^ 1, stop));
        if (!ok) break;
        const uint32_t dst = abase + (s % S) * kStageBytes;
        const int ch = g * kStageChunks + (lane & 7);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int grow = __shfl_sync(kFull, id, 4 * i + (lane >> 3));
          const int r = (warp - 8) * 32 + 4 * i + (lane >> 3);
          if (ch < chunks) {
            const uint32_t o = dst + r * 128 + (((lane & 7) ^ (r & 7)) << 4);
            const size_t src = static_cast<size_t>(grow) * dp + ch * 8;
            cp_async16(o, B.xh + src);
            cp_async16(o + kStageBytes / 2, B.xl + src);
          }
        }
        // the barrier is arrived at when this thread's copies have landed
        cp_async_arrive(tc5::smem_u32(&sh.full[s % S]));
      }
    }
    cp_async_wait_all();
  } else if (warp == 12) {
    const uint32_t abase = tc5::smem_u32(sm + L.o_a), bbase = tc5::smem_u32(sm + L.o_b);
    const uint32_t blo = static_cast<uint32_t>(kpad) * dp * 2;
    const int n0 = kpad <= 256 ? kpad : 256, n1 = kpad - n0;
    const uint32_t id0 = tc5::idesc_bf16(kRows, n0), id1 = n1 > 0 ? tc5::idesc_bf16(kRows, n1) : 0u;
    int s = pg.stages, it = pg.tiles;
    bool ok = true;
    for (int t = t0; ok && t < t1; ++t, ++it) {
      const int buf = it % nbuf;
      ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.aempty[buf]), ((it / nbuf) & 1) ^ 1, stop));
      if (!ok) break;
      tc5::fence_after();
      const uint32_t acc = tmem + buf * 256;
      for (int g = 0; g < groups; ++g, ++s) {
        ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.ready[s % S]), (s / S) & 1, stop));
        if (!ok) break;
        tc5::fence_after();
        const uint32_t as = abase + (s % S) * kStageBytes;
        // descriptors advance by 16-coordinate steps (their address field
        // counts 16 bytes)
        const int k1 = min(kStageChunks, chunks - g * kStageChunks) / 2;
        const uint32_t bo = bbase + static_cast<uint32_t>(g * kStageChunks * kpad) * 16;
        uint64_t ah = tc5::operand128(as), al = tc5::operand128(as + kStageBytes / 2);
        uint64_t bh = tc5::operand(bo, kpad), bl = tc5::operand(bo + blo, kpad);
#pragma unroll 4
        for (int q = 0; q < k1; ++q) {
          const bool add = g + q > 0;
          tc5::mma(acc, ah, bh, id0, add);
          tc5::mma(acc, ah, bl, id0, true);
          tc5::mma(acc, al, bh, id0, true);
          if (n1 > 0) {
            tc5::mma(acc + 256, ah, bh + 256, id1, add);
            tc5::mma(acc + 256, ah, bl + 256, id1, true);
            tc5::mma(acc + 256, al, bh + 256, id1, true);
          }
          ah += 2;
          al += 2;
          bh += 2 * kpad;
          bl += 2 * kpad;
        }
        tc5::commit(tc5::smem_u32(&sh.empty[s % S]));
      }
      if (ok) tc5::commit(tc5::smem_u32(&sh.afull[buf]));
    }
    if (!ok) {
      // the products still queued finish before the block ends
      int zero = 0;
      tc5::commit(tc5::smem_u32(&sh.drain));
      tc5::mbar_wait(tc5::smem_u32(&sh.drain), 0, &zero);
    }
  } else if (warp >= 13) {
    // ---- landed stages are handed to the tensor core by three threads in
    // turn: the proxy fence takes about 1000 cycles, in the copying threads it
    // would also wait for the copies of later stages, in the issuing thread it
    // would stand between the products.  No more threads than stages: a wait tells
    // a phase from the one after the next only, and a thread at stage s has seen
    // stage s - relays land, which has to be its slot's last use, s - S, or a later
    // one (three threads on a ring of two passed stages on before they had landed)
    const int relays = min(3, S);
    if (lane == 0 && warp - 13 < relays) {
      const int end = pg.stages + (t1 - t0) * groups;
      for (int s = pg.stages + (warp - 13); s < end; s += relays) {
        if (!tc5::mbar_wait(tc5::smem_u32(&sh.full[s % S]), (s / S) & 1, stop)) break;
        fence_async_proxy();
        tc5::mbar_arrive(tc5::smem_u32(&sh.ready[s % S]));
      }
    }
  } else if (warp < 8) {
    const int g = warp >> 2, rl = (warp & 3) * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    bool ok = true;
    // a single accumulator is the first group's; this group's tiles are nbuf
    // apart, the row ids two of them and the norms one of them ahead
    const int first = t0 + (g - pg.tiles % nbuf + nbuf) % nbuf;
    auto row_id = [&](int t) {
      const int r = min(t * kRows + rl, n - 1);
      return rows != nullptr ? rows[r] : r;
    };
    const int last = g < nbuf ? t1 : t0;
    int id = 0, id1 = 0;
    float pn1 = 0.0f;
    if (first < last) {
      id = row_id(first);
      id1 = row_id(first + nbuf);
      pn1 = B.pnorm[id];
    }
    for (int t = first; ok && t < last; t += nbuf) {
      const int it = pg.tiles + t - t0;
      const int buf = g, i = t * kRows + rl;
      const uint32_t acc = tmem + buf * 256 + lanes;
      const float pn = pn1;
      const int grow = id;
      pn1 = B.pnorm[id1];
      id = id1;
      id1 = row_id(t + 2 * nbuf);
      ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.afull[buf]), (it / nbuf) & 1, stop));
      if (!ok) break;
      tc5::fence_after();
      const float tol = 2.0f * fadd(pn, cmax) * B.tc_crel + 4e-35f;
      float low = INFINITY, mins[NCH];
      uint32_t mask[NCH];
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        mins[c] = INFINITY;
        mask[c] = 0u;
        if (c < L.nch) {
          float v[32];
          tc5::load32(acc + 32 * c, v);
          float m = INFINITY;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const float4 n4 = *reinterpret_cast<const float4*>(cn + 32 * c + e);
            v[e] = __fmaf_rn(v[e], -2.0f, n4.x);
            v[e + 1] = __fmaf_rn(v[e + 1], -2.0f, n4.y);
            v[e + 2] = __fmaf_rn(v[e + 2], -2.0f, n4.z);
            v[e + 3] = __fmaf_rn(v[e + 3], -2.0f, n4.w);
            m = tc5::min3(m, v[e], v[e + 1]);
            m = tc5::min3(m, v[e + 2], v[e + 3]);
          }
          low = fminf(low, m);
          mins[c] = m;
          const float thr = low + tol;
          if (__any_sync(kFull, m <= thr)) {
#pragma unroll
            for (int e = 0; e < 32; ++e) mask[c] |= v[e] <= thr ? 1u << e : 0u;
          }
        }
      }
      tc5::fence_before();
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(tc5::smem_u32(&sh.aempty[buf]));
      const bool plain = pn <= 1e37f && cmax <= 1e37f;
      const float thr = low + tol;
      int count = 0, best = 0;
#pragma unroll
      for (int c = NCH - 1; c >= 0; --c) {
        if (!plain) {
          const int left = k - 32 * c;
          mask[c] = left >= 32 ? ~0u : left > 0 ? (1u << left) - 1u : 0u;
        } else if (mins[c] > thr) {
          mask[c] = 0u;
        }
        count += __popc(mask[c]);
        if (mask[c] != 0u) best = 32 * c + __ffs(mask[c]) - 1;
      }
      const bool single = plain && count == 1;
      if (i < n && single) put(i, best);
      if (i < n && !single) {
        if (plain && count <= 4) {
          // up to 64 centroids the masks themselves, else 16 bits a candidate
          // (0xffff = none)
          unsigned long long cand = NCH == 2 ? mask[0] | (static_cast<unsigned long long>(mask[1]) << 32) : ~0ull;
#pragma unroll
          for (int c = 0; c < (NCH == 2 ? 0 : NCH); ++c) {
            while (mask[c] != 0u) {
              cand = (cand << 16) | static_cast<unsigned>(32 * c + __ffs(mask[c]) - 1);
              mask[c] &= mask[c] - 1u;
            }
          }
          list[atomicAdd(&sh.multi, 1)] =
              make_int4(i, grow, static_cast<int>(cand & 0xffffffffu), static_cast<int>(cand >> 32));
        } else {
          const int slot = cap - 1 - atomicAdd(&sh.many, 1);
          list[slot] = make_int4(i, grow, __float_as_int(pn), 0);
#pragma unroll
          for (int c = 0; c < NCH; ++c)
            if (c < L.nch) lmask[static_cast<size_t>(slot) * L.nch + c] = mask[c];
        }
      }
      __syncwarp();
    }
  }
  __syncwarp();
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  pg.tiles += t1 - t0;
  pg.stages += (t1 - t0) * groups;
  if (sh.stop != 0) return;

  // ---- exact distances of the listed rows.  Up to four candidates: a quad of
  // lanes per row, a candidate per lane, each dot whole in its lane
  for (int e0 = warp * 8; e0 < sh.multi; e0 += 8 * kWarps5) {
    const int e = e0 + (lane >> 2);
    int4 r = make_int4(0, 0, -1, -1);
    if (e < sh.multi) r = list[e];
    int c;
    if (NCH == 2) {
      unsigned long long m =
          static_cast<unsigned>(r.z) | (static_cast<unsigned long long>(static_cast<unsigned>(r.w)) << 32);
      if (lane & 1) m &= m - 1ull;
      if (lane & 2) {
        m &= m - 1ull;
        m &= m - 1ull;
      }
      c = m != 0ull && e < sh.multi ? __ffsll(static_cast<long long>(m)) - 1 : 0xffff;
    } else {
      const int half = (lane & 2) ? r.w : r.z;
      c = static_cast<int>((static_cast<unsigned>(half) >> (16 * (lane & 1))) & 0xffffu);
    }
    float dist = INFINITY;
    if (c != 0xffff) {
      const float* xr = B.x + static_cast<size_t>(r.y) * d;
      const float* cc = cent + static_cast<size_t>(c) * d;
      const float dot = dot_x86([&](int j) { return xr[j]; }, [&](int j) { return cc[j]; }, d);
      dist = __fsub_rn(fadd(B.pnorm[r.y], cn[c]), fmul(2.0f, dot));
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      const float od = __shfl_xor_sync(kFull, dist, o);
      const int oc = __shfl_xor_sync(kFull, c, o);
      if (od < dist || (od == dist && oc < c)) {
        dist = od;
        c = oc;
      }
    }
    if (e < sh.multi && (lane & 3) == 0) put(r.x, c);
  }
  // more candidates (or norms out of range): half a warp per row
  const int hl = lane & 15, hb = lane & 16;
  const unsigned hm = 0xffffu << hb;
  for (int e = warp * 2 + (hb >> 4); e < sh.many; e += 2 * kWarps5) {
    const int4 r = list[cap - 1 - e];
    const uint32_t mine = hl < L.nch ? lmask[static_cast<size_t>(cap - 1 - e) * L.nch + hl] : 0u;
    const float pn = __int_as_float(r.z);
    const float* xr = B.x + static_cast<size_t>(r.y) * d;
    int best = k;
    float bestd = INFINITY;
    unsigned words = (__ballot_sync(hm, mine != 0u) >> hb) & 0xffffu;
    while (words != 0u) {
      const int w = __ffs(words) - 1;
      words &= words - 1u;
      uint32_t bits = __shfl_sync(hm, mine, hb + w);
      while (bits != 0u) {
        const int c = 32 * w + __ffs(bits) - 1;
        bits &= bits - 1u;
        const float sum = half_warp_dot(xr, cent + static_cast<size_t>(c) * d, d);
        const float dist = __fsub_rn(fadd(pn, cn[c]), fmul(2.0f, sum));
        if (dist < bestd || (dist == bestd && c < best)) {
          bestd = dist;
          best = c;
        }
      }
    }
    if (!(bestd < INFINITY)) best = 0;  // no finite distance: the full scan keeps its first cluster
    if (hl == 0) put(r.x, best);
  }
  __syncthreads();
}

__device__ __forceinline__ uint32_t setup5(Shared5& sh) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      tc5::mbar_init(tc5::smem_u32(&sh.full[s]), 128);
      tc5::mbar_init(tc5::smem_u32(&sh.ready[s]), 1);
      tc5::mbar_init(tc5::smem_u32(&sh.empty[s]), 1);
    }
    for (int g = 0; g < 2; ++g) {
      tc5::mbar_init(tc5::smem_u32(&sh.afull[g]), 1);
      tc5::mbar_init(tc5::smem_u32(&sh.aempty[g]), 4);
    }
    tc5::mbar_init(tc5::smem_u32(&sh.drain), 1);
    tc5::mbar_fence_init();
    sh.stop = 0;
    sh.changed = 0;
  }
  if (threadIdx.x < 32) tc5::tmem_alloc(tc5::smem_u32(&sh.tmem), 512);
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  return __shfl_sync(kFull, sh.tmem, 0);
}

__device__ __forceinline__ void release5(uint32_t tmem) {
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  if (threadIdx.x < 32) tc5::tmem_free(tmem, 512);
}

// One assignment pass of the separate-launch path: CTA blockIdx.x of problem
// blockIdx.y takes tc_blocks tiles.
template <int NCH>
__global__ void __launch_bounds__(kThreads5, 1) assign5_kernel(KMeansBatch B, int final_pass) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  __shared__ Shared5 sh;
  const int p = blockIdx.y;
  if (!final_pass && !B.active[p]) return;
  const Layout5 L = layout5(B.n, B.k, B.dp, false);
  const uint32_t tmem = setup5(sh);
  const float* cent = B.cent + static_cast<size_t>(p) * B.k * B.d;
  stage_centroids(B, L, smraw, sh, cent);
  const int ntiles = (B.n + kRows - 1) / kRows;
  const int t0 = blockIdx.x * B.tc_blocks, t1 = min(ntiles, t0 + B.tc_blocks);
  int* as = B.assign + static_cast<size_t>(p) * B.n;
  int* lab = B.labels + static_cast<size_t>(p) * B.n;
  Progress pg;
  assign_tiles<NCH>(B, L, smraw, sh, tmem, p, t0, t1, cent, pg, [&](int i, int c) {
    if (final_pass) {
      lab[i] = c + 1;
    } else if (as[i] != c) {
      as[i] = c;
      sh.changed = 1;
    }
  });
  __syncthreads();
  if (sh.stop != 0) {
    // a wait ran out: the call fails (status), later stages still get labels
    for (int i = t0 * kRows + threadIdx.x; i < min(B.n, t1 * kRows); i += kThreads5) {
      as[i] = 0;
      if (final_pass) lab[i] = 1;
    }
    if (threadIdx.x == 0) *B.status = 2;
  }
  if (threadIdx.x == 0 && sh.changed != 0) B.changed[p] = 1;
  release5(tmem);
}

// Float Fenwick tree over donor weights (kodama_matrix.cpp:566-603).
struct Fenwick {
  float* tree;  // k+1
  float* vals;  // k
  int k;
  __device__ void set(int i, float v) {
    const float delta = __fsub_rn(v, vals[i]);
    vals[i] = v;
    for (unsigned j = static_cast<unsigned>(i) + 1u; j < static_cast<unsigned>(k) + 1u; j += j & (~j + 1u))
      tree[j] = fadd(tree[j], delta);
  }
  __device__ float total() const {
    float s = 0.0f;
    for (unsigned j = static_cast<unsigned>(k); j > 0; j -= j & (~j + 1u)) s = fadd(s, tree[j]);
    return s;
  }
  __device__ int select(float target) const {
    unsigned pos = 0, step = 1;
    const unsigned size = static_cast<unsigned>(k) + 1u;
    while ((step << 1) < size) step <<= 1;
    float prefix = 0.0f;
    for (; step > 0; step >>= 1) {
      const unsigned nxt = pos + step;
      if (nxt < size && fadd(prefix, tree[nxt]) <= target) {
        pos = nxt;
        prefix = fadd(prefix, tree[nxt]);
      }
    }
    return pos < static_cast<unsigned>(k) ? static_cast<int>(pos) : -1;
  }
};

// Empty clusters take half of a donor (kodama_matrix.cpp:604-662): a donor
// picked by the Fenwick tree, the two centroids moved apart by 1/1024.  fsize:
// the cluster sizes; the uniforms restart with every split.
__device__ __noinline__ void split_empty(const KMeansBatch& B, float* fsize, float* ftree, float* fvals, float* cent) {
  const int k = B.k, d = B.d;
  const float eps = 1.0f / 1024.0f;
  Fenwick fw{ftree, fvals, k};
  for (int i = 0; i <= k; ++i) ftree[i] = 0.0f;
  for (int i = 0; i < k; ++i) fvals[i] = 0.0f;
  for (int c = 0; c < k; ++c) fw.set(c, pos_part(__fsub_rn(fsize[c], 1.0f)));
  int u = 0;
  for (int e = 0; e < k; ++e) {
    if (fsize[e] != 0.0f) continue;
    const float total = fw.total();
    int donor = -1;
    if (total > 0.0f) donor = fw.select(fmul(B.split_uniform[u++], total));
    if (donor < 0) {
      donor = 0;
      for (int c = 1; c < k; ++c) if (fsize[c] > fsize[donor]) donor = c;
    }
    float* ec = cent + static_cast<size_t>(e) * d;
    float* dc = cent + static_cast<size_t>(donor) * d;
    for (int j = 0; j < d; ++j) ec[j] = dc[j];
    for (int j = 0; j < d; ++j) {
      if ((j & 1) == 0) {
        ec[j] = fmul(ec[j], fadd(1.0f, eps));
        dc[j] = fmul(dc[j], __fsub_rn(1.0f, eps));
      } else {
        ec[j] = fmul(ec[j], __fsub_rn(1.0f, eps));
        dc[j] = fmul(dc[j], fadd(1.0f, eps));
      }
    }
    fsize[e] = __fdiv_rn(fsize[donor], 2.0f);
    fsize[donor] = __fsub_rn(fsize[donor], fsize[e]);
    fw.set(e, pos_part(__fsub_rn(fsize[e], 1.0f)));
    fw.set(donor, pos_part(__fsub_rn(fsize[donor], 1.0f)));
  }
}

// Update step, part 1 (one CTA of 1024 threads per problem): stable grouping
// of the rows by cluster.  Each warp takes a contiguous range of rows, counts
// its clusters, then places its rows in order at per-(warp, cluster) offsets;
// members[] holds global row ids grouped by cluster in ascending row order.
__global__ void __launch_bounds__(1024) sort_kernel(KMeansBatch B) {
  extern __shared__ int sm[];
  const int p = blockIdx.x;
  if (!B.active[p]) return;
  const int k = B.k, n = B.n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* whist = sm;             // 32 x k
  int* cbase = whist + 32 * k; // k+1
  const int* as = B.assign + static_cast<size_t>(p) * n;
  int* mem = B.members + static_cast<size_t>(p) * n;
  int* off = B.offsets + static_cast<size_t>(p) * (k + 1);
  for (int i = threadIdx.x; i < 32 * k; i += blockDim.x) whist[i] = 0;
  __syncthreads();
  const int per = (n + 31) / 32;
  const int beg = warp * per, end = min(n, beg + per);
  for (int base = beg; base < end; base += 32) {
    const int r = base + lane;
    const int c = r < end ? as[r] : -1;
    const unsigned m = __match_any_sync(kFull, c);
    if (c >= 0 && (__ffs(m) - 1) == lane) whist[warp * k + c] += __popc(m);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    int run = 0;
    for (int w = 0; w < 32; ++w) {
      const int v = whist[w * k + c];
      whist[w * k + c] = run;
      run += v;
    }
    cbase[c] = run;  // size for now
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int c = 0; c < k; ++c) {
      const int sz = cbase[c];
      cbase[c] = run;
      off[c] = run;
      run += sz;
    }
    cbase[k] = run;
    off[k] = run;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * k; i += blockDim.x) whist[i] += cbase[i % k];
  __syncthreads();
  const int* rows = B.rows ? B.rows + static_cast<size_t>(p) * n : nullptr;
  for (int base = beg; base < end; base += 32) {
    const int r = base + lane;
    const int c = r < end ? as[r] : -1;
    const unsigned m = __match_any_sync(kFull, c);
    if (c >= 0) {
      const int rank = __popc(m & ((1u << lane) - 1u));
      mem[whist[warp * k + c] + rank] = rows ? rows[r] : r;
    }
    __syncwarp();
    if (c >= 0 && (__ffs(m) - 1) == lane) whist[warp * k + c] += __popc(m);
    __syncwarp();
  }
}

// Update step, part 2 (one CTA per problem and cluster): centroid sums in
// ascending row order, scaled by 1/size.  A cluster can hold thousands of
// rows (in high dimension one centroid often takes most of a mixture
// component), and its features are sequential float chains, so the rows are
// streamed through a ring of kSumStages chunks of kSumChunk rows in shared
// memory with cp.async: every thread copies, the member ids of a chunk are
// read one chunk ahead of its copies, and thread j adds feature j down each
// landed chunk in row order.  Features go in blocks of kSumCols.
constexpr int kSumChunk = 128;
constexpr int kSumStages = 4;
constexpr int kSumCols = 64;
constexpr int kSumThreads = 256;

size_t sums_smem(int d) {
  const int dw = d < kSumCols ? d : kSumCols;
  return sizeof(float) * kSumStages * kSumChunk * dw + sizeof(int) * kSumStages * kSumChunk;
}

__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__global__ void __launch_bounds__(kSumThreads) sums_kernel(KMeansBatch B) {
  extern __shared__ float sring[];
  const int p = blockIdx.x / B.k, c = blockIdx.x % B.k;
  if (p >= B.problems || !B.active[p]) return;
  const int d = B.d;
  const int* mem = B.members + static_cast<size_t>(p) * B.n;
  const int* off = B.offsets + static_cast<size_t>(p) * (B.k + 1);
  const int b0 = off[c], b1 = off[c + 1];
  float* cent = B.cent + (static_cast<size_t>(p) * B.k + c) * d;
  const int cnt = b1 - b0;
  const float inv = cnt != 0 ? __fdiv_rn(1.0f, static_cast<float>(cnt)) : 0.0f;
  const int nchunks = (cnt + kSumChunk - 1) / kSumChunk;
  for (int jb = 0; jb < d; jb += kSumCols) {
    const int dw = min(kSumCols, d - jb);
    float* rows_s = sring;                                              // [stage][kSumChunk][dw]
    int* ids_s = reinterpret_cast<int*>(sring + kSumStages * kSumChunk * dw);  // [stage][kSumChunk]
    // stage the ids of the first chunks, then copy chunk i while the ids of
    // chunk i + 1 are read
    auto load_ids = [&](int ch) {
      const int base = b0 + ch * kSumChunk;
      int* ids = ids_s + (ch % kSumStages) * kSumChunk;
      for (int r = threadIdx.x; r < kSumChunk; r += kSumThreads) ids[r] = base + r < b1 ? mem[base + r] : -1;
    };
    auto copy_rows = [&](int ch) {
      const int* ids = ids_s + (ch % kSumStages) * kSumChunk;
      float* dst = rows_s + (ch % kSumStages) * kSumChunk * dw;
      const int m = min(kSumChunk, b1 - (b0 + ch * kSumChunk));
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      for (int r = warp; r < m; r += kSumThreads / 32) {
        const float* src = B.x + static_cast<size_t>(ids[r]) * d + jb;
        for (int col = lane; col < dw; col += 32) cp_async4(dst + r * dw + col, src + col);
      }
    };
    float s = 0.0f;
    __syncthreads();
    if (nchunks > 0) load_ids(0);
    __syncthreads();
    // prologue: copies of chunks 0 .. kSumStages-2 in flight
    for (int ch = 0; ch < kSumStages - 1; ++ch) {
      if (ch < nchunks) {
        if (ch + 1 < nchunks) load_ids(ch + 1);
        copy_rows(ch);
      }
      cp_async_commit_group();
      __syncthreads();
    }
    for (int ch = 0; ch < nchunks; ++ch) {
      // keep kSumStages - 1 chunks in flight: issue chunk ch + kSumStages - 1
      const int nx = ch + kSumStages - 1;
      if (nx < nchunks) {
        if (nx + 1 < nchunks) load_ids(nx + 1);
        copy_rows(nx);
      }
      cp_async_commit_group();
      cp_async_wait_groups<kSumStages - 1>();
      __syncthreads();
      if (threadIdx.x < dw) {
        const int m = min(kSumChunk, b1 - (b0 + ch * kSumChunk));
        const float* sc = rows_s + (ch % kSumStages) * kSumChunk * dw + threadIdx.x;
#pragma unroll 8
        for (int r = 0; r < m; ++r) s = fadd(s, sc[r * dw]);
      }
      __syncthreads();
    }
    if (threadIdx.x < dw) cent[jb + threadIdx.x] = cnt != 0 ? fmul(s, inv) : s;
  }
}

// Update step, sort and sums in one (one CTA per cluster and problem, d up
// to kScanCols x kScanThreads): the CTA scans the problem's assignments, a run
// of rows per warp, first counting and then listing the cluster's members in
// ascending row order in shared memory (kScanCap at a time); thread j then adds
// columns j, j + 512 down them, 32 to 64 rows' loads in flight.  The size goes to
// offsets[c] (finalize_kernel reads sizes).  Without the member lists and the
// one-CTA sort this replaces sort_kernel and sums_kernel when each problem's
// assignments are read by its k CTAs anyway.
// What bounds it: the scan's and the rows' loads.  Scanning, listing and adding
// 1024 rows at a time waited for memory in every chunk: 20000 x 50 rows and 50
// clusters 80 -> 36 us, 100000 x 50 and 300 143 -> 81, 4999 x 37 and 100 19 -> 12
// (1000 x 10, one chunk before: 4.6 and 5.0).
constexpr int kScanThreads = 512;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanCols = 2;     // columns per thread
constexpr int kScanCap = 8192;   // members listed at a time

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(KMeansBatch B) {
  __shared__ int mem[kScanCap];
  __shared__ int wcount[kScanWarps];
  const int c = blockIdx.x, p = blockIdx.y;
  if (!B.active[p]) return;
  const int n = B.n, d = B.d, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int* as = B.assign + static_cast<size_t>(p) * n;
  const int* rows = B.rows != nullptr ? B.rows + static_cast<size_t>(p) * n : nullptr;
  const int per = ((n + kScanWarps - 1) / kScanWarps + 31) / 32 * 32;
  const int beg = min(n, warp * per), end = min(n, beg + per);
  // use(row, member, members of the 32 rows), eight steps' loads in flight
  auto walk = [&](auto&& use) {
    for (int b0 = beg; b0 < end; b0 += 8 * 32) {
      int a[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = b0 + 32 * u + lane;
        a[u] = r < end ? as[r] : -1;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const bool in = a[u] == c;
        use(b0 + 32 * u + lane, in, __ballot_sync(kFull, in));
      }
    }
  };
  int mine = 0;
  walk([&](int, bool, unsigned m) { mine += __popc(m); });
  if (lane == 0) wcount[warp] = mine;
  __syncthreads();
  int off = 0, count = 0;
#pragma unroll
  for (int q = 0; q < kScanWarps; ++q) {
    off += q < warp ? wcount[q] : 0;
    count += wcount[q];
  }
  float s[kScanCols];
#pragma unroll
  for (int q = 0; q < kScanCols; ++q) s[q] = 0.0f;
  for (int first = 0; first < count; first += kScanCap) {
    int pos = off - first;
    walk([&](int r, bool in, unsigned m) {
      const int at = pos + __popc(m & ((1u << lane) - 1u));
      if (in && at >= 0 && at < kScanCap) mem[at] = rows != nullptr ? rows[r] : r;
      pos += __popc(m);
    });
    __syncthreads();
    const int total = min(kScanCap, count - first);
#pragma unroll
    for (int q = 0; q < kScanCols; ++q) {
      const int j = tid + q * kScanThreads;
      if (j >= d) continue;
      const float* xj = B.x + j;
      float va[32], vb[32];
      auto fetch = [&](float (&v)[32], int m0) {
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = xj[static_cast<size_t>(mem[min(m0 + u, total - 1)]) * d];
      };
      auto add = [&](const float (&v)[32], int left) {
        if (left >= 32) {
#pragma unroll
          for (int u = 0; u < 32; ++u) s[q] = fadd(s[q], v[u]);
        } else {
#pragma unroll
          for (int u = 0; u < 32; ++u)
            if (u < left) s[q] = fadd(s[q], v[u]);
        }
      };
      fetch(va, 0);
      for (int m = 0; m < total; m += 64) {
        if (m + 32 < total) fetch(vb, m + 32);
        add(va, total - m);
        if (m + 64 < total) fetch(va, m + 64);
        if (m + 32 < total) add(vb, total - m - 32);
      }
    }
    __syncthreads();  // mem is rewritten by the next part
  }
  const float inv = count != 0 ? __fdiv_rn(1.0f, static_cast<float>(count)) : 0.0f;
  float* cent = B.cent + (static_cast<size_t>(p) * B.k + c) * d;
#pragma unroll
  for (int q = 0; q < kScanCols; ++q) {
    const int j = tid + q * kScanThreads;
    if (j < d) cent[j] = count != 0 ? fmul(s[q], inv) : s[q];
  }
  if (tid == 0) B.offsets[static_cast<size_t>(p) * (B.k + 1) + c] = count;
}

// Update step, part 3 (one thread per problem): empty-cluster splitting and
// the early-exit flag.  sizes: offsets[c] holds cluster c's size (after
// scan_sums_kernel) rather than its start (after sort_kernel).
__global__ void finalize_kernel(KMeansBatch B, int sizes) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= B.problems || !B.active[p]) return;
  const int k = B.k, d = B.d, n = B.n;
  const int* off = B.offsets + static_cast<size_t>(p) * (k + 1);
  float* cent = B.cent + static_cast<size_t>(p) * k * d;
  float* fsize = B.fscratch + static_cast<size_t>(p) * (3 * k + 1);
  float* ftree = fsize + k;
  float* fvals = ftree + k + 1;
  bool any_empty = false;
  for (int c = 0; c < k; ++c) {
    const int size = sizes ? off[c] : off[c + 1] - off[c];
    fsize[c] = static_cast<float>(size);
    any_empty |= size == 0;
  }
  if (any_empty && n > k) {
    split_empty(B, fsize, ftree, fvals, cent);
  }
  if (B.changed[p] == 0) B.active[p] = 0;
  B.changed[p] = 0;
}

// ---------------------------------------------------------------------------
// Persistent batched k-means: one CTA per problem runs every Lloyd iteration
// and the final assignment with block barriers only, so a batch of M problems
// is one launch instead of 3 per iteration.  Same arithmetic as the
// separate-launch path, hence the same labels bit for bit.
//
// Shared memory holds the centroids' bf16 operand and norms, the row ring, the
// problem's assignments (16 bits) and per-warp cluster histograms; the fp32
// centroids (read for the operand, the norms and the few exact rechecks) and
// the member lists (rows grouped by cluster, ascending) stay in L2.
//   assignment: assign_tiles;
//   grouping: per-warp counts over contiguous row ranges, prefix sums, stable
//     scatter of the row ids into the member lists;
//   sums: a warp per (cluster, 32 columns), the largest clusters first: a
//     cluster's chain bounds the phase; lane j keeps the float chain of its
//     column down the member rows in ascending order, 32 to 64 rows' loads in
//     flight;
//   split: one thread, as finalize_kernel.
// ---------------------------------------------------------------------------
template <int NCH>
__global__ void __launch_bounds__(kThreads5, 1) kmeans_persistent_kernel(KMeansBatch B) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  __shared__ Shared5 sh;
  const int p = blockIdx.x;
  const int k = B.k, d = B.d, n = B.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Layout5 L = layout5(n, k, B.dp, true);
  uint16_t* sas = reinterpret_cast<uint16_t*>(smraw + L.o_as);  // [n] assignments
  int* whist = reinterpret_cast<int*>(smraw + L.o_wh);          // [warps][k]
  int* soff = reinterpret_cast<int*>(smraw + L.o_off);          // [k + 1]
  float* fsize = reinterpret_cast<float*>(smraw + L.o_fs);      // [k], tree [k + 1], vals [k]
  const int* prow = B.rows + static_cast<size_t>(p) * n;
  int* mem = B.members + static_cast<size_t>(p) * n;
  int* lab = B.labels + static_cast<size_t>(p) * n;
  unsigned char* dirty = smraw + L.o_di;                        // [k] membership changed
  uint16_t* order = reinterpret_cast<uint16_t*>(smraw + L.o_or);  // [k] clusters, the largest first
  float* cent = B.cent + static_cast<size_t>(p) * k * d;
  const uint32_t tmem = setup5(sh);
  // initial centroids: the problem's rows init_rows[0..k)
  for (int i = tid; i < k * d; i += kThreads5) {
    const int c = i / d, j = i % d;
    cent[i] = B.x[static_cast<size_t>(prow[B.init_rows[static_cast<size_t>(p) * k + c]]) * d + j];
  }
  for (int i = tid; i < n; i += kThreads5) sas[i] = 0xffffu;
  for (int c = tid; c < k; c += kThreads5) dirty[c] = 1;
  __syncthreads();
  const int ntiles = (n + kRows - 1) / kRows;
  const int iters = B.max_iter > 1 ? B.max_iter : 1;
  Progress pg;
  for (int it = 0; it <= iters; ++it) {
    const bool final_pass = it == iters;
    if (tid == 0) sh.changed = 0;
    stage_centroids(B, L, smraw, sh, cent);
    assign_tiles<NCH>(B, L, smraw, sh, tmem, p, 0, ntiles, cent, pg, [&](int i, int c) {
      if (final_pass) {
        lab[i] = c + 1;
      } else {
        const int old = sas[i];
        if (old != c) {
          sas[i] = static_cast<uint16_t>(c);
          if (old < k) dirty[old] = 1;
          dirty[c] = 1;
          sh.changed = 1;
        }
      }
    });
    __syncthreads();
    if (sh.stop != 0) {
      // a wait ran out: the call fails (status), later stages still get labels
      for (int i = tid; i < n; i += kThreads5) lab[i] = 1;
      if (tid == 0) *B.status = 2;
      break;
    }
    if (final_pass) break;

    // ---- grouping: member lists in ascending row order per cluster ----
    for (int i = tid; i < kWarps5 * k; i += kThreads5) whist[i] = 0;
    __syncthreads();
    const int per = (n + kWarps5 - 1) / kWarps5;
    const int beg = min(n, warp * per), end = min(n, beg + per);
    for (int r = beg + lane; r < end; r += 32) atomicAdd(&whist[warp * k + sas[r]], 1);
    __syncthreads();
    bool empty = false;
    for (int c = tid; c < k; c += kThreads5) {
      int run = 0;
      for (int w = 0; w < kWarps5; ++w) {
        const int v = whist[w * k + c];
        whist[w * k + c] = run;
        run += v;
      }
      soff[c] = run;  // size for now
      fsize[c] = static_cast<float>(run);
      empty = empty || run == 0;
    }
    const bool any_empty = __syncthreads_or(empty) != 0;
    if (warp == 0) {
      // exclusive prefix sums of the sizes
      int run = 0;
      for (int c0 = 0; c0 < k; c0 += 32) {
        const int c = c0 + lane, sz = c < k ? soff[c] : 0;
        int incl = sz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += v;
        }
        if (c < k) soff[c] = run + incl - sz;
        run += __shfl_sync(kFull, incl, 31);
      }
      if (lane == 0) {
        soff[k] = run;
        sh.queue = 0;
      }
    }
    __syncthreads();
    for (int i = tid; i < kWarps5 * k; i += kThreads5) whist[i] += soff[i % k];
    for (int c = tid; c < k; c += kThreads5) {
      const float size = fsize[c];
      int rank = 0;
      for (int q = 0; q < k; ++q) rank += fsize[q] > size || (fsize[q] == size && q < c);
      order[rank] = static_cast<uint16_t>(c);
    }
    __syncthreads();
    for (int base = beg; base < end; base += 128) {
      int cl[4], id[4];
      unsigned mm[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = base + 32 * u + lane;
        cl[u] = r < end ? sas[r] : -1;
        id[u] = r < end ? prow[r] : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mm[u] = __match_any_sync(kFull, cl[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (cl[u] >= 0) mem[whist[warp * k + cl[u]] + __popc(mm[u] & ((1u << lane) - 1u))] = id[u];
        __syncwarp();
        if (cl[u] >= 0 && (__ffs(mm[u]) - 1) == lane) whist[warp * k + cl[u]] += __popc(mm[u]);
        __syncwarp();
      }
    }
    __syncthreads();

    // ---- centroid sums in ascending row order (a cluster whose members did
    // not change keeps its centroid) ----
    const int nblk = (d + 31) / 32;
    for (;;) {
      int item = 0;
      if (lane == 0) item = atomicAdd(&sh.queue, 1);
      item = __shfl_sync(kFull, item, 0);
      if (item >= k * nblk) break;
      const int c = order[item / nblk], j = (item % nblk) * 32 + lane;
      if (!dirty[c]) continue;
      const int b0 = soff[c], cnt = soff[c + 1] - b0;
      const bool in = j < d;
      const float* xj = B.x + (in ? j : 0);
      float sum = 0.0f, va[32], vb[32];
      // the rows at batch m (ids held by the lanes) into v, zero past the end
      auto fetch = [&](float (&v)[32], int ids) {
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = xj[static_cast<size_t>(__shfl_sync(kFull, ids, u)) * d];
      };
      auto members = [&](int m) { return mem[b0 + min(m + lane, cnt - 1)]; };
      auto add = [&](const float (&v)[32], int left) {
        if (left >= 32) {
#pragma unroll
          for (int u = 0; u < 32; ++u) sum = fadd(sum, v[u]);
        } else {
#pragma unroll
          for (int u = 0; u < 32; ++u)
            if (u < left) sum = fadd(sum, v[u]);
        }
      };
      if (cnt > 0) {
        int ids = members(0);
        fetch(va, ids);
        ids = members(32);
        for (int m = 0; m < cnt; m += 64) {
          const int id2 = members(m + 64);
          if (m + 32 < cnt) fetch(vb, ids);
          add(va, cnt - m);
          ids = members(m + 96);
          if (m + 64 < cnt) fetch(va, id2);
          if (m + 32 < cnt) add(vb, cnt - m - 32);
        }
      }
      const float inv = cnt != 0 ? __fdiv_rn(1.0f, static_cast<float>(cnt)) : 0.0f;
      if (in) cent[static_cast<size_t>(c) * d + j] = cnt != 0 ? fmul(sum, inv) : sum;
    }
    __syncthreads();

    // ---- empty-cluster split (finalize_kernel) ----
    // (it moves donors too: the next sums form every centroid again)
    for (int c = tid; c < k; c += kThreads5) dirty[c] = any_empty ? 1 : 0;
    if (any_empty && n > k && tid == 0) split_empty(B, fsize, fsize + k, fsize + 2 * k + 1, cent);
    // early exit: no assignment changed in this iteration (checked after the
    // update, as the reference does); go to the final assignment
    const bool done = sh.changed == 0;
    __syncthreads();
    if (done) it = iters - 1;
  }
  release5(tmem);
}

}  // namespace

bool kmeans_tc_supported(int d, int k) {
  if (d < 1 || d > 256 || k < 1 || k > kMaxK) return false;
  return layout5(0, k, (d + 15) / 16 * 16, false).total + kShared5Room <= kSmemLimit;
}

size_t kmeans_mask_words(int k) { return (static_cast<size_t>(k) + 31) / 32; }

size_t kmeans_sort_smem(int k) { return sizeof(int) * (33 * static_cast<size_t>(k) + 1); }

int kmeans_row_norms(const float* x, int n, int d, float* out, cudaStream_t st) {
  row_norms_kernel<<<(n + 255) / 256, 256, 0, st>>>(x, n, d, out);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

namespace {

// |a + |x|^2 - dist| <= (|x|^2 + max |c|^2) * crel: 2 |dot_tc - dot_x86| <=
// 2 (3.1 * 2^-16 [the hi + lo split] + 3 dp * 2^-22 [f32 accumulation of 3 dp
// products, two ulps per add] + (d / 16 + 5) 2^-24 [the x86-order dot])
// sum|x_i c_i|, with sum|x_i c_i| <= 0.51 (|x|^2 + |c|^2); the canonical sum of
// norms and the final subtractions round values of at most 2.03 (|x|^2 +
// |c|^2) each
float tc_error_factor(int d, int dp) {
  const double tc = 3.1 * std::ldexp(1.0, -16) + 3.0 * dp * std::ldexp(1.0, -22) + (d / 16 + 5) * std::ldexp(1.0, -24);
  return static_cast<float>(1.05 * (1.02 * tc + 6.0 * std::ldexp(1.0, -24)) + 1e-7);
}

// The persistent kernel applies: a batch of several problems given by row
// lists, and its shared memory fits.
bool persistent_supported(const KMeansBatch& B) {
  if (B.problems < 2 || B.rows == nullptr || B.xh == nullptr || B.members == nullptr || B.n < 1) return false;
  return kmeans_tc_supported(B.d, B.k) && layout5(B.n, B.k, B.dp, true).total + kShared5Room <= kSmemLimit;
}

}  // namespace

int kmeans_run(const KMeansBatch& B, cudaStream_t st) {
  if (B.problems <= 0) return 0;
  const bool tc = B.xh != nullptr && kmeans_tc_supported(B.d, B.k);
  KMeansBatch T = B;
  T.tc_crel = tc_error_factor(B.d, B.dp);
  const int nch = (B.k + 31) / 32;
  // kernels with room for 2, 4, 8 or 16 chunks of 32 centroids in registers
  auto go = [&](auto kern, dim3 grid, size_t bytes, auto... more) {
    const cudaError_t err = allow_shared_memory(kern);
    if (err != cudaSuccess) return err;
    kern<<<grid, kThreads5, bytes, st>>>(T, more...);
    return cudaGetLastError();
  };
  if (persistent_supported(B)) {
    const size_t bytes = layout5(B.n, B.k, B.dp, true).total;
    const dim3 grid(B.problems);
    count_launch();
    return static_cast<int>(nch <= 2   ? go(kmeans_persistent_kernel<2>, grid, bytes)
                            : nch <= 4 ? go(kmeans_persistent_kernel<4>, grid, bytes)
                            : nch <= 8 ? go(kmeans_persistent_kernel<8>, grid, bytes)
                                       : go(kmeans_persistent_kernel<16>, grid, bytes));
  }
  init_centroids_kernel<<<dim3(B.k, B.problems), 64, 0, st>>>(B);
  const size_t cs_bytes = sizeof(float) * (static_cast<size_t>(B.k) * ((B.d + 3) & ~3) + B.k);
  const size_t sort_bytes = kmeans_sort_smem(B.k);
  const dim3 agrid((B.n + 128 * kAssignRows - 1) / (128 * kAssignRows), B.problems);
  const dim3 ngrid((B.k + 127) / 128, B.problems);
  const size_t sum_bytes = sums_smem(B.d);
  const size_t tc_bytes = tc ? layout5(B.n, B.k, B.dp, false).total : 0;
  // 128-row tiles per CTA: the centroids are staged once per CTA, the grid is
  // about one CTA per SM
  dim3 tgrid;
  {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long tiles = (B.n + kRows - 1) / kRows;
    const long long per = (tiles * B.problems + sms - 1) / sms;
    T.tc_blocks = static_cast<int>(per < 1 ? 1 : (per > tiles ? tiles : per));
    tgrid = dim3(static_cast<unsigned>((tiles + T.tc_blocks - 1) / T.tc_blocks), B.problems);
  }
  cudaError_t err = cudaSuccess;
  auto launch_assign = [&](int final_pass) {
    if (tc) {
      const cudaError_t e = nch <= 2   ? go(assign5_kernel<2>, tgrid, tc_bytes, final_pass)
                            : nch <= 4 ? go(assign5_kernel<4>, tgrid, tc_bytes, final_pass)
                            : nch <= 8 ? go(assign5_kernel<8>, tgrid, tc_bytes, final_pass)
                                       : go(assign5_kernel<16>, tgrid, tc_bytes, final_pass);
      if (err == cudaSuccess) err = e;
      return;
    }
    centroid_norms_kernel<<<ngrid, 128, 0, st>>>(B, final_pass);
    count_launch();
    if (B.d <= 16) assign_kernel<1><<<agrid, 128, cs_bytes, st>>>(B, final_pass);
    else if (B.d <= 32) assign_kernel<2><<<agrid, 128, cs_bytes, st>>>(B, final_pass);
    else if (B.d <= 64) assign_kernel<4><<<agrid, 128, cs_bytes, st>>>(B, final_pass);
    else assign_kernel<0><<<agrid, 128, cs_bytes, st>>>(B, final_pass);
  };
  if (!tc) {
    allow_shared_memory(assign_kernel<1>);
    allow_shared_memory(assign_kernel<2>);
    allow_shared_memory(assign_kernel<4>);
    allow_shared_memory(assign_kernel<0>);
  }
  allow_shared_memory(sort_kernel);
  allow_shared_memory(sums_kernel);
  const int iters = B.max_iter > 1 ? B.max_iter : 1;
  const bool scan = B.d <= kScanCols * kScanThreads;
  for (int it = 0; it < iters; ++it) {
    launch_assign(0);
    if (scan) {
      scan_sums_kernel<<<dim3(B.k, B.problems), kScanThreads, 0, st>>>(B);
    } else {
      sort_kernel<<<B.problems, 1024, sort_bytes, st>>>(B);
      sums_kernel<<<B.problems * B.k, kSumThreads, sum_bytes, st>>>(B);
    }
    finalize_kernel<<<(B.problems + 63) / 64, 64, 0, st>>>(B, scan ? 1 : 0);
  }
  launch_assign(1);
  count_launch(1 + (scan ? 3 : 4) * iters + 1);
  if (err != cudaSuccess) return static_cast<int>(err);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace kgb
