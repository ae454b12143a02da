// Exact nearest neighbours through a tensor-core candidate search (knn.cuh).
//
// The canonical result (knn.cu: a float32 chain over the coordinates in order,
// each term separately rounded, ties by row) is found in three steps, for the
// squared L2 distance or minus the inner product, over all other rows or over
// the rows of other folds:
//
//  1. prep: every row is split once into bfloat16 hi + lo parts
//     (x = hi + lo + r, |r| <= 2^-16 |x|), stored in blocks of 256 rows as
//     [chunk of 8 coordinates][row], the layout the tensor core reads, so that
//     a tile is one contiguous copy;
//  2. candidates: a persistent CTA per SM multiplies 128 queries with tiles of
//     256 candidates (hi.hi + hi.lo + lo.hi, tcgen05.mma into TMEM).  A thread
//     owns one query row of the accumulator, so it compares a = |c|^2 - 2 q.c
//     (|q|^2 dropped; -q.c for inner products) with the row's threshold without
//     talking to other lanes and appends the few values below it to the row's
//     list.  When a list grows past its trigger the warp cuts it back: tau =
//     A + 2 delta, A an upper bound of the K-th smallest value of the list;
//  3. re-rank: one warp per query joins the row's lists, bounds the K-th
//     smallest value A_K again, computes the canonical distances of the values
//     within A_K + 2 delta and keeps the K smallest by (distance, row).
//
// Certificate.  A value is only ever dropped at a threshold >= A_K + 2 delta,
// with delta >= |a - (e - |q|^2)| for every row that matters: the K smallest
// a's rows have e - |q|^2 <= A_K + delta, so a row of the true top K does too,
// and its a is at most A_K + 2 delta.  Rows whose lists overflow, hold too few
// values, or lie outside the value range below go to the brute force.
//
// Error bound (u = 2^-24), N = |q|^2 + |c|^2: the split drops at most
// 3.1 * 2^-16 sum|q_i c_i|; 3 dp accumulated products, allowed two ulps each,
// add 3 dp 2^-22 sum|q_i c_i|; twice their sum is at most N times that for L2
// (sum|q_i c_i| <= |q||c|), and |q||c| times that for inner products.  The
// canonical chain adds 2 (d + 4) u N, the float norms and the last fma
// (d + 4) u N.  delta = N crel, crel = 5e-5 + 1e-6 dp, covers the sum
// (4.8e-5 + 7.2e-7 dp + 1.8e-7 (d + 4)).  The rows that matter lie within
// R = sqrt(A + |q|^2 + 2 delta_max) of the query, so |c| <= |q| + R replaces
// the largest norm of the data there; delta falls with A, so an earlier
// threshold is never below a later one.  Norms outside [1e-20, 1e36] (or
// non-finite values) send every row to the brute force; kDeltaFloor covers
// products lost to underflow.
#include "knn.cuh"
#include "launch_count.cuh"
#include "smem_limit.cuh"

#include "bf16_split.cuh"
#include "tcgen05.cuh"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

namespace kgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBlockRows = 256;   // rows of an operand block = candidates per tile (mma N)
constexpr int kQRows = 128;       // queries per tile (mma M = TMEM lanes)
constexpr int kMaxDp = 256;
constexpr int kThreads = 320;     // 8 epilogue warps, the copy warp, the mma warp
constexpr int kMaxStages = 4;
constexpr int kNormSlots = 8;     // candidate tiles whose additive terms are staged
constexpr size_t kSmemLimit = 227 * 1024;
constexpr float kDeltaFloor = 2e-35f;
constexpr int kSurvivors = 512;   // joined list entries of a query in the re-rank

// status words: [0] largest norm (float bits), [1] non-finite value seen,
// [2] fallback rows, [3] a wait of the candidate kernel ran out
enum { kStNorm = 0, kStBad = 1, kStFallback = 2, kStTimeout = 3 };

// Rows perm[pos] (pos itself without perm; -1 = padding) of x split into the
// operand blocks.  A warp's lanes take 32 rows of one chunk, so the 16-byte
// stores of a chunk are contiguous; the block's warps share the chunks.
// cn: the additive term of a candidate (|c|^2, or 0 for inner products; +inf
// for padding), qn: |q|^2 (-1 for padding).  xp != nullptr also gets the rows
// as floats padded to d4 (a multiple of 4), for the re-rank's vector loads.
__global__ void __launch_bounds__(256) prep_kernel(const float* __restrict__ x, int n, int d, int chunks, int npos,
                                                   const int* __restrict__ perm, int inner,
                                                   uint16_t* __restrict__ xh, uint16_t* __restrict__ xl,
                                                   float* __restrict__ cn, float* __restrict__ qn,
                                                   float* __restrict__ xp, int d4, unsigned* __restrict__ status) {
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos = blockIdx.x * 32 + lane;  // npos is a multiple of 256
  const int row = perm != nullptr ? perm[pos] : (pos < n ? pos : -1);
  const size_t base = static_cast<size_t>(pos / kBlockRows) * chunks * kBlockRows + pos % kBlockRows;
  float s = 0.0f;
  bool fin = true;
  for (int c = warp; c < chunks; c += 8) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = c * 8 + e;
      v[e] = row >= 0 && k < d ? x[static_cast<size_t>(row) * d + k] : 0.0f;
      fin = fin && isfinite(v[e]);
      s = __fadd_rn(s, __fmul_rn(v[e], v[e]));
    }
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t h0 = bf16_bits(v[2 * e]), h1 = bf16_bits(v[2 * e + 1]);
      h[e] = h0 | (h1 << 16);
      l[e] = bf16_bits(__fsub_rn(v[2 * e], __uint_as_float(h0 << 16))) |
             (bf16_bits(__fsub_rn(v[2 * e + 1], __uint_as_float(h1 << 16))) << 16);
    }
    reinterpret_cast<uint4*>(xh)[base + static_cast<size_t>(c) * kBlockRows] = make_uint4(h[0], h[1], h[2], h[3]);
    reinterpret_cast<uint4*>(xl)[base + static_cast<size_t>(c) * kBlockRows] = make_uint4(l[0], l[1], l[2], l[3]);
    if (xp != nullptr && row >= 0) {
      float4* o = reinterpret_cast<float4*>(xp + static_cast<size_t>(row) * d4);
      if (c * 8 < d4) o[c * 2] = make_float4(v[0], v[1], v[2], v[3]);
      if (c * 8 + 4 < d4) o[c * 2 + 1] = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  part[warp][lane] = s;
  if (__any_sync(kFull, !fin) && lane == 0) atomicExch(&status[kStBad], 1u);
  __syncthreads();
  if (warp == 0) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t = __fadd_rn(t, part[w][lane]);
    cn[pos] = row < 0 ? INFINITY : (inner ? 0.0f : t);
    qn[pos] = row < 0 ? -1.0f : t;
    // finite sums only: an infinite one is caught by the range check
    const unsigned m = __reduce_max_sync(kFull, row < 0 || !(t >= 0.0f) ? 0u : __float_as_uint(t));
    if (lane == 0) atomicMax(&status[kStNorm], m);
  }
}

// The tiles of a query tile, in the order they are visited.  All candidate
// tiles but a contiguous range [skip, skip + skipn) (its own fold), starting
// at the query's own block (without a skip) or after the range, in steps of a
// stride coprime to their number: near rows are often near in memory, so the
// thresholds fall at once, and no slow order of the data is followed.
struct TileOrder {
  int ntiles, skip, skipn, count, first, stride;
  __device__ __forceinline__ TileOrder(int ntiles_, int own, int skip_, int skipn_)
      : ntiles(ntiles_), skip(skip_), skipn(skipn_) {
    count = ntiles - skipn;
    first = skipn > 0 ? 0 : own;
    stride = count > 0 ? 1000003 % count : 0;
    if (stride == 0) stride = 1;
  }
  __device__ __forceinline__ int at(int k) const {
    int t = static_cast<int>((first + static_cast<long long>(k) * stride) % count);
    if (skipn > 0) {
      t += skip + skipn;
      if (t >= ntiles) t -= ntiles;
    }
    return t;
  }
};

struct SearchArgs {
  const uint16_t* xh;      // blocks of [chunk][256 rows][8]
  const uint16_t* xl;
  const float* cn;
  const float* qn;
  unsigned* status;
  int chunks, kg, stages;  // 8-coordinate chunks of a row / per stage; stages
  int ntiles, qtiles;
  int Kq;                  // values a list has to keep: K, plus the query itself
  int cap;                 // entries per list
  float scale, crel;       // a = cn + scale * acc
  int inner;
  // stream-K split: the (query tile, candidate tile) pairs of all query tiles
  // in a row, `per` of them per CTA.  off: first pair of every query tile
  // (nullptr: q * ntiles), skip: the tile range a query tile leaves out
  const int* off;
  const int2* skip;
  long long pairs;         // past 2^31 from 8.4 million rows on; a CTA's own are counted
  int per, segs;           // from its first, and so are the query tiles' starts there
  float2* list;            // [query position][segment][group][cap] (a, position)
  int* cnt;                // [query position][segment][group], -1 = overflow
  float* tau;
};

__device__ __forceinline__ float delta_of(float A, float nq, float nmax, float crel, int inner) {
  if (inner) return crel * sqrtf(nq) * sqrtf(nmax) * 1.00001f + kDeltaFloor;
  const float dmax = crel * (nq + nmax) + kDeltaFloor;
  const float r2 = fmaxf(0.0f, A + nq + 2.0f * dmax) * 1.0001f + 1e-6f * nq;
  const float cm = fminf(sqrtf(nmax), sqrtf(nq) + sqrtf(r2)) * 1.00001f;
  return fminf(dmax, crel * (nq + cm * cm) + kDeltaFloor);
}

// order-preserving image of a float as an unsigned
__device__ __forceinline__ unsigned ord_float(float v) {
  const unsigned u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ord(unsigned o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// An upper bound of the Kq-th smallest of the warp's values (v[t] of lane l,
// +inf = none; at least Kq of them finite): bisection between their extremes
// until at most Kq + slack values lie below the bound.
template <int P>
__device__ __forceinline__ float kth_bound(const float (&v)[P], int Kq, int slack, int rounds) {
  float lo = INFINITY, hi = -INFINITY;
#pragma unroll
  for (int t = 0; t < P; ++t) {
    lo = fminf(lo, v[t]);
    if (v[t] < INFINITY) hi = fmaxf(hi, v[t]);
  }
  lo = from_ord(__reduce_min_sync(kFull, ord_float(lo)));
  hi = from_ord(__reduce_max_sync(kFull, ord_float(hi)));
  for (int it = 0; it < rounds; ++it) {
    const float mid = 0.5f * lo + 0.5f * hi;
    if (!(mid > lo) || !(mid < hi)) break;
    int c = 0;
#pragma unroll
    for (int t = 0; t < P; ++t) c += v[t] <= mid;
    c = __reduce_add_sync(kFull, c);
    if (c >= Kq) {
      hi = mid;
      if (c <= Kq + slack) break;
    } else {
      lo = mid;
    }
  }
  return hi;
}

// Cuts the list of lane `src`'s row (m entries, P * 32 = cap) back to the
// values below its new threshold; returns the entries left.
template <int P>
__device__ __forceinline__ int cut_list(float2* list, int m, int Kq, float nq, float nmax, float crel, int inner,
                                        float* tau, int lane) {
  float2 e[P];
  float v[P];
#pragma unroll
  for (int t = 0; t < P; ++t) {
    const int i = lane + 32 * t;
    e[t] = i < m ? list[i] : make_float2(INFINITY, 0.0f);
    v[t] = e[t].x;
  }
  // a quarter more than Kq values may stay: every bisection round is a reduction
  const float A = kth_bound<P>(v, Kq, Kq >> 2, 14);
  const float lim = fminf(*tau, A + 2.0f * delta_of(A, nq, nmax, crel, inner));
  int left = 0;
  __syncwarp();
#pragma unroll
  for (int t = 0; t < P; ++t) {
    const bool keep = v[t] < lim;
    const unsigned b = __ballot_sync(kFull, keep);
    if (keep) list[left + __popc(b & ((1u << lane) - 1u))] = e[t];
    left += __popc(b);
  }
  __syncwarp();
  *tau = lim;
  return left;
}

struct SearchShared {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t afull[2], aempty[2], qfull, qempty, nfull[kNormSlots];
  uint32_t tmem;
  int stop;
  unsigned long long tau[2][kQRows];  // (query tile, threshold) of every row, per group
};

constexpr size_t kSharedRoom = 2432;  // static shared memory of candidates_kernel
static_assert(sizeof(SearchShared) <= kSharedRoom, "static shared memory");

// What bounds it: the epilogue's issue slots (about 4 per value) and the list
// cuts; the tensor pipe needs 12 instructions of 128 cycles for a 128 x 256
// tile of 64 padded coordinates.  N = 256 is the widest instruction; two
// accumulators (all 512 TMEM columns) let one group of four warps work on a
// tile while the tensor core fills the other.  Against the mma.sync kernel with
// per-lane heaps that this replaces, and its brute-force fallback rows:
// 100000 x 50, K = 30: 24.8 + 9.7 -> 6.1 ms; against the brute force, which
// took K > 96, inner products and the fold-wise searches: 20011 x 50, K = 100
// 62.9 -> 0.89 ms; 12000 x 100 cosine, K = 30 38.3 -> 0.3 ms; 10000 x 50,
// 10 folds, K = 10 1.5 -> 0.16 ms.
template <int P>
__global__ void __launch_bounds__(kThreads, 1) candidates_kernel(SearchArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ SearchShared sh;
  const int warp = tc5::warp_index(), lane = threadIdx.x & 31;
  const long long first_pair = static_cast<long long>(blockIdx.x) * A.per;
  const int span = static_cast<int>(min(A.pairs - first_pair, static_cast<long long>(A.per)));
  // first pair of a query tile, counted from the CTA's first
  auto start_of = [&](int qt) {
    return static_cast<int>((A.off != nullptr ? A.off[qt] : static_cast<long long>(qt) * A.ntiles) - first_pair);
  };
  const uint32_t qbytes = static_cast<uint32_t>(A.chunks) * kQRows * 16;       // one of hi / lo
  const uint32_t sbytes = static_cast<uint32_t>(A.kg) * kBlockRows * 16;       // one of hi / lo of a stage
  float* const norms = reinterpret_cast<float*>(smem);  // [slot][256]
  const uint32_t qs = tc5::smem_u32(smem) + kNormSlots * kBlockRows * 4, ss = qs + 2 * qbytes;
  volatile int* stop = &sh.stop;
  if (threadIdx.x == 0) {
    for (int s = 0; s < A.stages; ++s) {
      tc5::mbar_init(tc5::smem_u32(&sh.full[s]), 1);
      tc5::mbar_init(tc5::smem_u32(&sh.empty[s]), 1);
    }
    for (int g = 0; g < 2; ++g) {
      tc5::mbar_init(tc5::smem_u32(&sh.afull[g]), 1);
      tc5::mbar_init(tc5::smem_u32(&sh.aempty[g]), 4);
    }
    for (int g = 0; g < kNormSlots; ++g) tc5::mbar_init(tc5::smem_u32(&sh.nfull[g]), 1);
    tc5::mbar_init(tc5::smem_u32(&sh.qfull), 1);
    tc5::mbar_init(tc5::smem_u32(&sh.qempty), 1);
    tc5::mbar_fence_init();
    sh.stop = 0;
  }
  if (threadIdx.x < 2 * kQRows) sh.tau[threadIdx.x / kQRows][threadIdx.x % kQRows] = ~0ull;
  if (warp == 9) tc5::tmem_alloc(tc5::smem_u32(&sh.tmem), 512);
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  const uint32_t tmem = __shfl_sync(kFull, sh.tmem, 0);

  // first query tile of the range
  int q = 0;
  if (A.off == nullptr) {
    q = static_cast<int>(first_pair / A.ntiles);
  } else {
    int lo = 0, hi = A.qtiles - 1;  // last q with off[q] <= first_pair
    while (lo < hi) {
      const int m = (lo + hi + 1) >> 1;
      if (A.off[m] <= first_pair) lo = m;
      else hi = m - 1;
    }
    q = lo;
  }

  // every role walks the same (query tile, candidate tile) sequence
  if (warp == 8) {
    if (lane == 0) {
      int stage = 0, qn = 0;
      uint32_t phase = 0;
      bool ok = true;
      int issued = 0, it = 0;
      for (int pair = 0, qt = q; ok && pair < span; ++qt) {
        const int o = start_of(qt);
        const int2 sk = A.skip != nullptr ? A.skip[qt] : make_int2(0, 0);
        const TileOrder ord(A.ntiles, qt * kQRows / kBlockRows, sk.x, sk.y);
        const int end = min(span, o + ord.count);
        if (pair >= end) continue;
        // the query tile: half of a block, 2 KB of every chunk
        if (qn > 0) ok = tc5::mbar_wait(tc5::smem_u32(&sh.qempty), (qn - 1) & 1, stop);
        if (!ok) break;
        ++qn;
        const uint32_t qb = tc5::smem_u32(&sh.qfull);
        tc5::mbar_expect(qb, 2 * qbytes);
        const size_t src0 = (static_cast<size_t>(qt / 2) * A.chunks * kBlockRows + (qt & 1) * kQRows) * 8;
        for (int c = 0; c < A.chunks; ++c) {
          const size_t src = src0 + static_cast<size_t>(c) * kBlockRows * 8;
          tc5::bulk_load(qs + c * kQRows * 16, A.xh + src, kQRows * 16, qb);
          tc5::bulk_load(qs + qbytes + c * kQRows * 16, A.xl + src, kQRows * 16, qb);
        }
        for (; ok && pair < end; ++pair) {
          const int tile = ord.at(pair - o);
          for (int c0 = 0; c0 < A.chunks; c0 += A.kg) {
            ok = tc5::mbar_wait(tc5::smem_u32(&sh.empty[stage]), phase ^ 1u, stop);
            if (!ok) break;
            if (c0 == 0) {
              // the tile's additive terms.  At most kMaxStages tiles are
              // multiplied after the one whose stage was just freed, and a
              // tile is multiplied once the tile two before it is read out, so
              // the tile kNormSlots before this one is done with its slot
              const uint32_t nb = tc5::smem_u32(&sh.nfull[it % kNormSlots]);
              tc5::mbar_expect(nb, kBlockRows * 4);
              tc5::bulk_load(tc5::smem_u32(norms + (it % kNormSlots) * kBlockRows),
                             A.cn + static_cast<size_t>(tile) * kBlockRows, kBlockRows * 4, nb);
              ++it;
            }
            const int nc = min(A.kg, A.chunks - c0);
            const uint32_t bytes = static_cast<uint32_t>(nc) * kBlockRows * 16;
            const uint32_t bar = tc5::smem_u32(&sh.full[stage]), dst = ss + stage * 2 * sbytes;
            const size_t src = (static_cast<size_t>(tile) * A.chunks + c0) * kBlockRows * 8;
            tc5::mbar_expect(bar, 2 * bytes);
            tc5::bulk_load(dst, A.xh + src, bytes, bar);
            tc5::bulk_load(dst + sbytes, A.xl + src, bytes, bar);
            ++issued;
            if (++stage == A.stages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (!ok) {
        // the copies in flight land before the block's memory is given up
        int zero = 0;
        for (int b = 1; b <= min(issued, A.stages); ++b) {
          const int s = (stage - b + A.stages) % A.stages;
          tc5::mbar_wait(tc5::smem_u32(&sh.full[s]), s < stage ? phase : phase ^ 1u, &zero);
        }
        if (qn > 0) tc5::mbar_wait(tc5::smem_u32(&sh.qfull), (qn - 1) & 1, &zero);
        for (int i = it - min(it, kNormSlots); i < it; ++i)
          tc5::mbar_wait(tc5::smem_u32(&sh.nfull[i % kNormSlots]), (i / kNormSlots) & 1, &zero);
      }
    }
  } else if (warp == 9) {
    const uint32_t idesc = tc5::idesc_bf16(kQRows, kBlockRows);
    int stage = 0, qn = 0, it = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int pair = 0, qt = q; ok && pair < span; ++qt) {
      const int o = start_of(qt);
      const int2 sk = A.skip != nullptr ? A.skip[qt] : make_int2(0, 0);
      const int end = min(span, o + A.ntiles - sk.y);
      if (pair >= end) continue;
      ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.qfull), qn & 1, stop));
      ++qn;
      for (; ok && pair < end; ++pair, ++it) {
        const int buf = it & 1;
        ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.aempty[buf]), ((it >> 1) & 1) ^ 1, stop));
        if (!ok) break;
        tc5::fence_after();
        const uint32_t dcol = tmem + buf * kBlockRows;
        for (int c0 = 0; c0 < A.chunks; c0 += A.kg) {
          ok = __all_sync(kFull, tc5::mbar_wait(tc5::smem_u32(&sh.full[stage]), phase, stop));
          if (!ok) break;
          tc5::fence_after();
          // descriptors advance by whole 16-coordinate steps (their address
          // field counts 16 bytes)
          const uint32_t bs = ss + stage * 2 * sbytes, ao = static_cast<uint32_t>(c0) * kQRows * 16;
          uint64_t ah = tc5::operand(qs + ao, kQRows), al = tc5::operand(qs + qbytes + ao, kQRows);
          uint64_t bh = tc5::operand(bs, kBlockRows), bl = tc5::operand(bs + sbytes, kBlockRows);
          const int k1 = min(A.kg, A.chunks - c0) / 2;
#pragma unroll 2
          for (int k = 0; k < k1; ++k) {
            tc5::mma(dcol, ah, bh, idesc, c0 + k > 0);
            tc5::mma(dcol, ah, bl, idesc, true);
            tc5::mma(dcol, al, bh, idesc, true);
            ah += 2 * kQRows;
            al += 2 * kQRows;
            bh += 2 * kBlockRows;
            bl += 2 * kBlockRows;
          }
          tc5::commit(tc5::smem_u32(&sh.empty[stage]));
          if (++stage == A.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) tc5::commit(tc5::smem_u32(&sh.afull[buf]));
      }
      if (ok) tc5::commit(tc5::smem_u32(&sh.qempty));
    }
    // on an early end the instructions still queued finish first
    if (!ok) {
      int zero = 0;
      tc5::commit(tc5::smem_u32(&sh.qempty));
      tc5::mbar_wait(tc5::smem_u32(&sh.qempty), qn > 0 ? (qn - 1) & 1 : 0, &zero);
    }
  } else {
    const int g = warp >> 2;                 // this warp's accumulator / tile parity
    const int r = (warp & 3) * 32 + lane;    // its row of the query tile
    const uint32_t acc = tmem + g * kBlockRows + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float nmax = __uint_as_float(A.status[kStNorm]);
    const int trig0 = A.Kq + max(32, A.Kq / 2), room = A.cap - 32;
    int it = 0;
    bool ok = true;
    for (int pair = 0, qt = q; ok && pair < span; ++qt) {
      const int o = start_of(qt);
      const int2 sk = A.skip != nullptr ? A.skip[qt] : make_int2(0, 0);
      const TileOrder ord(A.ntiles, qt * kQRows / kBlockRows, sk.x, sk.y);
      const int end = min(span, o + ord.count);
      if (pair >= end) continue;
      const int seg = blockIdx.x - static_cast<int>((first_pair + o) / A.per);
      const size_t qpos = static_cast<size_t>(qt) * kQRows + r;
      const size_t slot = (qpos * A.segs + seg) * 2 + g;
      float2* const list = A.list + slot * A.cap;
      const float nq = A.qn[qpos];
      float tau = nq < 0.0f ? -INFINITY : INFINITY;
      int cnt = 0, trig = min(trig0, room);
      bool fresh = true, failed = false;
      for (; ok && pair < end; ++pair, ++it) {
        if ((it & 1) != g) continue;
        const int tile = ord.at(pair - o);
        const float* cn = norms + (it % kNormSlots) * kBlockRows;
        ok = tc5::mbar_wait(tc5::smem_u32(&sh.nfull[it % kNormSlots]), (it / kNormSlots) & 1, stop);
        ok = __all_sync(kFull, ok && tc5::mbar_wait(tc5::smem_u32(&sh.afull[g]), (it >> 1) & 1, stop));
        if (!ok) break;
        tc5::fence_after();
        if (fresh) {
          // The list's first tile: bound the row's Kq-th smallest value of the
          // tile by bisection on the accumulator, each thread for its own row,
          // so that the list starts with about Kq values instead of 256.
          fresh = false;
          float lo = INFINITY, hi = -INFINITY;
          int fin = 0;
          for (int c = 0; c < kBlockRows; c += 32) {
            float v[32];
            tc5::load32(acc + c, v);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 n4 = *reinterpret_cast<const float4*>(cn + c + i);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float a = __fmaf_rn(v[i + e], A.scale, e == 0 ? n4.x : e == 1 ? n4.y : e == 2 ? n4.z : n4.w);
                lo = fminf(lo, a);
                if (a < INFINITY) {
                  hi = fmaxf(hi, a);
                  ++fin;
                }
              }
            }
          }
          bool active = fin >= A.Kq;
          for (int round = 0; round < 10; ++round) {
            if (!__any_sync(kFull, active)) break;
            const float mid = 0.5f * lo + 0.5f * hi;
            int below = 0;
            for (int c = 0; c < kBlockRows; c += 32) {
              float v[32];
              tc5::load32(acc + c, v);
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 n4 = *reinterpret_cast<const float4*>(cn + c + i);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  below += __fmaf_rn(v[i + e], A.scale, e == 0 ? n4.x : e == 1 ? n4.y : e == 2 ? n4.z : n4.w) <= mid;
              }
            }
            if (active) {
              if (below >= A.Kq) {
                hi = mid;
                if (below <= A.Kq + (A.Kq >> 3)) active = false;
              } else {
                lo = mid;
              }
            }
          }
          if (fin >= A.Kq && nq >= 0.0f) tau = hi + 2.0f * delta_of(hi, nq, nmax, A.crel, A.inner);
        }
        // the other group's threshold for the same query holds for this group
        // too: it is at least the row's final limit
        const unsigned long long other = *const_cast<volatile unsigned long long*>(&sh.tau[g ^ 1][r]);
        if (!failed && static_cast<int>(other >> 32) == qt)
          tau = fminf(tau, __uint_as_float(static_cast<unsigned>(other)));
        const int pos0 = tile * kBlockRows;
        for (int c = 0; c < kBlockRows; c += 32) {
          float v[32];
          tc5::load32(acc + c, v);
          float m = INFINITY;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 n4 = *reinterpret_cast<const float4*>(cn + c + i);
            v[i] = __fmaf_rn(v[i], A.scale, n4.x);
            v[i + 1] = __fmaf_rn(v[i + 1], A.scale, n4.y);
            v[i + 2] = __fmaf_rn(v[i + 2], A.scale, n4.z);
            v[i + 3] = __fmaf_rn(v[i + 3], A.scale, n4.w);
            m = tc5::min3(m, v[i], v[i + 1]);
            m = tc5::min3(m, v[i + 2], v[i + 3]);
          }
          if (!__any_sync(kFull, m < tau)) continue;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (v[i] < tau) list[cnt++] = make_float2(v[i], __int_as_float(pos0 + c + i));
          }
          unsigned todo = __ballot_sync(kFull, cnt > trig);
          while (todo != 0u) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            __syncwarp();
            float2* const l2 = reinterpret_cast<float2*>(
                __shfl_sync(kFull, reinterpret_cast<unsigned long long>(list), src));
            float t2 = __shfl_sync(kFull, tau, src);
            const int left = cut_list<P>(l2, __shfl_sync(kFull, cnt, src), A.Kq, __shfl_sync(kFull, nq, src), nmax,
                                         A.crel, A.inner, &t2, lane);
            if (lane == src) {
              cnt = left;
              tau = t2;
              trig = min(room, max(trig0, left + max(32, A.Kq / 2)));
              if (left > room) {  // too many values within 2 delta: the row goes to the brute force
                failed = true;
                cnt = 0;
                tau = -INFINITY;
              } else {
                *const_cast<volatile unsigned long long*>(&sh.tau[g][r]) =
                    (static_cast<unsigned long long>(qt) << 32) | __float_as_uint(tau);
              }
            }
          }
        }
        tc5::fence_before();
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(tc5::smem_u32(&sh.aempty[g]));
      }
      if (pair < end) pair = end;
      A.cnt[slot] = failed ? -1 : cnt;
      A.tau[slot] = failed ? -INFINITY : tau;
    }
  }
  __syncwarp();
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  if (warp == 9) tc5::tmem_free(tmem, 512);
  if (threadIdx.x == 0 && sh.stop != 0) atomicExch(&A.status[kStTimeout], 1u);
}

struct RerankArgs {
  SearchArgs s;
  const float* x;      // n x d4 floats, 16-byte aligned rows
  int d, d4, K, npos, mode;
  const int* perm;
  int* idx;
  float* dist;
  int* fb_rows;
};

// One warp per query position.
__global__ void __launch_bounds__(128) rerank_kernel(RerankArgs R) {
  __shared__ float2 room[4][kSurvivors];
  const SearchArgs& A = R.s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos = blockIdx.x * 4 + warp;
  if (pos >= R.npos) return;
  const int row = R.perm != nullptr ? R.perm[pos] : pos;
  const float nq = A.qn[pos];
  if (nq < 0.0f) return;  // padding
  const float nmax = __uint_as_float(A.status[kStNorm]);
  const unsigned below = (1u << lane) - 1u;
  float2* list = room[warp];
  bool bad = A.status[kStBad] != 0u || A.status[kStTimeout] != 0u || !(nmax >= 1e-20f && nmax <= 1e36f);
  int m = 0;
  if (!bad) {
    const int qt = pos / kQRows;
    const long long o = A.off != nullptr ? A.off[qt] : static_cast<long long>(qt) * A.ntiles;
    const int count = A.ntiles - (A.skip != nullptr ? A.skip[qt].y : 0);
    // this row's lists
    const int nl = count > 0 ? 2 * (static_cast<int>((o + count - 1) / A.per - o / A.per) + 1) : 0;
    const size_t slot = static_cast<size_t>(pos) * A.segs * 2;
    float tau = INFINITY;
    int low = 0;
    for (int l = lane; l < nl; l += 32) {
      tau = fminf(tau, A.tau[slot + l]);
      low = min(low, A.cnt[slot + l]);
    }
    tau = from_ord(__reduce_min_sync(kFull, ord_float(tau)));
    bad = __reduce_min_sync(kFull, low) < 0;
    for (int l = 0; l < nl && !bad; ++l) {
      const int c = A.cnt[slot + l];
      const float2* src = A.list + (slot + l) * A.cap;
      for (int e0 = 0; e0 < c; e0 += 32) {
        const float2 v = e0 + lane < c ? src[e0 + lane] : make_float2(INFINITY, 0.0f);
        const bool keep = v.x < tau;
        const unsigned b = __ballot_sync(kFull, keep);
        if (m + __popc(b) > kSurvivors) {
          // many short segments each hold about Kq values: cut the joined list
          __syncwarp();
          m = cut_list<kSurvivors / 32>(list, m, A.Kq, nq, nmax, A.crel, A.inner, &tau, lane);
          if (m + __popc(b) > kSurvivors) {
            bad = true;
            break;
          }
        }
        if (keep) list[m + __popc(b & below)] = v;
        m += __popc(b);
      }
    }
    __syncwarp();
    bad = bad || m < A.Kq;
  }
  if (bad) {
    if (lane == 0) R.fb_rows[atomicAdd(&A.status[kStFallback], 1u)] = row;
    return;
  }
  float v[kSurvivors / 32];
#pragma unroll
  for (int t = 0; t < kSurvivors / 32; ++t) v[t] = lane + 32 * t < m ? list[lane + 32 * t].x : INFINITY;
  const float AK = kth_bound<kSurvivors / 32>(v, A.Kq, 0, 24);
  const float lim = AK + 2.0f * delta_of(AK, nq, nmax, A.crel, A.inner);
  // keep the values within the limit, except the query itself
  int m2 = 0;
#pragma unroll
  for (int t = 0; t < kSurvivors / 32; ++t) {
    if (32 * t >= m) break;
    const int i = lane + 32 * t;
    const float2 e = i < m ? list[i] : make_float2(INFINITY, 0.0f);
    const int p = __float_as_int(e.y);
    const bool keep = i < m && e.x <= lim && p != pos;
    const unsigned b = __ballot_sync(kFull, keep);
    __syncwarp();
    if (keep) list[m2 + __popc(b & below)] = make_float2(0.0f, e.y);
    __syncwarp();
    m2 += __popc(b);
  }
  if (m2 < R.K) {
    if (lane == 0) R.fb_rows[atomicAdd(&A.status[kStFallback], 1u)] = row;
    return;
  }
  // canonical distances, a lane per candidate; the keys replace the entries
  unsigned long long* key = reinterpret_cast<unsigned long long*>(list);
  const float4* xq = reinterpret_cast<const float4*>(R.x + static_cast<size_t>(row) * R.d4);
  const int full4 = R.d / 4, rest = R.d & 3;
  for (int i = lane; i < m2; i += 32) {
    const int p = __float_as_int(list[i].y);
    const int j = R.perm != nullptr ? R.perm[p] : p;
    const float4* xj = reinterpret_cast<const float4*>(R.x + static_cast<size_t>(j) * R.d4);
    float a = 0.0f;
    if (A.inner) {
#pragma unroll 4
      for (int k = 0; k < full4; ++k) {
        const float4 u = xq[k], w = xj[k];
        a = __fadd_rn(a, __fmul_rn(u.x, w.x));
        a = __fadd_rn(a, __fmul_rn(u.y, w.y));
        a = __fadd_rn(a, __fmul_rn(u.z, w.z));
        a = __fadd_rn(a, __fmul_rn(u.w, w.w));
      }
      if (rest) {
        const float4 u = xq[full4], w = xj[full4];
        a = __fadd_rn(a, __fmul_rn(u.x, w.x));
        if (rest > 1) a = __fadd_rn(a, __fmul_rn(u.y, w.y));
        if (rest > 2) a = __fadd_rn(a, __fmul_rn(u.z, w.z));
      }
      a = __fsub_rn(0.0f, a);  // +0 for a zero product, so that equal values have equal keys
    } else {
#pragma unroll 4
      for (int k = 0; k < full4; ++k) {
        const float4 u = xq[k], w = xj[k];
        float f = __fsub_rn(u.x, w.x);
        a = __fadd_rn(a, __fmul_rn(f, f));
        f = __fsub_rn(u.y, w.y);
        a = __fadd_rn(a, __fmul_rn(f, f));
        f = __fsub_rn(u.z, w.z);
        a = __fadd_rn(a, __fmul_rn(f, f));
        f = __fsub_rn(u.w, w.w);
        a = __fadd_rn(a, __fmul_rn(f, f));
      }
      if (rest) {
        const float4 u = xq[full4], w = xj[full4];
        float f = __fsub_rn(u.x, w.x);
        a = __fadd_rn(a, __fmul_rn(f, f));
        if (rest > 1) {
          f = __fsub_rn(u.y, w.y);
          a = __fadd_rn(a, __fmul_rn(f, f));
        }
        if (rest > 2) {
          f = __fsub_rn(u.z, w.z);
          a = __fadd_rn(a, __fmul_rn(f, f));
        }
      }
    }
    key[i] = (static_cast<unsigned long long>(ord_float(a)) << 32) | static_cast<unsigned>(j);
  }
  __syncwarp();
  // rank of every key; the first K are the row's neighbours
  for (int i = lane; i < m2; i += 32) {
    const unsigned long long mine = key[i];
    int rank = 0;
#pragma unroll 4
    for (int e = 0; e < m2; ++e) rank += key[e] < mine;
    if (rank < R.K) {
      float a = from_ord(static_cast<unsigned>(mine >> 32));
      // the brute force reports minus a float sum: a zero sum gives -0
      if (A.inner && a == 0.0f) a = -0.0f;
      const size_t out = static_cast<size_t>(row) * R.K + rank;
      R.idx[out] = static_cast<int>(mine & 0xffffffffu);
      R.dist[out] = knn_output_distance(a, R.mode);
    }
  }
}

}  // namespace

// a 16-byte chunk (8 coordinates) of a row per thread
__global__ void split_rows_kernel(const float* __restrict__ x, int n, int d, int chunks, uint4* __restrict__ xh,
                                  uint4* __restrict__ xl) {
  const size_t e = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<size_t>(n) * chunks) return;
  const size_t r = e / chunks;
  const int c = static_cast<int>(e % chunks);
  uint32_t h[4], l[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t hb[2], lb[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int k = 8 * c + 2 * q + s;
      const float v = k < d ? x[r * d + k] : 0.0f;
      hb[s] = bf16_bits(v);
      lb[s] = bf16_bits(__fsub_rn(v, __uint_as_float(hb[s] << 16)));
    }
    h[q] = hb[0] | (hb[1] << 16);
    l[q] = lb[0] | (lb[1] << 16);
  }
  xh[e] = make_uint4(h[0], h[1], h[2], h[3]);
  xl[e] = make_uint4(l[0], l[1], l[2], l[3]);
}

int bf16_split_rows(const float* x, int n, int d, int dp, uint16_t* xh, uint16_t* xl, cudaStream_t st) {
  const size_t total = static_cast<size_t>(n) * (dp / 8);
  if (total == 0) return 0;
  split_rows_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(
      x, n, d, dp / 8, reinterpret_cast<uint4*>(xh), reinterpret_cast<uint4*>(xl));
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

namespace {

// Up to 223 neighbours: lists of 512 entries.  Up to 2^26 rows: their lists, 4 KB a row
// at least, take all of the memory.
constexpr int kMinRows = 97;
constexpr int kMaxRows = 1 << 26;

struct TcLayout {
  int dp, chunks, kg, stages, npos, ntiles, qtiles, cap, Kq, per, segs, d4, ctas;
  long long pairs;
  size_t smem;
  size_t o_xh, o_xl, o_cn, o_qn, o_status, o_xp, o_cnt, o_tau, o_list, o_fb, o_brute, total;
};

int list_entries(int Kq) { return Kq <= 36 ? 128 : Kq <= 112 ? 256 : 512; }

// The operand blocks, the stream-K split over `sms` CTAs and the scratch
// offsets.  fp: the fold-wise search's row order, or null.
TcLayout tc_layout(int n, int d, int K, int segments, int sms, const KnnFoldPlan* fp) {
  TcLayout L{};
  L.dp = (d + 15) / 16 * 16;
  L.chunks = L.dp / 8;
  L.d4 = (d + 3) / 4 * 4;
  L.Kq = fp != nullptr ? K : K + 1;
  L.cap = list_entries(L.Kq);
  L.ntiles = fp != nullptr ? fp->tiles : (n + kBlockRows - 1) / kBlockRows;
  L.qtiles = fp != nullptr ? 2 * fp->tiles : (n + kQRows - 1) / kQRows;
  L.pairs = fp != nullptr ? fp->pairs : static_cast<long long>(L.ntiles) * L.qtiles;
  L.npos = L.ntiles * kBlockRows;
  L.ctas = L.pairs < sms ? (L.pairs > 0 ? static_cast<int>(L.pairs) : 1) : sms;
  L.per = static_cast<int>((L.pairs + L.ctas - 1) / L.ctas);
  if (L.per < 1) L.per = 1;
  L.segs = (L.ntiles - 1) / L.per + 2;
  // stages of 32 coordinates (32 KB), four where the query tile (up to 128 KB)
  // leaves the room; never less than half an SM's shared memory, so that one
  // CTA owns the SM's TMEM
  L.kg = L.chunks < 4 ? L.chunks : 4;
  const size_t query = static_cast<size_t>(2) * L.chunks * kQRows * 16 + kNormSlots * kBlockRows * 4;
  const size_t stage = static_cast<size_t>(2) * L.kg * kBlockRows * 16;
  L.stages = kMaxStages;
  while (L.stages > 2 && query + L.stages * stage > kSmemLimit - kSharedRoom) --L.stages;
  L.smem = query + L.stages * stage;
  if (L.smem < 116 * 1024) L.smem = 116 * 1024;
  auto al = [](size_t v) { return (v + 255) / 256 * 256; };
  size_t o = 0;
  const size_t lists = static_cast<size_t>(L.qtiles) * kQRows * L.segs * 2;
  L.o_xh = o; o = al(o + static_cast<size_t>(L.npos) * L.dp * 2);
  L.o_xl = o; o = al(o + static_cast<size_t>(L.npos) * L.dp * 2);
  L.o_cn = o; o = al(o + static_cast<size_t>(L.npos) * 4);
  L.o_qn = o; o = al(o + static_cast<size_t>(L.npos) * 4);
  L.o_status = o; o = al(o + 16);
  L.o_xp = o; o = al(o + static_cast<size_t>(n) * L.d4 * 4);
  L.o_cnt = o; o = al(o + lists * 4);
  L.o_tau = o; o = al(o + lists * 4);
  L.o_list = o; o = al(o + lists * L.cap * sizeof(float2));
  L.o_fb = o; o = al(o + static_cast<size_t>(n) * 4);
  L.o_brute = o; o = al(o + knn_bruteforce_scratch(n, K, segments));
  L.total = o;
  return L;
}

template <int P>
cudaError_t launch_candidates(const SearchArgs& S, const TcLayout& L, cudaStream_t st) {
  const cudaError_t e = allow_shared_memory(candidates_kernel<P>);
  if (e != cudaSuccess) return e;
  candidates_kernel<P><<<L.ctas, kThreads, L.smem, st>>>(S);
  return cudaGetLastError();
}

int tc_search(const TcLayout& L, const float* x, int n, int d, int K, bool inner, int mode, const int* d_folds,
              const int* perm, const int* off, const int2* skip, int segments, unsigned char* b, int* idx,
              float* dist, cudaStream_t st) {
  unsigned* status = reinterpret_cast<unsigned*>(b + L.o_status);
  cudaError_t e = cudaMemsetAsync(status, 0, 16, st);
  if (e != cudaSuccess) return static_cast<int>(e);
  // rows the re-rank can load as 16-byte vectors, or a padded copy of them
  const bool in_place = d % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  float* xp = in_place ? nullptr : reinterpret_cast<float*>(b + L.o_xp);
  uint16_t* xh = reinterpret_cast<uint16_t*>(b + L.o_xh);
  uint16_t* xl = reinterpret_cast<uint16_t*>(b + L.o_xl);
  float* cn = reinterpret_cast<float*>(b + L.o_cn);
  float* qn = reinterpret_cast<float*>(b + L.o_qn);
  int* fb = reinterpret_cast<int*>(b + L.o_fb);
  prep_kernel<<<L.npos / 32, 256, 0, st>>>(x, n, d, L.chunks, L.npos, perm, inner ? 1 : 0, xh, xl, cn, qn, xp, L.d4,
                                          status);
  SearchArgs S{};
  S.xh = xh;
  S.xl = xl;
  S.cn = cn;
  S.qn = qn;
  S.status = status;
  S.chunks = L.chunks;
  S.kg = L.kg;
  S.stages = L.stages;
  S.ntiles = L.ntiles;
  S.qtiles = L.qtiles;
  S.Kq = L.Kq;
  S.cap = L.cap;
  S.scale = inner ? -1.0f : -2.0f;
  S.crel = 5e-5f + 1e-6f * static_cast<float>(L.dp);
  S.inner = inner ? 1 : 0;
  S.off = off;
  S.skip = skip;
  S.pairs = L.pairs;
  S.per = L.per;
  S.segs = L.segs;
  S.list = reinterpret_cast<float2*>(b + L.o_list);
  S.cnt = reinterpret_cast<int*>(b + L.o_cnt);
  S.tau = reinterpret_cast<float*>(b + L.o_tau);
  e = L.cap == 128   ? launch_candidates<4>(S, L, st)
      : L.cap == 256 ? launch_candidates<8>(S, L, st)
                     : launch_candidates<16>(S, L, st);
  if (e != cudaSuccess) return static_cast<int>(e);
  RerankArgs R{};
  R.s = S;
  R.x = in_place ? x : xp;
  R.d = d;
  R.d4 = L.d4;
  R.K = K;
  R.npos = perm != nullptr ? L.npos : n;
  R.mode = mode;
  R.perm = perm;
  R.idx = idx;
  R.dist = dist;
  R.fb_rows = fb;
  rerank_kernel<<<(R.npos + 3) / 4, 128, 0, st>>>(R);
  count_launch(3);
  e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  return knn_bruteforce_rows(x, n, d, K, inner, d_folds, mode, segments, fb,
                             reinterpret_cast<const int*>(status + kStFallback), b + L.o_brute, idx, dist, st);
}

}  // namespace

bool knn_tc_supported(int n, int d, int K) {
  return d >= 1 && d <= kMaxDp && K >= 1 && K + 1 <= 224 && n >= kMinRows && n <= kMaxRows && n > K;
}

bool knn_tc_explicit(int n, int d, int K) {
  const int heaps = 2 * (K <= 40 ? 8 : 4);
  int kp = (2 * ((K + heaps - 1) / heaps) + 15) / 8 * 8;
  kp = kp < 16 ? 16 : kp;
  return d >= 1 && d <= kMaxDp && K >= 1 && K <= 96 && n > 2 * kp + 64 && n <= kMaxRows;
}

size_t knn_tc_scratch(int n, int d, int K, int segments, int sms, const KnnFoldPlan* fp) {
  return tc_layout(n, d, K, segments, sms, fp).total;
}

int knn_tc_graph(const float* x, int n, int d, int K, int metric, int segments, int sms, void* scratch, int* idx,
                 float* dist, cudaStream_t st) {
  const TcLayout L = tc_layout(n, d, K, segments, sms, nullptr);
  const int mode = metric == 2 ? kKnnOutSqrt : metric == 0 ? kKnnOutCosine : kKnnOutInner;
  return tc_search(L, x, n, d, K, metric != 2, mode, nullptr, nullptr, nullptr, nullptr, segments,
                   static_cast<unsigned char*>(scratch), idx, dist, st);
}

int knn_tc_fallback_count(const void* scratch, int n, int d, int K, int segments, int sms, int* out,
                          cudaStream_t st) {
  const TcLayout L = tc_layout(n, d, K, segments, sms, nullptr);
  const unsigned char* b = static_cast<const unsigned char*>(scratch);
  return static_cast<int>(
      cudaMemcpyAsync(out, b + L.o_status + 4 * kStFallback, sizeof(int), cudaMemcpyDeviceToHost, st));
}

namespace {

// The brute force's time in ns: its scan of the rows (another kernel above 64
// coordinates; at few rows the latency of a row's chain over a segment) and the
// insertions into the kept neighbours, which grow with their number.
double brute_ns(int n, int d, int K) {
  const double rows = n, k = K;
  const double scan = d <= 64 ? std::max(2.2e-4 * rows * rows * (d + 1), 1.2 * rows * (d + 6))
                              : std::max(7e-3 * rows * rows * d, 18.0 * rows * d);
  return scan + std::max(450.0 * k * std::sqrt(rows), 0.4 * rows * k * std::min(k, 64.0));
}

// ... and that of a 128 x 256 tile's products and lists.
double pair_ns(int d) { return 6.0 + 0.03 * d; }

// Points on a line, or on a circle once scaled to length one: from some thousands of
// rows on more of them lie within the products' error bound of a row than its list
// holds, and nearly all rows would go on to the brute force as well.  30000 rows, line
// and circle, K = 10: 1.2 and 1.0 of the brute force's time, K = 30 0.7 and 0.6; 100000
// rows, K = 30 1.1, K = 90 0.7 and 1.0; 8000 rows, K = 1 1.3 and below 1.
bool too_close(int n, int d, int K, int metric) {
  return metric != 1 && d <= (metric == 0 ? 2 : 1) && K <= n / 3000;
}

// Whether the fold-wise search is the faster by tensor cores.  Every fold is padded
// to whole tiles, so the products grow with the number of folds: leave-one-out of n
// rows would take n (n - 1) tiles' products and 4 KB or more of lists for 256 n
// positions.  Both sides' times in ns, fitted to 2267 whole calls of either (256 to
// 65000 rows, 2 to 128 coordinates, 1 to 50 neighbours, 2 to 400 folds; the rule is
// 0.2% behind the better side on average, 1.15x at worst up to 100 folds and 1.36x
// beyond; always the tensor search 8.5% and 3.3x): 10000 x 50, K = 10, 300 folds take 2.45 ms here and
// 2.51 by the brute force, 1000 folds 10.8 and 3.1; 1000 x 8, K = 10, 60 folds 0.45
// and 0.47, 300 folds 1.20 and 0.66; 10000 x 128, 1000 folds 13.7 and 100.
bool fold_plan_pays(int n, int d, int K, long long tiles, long long pairs) {
  // room: lists of up to 16 KB a position; pairs and positions are counted in ints
  if (tiles * kBlockRows > std::max(131072ll, 16ll * n) || pairs > (1ll << 30)) return false;
  return 50e3 + 8.0 * n + static_cast<double>(pairs) * pair_ns(d) < brute_ns(n, d, K);
}

}  // namespace

// The graph's search, measured against the brute force over 97 to 100000 rows, 1 to 256
// coordinates, 1 to 90 neighbours and the three metrics.  Its launches take some 65 us
// more, which few neighbours of few rows do not earn: 256 x 8, K = 1 0.145 and 0.101 ms
// a call, 512 x 8, K = 5 0.13 and 0.12, K = 10 0.18 and 0.23, 2000 x 8, K = 1 equal; 100 x
// 100, K = 30 0.19 and 0.45.
bool knn_tc_pays(int n, int d, int K, int metric) {
  if (!knn_tc_supported(n, d, K) || too_close(n, d, K, metric)) return false;
  const double pairs = static_cast<double>((n + kBlockRows - 1) / kBlockRows) * ((n + kQRows - 1) / kQRows);
  return 65e3 + pairs * pair_ns(d) < brute_ns(n, d, K);
}

KnnFoldPlan knn_fold_plan(const std::vector<int>& folds, int d, int K, int metric) {
  KnnFoldPlan p;
  const int n = static_cast<int>(folds.size());
  if (!knn_tc_supported(n, d, K) || too_close(n, d, K, metric) || n < 256) return p;
  // the rows by fold, ascending within one (fold numbers lie below n: make_folds)
  std::vector<int> size;
  for (int f : folds) {
    if (static_cast<size_t>(f) >= size.size()) size.resize(static_cast<size_t>(f) + 1, 0);
    ++size[f];
  }
  long long tiles = 0, pairs = 0;
  for (int v : size) tiles += (v + kBlockRows - 1) / kBlockRows;
  for (int v : size) pairs += (v + kQRows - 1) / kQRows * (tiles - (v + kBlockRows - 1) / kBlockRows);
  if (!fold_plan_pays(n, d, K, tiles, pairs)) return p;
  p.tiles = static_cast<int>(tiles);
  p.perm.assign(static_cast<size_t>(tiles) * kBlockRows, -1);
  std::vector<int> at(size.size(), 0);
  int first = 0;
  for (size_t f = 0; f < size.size(); ++f) {
    const int own = (size[f] + kBlockRows - 1) / kBlockRows;
    at[f] = first * kBlockRows;
    for (int q = 0; q < 2 * own; ++q) {
      const bool rows = q * kQRows < size[f];  // a query tile of padding alone has no pairs
      p.off.push_back(p.pairs);
      p.skip.push_back(rows ? first : 0);
      p.skip.push_back(rows ? own : p.tiles);
      if (rows) p.pairs += p.tiles - own;
    }
    first += own;
  }
  for (int i = 0; i < n; ++i) p.perm[at[folds[i]]++] = i;
  return p;
}

int knn_tc_fold_search(const float* x, int n, int d, int K, bool inner, const int* d_folds, const KnnFoldPlan& fp,
                       const int* d_perm, const int* d_off, const int* d_skip, int segments, int sms, void* scratch,
                       int* idx, float* dist, cudaStream_t st) {
  const TcLayout L = tc_layout(n, d, K, segments, sms, &fp);
  return tc_search(L, x, n, d, K, inner, kKnnOutRaw, d_folds, d_perm, d_off, reinterpret_cast<const int2*>(d_skip),
                   segments, static_cast<unsigned char*>(scratch), idx, dist, st);
}

}  // namespace kgb
