// Per-run landmark planning on the device.
//
//   strata_kernel (one CTA): index_strata (kodama_matrix.cpp:806-854): the
//     rows of every atlas cluster in ascending row order (counting sort by
//     warps of consecutive rows, each with counters of its own), and the
//     run-independent parts of the quota allocation
//     (kodama_matrix.cpp:880-903): floor of target*count/n and its fractional
//     part, both in x86 extended precision (ext80.h).
//   plan_runs_kernel (one CTA per run): the run's std::mt19937_64 stream
//     (seed + run, one output discarded), the shuffle of the non-empty strata,
//     the systematic residual allocation, std::sample inside each stratum
//     (selection sampling with two positions per draw), then the init k-means
//     seed; the selected rows are compacted in ascending order by the whole
//     CTA, and the first init_k entries of the FAISS-compatible permutation
//     (std::mt19937 seeded (draw & 0x7fffffff) + 1, swaps r <-> r + u % (L-r),
//     kodama_matrix.cpp:535-564) give the initial centroid rows.
//
// The serial parts restate the libstdc++ 13 algorithms the reference calls:
// std::shuffle and std::sample draw two positions per engine call when the
// engine range allows it (uniform integer in [0, b0*b1) split as x / b1,
// x % b1), and uniform_int_distribution downscales one 64-bit output by
// Lemire's method (rng.cuh).
#include "ext80.h"
#include "launch_count.cuh"
#include "smem_limit.cuh"
#include "plan.cuh"
#include "rng.cuh"
#include "warp_match.cuh"

#include <algorithm>

namespace kgb {
namespace {

constexpr int kPlanThreads = 256;
constexpr int kCounterBytes = 128 * 1024;  // strata_kernel: warps' counters in shared memory
// plan_runs_kernel: order, quotas and fractions in shared memory.  No more than
// that, so that a CTA fits beside one of the exact graph's, which runs meanwhile.
constexpr int kSharedStrata = 2048;
constexpr int kRounded = 0x40000000;  // marks a stratum of the shuffled order that took a residual slot

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

struct PlanScratch {
  int* counts;    // strata
  int* offsets;   // strata + 1
  int* cursor;    // strata
  int* rows;      // n
  int* base;      // strata
  Ext80* frac;    // strata
  int* assigned;  // 1
  int* order;     // runs x strata
  int* quota;     // runs x strata
  uint8_t* flags; // runs x n
  int* perm;      // runs x target
};

PlanScratch carve(const PlanArgs& a) {
  PlanScratch s{};
  char* p = static_cast<char*>(a.scratch);
  auto take = [&](size_t bytes) {
    char* q = p;
    p += align256(bytes);
    return q;
  };
  const size_t S = static_cast<size_t>(a.strata), R = static_cast<size_t>(a.runs);
  s.counts = reinterpret_cast<int*>(take(sizeof(int) * S));
  s.offsets = reinterpret_cast<int*>(take(sizeof(int) * (S + 1)));
  s.cursor = reinterpret_cast<int*>(take(sizeof(int) * S));
  s.rows = reinterpret_cast<int*>(take(sizeof(int) * a.n));
  s.base = reinterpret_cast<int*>(take(sizeof(int) * S));
  s.frac = reinterpret_cast<Ext80*>(take(sizeof(Ext80) * S));
  s.assigned = reinterpret_cast<int*>(take(sizeof(int)));
  s.order = reinterpret_cast<int*>(take(sizeof(int) * S * R));
  s.quota = reinterpret_cast<int*>(take(sizeof(int) * S * R));
  s.flags = reinterpret_cast<uint8_t*>(take(static_cast<size_t>(a.n) * R));
  s.perm = reinterpret_cast<int*>(take(sizeof(int) * static_cast<size_t>(a.target) * R));
  return s;
}

// Each of nw warps takes a run of rows and counts them per stratum; after a scan
// over warps and strata it walks them again and places them, so the rows of a
// stratum keep ascending order.  One warp placing all rows took 0.94 ms at
// 100000 rows.  With too many strata for two warps' counters in shared memory, one
// warp counts in global memory.
__global__ void __launch_bounds__(1024) strata_kernel(PlanArgs a, PlanScratch s) {
  extern __shared__ int counters[];  // nw x strata
  __shared__ int bad;
  __shared__ unsigned long long asum;
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int fit = kCounterBytes / static_cast<int>(sizeof(int)) / a.strata;
  const int nw = fit >= 2 ? min(32, fit) : 1;
  int* count = fit >= 2 ? counters : s.counts;
  if (tid == 0) {
    bad = 0;
    asum = 0;
  }
  for (int t = tid; t < nw * a.strata; t += blockDim.x) count[t] = 0;
  __syncthreads();
  const int chunk = ((a.n + nw - 1) / nw + 31) / 32 * 32;
  const int beg = warp < nw ? min(a.n, warp * chunk) : 0, end = warp < nw ? min(a.n, beg + chunk) : 0;
  int* mine = count + min(warp, nw - 1) * a.strata;
  // the labels of eight 32-row steps are loaded ahead of their step
  auto walk = [&](auto&& use) {
    for (int b0 = beg; b0 < end; b0 += 8 * 32) {
      int lv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = b0 + 32 * u + lane;
        lv[u] = r < end ? a.atlas[r] - 1 : -1;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (b0 + 32 * u < end) use(b0 + 32 * u + lane, lv[u]);
    }
  };
  walk([&](int r, int l) {
    if (r >= end) return;
    if (l < 0 || l >= a.strata) bad = 1;
    else atomicAdd(&mine[l], 1);
  });
  __syncthreads();
  if (bad) {
    if (tid == 0) atomicExch(a.status, 1);
    return;
  }
  // per stratum the warps' starts within it, then the strata's offsets: a run of
  // consecutive strata per thread
  const int per = (a.strata + static_cast<int>(blockDim.x) - 1) / static_cast<int>(blockDim.x);
  const int t0 = min(a.strata, tid * per), t1 = min(a.strata, t0 + per);
  int local = 0;
  for (int t = t0; t < t1; ++t)
    for (int w = 0; w < nw; ++w) local += count[w * a.strata + t];
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int run = incl - local;
  for (int w = 0; w < warp; ++w) run += wsum[w];
  for (int t = t0; t < t1; ++t) {
    s.offsets[t] = run;
    for (int w = 0; w < nw; ++w) {
      const int c = count[w * a.strata + t];
      count[w * a.strata + t] = run;
      run += c;
    }
  }
  if (tid == 0) s.offsets[a.strata] = a.n;
  __syncthreads();
  const int bits = 32 - __clz(a.strata);
  walk([&](int r, int l) {
    const bool in = r < end;
    const unsigned m = same_code(in ? l : 0, __ballot_sync(0xffffffffu, in), bits);
    const int at = in ? mine[l] : 0;
    const unsigned before = m & ((1u << lane) - 1u);
    if (in) s.rows[at + __popc(before)] = r;
    __syncwarp();
    if (in && before == 0u) mine[l] = at + __popc(m);
    __syncwarp();
  });
  // quota parts (run-independent)
  const Ext80 total = ext80_from_u64(static_cast<uint64_t>(a.n));
  unsigned long long bases = 0;
  for (int t = tid; t < a.strata; t += blockDim.x) {
    const int c = s.offsets[t + 1] - s.offsets[t];
    int base = 0;
    Ext80 frac{0, 0};
    if (c > 0) {
      const Ext80 expected =
          ext80_div(ext80_from_u64(static_cast<uint64_t>(a.target) * static_cast<uint64_t>(c)), total);
      base = min(c, ext80_floor_int(expected));
      frac = ext80_sub(expected, ext80_from_u64(static_cast<uint64_t>(base)));
    }
    s.base[t] = base;
    s.frac[t] = frac;
    bases += static_cast<unsigned long long>(base);
  }
  atomicAdd(&asum, bases);
  __syncthreads();
  if (tid == 0) *s.assigned = static_cast<int>(asum);
}

// x / b and x % b: 32-bit division when both fit.
__device__ __forceinline__ void divmod_u64(uint64_t x, uint64_t b, uint64_t& q, uint64_t& r) {
  if (x <= 0xffffffffull) {
    const uint32_t x32 = static_cast<uint32_t>(x), b32 = static_cast<uint32_t>(b);
    const uint32_t q32 = x32 / b32;
    q = q32;
    r = x32 - q32 * b32;
  } else {
    q = x / b;
    r = x % b;
  }
}

// std::shuffle of a[0..n) (random-access, 64-bit engine): one swap with a
// {0,1} draw first when n is even, then pairs from one draw each.
__device__ void shuffle_serial(int* a, int n, Mt64State& rng) {
  if (n <= 0) return;
  int i = 1;
  if ((n % 2) == 0) {
    const int j = static_cast<int>(draw_below_serial(rng, 2));
    const int t = a[i];
    a[i] = a[j];
    a[j] = t;
    ++i;
  }
  while (i != n) {
    const uint64_t r = static_cast<uint64_t>(i) + 1;
    uint64_t p1, p2;
    divmod_u64(draw_below_serial(rng, r * (r + 1)), r + 1, p1, p2);
    int t = a[i];
    a[i] = a[p1];
    a[p1] = t;
    ++i;
    t = a[i];
    a[i] = a[p2];
    a[p2] = t;
    ++i;
  }
}

// Lemire draw in [0, range) by a whole warp in lockstep (every lane computes
// the same value; the warp regenerates the state block when it runs out).
__device__ uint64_t draw_below_warp(Mt64State& rng, uint64_t range, int lane) {
  for (;;) {
    if (rng.pos >= kMtN) mt64_refill_warp(rng, lane);
    const uint64_t u = rng.out[rng.pos];
    __syncwarp();
    if (lane == 0) rng.pos += 1;
    __syncwarp();
    const uint64_t lo = u * range;
    if (lo >= range || lo >= (0ull - range) % range) return __umul64hi(u, range);
  }
}

// std::sample in strata (forward population), by one warp: selection sampling with
// two acceptance positions per draw while two or more rows remain.  A step's
// range depends only on how many rows remain, so the lanes draw the positions of
// up to 32 steps at once (one engine output per step) and the acceptance
// recursion -- a compare and a decrement per row -- runs over them in every lane
// alike; a taken row's flag is set a batch later, when its number has come from
// memory.  A draw that Lemire's method would reject (probability about
// range / 2^64) ends the batch and is drawn one output at a time, as are the
// single draws once fewer than two rows remain.
// What bounds it is the recursion, some 20 cycles a step.  By the whole CTA, with
// six barriers and a trip to memory per batch, 100 strata of 10 rows took 430k
// cycles and 300 of 333 rows 3.8 M.
struct Sampler {
  Mt64State& rng;
  const int* rows;
  uint8_t* flags;
  int lane;
  int wait_a = -1, wait_b = -1;  // rows of the batch before whose flags are to be set

  __device__ void settle() {
    if (wait_a >= 0) flags[wait_a] = 1;
    if (wait_b >= 0) flags[wait_b] = 1;
    wait_a = wait_b = -1;
  }

  // min(q, size) of the size rows at position first of the strata's row list
  __device__ int take(int first, int size, int q) {
    int uns = size, nq = min(q, size), at = first;
    const int wanted = nq;
    while (nq != 0 && uns >= 2) {
      if (rng.pos >= kMtN) mt64_refill_warp(rng, lane);
      const int pos = rng.pos, batch = min(32, min(kMtN - pos, uns >> 1));
      const bool in = lane < batch;
      const int ra = in ? rows[at + 2 * lane] : -1, rb = in ? rows[at + 2 * lane + 1] : -1;
      settle();
      const uint64_t left = static_cast<uint64_t>(in ? uns - 2 * lane : 2), b1 = left - 1, range = left * b1;
      const uint64_t u = in ? rng.out[pos + lane] : 0;
      const uint64_t lo = u * range;
      const unsigned bad = __ballot_sync(0xffffffffu, in && lo < range && lo < (0ull - range) % range);
      const int usable = bad != 0u ? __ffs(bad) - 1 : batch;
      // floor(u left b1 / 2^64) by b1: the quotient is floor(u left / 2^64)
      uint64_t d1 = __umul64hi(u, left), d2 = __umul64hi(u, range) - d1 * b1;
      // positions of steps past the usable ones take nothing
      const unsigned p1 = lane < usable ? static_cast<unsigned>(d1) : 0xffffffffu;
      const unsigned p2 = lane < usable ? static_cast<unsigned>(d2) : 0xffffffffu;
      // once nn is 0 every later compare fails, so the last row taken ends it
      unsigned nn = static_cast<unsigned>(nq), m1 = 0, m2 = 0;
      for (int j = 0; j < usable && nn != 0u; j += 8) {
        unsigned a1[8], a2[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          a1[e] = __shfl_sync(0xffffffffu, p1, j + e);
          a2[e] = __shfl_sync(0xffffffffu, p2, j + e);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const unsigned t1 = a1[e] < nn ? 1u : 0u;
          nn -= t1;
          const unsigned t2 = a2[e] < nn ? 1u : 0u;
          nn -= t2;
          m1 |= t1 << (j + e);
          m2 |= t2 << (j + e);
        }
      }
      int steps = usable, visited = 2 * usable;
      if (nn == 0u) {
        const int last = 31 - __clz(m1 | m2);
        steps = last + 1;
        visited = 2 * last + 1 + static_cast<int>((m2 >> last) & 1u);
      }
      __syncwarp();
      if (lane == 0) rng.pos = pos + steps;
      __syncwarp();
      wait_a = (m1 >> lane) & 1u ? ra : -1;
      wait_b = (m2 >> lane) & 1u ? rb : -1;
      uns -= visited;
      at += visited;
      nq = static_cast<int>(nn);
      if (nq != 0 && usable < batch) {
        // the rejected step, drawn one output at a time
        const uint64_t c1 = static_cast<uint64_t>(uns) - 1;
        divmod_u64(draw_below_warp(rng, static_cast<uint64_t>(uns) * c1, lane), c1, d1, d2);
        for (const uint64_t d : {d1, d2}) {
          if (nq == 0) break;
          if (d < static_cast<uint64_t>(nq)) {
            if (lane == 0) flags[rows[at]] = 1;
            --nq;
          }
          --uns;
          ++at;
        }
      }
    }
    for (; nq != 0; ++at) {
      --uns;
      if (draw_below_warp(rng, static_cast<uint64_t>(uns) + 1, lane) < static_cast<uint64_t>(nq)) {
        if (lane == 0) flags[rows[at]] = 1;
        --nq;
      }
    }
    return wanted;
  }
};

// std::mt19937 (Matsumoto & Nishimura 1998: n=624, m=397) by the whole CTA:
// seeding is a chain, a block of outputs is formed in three parts, each from words
// that are ready.
constexpr int kMt32N = 624, kMt32M = 397;

__device__ void mt32_seed(uint32_t* mt, uint32_t seed) {
  uint32_t p = seed;
  mt[0] = p;
  for (int i = 1; i < kMt32N; ++i) {
    p = 1812433253u * (p ^ (p >> 30)) + static_cast<uint32_t>(i);
    mt[i] = p;
  }
}

__device__ void mt32_block(uint32_t* mt, int tid) {
  for (int part = 0; part < kMt32N; part += kMt32N - kMt32M) {
    const int i = part + tid;
    const bool in = tid < kMt32N - kMt32M && i < kMt32N;
    uint32_t v = 0;
    if (in) {
      const uint32_t y = (mt[i] & 0x80000000u) | (mt[i + 1 < kMt32N ? i + 1 : 0] & 0x7fffffffu);
      v = mt[i + kMt32M < kMt32N ? i + kMt32M : i + kMt32M - kMt32N] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
    }
    __syncthreads();
    if (in) mt[i] = v;
    __syncthreads();
  }
}

__device__ __forceinline__ uint32_t mt32_temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}

// Bytes of shared memory for the strata's order, quotas and fractions.
size_t plan_smem_bytes(int strata) {
  return strata <= kSharedStrata ? static_cast<size_t>(strata) * (sizeof(Ext80) + 2 * sizeof(int)) : 0;
}

// The chains of dependent steps (the shuffle's swaps, the residual allocation,
// each stratum's sample) run on one thread or warp, so what they read is brought
// into shared memory first: from global memory each step waited for L2.
__global__ void __launch_bounds__(kPlanThreads) plan_runs_kernel(PlanArgs a, PlanScratch s) {
  extern __shared__ __align__(16) unsigned char plan_smem[];
  __shared__ Mt64State rng;
  __shared__ uint32_t mt32[kMt32N];
  __shared__ uint32_t swap_to[kMt32N];
  __shared__ int sh_bad, sh_strata;
  __shared__ uint32_t sh_kseed;
  __shared__ int sh_warp[kPlanThreads / 32];
  const int run = blockIdx.x, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  uint8_t* flags = s.flags + static_cast<size_t>(run) * a.n;
  const bool shared_strata = a.strata <= kSharedStrata;
  Ext80* sh_frac = reinterpret_cast<Ext80*>(plan_smem);  // by position in the shuffled order
  int* quota = shared_strata ? reinterpret_cast<int*>(sh_frac + a.strata) : s.quota + static_cast<size_t>(run) * a.strata;
  int* order = shared_strata ? quota + a.strata : s.order + static_cast<size_t>(run) * a.strata;
  for (int r = tid; r < a.n; r += kPlanThreads) flags[r] = 0;
  for (int t = tid; t < a.strata; t += kPlanThreads) quota[t] = s.base[t];
  if (tid == 0) mt64_seed(rng, a.seed + static_cast<uint64_t>(a.first_run + run));
  if (warp == 1) {
    // the non-empty strata in order
    int S = 0;
    for (int b = 0; b < a.strata; b += 32) {
      const int t = b + lane;
      const bool in = t < a.strata && s.offsets[t + 1] > s.offsets[t];
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) order[S + __popc(m & ((1u << lane) - 1u))] = t;
      S += __popc(m);
    }
    if (lane == 0) sh_strata = S;
  }
  __syncthreads();
  if (warp == 0) mt64_refill_warp(rng, lane);
  __syncthreads();
  const int S = sh_strata;
  if (tid == 0) {
    (void)mt64_next_serial(rng);
    shuffle_serial(order, S, rng);
    sh_bad = 0;
  }
  __syncthreads();
  if (shared_strata)
    for (int i = tid; i < S; i += kPlanThreads) sh_frac[i] = s.frac[order[i]];
  __syncthreads();
  if (tid == 0) {
    const int residual = a.target - *s.assigned;
    if (residual > 0) {
      auto frac = [&](int i) { return shared_strata ? sh_frac[i] : s.frac[order[i] & ~kRounded]; };
      const Ext80 offset = ext80_canonical(mt64_next_serial(rng));
      Ext80 cumulative{0, 0};
      int selected = 0;
      for (int i = 0; i < S; ++i) {
        cumulative = ext80_add(cumulative, frac(i));
        const Ext80 next = ext80_add(offset, ext80_from_u64(static_cast<uint64_t>(selected)));
        if (selected < residual && ext80_lt(next, cumulative)) {
          const int t = order[i];
          ++quota[t];
          order[i] = t | kRounded;
          ++selected;
        }
      }
      while (selected < residual) {
        int besti = -1;
        Ext80 bestv{0, 0};
        for (int i = 0; i < S; ++i) {
          if (order[i] & kRounded) continue;
          if (besti < 0 || ext80_lt(bestv, frac(i))) {
            bestv = frac(i);
            besti = i;
          }
        }
        if (besti < 0) {
          sh_bad = 4;
          break;
        }
        const int best = order[besti];
        ++quota[best];
        order[besti] = best | kRounded;
        ++selected;
      }
    }
  }
  __syncthreads();
  if (warp == 0 && sh_bad == 0) {
    Sampler sampler{rng, s.rows, flags, lane};
    int total = 0;
    for (int t0 = 0; t0 < a.strata; t0 += 32) {
      // 32 strata's ranges and quotas at a time
      const int t = min(t0 + lane, a.strata - 1);
      const int first = s.offsets[t], size = s.offsets[t + 1] - first, q = t0 + lane < a.strata ? quota[t] : 0;
      for (unsigned m = __ballot_sync(0xffffffffu, q > 0 && size > 0); m != 0u; m &= m - 1) {
        const int l = __ffs(m) - 1;
        total += sampler.take(__shfl_sync(0xffffffffu, first, l), __shfl_sync(0xffffffffu, size, l),
                              __shfl_sync(0xffffffffu, q, l));
      }
    }
    sampler.settle();
    if (lane == 0 && total != a.target) sh_bad = 3;
  }
  __syncthreads();
  if (tid == 0) sh_kseed = static_cast<uint32_t>((mt64_next_serial(rng) & 0x7fffffffull) + 1ull);
  __syncthreads();
  if (sh_bad) {
    if (tid == 0) atomicExch(a.status, sh_bad);
    return;
  }
  const int L = a.target;
  const int k = max(1, min(a.init_k, L));
  // ascending compaction of the selected rows (and of the others): a run of rows
  // per warp, eight 32-row steps' flags in flight; the last warp seeds the
  // permutation's engine beside it
  constexpr int kCompactWarps = kPlanThreads / 32 - 1;
  int* land = a.land + static_cast<size_t>(run) * a.target;
  int* nonland = a.nonland == nullptr ? nullptr : a.nonland + static_cast<size_t>(run) * (a.n - a.target);
  const int chunk = ((a.n + kCompactWarps - 1) / kCompactWarps + 31) / 32 * 32;
  const int beg = warp < kCompactWarps ? min(a.n, warp * chunk) : 0;
  const int end = warp < kCompactWarps ? min(a.n, beg + chunk) : 0;
  auto walk = [&](auto&& use) {
    for (int b0 = beg; b0 < end; b0 += 8 * 32) {
      unsigned f[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = b0 + 32 * u + lane;
        f[u] = r < end ? flags[r] : 0u;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) use(b0 + 32 * u + lane, f[u] != 0u);
    }
  };
  int taken = 0;
  walk([&](int, bool f) { taken += __popc(__ballot_sync(0xffffffffu, f)); });
  if (lane == 0) sh_warp[warp] = taken;
  if (tid == kPlanThreads - 32) mt32_seed(mt32, sh_kseed);
  __syncthreads();
  int pos0 = 0;
  for (int w = 0; w < warp; ++w) pos0 += sh_warp[w];
  walk([&](int r, bool f) {
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int pos = pos0 + __popc(m & ((1u << lane) - 1u));
    if (r < end) {
      if (f) land[pos] = r;
      else if (nonland != nullptr) nonland[r - pos] = r;
    }
    pos0 += __popc(m);
  });
  __syncthreads();
  // initial centroid rows: head of the permutation of 0..L-1.  Step i swaps
  // positions i and to(i) >= i.  Position x holds x until a step j with to(j) == x
  // moves there what was at j; so before its own step, position j holds the root
  // of the chain j -> last i < j with to(i) == j, and entry r of the head is the
  // root of the last j < r with to(j) == to(r), or to(r) itself.
  const int steps = min(k, L - 1);
  int* out = a.init_rows + static_cast<size_t>(run) * a.init_k;
  if (steps <= kMt32N) {
    mt32_block(mt32, tid);
    for (int i = tid; i < steps; i += kPlanThreads)
      swap_to[i] = static_cast<uint32_t>(i) + mt32_temper(mt32[i]) % static_cast<uint32_t>(L - i);
    __syncthreads();
    // the last step before `upto` that swaps with position x, or -1
    auto last_to = [&](int x, int upto) {
      int at = -1;
      for (int j = 0; j < upto; ++j) at = swap_to[j] == static_cast<uint32_t>(x) ? j : at;
      return at;
    };
    for (int j = tid; j < steps; j += kPlanThreads) mt32[j] = static_cast<uint32_t>(last_to(j, j));
    __syncthreads();
    for (int r = tid; r < k; r += kPlanThreads) {
      // past the last step (k = L) the entry is what its position holds
      const int x = r < steps ? static_cast<int>(swap_to[r]) : r;
      int j = last_to(x, min(r, steps));
      if (j >= 0)
        for (int up = static_cast<int>(mt32[j]); up >= 0; up = static_cast<int>(mt32[j])) j = up;
      out[r] = j >= 0 ? j : x;
    }
  } else {
    int* perm = s.perm + static_cast<size_t>(run) * L;
    for (int i = tid; i < L; i += kPlanThreads) perm[i] = i;
    for (int r0 = 0; r0 < steps; r0 += kMt32N) {
      mt32_block(mt32, tid);
      const int m = min(kMt32N, steps - r0);
      for (int i = tid; i < m; i += kPlanThreads)
        swap_to[i] = static_cast<uint32_t>(r0 + i) + mt32_temper(mt32[i]) % static_cast<uint32_t>(L - r0 - i);
      __syncthreads();
      if (tid == 0) {
        for (int i = 0; i < m; ++i) {
          const int r = r0 + i, other = static_cast<int>(swap_to[i]), t = perm[r];
          perm[r] = perm[other];
          perm[other] = t;
        }
      }
      __syncthreads();
    }
    for (int r = tid; r < k; r += kPlanThreads) out[r] = perm[r];
  }
}

// FNV-1a over each run's landmark rows (hash_integer_vector,
// kodama_matrix.cpp:1689-1699).
__global__ void land_hash_kernel(const int* __restrict__ land, int runs, int L, uint64_t* __restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= runs) return;
  const int* v = land + static_cast<size_t>(r) * L;
  uint64_t h = 1469598103934665603ull;
  for (int i = 0; i < L; ++i) {
    const uint32_t b = static_cast<uint32_t>(v[i]);
#pragma unroll
    for (int sft = 0; sft < 32; sft += 8) {
      h ^= static_cast<uint8_t>((b >> sft) & 0xffu);
      h *= 1099511628211ull;
    }
  }
  out[r] = h;
}

}  // namespace

size_t plan_scratch_bytes(int n, int strata, int target, int runs) {
  const size_t S = static_cast<size_t>(strata), R = static_cast<size_t>(runs);
  return align256(sizeof(int) * S) * 3 + align256(sizeof(int) * (S + 1)) + align256(sizeof(int) * n) +
         align256(sizeof(Ext80) * S) + align256(sizeof(int)) + align256(sizeof(int) * S * R) * 2 +
         align256(static_cast<size_t>(n) * R) + align256(sizeof(int) * static_cast<size_t>(target) * R);
}

int plan_landmarks(const PlanArgs& a, cudaStream_t st) {
  if (a.n < 1 || a.strata < 1 || a.target < 1 || a.target > a.n || a.runs < 1 || a.init_k < 1 ||
      a.init_k > a.target)
    return static_cast<int>(cudaErrorInvalidValue);
  const PlanScratch s = carve(a);
  const int fit = kCounterBytes / static_cast<int>(sizeof(int)) / a.strata;
  const int counter_bytes = fit >= 2 ? std::min(32, fit) * a.strata * static_cast<int>(sizeof(int)) : 0;
  cudaError_t e = allow_shared_memory(strata_kernel);
  if (e != cudaSuccess) return static_cast<int>(e);
  strata_kernel<<<1, 1024, counter_bytes, st>>>(a, s);
  count_launch();
  const size_t smem = plan_smem_bytes(a.strata);
  e = allow_shared_memory(plan_runs_kernel);
  if (e != cudaSuccess) return static_cast<int>(e);
  plan_runs_kernel<<<a.runs, kPlanThreads, smem, st>>>(a, s);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int plan_land_hash(const PlanArgs& a, cudaStream_t st) {
  land_hash_kernel<<<(a.runs + 127) / 128, 128, 0, st>>>(a.land, a.runs, a.target, a.land_hash);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

}  // namespace kgb
