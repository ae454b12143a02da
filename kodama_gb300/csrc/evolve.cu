// Persistent label-evolution kernel: every problem (KODAMA.matrix run, or
// CoreKNNGraph call) runs all of its Tcycle perturb / vote / score / accept
// steps inside one CTA, in one launch, with the labels resident in shared
// memory and the fold-filtered neighbour table streamed from HBM/L2.
//
// It restates maximize_core (core.cpp:1269-1549) with the precomputed-kNN
// predictor predict_precomputed_knn (core.cpp:784-914) and the training-fold
// fallbacks (core.cpp:274-309):
//   proposal size   sample_proposal_group_count  core.cpp:1228-1254
//   group shuffle   std::shuffle of the group ids core.cpp:1363-1365
//   relabel         prediction-guided draw        core.cpp:1384-1419
//   absorption      propose_many_to_one_absorption core.cpp:1110-1226
//   score           core_objective_score          core.cpp:916-972
//   accept          greedy / annealed              core.cpp:1471-1508
// Labels are carried as 16-bit codes: the rank of the label among the sorted
// distinct initial labels, so every label comparison of the reference (ties to
// the smaller label, ordered maps) is a code comparison.
//
// Exactness: all double arithmetic uses explicit round-to-nearest intrinsics
// (no contraction), random draws follow rng.cuh, and the unordered_map
// iteration order that fixes the summation order of the diversity term is
// reproduced (reverse first-insertion order, bucket runs on collisions).
//
// What bounds it: a cycle is a chain of short phases in one CTA, 40k to 100k
// cycles long, about half of them issuing (208k warp instructions a cycle at 10000
// rows and 30 neighbours), the rest barriers and latency.  So per-row passes take
// eight rows a thread, one thread's work is kept to what is serial, and double
// arithmetic, 64 cycles a dependent operation and 512 for all 1024 threads, is
// left to single warps.
#include "evolve.cuh"
#include "launch_count.cuh"
#include "smem_limit.cuh"
#include "rng.cuh"
#include "crmath.cuh"
#include "mlp.cuh"
#include "warp_match.cuh"

#include <cuda_runtime.h>
#include <float.h>
#include <math.h>

namespace kgb {

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kRowArrays = 8;  // cl, cur, curpred, pred/perm, J, list, 2 x (32-bit scratch)

// The run's scores and counters, kept by thread 0.
struct RunState {
  double accbest, scorebest, cur_acc, cur_score;
  int nc_cur, nc_best;
  int best_updates, accepts, st_att, st_acc, rejections, absorb_moves, tr_acc, success;
};

struct Fixed {
  RunState run;
  Mt64State rng;
  union {
    uint64_t mt_alt[kMtN];  // the engine state's second buffer (produce_outputs_group)
    int sel_hist[256];      // digit counts of learned_flip; labels of vote_empty_rows
  };
  int rejected;
  int i0;
  int ns;
  int red_i[kWarps];
  int flag;
  int nc;          // distinct labels of the proposal
  int changed_cnt;  // dirty_rows_block: rows whose label changed
  int dirty_cnt;    // dirty_rows_block: rows listed for the vote
  int walk_cnt;    // groups whose final position is walked
  int empty_cnt;   // rows without out-of-fold neighbours
  unsigned empty_folds[8];  // the folds they are in
  int selected_target;
  int rev_total;   // this problem's reverse-neighbour entries (rev_off[L])
  double acc;
  double score;
  double cooling[2];  // annealing factors of this and the next acceptance test, by cycle parity
  int max_groups;  // largest size of the coming proposal
  int accept;
  // this problem's groups and fixed flags (bind_groups)
  const int* goff;
  const int* gmem;
  const int* fxd;
  int G;
  // learned proposal: candidate count and radix-select state
  int sel_count;
  int sel_digit;
  int sel_need;
};
// The room the struct is given, part of how many labels fit (evolve_place).
constexpr size_t kFixedBytes = 8768;
static_assert(sizeof(Fixed) <= kFixedBytes, "evolve_place's limit");

struct Smem {
  Fixed* f;
  uint16_t* cl;      // proposal
  uint16_t* cur;     // current state (evolutionary) or best state (greedy)
  uint16_t* curpred; // CV predictions of cur
  uint16_t* pred;    // CV predictions of the proposal
  uint16_t* perm;    // shuffled group ids (first ns positions; aliases pred during the shuffle)
  uint16_t* jarr;    // swap target of every shuffle step
  uint16_t* list;    // shuffle steps bucketed by swap target
  int* scratch32;    // per-position counts / bucket offsets
  int* hist;         // per warp: one counter per code, all zero between uses
  int hist_stride;   // counters per warp
  int hist_warps;    // warps that have counters
  uint64_t* save;    // the engine's state before a shuffle (global scratch)
  int* cnt;          // per code: count in proposal
  int* firstpos;     // per code: first row
  int* movable;      // per code: non-fixed rows
  int* order;        // per code: unordered_map iteration order / scratch
  int* bt;           // per code: absorption target (-1 none)
  int* aux;          // per code: scratch counts
  double* bsur;      // per code: absorption surplus
  double* weight;    // per code: per-target weight / discrete weights
  double* cp;        // discrete cumulative scratch
};

__device__ __forceinline__ size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Where the per-row arrays lie is a property of the kernel, and the struct is only
// ever inlined, so that the accesses are known to be to shared memory.
template <bool kRows>
__device__ __forceinline__ Smem carve_smem(const EvolveParams& P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem s;
  size_t off = 0;
  s.f = reinterpret_cast<Fixed*>(smem_raw);
  off = kFixedBytes;
  const int C = P.C0max;
  s.cnt = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * C, 16);
  s.firstpos = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * C, 16);
  s.movable = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * C, 16);
  s.order = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * (C + 1), 16);
  s.bt = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * C, 16);
  s.aux = reinterpret_cast<int*>(smem_raw + off); off += align_up(sizeof(int) * C, 16);
  s.bsur = reinterpret_cast<double*>(smem_raw + off); off += align_up(sizeof(double) * C, 16);
  s.weight = reinterpret_cast<double*>(smem_raw + off); off += align_up(sizeof(double) * C, 16);
  s.cp = reinterpret_cast<double*>(smem_raw + off); off += align_up(sizeof(double) * 2 * C, 16);
  const size_t Lp = align_up(static_cast<size_t>(P.L), 8);
  s.save = P.engine_save + static_cast<size_t>(blockIdx.x) * kEvolveEngineSave;
  s.hist_stride = static_cast<int>(align_up(C, 4));
  s.hist_warps = P.hist_warps;
  s.hist = reinterpret_cast<int*>(smem_raw + off);
  off += sizeof(int) * static_cast<size_t>(s.hist_stride) * s.hist_warps;
  uint16_t* rows = kRows ? reinterpret_cast<uint16_t*>(smem_raw + off)
                         : P.rows_scratch + static_cast<size_t>(blockIdx.x) * kRowArrays * Lp;
  s.cl = rows;
  s.cur = rows + Lp;
  s.curpred = rows + 2 * Lp;
  s.pred = rows + 3 * Lp;
  s.perm = s.pred;
  s.jarr = rows + 4 * Lp;
  s.list = rows + 5 * Lp;
  s.scratch32 = reinterpret_cast<int*>(rows + 6 * Lp);  // 2 * Lp u16 = Lp ints
  return s;
}

// The same layout for the functions kept out of line, where the two are looked up
// instead.
__device__ Smem carve_smem_any(const EvolveParams& P) {
  return P.smem_rows ? carve_smem<true>(P) : carve_smem<false>(P);
}

__device__ __forceinline__ int block_sum(int v, Fixed& f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = __reduce_add_sync(kFull, v);
  if (lane == 0) f.red_i[warp] = v;
  __syncthreads();
  const int out = __reduce_add_sync(kFull, f.red_i[lane]);
  __syncthreads();
  return out;
}

// The per-row arrays start on 16-byte boundaries and are padded to whole
// 8-row vectors; row_code unpacks row e of a vector.
__device__ __forceinline__ int row_vectors(int L) { return (L + 7) >> 3; }
__device__ __forceinline__ int row_code(const uint4& v, int e) {
  const unsigned w = e < 2 ? v.x : e < 4 ? v.y : e < 6 ? v.z : v.w;
  return static_cast<int>((w >> (16 * (e & 1))) & 0xffffu);
}
__device__ __forceinline__ uint4 load_rows(const uint16_t* a, int i) { return reinterpret_cast<const uint4*>(a)[i]; }
__device__ __forceinline__ void copy_rows(uint16_t* dst, const uint16_t* src, int L) {
  for (int i = threadIdx.x; i < row_vectors(L); i += kThreads) reinterpret_cast<uint4*>(dst)[i] = load_rows(src, i);
}

// acc plus n doubles from shared memory in order.  The FP64 pipe takes 64 cycles
// for a dependent sum, so the values are read eight ahead of the chain.
__device__ __forceinline__ double chain_add(double acc, const double* v, int n) {
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    double t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = v[i + q];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc = __dadd_rn(acc, t[q]);
  }
  for (; i < n; ++i) acc = __dadd_rn(acc, v[i]);
  return acc;
}

// std::discrete_distribution (discrete_serial) by one warp: the divisions run a
// lane each, the two running sums stay in order.  w is overwritten.
__device__ __forceinline__ int discrete_warp(Mt64State& g, double* w, int n, double* cp, int lane) {
  if (n < 2) return 0;
  const double sum = chain_add(0.0, w, n);
  __syncwarp();
  for (int i = lane; i < n; i += 32) w[i] = __ddiv_rn(w[i], sum);
  __syncwarp();
  int at = 0;
  if (lane == 0) {
    double acc = 0.0;
    for (int q0 = 0; q0 < n; q0 += 8) {
      double t[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) t[q] = q0 + q < n ? w[q0 + q] : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q0 + q >= n) break;
        acc = q0 + q == 0 ? t[q] : __dadd_rn(acc, t[q]);
        cp[q0 + q] = acc;
      }
    }
    cp[n - 1] = 1.0;
    at = discrete_probe(cp, n, canonical_serial(g));
  }
  return __shfl_sync(kFull, at, 0);
}

// ---------------------------------------------------------------------------
// Group shuffle (std::shuffle of iota(G) with a 64-bit engine).  For an engine
// range wider than G^2 the draws come two at a time: one downscaled draw over
// (i+1)*(i+2) gives the swap targets of positions i and i+1 (quotient and
// remainder by i+2); an even G first swaps position 1 with a draw over {0,1}.
//
// Only the groups at positions [0, ns) are used, so the permutation is not
// materialised serially.  Step i (swap of positions i and J[i] <= i) moves
// group i, which is still at position i, to J[i].  Hence the final occupant of
// position q is the last step i > q with J[i] == q if there is one; otherwise
// it is whatever step q pulled into position q, i.e. the occupant of position
// J[q] just before step q (q itself when J[q] == q; 0 for position 0).  The
// CTA computes all J[i] in parallel from the engine blocks, buckets the steps
// by target, and walks each wanted position down this chain.
// ---------------------------------------------------------------------------
// Exclusive prefix sum of a[0..n) in place (block-wide); returns the total.
__device__ __forceinline__ int block_exclusive_scan(int* a, int n, Fixed& f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunk = (n + kThreads - 1) / kThreads;
  const int b = threadIdx.x * chunk, e = min(n, b + chunk);
  int local = 0;
  for (int i = b; i < e; ++i) local += a[i];
  int incl = local;
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(kFull, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) f.red_i[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = f.red_i[lane];
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(kFull, w, off);
      if (lane >= off) w += v;
    }
    f.red_i[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  int run = (warp > 0 ? f.red_i[warp - 1] : 0) + incl - local;
  for (int i = b; i < e; ++i) {
    const int v = a[i];
    a[i] = run;
    run += v;
  }
  const int total = f.red_i[kWarps - 1];
  __syncthreads();
  return total;
}

// Engine producer group: the first 160 threads (warps 0-4) synchronised by
// named barrier 1.
constexpr int kProducerThreads = 160;
__device__ __forceinline__ void producer_sync() { asm volatile("bar.sync 1, 160;" ::: "memory"); }
__device__ __forceinline__ void shuffle_step_sync() { asm volatile("bar.sync 2, 1024;" ::: "memory"); }

// Advances the CTA's engine by the next `count` outputs (producer group), with a
// shuffle_step_sync after every regeneration (one in all if the outputs left
// suffice).  The state and its position go to `save` first.
// Thread t < 156 keeps words t and t + 156 of the state in registers: the new word
// t takes old words t, t + 1 and t + 156, the new word t + 156 old words t + 156,
// t + 157 and the new word t; word 311 takes the new word 0, which thread 156
// forms for its neighbour.  Regeneration r goes to f.mt_alt for even r, f.rng.mt
// for odd r, where the other warps read its words, still to be tempered, until
// the next step; the last block's outputs and the state go to f.rng once at the
// end, after the last step's barrier: until then the other warps read the old
// position and, for an odd number of regenerations, the block before in f.rng.mt.
// The caller's block barrier publishes them.
// Tempering every block here and writing it to global memory, the state's words
// reloaded, took 860 cycles a regeneration; this takes 270, as a function of its
// own with its own registers (640 within the kernel's).
__device__ __noinline__ void produce_outputs_group(int count, uint64_t* save) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Fixed& f = *reinterpret_cast<Fixed*>(smem_raw);
  Mt64State& g = f.rng;
  const int t = threadIdx.x, h = t + kMtM;
  const int pos0 = g.pos;
  const int lead = min(kMtN - pos0, count);
  const bool live = t < kMtM, spare = t == kMtM;
  const int i0 = live ? t : 0;
  uint64_t a = g.mt[i0], b = g.mt[i0 + kMtM];
  if (live) {
    save[t] = a;
    save[h] = b;
  }
  if (t == 0) save[kMtN] = static_cast<uint64_t>(pos0);
  int done = lead, pos = pos0 + lead;
  uint64_t* cur = g.mt;
  uint64_t* nxt = f.mt_alt;
  while (done < count) {
    const uint64_t an = cur[i0 + 1];
    uint64_t bn = cur[min(i0 + kMtM + 1, kMtN - 1)];
    const uint64_t lo = mt64_mix(a, an, b);
    const uint64_t first = __shfl_down_sync(kFull, lo, 1);  // thread 156's word 0, for thread 155
    if (t == kMtM - 1) bn = first;
    const uint64_t hi = mt64_mix(b, bn, lo);
    if (live) {
      nxt[t] = lo;
      nxt[h] = hi;
    }
    a = lo;
    b = hi;
    pos = min(kMtN, count - done);
    done += pos;
    // the next regeneration reads what this one wrote and overwrites what it
    // read, and what the other warps read of the one before
    producer_sync();
    if (spare) b = nxt[kMtM];  // thread 156 stands in for word 0 only
    uint64_t* const tmp = cur;
    cur = nxt;
    nxt = tmp;
    if (done < count) shuffle_step_sync();
  }
  // the other warps' last reads of the state and its position lie before this
  // barrier; of the last regeneration they read what is in `cur`
  shuffle_step_sync();
  if (live && done > lead) {
    if (cur != g.mt) {
      g.mt[t] = a;
      g.mt[h] = b;
    }
    g.out[t] = mt64_temper(a);
    g.out[h] = mt64_temper(b);
  }
  if (t == 0) g.pos = pos;
}

// Swap targets J[i] of every step of the shuffle of G groups.  The producer
// group runs the engine on by the outputs of the pair draws; the other warps
// downscale each regeneration while the next is formed.  One after the other,
// through global memory, the two took 16.2k cycles for 10000 groups.  A rejected
// draw (Lemire resampling, about one in 2^64/G^2) shifts every later pair by one
// output: the shuffle is then drawn again from the saved state, in order.
__device__ __forceinline__ void shuffle_targets_block(Fixed& f, uint16_t* J, int G, uint64_t* save) {
  if (threadIdx.x == 0) {
    f.i0 = 1;
    if (G >= 2 && (G & 1) == 0) {
      J[1] = static_cast<uint16_t>(draw_below_serial(f.rng, 2));
      f.i0 = 2;
    }
    f.rejected = 0;
  }
  __syncthreads();
  const int i0 = f.i0;
  const int npairs = (G - i0) >> 1;
  if (npairs <= 0) return;
  if (threadIdx.x < kProducerThreads) {
    produce_outputs_group(npairs, save);
  } else {
    const int t = threadIdx.x - kProducerThreads, pos0 = f.rng.pos, lead = min(kMtN - pos0, npairs);
    // x = floor(u b0 b1 / 2^64) is below (G-1)*G < 2^32 for G <= 65535, and its
    // quotient by b1 is floor(u b0 / 2^64)
    auto place = [&](int p, uint64_t word) {
      const uint32_t b0 = static_cast<uint32_t>(i0 + 2 * p) + 1u, b1 = b0 + 1u;
      const uint64_t range = static_cast<uint64_t>(b0) * b1;
      const uint64_t u = mt64_temper(word);
      const uint64_t lo = u * range;
      if (lo < range && lo < (0ull - range) % range) f.rejected = 1;
      const uint32_t x = static_cast<uint32_t>(__umul64hi(u, range));
      const uint32_t qv = static_cast<uint32_t>(__umul64hi(u, b0));
      J[i0 + 2 * p] = static_cast<uint16_t>(qv);
      J[i0 + 2 * p + 1] = static_cast<uint16_t>(x - qv * b1);
    };
    // what is left of the old block, while the first regeneration is formed
    if (t < lead) place(t, f.rng.mt[pos0 + t]);
    const uint64_t* words = f.mt_alt;
    const uint64_t* next = f.rng.mt;
    for (int from = lead; from < npairs; from += kMtN) {
      shuffle_step_sync();
      if (t < kMtN && from + t < npairs) place(from + t, words[t]);
      const uint64_t* const tmp = words;
      words = next;
      next = tmp;
    }
    if (lead == npairs) shuffle_step_sync();
  }
  __syncthreads();
  if (f.rejected == 0) return;
  __syncthreads();
  for (int k = threadIdx.x; k < kMtN; k += kThreads) {
    f.rng.mt[k] = save[k];
    f.rng.out[k] = mt64_temper(save[k]);
  }
  if (threadIdx.x == 0) f.rng.pos = static_cast<int>(save[kMtN]);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = i0; i < G; i += 2) {
      const uint64_t b1 = static_cast<uint64_t>(i) + 2ull;
      const uint64_t x = draw_below_serial(f.rng, (b1 - 1ull) * b1);
      J[i] = static_cast<uint16_t>(x / b1);
      J[i + 1] = static_cast<uint16_t>(x % b1);
    }
  }
  __syncthreads();
}

// Bucket the steps by swap target, for the targets below lim (the used
// positions [0, ns)): afterwards cnt[q] is the end of bucket q in `list` and
// the start of bucket q+1.  A group only moves to higher positions (a later
// step targeting its position p sits at a position above p), so walks that
// decide membership of [0, lim) never need a bucket at or above lim.
__device__ __forceinline__ void bucket_steps_block(const Smem& s, int G, int lim) {
  const uint16_t* J = s.jarr;
  int* cnt = s.scratch32;
  uint16_t* list = s.list;
  for (int q = threadIdx.x; q < lim; q += kThreads) cnt[q] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < row_vectors(G); i += kThreads) {
    const uint4 v = load_rows(J, i);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int st = 8 * i + e, j = row_code(v, e);
      if (st >= 1 && st < G && j < lim) atomicAdd(&cnt[j], 1);
    }
  }
  __syncthreads();
  block_exclusive_scan(cnt, lim, *s.f);
  for (int i = threadIdx.x; i < row_vectors(G); i += kThreads) {
    const uint4 v = load_rows(J, i);
    int slot[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int st = 8 * i + e, j = row_code(v, e);
      slot[e] = st >= 1 && st < G && j < lim ? atomicAdd(&cnt[j], 1) : -1;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (slot[e] >= 0) list[slot[e]] = static_cast<uint16_t>(8 * i + e);
  }
  __syncthreads();
}

// Group at final position p: last step > q targeting q, else what step q
// pulled into q (see above).
__device__ __forceinline__ int occupant_of(const Smem& s, int G, int p) {
  const uint16_t* J = s.jarr;
  const int* cnt = s.scratch32;
  int q = p, t = G - 1;
  for (;;) {
    const int b = q > 0 ? cnt[q - 1] : 0, e = cnt[q];
    int best = -1;
    for (int k = b; k < e; ++k) {
      const int st = s.list[k];
      if (st > q && st <= t && st > best) best = st;
    }
    if (best >= 0) return best;
    if (q == 0) return 0;
    const int jq = J[q];
    if (jq == q) return q;
    t = q - 1;
    q = jq;
  }
}

// Final position of group e: it lands on J[e] at step e (group 0 starts at
// 0), then every later step targeting its position moves it to that step's
// own position.  Positions only grow, so once the position reaches lim (the
// buckets' limit) the walk stops and returns that position, which is enough
// for a `< lim` test.
__device__ __forceinline__ int final_position_of(const Smem& s, int e, int lim) {
  const int* cnt = s.scratch32;
  int pos = e == 0 ? 0 : s.jarr[e];
  int time = e;
  for (;;) {
    if (pos >= lim) return pos;
    const int b = pos > 0 ? cnt[pos - 1] : 0, en = cnt[pos];
    int next = 0x7fffffff;
    for (int k = b; k < en; ++k) {
      const int st = s.list[k];
      if (st > time && st < next) next = st;
    }
    if (next == 0x7fffffff) return pos;
    pos = next;
    time = next;
  }
}

// ---------------------------------------------------------------------------
// Tie-break of a vote among the labels reaching the top count `maxc`
// (`tied`: one lane per such label).  The larger double score sum wins, then
// the smaller code.  With |s| = mant * 2^ex, if the non-zero magnitudes of the
// row span at most 24 binades every sequential double partial sum of <= 32 of
// them is exact, so when all scores share a sign (-(d*d) <= 0 for squared L2,
// inner products >= 0 among near neighbours) exact integer sums of the
// magnitudes order the tied labels exactly as the reference's double sums do
// (smaller magnitude first for non-positive scores, larger for non-negative);
// otherwise the double sums are formed in neighbour order.
// ---------------------------------------------------------------------------
__device__ __noinline__ int vote_tiebreak(int code, unsigned tied, const float* scrow, int w, int lane) {
  const float my = lane < w ? scrow[lane] : 0.0f;
  const uint32_t bits = __float_as_uint(my);
  const uint32_t ef = (bits >> 23) & 0xffu;
  const uint32_t mant = ef ? ((bits & 0x7fffffu) | 0x800000u) : (bits & 0x7fffffu);
  const int ex = ef ? static_cast<int>(ef) - 150 : -149;
  const bool live = code >= 0 && mant != 0u;
  const bool bad = code >= 0 && ef == 0xffu;
  const int emin = __reduce_min_sync(kFull, live ? ex : 0x7fffffff);
  const int emax = __reduce_max_sync(kFull, live ? ex : -0x7fffffff);
  const bool any_neg = __any_sync(kFull, live && (bits >> 31) != 0u);
  const bool any_pos = __any_sync(kFull, live && (bits >> 31) == 0u);
  const bool exact_ok = !__any_sync(kFull, bad) && !(any_neg && any_pos) &&
                        (emin == 0x7fffffff || emax - emin <= 24);
  uint32_t p0 = 0, p1 = 0, p2 = 0;
  if (exact_ok && live) {
    const uint64_t contrib = static_cast<uint64_t>(mant) << (ex - emin);
    p0 = static_cast<uint32_t>(contrib & 0x1fffffu);
    p1 = static_cast<uint32_t>((contrib >> 21) & 0x1fffffu);
    p2 = static_cast<uint32_t>(contrib >> 42);
  }
  uint64_t bmag = any_pos ? 0ull : ~0ull;
  double bsum = -INFINITY;
  int bc = 0x7fffffff;
  unsigned rem = tied;
  while (rem) {
    const int ld = __ffs(rem) - 1;
    rem &= rem - 1;
    const int v = __shfl_sync(kFull, code, ld);
    const bool in = code == v;
    if (exact_ok) {
      const uint64_t s0 = __reduce_add_sync(kFull, in ? p0 : 0u);
      const uint64_t s1 = __reduce_add_sync(kFull, in ? p1 : 0u);
      const uint64_t s2 = __reduce_add_sync(kFull, in ? p2 : 0u);
      const uint64_t mag = s0 + (s1 << 21) + (s2 << 42);
      if ((any_pos ? mag > bmag : mag < bmag) || (mag == bmag && v < bc)) {
        bmag = mag;
        bc = v;
      }
    } else {
      const unsigned msk = __ballot_sync(kFull, in);
      double sum = 0.0;
      for (int t = 0; t < w; ++t) {
        const float st = __shfl_sync(kFull, my, t);
        if ((msk >> t) & 1u) sum = __dadd_rn(sum, static_cast<double>(st));
      }
      // (the first label stands until a larger sum: a sum that is not a number never is
      // one, and the result is a label of the row all the same)
      if (bc == 0x7fffffff || sum > bsum || (sum == bsum && v < bc)) {
        bsum = sum;
        bc = v;
      }
    }
  }
  return bc;
}

__device__ __forceinline__ int code_bits(int C0) { return 32 - __clz((C0 - 1) | 1); }

// Fold votes of R rows by one warp (lane j holds neighbour slot j of every
// row).  Lanes holding the same label find each other with __match_any_sync,
// so a label's count is a popcount; winner: largest count, then (tie-break)
// largest double score sum, then the smallest code.  The R rows' steps are
// interleaved so their latencies overlap.  out[q] = -1 for a row without
// valid neighbours.
template <int R>
__device__ __forceinline__ void vote_rows_match(const uint16_t* lab, const uint16_t* id, const float* const* sc, int w,
                                                int lane, int* out) {
  int c[R], cnt[R], mx[R], best[R];
  unsigned m[R], tied[R];
#pragma unroll
  for (int q = 0; q < R; ++q) c[q] = id[q] != kNoRow ? static_cast<int>(lab[id[q]]) : -1;
#pragma unroll
  for (int q = 0; q < R; ++q) m[q] = __match_any_sync(kFull, c[q]);
#pragma unroll
  for (int q = 0; q < R; ++q) cnt[q] = c[q] >= 0 ? __popc(m[q]) : 0;
#pragma unroll
  for (int q = 0; q < R; ++q) mx[q] = __reduce_max_sync(kFull, cnt[q]);
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const bool top = c[q] >= 0 && cnt[q] == mx[q];
    best[q] = static_cast<int>(__reduce_min_sync(kFull, top ? static_cast<unsigned>(c[q]) : 0xffffffffu));
    // one lane (the lowest) per label reaching the top count
    tied[q] = __ballot_sync(kFull, top && (__ffs(m[q]) - 1) == lane);
  }
#pragma unroll
  for (int q = 0; q < R; ++q)
    out[q] = mx[q] == 0 ? -1 : (__popc(tied[q]) == 1 ? best[q] : vote_tiebreak(c[q], tied[q], sc[q], w, lane));
}

// Rows with no out-of-fold neighbour take the majority label of their training
// folds (ties to the smaller code).  P.foldcnt holds the rows per code of every
// fold and, after the last, of all of them, for the labels being voted on: it is
// counted once (count_folds) and follows the rows whose label changes
// (move_fold).  Counting every row again for each vote took 30k cycles of a
// cycle at 10000 rows and 300 codes.
__device__ __forceinline__ int* fold_counts(const EvolveParams& P, int prob) {
  return P.foldcnt + static_cast<size_t>(prob) * (P.F + 1) * P.C0max;
}

__device__ __forceinline__ void move_fold(const EvolveParams& P, int prob, int row, int from, int to) {
  int* fc = fold_counts(P, prob);
  const size_t fold = static_cast<size_t>(P.folds[static_cast<size_t>(prob) * P.L + row]) * P.C0max;
  const size_t all = static_cast<size_t>(P.F) * P.C0max;
  atomicSub(&fc[fold + from], 1);
  atomicAdd(&fc[fold + to], 1);
  atomicSub(&fc[all + from], 1);
  atomicAdd(&fc[all + to], 1);
}

// Lists the rows without neighbours in P.empty_rows (f.empty_cnt of them) and
// counts the folds of s.cur.
__device__ __noinline__ void count_folds(const EvolveParams& P, int prob, int C0) {
  const Smem s = carve_smem_any(P);
  Fixed& f = *s.f;
  const uint16_t* nbp = P.nb + static_cast<size_t>(prob) * P.L * P.w;
  const uint8_t* fo = P.folds + static_cast<size_t>(prob) * P.L;
  uint16_t* list = P.empty_rows + static_cast<size_t>(blockIdx.x) * P.L;
  int* fc = fold_counts(P, prob);
  if (threadIdx.x == 0) f.empty_cnt = 0;
  if (threadIdx.x < 8) f.empty_folds[threadIdx.x] = 0u;
  for (int i = threadIdx.x; i < (P.F + 1) * P.C0max; i += kThreads) fc[i] = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < P.L; r += kThreads) {
    if (nbp[static_cast<size_t>(r) * P.w] == kNoRow) {
      list[atomicAdd(&f.empty_cnt, 1)] = static_cast<uint16_t>(r);
      atomicOr(&f.empty_folds[fo[r] >> 5], 1u << (fo[r] & 31));
    }
    atomicAdd(&fc[fo[r] * P.C0max + s.cur[r]], 1);
    atomicAdd(&fc[P.F * P.C0max + s.cur[r]], 1);
  }
  __syncthreads();
}

__device__ __noinline__ void vote_empty_rows(const EvolveParams& P, int prob, uint16_t* out, int C0) {
  const Smem s = carve_smem_any(P);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint8_t* fo = P.folds + static_cast<size_t>(prob) * P.L;
  const uint16_t* list = P.empty_rows + static_cast<size_t>(blockIdx.x) * P.L;
  const int* fc = fold_counts(P, prob);
  const int* all = fc + P.F * P.C0max;
  // one warp per fold, its lanes over the codes: the largest training count,
  // ties to the smaller code (the reference scans the codes in ascending
  // order keeping strict improvements)
  for (int fo_i = warp; fo_i < P.F; fo_i += kWarps) {
    if (((s.f->empty_folds[fo_i >> 5] >> (fo_i & 31)) & 1u) == 0u) continue;
    int bl = 0x7fffffff, bcount = -1;
    for (int c = lane; c < C0; c += 32) {
      const int cnt = __ldcg(&all[c]) - __ldcg(&fc[fo_i * P.C0max + c]);
      if (cnt > bcount) {
        bl = c;
        bcount = cnt;
      }
    }
    const int top = __reduce_max_sync(kFull, bcount);
    bl = __reduce_min_sync(kFull, bcount == top ? bl : 0x7fffffff);
    if (lane == 0) s.f->sel_hist[fo_i] = bl;  // F <= 255
  }
  __syncthreads();
  for (int i = threadIdx.x; i < s.f->empty_cnt; i += kThreads) {
    const int r = list[i];
    out[r] = static_cast<uint16_t>(s.f->sel_hist[fo[r]]);
  }
}

// Rows per warp batch of the vote (a multiple of kVoteRows): the batch loop
// is unrolled, so this also sets how many copies of the vote code the kernel
// carries.
constexpr int kVoteBatch = 8;
constexpr int kVoteRows = 4;

// Vote rows into `out`: every row (rows == nullptr) or the nrows rows listed
// in `rows` (the caller has filled the others).  Rows with no out-of-fold
// neighbour take the majority label of their training folds (ties to the
// smaller label).  Neighbour ids are fetched 8 rows at a time per warp so the
// memory latency is paid once per batch; scores only for tied rows.
__device__ __forceinline__ void vote_block(const EvolveParams& P, const Smem& s, int prob, const uint16_t* lab,
                           uint16_t* out, int C0, bool has_empty, const uint16_t* rows = nullptr,
                           int nrows = -1) {
  const int L = P.L, w = P.w;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint16_t* nbp = P.nb + static_cast<size_t>(prob) * L * w;
  const float* scp = P.sc + static_cast<size_t>(prob) * L * w;
  const int count = rows ? nrows : L;
  constexpr int kB = kVoteBatch;
  for (int i0 = warp * kB; i0 < count; i0 += kWarps * kB) {
    uint16_t ids[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 + u;
      const int r = i < count ? (rows ? static_cast<int>(rows[i]) : i) : 0;
      ids[u] = (i < count && lane < w) ? nbp[static_cast<size_t>(r) * w + lane] : kNoRow;
    }
#pragma unroll
    for (int u = 0; u < kB; u += kVoteRows) {
      const int i = i0 + u;
      if (i >= count) break;
      int rr[kVoteRows], best[kVoteRows];
      uint16_t id[kVoteRows];
      const float* sc[kVoteRows];
#pragma unroll
      for (int q = 0; q < kVoteRows; ++q) {
        const bool in = i + q < count;
        rr[q] = in ? (rows ? static_cast<int>(rows[i + q]) : i + q) : -1;
        id[q] = in ? ids[u + q] : kNoRow;
        sc[q] = scp + static_cast<size_t>(in ? rr[q] : 0) * w;
      }
      vote_rows_match<kVoteRows>(lab, id, sc, w, lane, best);
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < kVoteRows; ++q)
          if (rr[q] >= 0 && best[q] >= 0) out[rr[q]] = static_cast<uint16_t>(best[q]);
      }
    }
  }
  if (has_empty) vote_empty_rows(P, prob, out, C0);
  __syncthreads();
}

// Rows whose vote may differ from the current state's: reverse neighbours of
// the rows whose label changed.  Lists them in s.jarr (free after the
// relabel) and returns how many, or returns -1 when so many rows changed that
// a full vote is cheaper; either way s.pred starts as a copy of s.curpred.
//   pass: eight rows a thread, predictions copied and the changed rows'
//     reverse-list bounds appended to s.list;
//   gather: each warp takes four changed rows at a time, its lanes reading 32
//     reverse entries of each per step (all four rows' loads in flight) and
//     setting the entries' bits, which returns nothing and waits for nothing;
//   list: a word of bits per thread, places from a scan over the warp.
// The list is in no particular order: every listed row is voted on its own.
// Testing each entry's flag and appending it at once made every 32 entries wait
// for two atomics: 11.0k cycles at 132 changed of 10000 rows.
__device__ __forceinline__ int dirty_rows_block(const EvolveParams& P, const Smem& s, int prob, bool has_empty) {
  Fixed& f = *s.f;
  const int L = P.L, words = (L + 31) >> 5;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* mark = reinterpret_cast<unsigned*>(s.scratch32);
  int* bounds = reinterpret_cast<int*>(s.list);  // 2 ints per changed row, room for L / 4 rows
  uint16_t* dirty = s.jarr;
  const int cap = L / 4;
  const int* roff = P.rev_off + static_cast<size_t>(prob) * (L + 1);
  const uint16_t* ridx = P.rev_idx + static_cast<size_t>(prob) * L * P.w;
  if (threadIdx.x == 0) {
    f.changed_cnt = 0;
    f.dirty_cnt = 0;
  }
  for (int i = threadIdx.x; i < words; i += kThreads) mark[i] = 0u;
  __syncthreads();
  for (int i = threadIdx.x; i < row_vectors(L); i += kThreads) {
    reinterpret_cast<uint4*>(s.pred)[i] = load_rows(s.curpred, i);
    const uint4 a = load_rows(s.cl, i), b = load_rows(s.cur, i);
    if (a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w) continue;
    for (int e = 0; e < 8; ++e) {
      const int r = 8 * i + e;
      if (r >= L || row_code(a, e) == row_code(b, e)) continue;
      if (has_empty) move_fold(P, prob, r, row_code(b, e), row_code(a, e));
      const int slot = atomicAdd(&f.changed_cnt, 1);
      if (slot < cap) {
        bounds[2 * slot] = roff[r];
        bounds[2 * slot + 1] = roff[r + 1];
      }
    }
  }
  __syncthreads();
  const int changed = f.changed_cnt;
  // changed * mean in-degree reverse entries mark about L (1 - exp(-e / L))
  // distinct rows for e entries; the gather costs little next to a vote, so
  // the full vote is kept for e > 3 L (about 95% of the rows dirty), and for
  // more changed rows than the bounds' room
  if (static_cast<long long>(changed) * f.rev_total > 3ll * L * L || changed > cap) return -1;
  for (int i0 = 4 * warp; i0 < changed; i0 += 4 * kWarps) {
    int b[4], e[4];
    int span = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + q;
      b[q] = i < changed ? bounds[2 * i] : 0;
      e[q] = i < changed ? bounds[2 * i + 1] : 0;
      span = max(span, e[q] - b[q]);
    }
    for (int k0 = 0; k0 < span; k0 += 32) {
      uint16_t v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = b[q] + k0 + lane;
        v[q] = k < e[q] ? ridx[k] : kNoRow;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v[q] != kNoRow) atomicOr(&mark[v[q] >> 5], 1u << (v[q] & 31u));
    }
  }
  __syncthreads();
  for (int i0 = warp * 32; i0 < words; i0 += kThreads) {
    unsigned bits = i0 + lane < words ? mark[i0 + lane] : 0u;
    const int n = __popc(bits);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += v;
    }
    int at = 0;
    if (lane == 31 && incl > 0) at = atomicAdd(&f.dirty_cnt, incl);
    at = __shfl_sync(kFull, at, 31) + incl - n;
    for (; bits != 0u; bits &= bits - 1) dirty[at++] = static_cast<uint16_t>((i0 + lane) * 32 + __ffs(bits) - 1);
  }
  __syncthreads();
  return f.dirty_cnt;
}

// Count labels of `lab` per code, first positions and distinct count.
// have_cnt: s.cnt already holds the counts of `lab`.  The first kThreads rows
// set the first positions; of the others, taken eight to a thread, only those
// before their code's first position so far need an atomicMin: nearly none.
// pred != nullptr: *ok also receives the count of rows with lab == pred
// (both totals from one block reduction: ok + 2^16 nc, L and C0 < 2^15).
__device__ __forceinline__ int label_census(const EvolveParams& P, const Smem& s, const uint16_t* lab, int C0,
                            bool have_cnt = false, const uint16_t* pred = nullptr, int* ok = nullptr) {
  for (int c = threadIdx.x; c < C0; c += kThreads) {
    if (!have_cnt) s.cnt[c] = 0;
    s.firstpos[c] = 0x7fffffff;
  }
  __syncthreads();
  if (threadIdx.x < P.L) {
    const int r = threadIdx.x, code = lab[r];
    if (!have_cnt) atomicAdd(&s.cnt[code], 1);
    atomicMin(&s.firstpos[code], r);
  }
  __syncthreads();
  int hits = 0;
  for (int i = threadIdx.x; i < row_vectors(P.L); i += kThreads) {
    const uint4 v = load_rows(lab, i);
    const uint4 u = pred != nullptr ? load_rows(pred, i) : v;
    int first[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) first[e] = 8 * i + e < P.L ? s.firstpos[row_code(v, e)] : 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = 8 * i + e;
      if (r >= P.L) break;
      const int code = row_code(v, e);
      hits += code == row_code(u, e);
      if (!have_cnt && r >= kThreads) atomicAdd(&s.cnt[code], 1);
      if (r < first[e]) atomicMin(&s.firstpos[code], r);
    }
  }
  __syncthreads();
  int local = 0;
  for (int c = threadIdx.x; c < C0; c += kThreads) local += s.cnt[c] > 0;
  if (pred == nullptr) return block_sum(local, *s.f);
  const int packed = block_sum(hits + (local << 16), *s.f);
  *ok = packed & 0xffff;
  return packed >> 16;
}

// s.order[0..nc) = the codes of the census in the iteration order of
// std::unordered_map<int,int> after reserve(L) and insertion in row order.
__device__ __forceinline__ void map_order(const EvolveParams& P, const Smem& s, int prob, int C0) {
  const bool nocollide = P.nocollide[prob] != 0;
  if (nocollide) {
    // every key has its own bucket: each new key goes to the list front, so
    // a key's rank counts the keys first seen after it (one warp per key)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kHeld = 10;  // first positions a lane keeps in registers
    int held[kHeld];
#pragma unroll
    for (int q = 0; q < kHeld; ++q) {
      const int c = lane + 32 * q;
      held[q] = c < C0 && s.cnt[c] > 0 ? s.firstpos[c] : -1;
    }
    for (int c = warp; c < C0; c += kWarps) {
      if (s.cnt[c] == 0) continue;
      int rank = 0;
      const int fp = s.firstpos[c];
#pragma unroll
      for (int q = 0; q < kHeld; ++q) rank += held[q] > fp;
      for (int c2 = lane + 32 * kHeld; c2 < C0; c2 += 32) rank += (s.cnt[c2] > 0 && s.firstpos[c2] > fp);
      rank = __reduce_add_sync(kFull, rank);
      if (lane == 0) s.order[rank] = c;
    }
    __syncthreads();
  } else if (threadIdx.x == 0) {
    // keys in insertion order, then simulate bucket-run insertion
    int* ins = s.bt;   // scratch
    int k = 0;
    for (int c = 0; c < C0; ++c) if (s.cnt[c] > 0) ins[k++] = c;
    for (int a = 1; a < k; ++a) {  // insertion sort by first position
      const int v = ins[a];
      int b = a - 1;
      while (b >= 0 && s.firstpos[ins[b]] > s.firstpos[v]) {
        ins[b + 1] = ins[b];
        --b;
      }
      ins[b + 1] = v;
    }
    const int* c2l = P.code2label + static_cast<size_t>(prob) * P.C0max;
    int* list = s.order;  // list[0..len) in iteration order
    int len = 0;
    for (int a = 0; a < k; ++a) {
      const int code = ins[a];
      const uint64_t bkt = static_cast<uint64_t>(static_cast<int64_t>(c2l[code])) % P.bucket_count;
      int at = -1;
      for (int q = 0; q < len; ++q) {
        const uint64_t bq = static_cast<uint64_t>(static_cast<int64_t>(c2l[list[q]])) % P.bucket_count;
        if (bq == bkt) {
          at = q;
          break;
        }
      }
      if (at < 0) at = 0;
      for (int q = len; q > at; --q) list[q] = list[q - 1];
      list[at] = code;
      ++len;
    }
  }
  __syncthreads();
}

// Accuracy of `ok` hits and core_objective_score for the kNN classifier, in
// f.acc and f.score; census must be current.  Double operations are left to
// single warps: one of the whole block takes the FP64 pipe 512 cycles, a
// division 4400.
__device__ __forceinline__ void objective(const EvolveParams& P, const Smem& s, int prob, int ok, int nc, int C0) {
  Fixed& f = *s.f;
  const bool use_div = P.guarded && P.pol_diversity;
  const bool reject1 = P.guarded && P.pol_reject1;
  if (threadIdx.x == 32) f.acc = __ddiv_rn(static_cast<double>(ok), static_cast<double>(P.L));
  const bool ranked = use_div && !(reject1 && nc == 1);
  if (ranked) {
    map_order(P, s, prob, C0);
    // psq[c] = (c/L)*(c/L) rounded as the reference rounds each step
    for (int q = threadIdx.x; q < nc; q += kThreads) s.cp[q] = P.psq[s.cnt[s.order[q]]];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double acc = f.acc;
    double score = reject1 && nc == 1 ? -INFINITY : acc;
    if (ranked) {
      const double diff = __dsub_rn(1.0, chain_add(0.0, s.cp, nc));
      score = __dmul_rn(acc, __dsqrt_rn((0.0 < diff) ? diff : 0.0));
    }
    if (threadIdx.x == 0) f.score = score;
  }
}

// Groups the rows of s.cl by code: s.cnt[c] rows of which s.movable[c] are not
// fixed, their predictions pp at s.list[class_start(s, c)..], in no particular
// order.  A row's place in its class is what the count's atomicAdd returned
// (kept in s.jarr).  Returns the number of codes in use.
__device__ __forceinline__ int class_start(const Smem& s, int c) { return s.aux[c] & 0xffff; }
__device__ __forceinline__ int class_groups(const EvolveParams& P, const Smem& s, const uint16_t* pp, int C0) {
  const bool any_fixed = s.f->fxd != nullptr;
  for (int c = threadIdx.x; c < C0; c += kThreads) {
    s.cnt[c] = 0;
    s.movable[c] = 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < row_vectors(P.L); i += kThreads) {
    const uint4 v = load_rows(s.cl, i);
    unsigned at[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = 8 * i + e;
      at[e] = r < P.L ? atomicAdd(&s.cnt[row_code(v, e)], 1) : 0;
      if (any_fixed && r < P.L && s.f->fxd[r] != 1) atomicAdd(&s.movable[row_code(v, e)], 1);
    }
    reinterpret_cast<uint4*>(s.jarr)[i] =
        make_uint4(at[0] | at[1] << 16, at[2] | at[3] << 16, at[4] | at[5] << 16, at[6] | at[7] << 16);
  }
  __syncthreads();
  // starts (below 2^16) and codes in use in one scan
  for (int c = threadIdx.x; c < C0; c += kThreads) s.aux[c] = s.cnt[c] > 0 ? s.cnt[c] + 0x10000 : 0;
  __syncthreads();
  const int nc = static_cast<int>(static_cast<unsigned>(block_exclusive_scan(s.aux, C0, *s.f) - P.L) >> 16);
  for (int i = threadIdx.x; i < row_vectors(P.L); i += kThreads) {
    const uint4 v = load_rows(s.cl, i), u = load_rows(pp, i), at = load_rows(s.jarr, i);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if (8 * i + e >= P.L) break;
      s.list[class_start(s, row_code(v, e)) + row_code(at, e)] = static_cast<uint16_t>(row_code(u, e));
    }
  }
  if (!any_fixed)
    for (int c = threadIdx.x; c < C0; c += kThreads) s.movable[c] = s.cnt[c];
  __syncthreads();
  return nc;
}

// Calls use(src, n, items, each, h) for every code src in use with movable rows,
// by one warp of those that have counters: n rows, h[c] of them predicted as c
// (zero again afterwards).  each(i) for i < items runs over the codes
// predicted, some of them repeatedly (a small class: its rows' predictions) or
// not at all (a large one: all codes).
template <class Use>
__device__ __forceinline__ void for_each_source(const Smem& s, int C0, Use&& use) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp >= s.hist_warps) return;
  int* h = s.hist + static_cast<size_t>(warp) * s.hist_stride;
  for (int src = warp; src < C0; src += s.hist_warps) {
    const int n = s.cnt[src];
    if (n == 0 || s.movable[src] <= 0) continue;
    const uint16_t* seg = s.list + class_start(s, src);
    int i = lane;
    for (; i + 96 < n; i += 128) {
      int c[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) c[q] = seg[i + 32 * q];
#pragma unroll
      for (int q = 0; q < 4; ++q) atomicAdd(&h[c[q]], 1);
    }
    for (; i < n; i += 32) atomicAdd(&h[seg[i]], 1);
    __syncwarp();
    const bool members = n < C0;
    const int items = members ? n : C0;
    auto each = [&](int k) { return members ? static_cast<int>(seg[k]) : k; };
    use(src, n, items, each, h);
    __syncwarp();
    for (int k = lane; k < items; k += 32) h[each(k)] = 0;
    __syncwarp();
  }
}

// propose_many_to_one_absorption on s.cl given proposal predictions pp.
// Returns 1 if the labels changed.  On return s.cnt holds the counts of s.cl.
// The class x prediction counts are never laid out: a source only meets the
// predictions of its own rows, which its warp counts and reads back.  With a
// C0 x C0 table (in global memory past 200 codes), a scan of it, double
// divisions in every warp and the choice in one thread this took 18.6k cycles
// of a cycle at 10000 rows and 50 codes, 54k at 750 and 100, 138k at 10000 and 300.
__device__ __forceinline__ int absorption_block(const EvolveParams& P, const Smem& s, int prob, const uint16_t* pp, int C0) {
  Fixed& f = *s.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = threadIdx.x; c < C0; c += kThreads) s.bt[c] = -1;
  const int nc = class_groups(P, s, pp, C0);
  if (nc <= 2) return 0;
  const double n = static_cast<double>(P.L);
  const double nmax = (1.0 < n) ? n : 1.0;  // std::max(1.0, n)
  // The reference scans the destinations in ascending order keeping the best by
  // (surplus, count, destination size, smaller destination), starting from
  // (0, 0, source size, source).  Exact surplus x n = cnt*n - ssize*dsize; only
  // the candidates at the exact maximum can win the double comparison chain
  // (double rounding is far below the 1/n spacing of distinct exact surpluses).
  // Candidates there with one count have one size and one double surplus, so
  // the smallest wins; with several counts (rare) the doubles are compared.
  for_each_source(s, C0, [&](int src, int ssize, int items, auto&& each, const int* h) {
    const int stay = h[src];
    // both products are below 2^32, and a surplus of zero or less is no move
    unsigned kmax = 0;
    int kcnt = 0, kdst = 0x7fffffff;
    bool mixed = false;
    const unsigned size = static_cast<unsigned>(ssize), rows = static_cast<unsigned>(P.L);
    for (int i = lane; i < items; i += 32) {
      const int dst = each(i), cntd = h[dst], dsize = s.cnt[dst];
      const unsigned a = cntd * rows, b = size * dsize;
      if (dst == src || dsize == 0 || a <= b) continue;  // (a count of zero is never a surplus)
      if (a - b > kmax) {
        kmax = a - b;
        kcnt = cntd;
        kdst = dst;
        mixed = false;
      } else if (a - b == kmax) {
        mixed |= cntd != kcnt;
        kdst = min(kdst, dst);
      }
    }
    const unsigned top = __reduce_max_sync(kFull, kmax);
    if (top == 0u) return;
    const bool cand = kmax == top;
    const int bcount = __reduce_max_sync(kFull, cand ? kcnt : 0);
    int bt = __reduce_min_sync(kFull, cand ? kdst : 0x7fffffff);
    int count = bcount;
    if (__any_sync(kFull, cand && (mixed || kcnt != bcount))) {
      int bsize = ssize;
      double bsur = 0.0;
      bt = src;
      count = 0;
      for (int i = lane; i < items; i += 32) {
        const int dst = each(i), cntd = h[dst], dsize = s.cnt[dst];
        if (dst == src || dsize == 0) continue;
        const unsigned a = cntd * rows, b = size * dsize;
        if (a <= b || a - b != top) continue;
        const double expected = __ddiv_rn(__dmul_rn(static_cast<double>(ssize), static_cast<double>(dsize)), nmax);
        const double sur = __dsub_rn(static_cast<double>(cntd), expected);
        if (sur > bsur || (sur == bsur && cntd > count) || (sur == bsur && cntd == count && dsize > bsize) ||
            (sur == bsur && cntd == count && dsize == bsize && dst < bt)) {
          bt = dst;
          bsize = dsize;
          count = cntd;
          bsur = sur;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double osur = __shfl_xor_sync(kFull, bsur, o);
        const int ocount = __shfl_xor_sync(kFull, count, o);
        const int osize = __shfl_xor_sync(kFull, bsize, o);
        const int obt = __shfl_xor_sync(kFull, bt, o);
        if (osur > bsur || (osur == bsur && ocount > count) || (osur == bsur && ocount == count && osize > bsize) ||
            (osur == bsur && ocount == count && osize == bsize && obt < bt)) {
          bt = obt;
          bsize = osize;
          count = ocount;
          bsur = osur;
        }
      }
    }
    if (lane == 0 && bt != src && count > stay) {
      s.bt[src] = bt;
      s.order[src] = count;
    }
  });
  __syncthreads();
  // the surpluses, a thread per source; s.firstpos[t] becomes the last source of
  // target t and s.aux[t] (whose class starts are not needed any more) how many
  for (int c = threadIdx.x; c < C0; c += kThreads) {
    s.aux[c] = 0;
    s.firstpos[c] = 0;
  }
  __syncthreads();
  for (int src = threadIdx.x; src < C0; src += kThreads) {
    const int bt = s.bt[src];
    if (bt < 0) continue;
    const double expected =
        __ddiv_rn(__dmul_rn(static_cast<double>(s.cnt[src]), static_cast<double>(s.cnt[bt])), nmax);
    const double sur = __dsub_rn(static_cast<double>(s.order[src]), expected);
    if (sur > 0.0) {
      s.bsur[src] = sur;
      atomicAdd(&s.aux[bt], 1);
      atomicMax(&s.firstpos[bt], src);
    } else {
      s.bt[src] = -1;
    }
  }
  __syncthreads();
  // per-target weights accumulated in ascending source order, a warp per target
  // of several sources
  for (int t = warp; t < C0; t += kWarps) {
    const int k = s.aux[t];
    if (k == 0) continue;
    if (k == 1) {
      if (lane == 0) s.weight[t] = s.bsur[s.firstpos[t]];
      continue;
    }
    double weight = 0.0;
    for (int c0 = 0; c0 < C0; c0 += 32) {
      const unsigned m = __ballot_sync(kFull, c0 + lane < C0 && s.bt[min(c0 + lane, C0 - 1)] == t);
      if (m == 0u) continue;
      const double mine = (m >> lane) & 1u ? s.bsur[c0 + lane] : 0.0;
      for (unsigned rem = m; rem != 0u; rem &= rem - 1)
        weight = __dadd_rn(weight, __shfl_sync(kFull, mine, __ffs(rem) - 1));
    }
    if (lane == 0) s.weight[t] = weight;
  }
  __syncthreads();
  if (warp == 0) {
    // the targets of several sources, or where there are none those of one
    bool multi = false;
    for (int c = lane; c < C0; c += 32) multi |= s.aux[c] > 1;
    multi = __any_sync(kFull, multi);
    int k = 0;
    for (int c0 = 0; c0 < C0; c0 += 32) {
      const int t = c0 + lane;
      const int a = t < C0 ? s.aux[t] : 0;
      const bool in = multi ? a > 1 : a == 1;
      const unsigned m = __ballot_sync(kFull, in);
      if (in) {
        const int at = k + __popc(m & ((1u << lane) - 1u));
        s.order[at] = t;
        s.cp[C0 + at] = s.weight[t] > DBL_MIN ? s.weight[t] : DBL_MIN;  // std::max(weight, DBL_MIN)
      }
      k += __popc(m);
    }
    __syncwarp();
    int sel = -1, apply = 0;
    if (k > 0) {
      sel = s.order[discrete_warp(f.rng, s.cp + C0, k, s.cp, lane)];
      // sizes after remapping every non-fixed row of the selected sources
      int moved = 0, after = 0;
      for (int c = lane; c < C0; c += 32) {
        int size = s.cnt[c];
        if (s.bt[c] == sel && c != sel) {
          moved += s.movable[c];
          size -= s.movable[c];
        }
        s.aux[c] = size;
        after += c != sel && size > 0;
      }
      moved = __reduce_add_sync(kFull, moved);
      __syncwarp();
      if (lane == 0) {
        s.aux[sel] += moved;
        after += s.aux[sel] > 0;
      }
      after = __reduce_add_sync(kFull, after);
      apply = moved > 0 && after > 1 && after < nc;
    }
    if (lane == 0) {
      f.selected_target = sel;
      f.flag = apply;
    }
  }
  __syncthreads();
  const int sel = f.selected_target, apply = f.flag;
  if (apply) {
    for (int i = threadIdx.x; i < row_vectors(P.L); i += kThreads) {
      const uint4 v = load_rows(s.cl, i);
      int to[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) to[e] = 8 * i + e < P.L ? s.bt[row_code(v, e)] : -1;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int r = 8 * i + e;
        if (to[e] != sel || row_code(v, e) == sel) continue;
        if (s.f->fxd != nullptr && s.f->fxd[r] == 1) continue;
        s.cl[r] = static_cast<uint16_t>(sel);
      }
    }
    for (int c = threadIdx.x; c < C0; c += kThreads) s.cnt[c] = s.aux[c];
  }
  __syncthreads();
  return apply;
}

// Relabel of sampled groups when draws are needed (groups of several rows, or
// no prediction guidance).  Thread 0, in shuffled order.
__device__ __noinline__ void relabel_serial(const EvolveParams& P, const uint16_t* pp, int ns, int C0) {
  const Smem s = carve_smem_any(P);
  Fixed& f = *s.f;
  int* hist = s.aux;
  for (int c = 0; c < C0; ++c) hist[c] = 0;
  int nemp = 0;
  if (!P.pol_guidance) {
    // empirical distribution of the labels at the start of the cycle
    for (int r = 0; r < P.L; ++r) hist[s.cl[r]]++;
    for (int c = 0; c < C0; ++c) {
      if (hist[c] > 0) {
        s.order[nemp] = c;
        s.weight[nemp] = static_cast<double>(hist[c]);
        ++nemp;
      }
      hist[c] = 0;
    }
  }
  for (int q = 0; q < ns; ++q) {
    const int g = s.perm[q];
    const int beg = s.f->goff[g], end = s.f->goff[g + 1];
    int neligible = 0;
    for (int a = beg; a < end; ++a) neligible += (s.f->fxd == nullptr || s.f->fxd[s.f->gmem[a]] != 1);
    if (neligible == 0) continue;
    int rep;
    if (P.pol_guidance) {
      // candidate labels: predictions of the eligible members, ascending, with counts
      int k = 0;
      for (int a = beg; a < end; ++a) {
        const int row = s.f->gmem[a];
        if (s.f->fxd != nullptr && s.f->fxd[row] == 1) continue;
        const int c = pp[row];
        if (hist[c]++ == 0) s.bt[k++] = c;
      }
      for (int a = 1; a < k; ++a) {
        const int v = s.bt[a];
        int b = a - 1;
        while (b >= 0 && s.bt[b] > v) {
          s.bt[b + 1] = s.bt[b];
          --b;
        }
        s.bt[b + 1] = v;
      }
      for (int a = 0; a < k; ++a) {
        s.cp[C0 + a] = static_cast<double>(hist[s.bt[a]]);
        hist[s.bt[a]] = 0;
      }
      rep = s.bt[discrete_serial(f.rng, s.cp + C0, k, s.cp)];
    } else {
      if (nemp == 0) continue;
      rep = s.order[discrete_serial(f.rng, s.weight, nemp, s.cp)];
    }
    for (int a = beg; a < end; ++a) {
      const int row = s.f->gmem[a];
      if (s.f->fxd != nullptr && s.f->fxd[row] == 1) continue;
      s.cl[row] = static_cast<uint16_t>(rep);
    }
  }
}

// ---------------------------------------------------------------------------
// Learned relabelling proposal (mlp.cuh)
// ---------------------------------------------------------------------------

// Features of `row` in the current state (s.cur / s.curpred), census of
// s.cur in `cnt_cur`: among the row's fold-filtered neighbours, the fractions
// sharing its label, holding its prediction as label, predicting its
// prediction and whose label equals their prediction; the sizes of its label
// and prediction classes; the run's progress; the fraction of valid
// neighbours.
__device__ __forceinline__ void proposal_features(const EvolveParams& P, const Smem& s, int prob, int row, const int* cnt_cur,
                                  float progress, float* f) {
  const uint16_t* nbr = P.nb + (static_cast<size_t>(prob) * P.L + row) * P.w;
  const int c = s.cur[row], q = s.curpred[row];
  int nv = 0, same_cur = 0, same_pred = 0, pred_pred = 0, stable = 0;
  for (int j = 0; j < P.w; ++j) {
    const int id = nbr[j];
    if (id == kNoRow) break;
    ++nv;
    const int lc = s.cur[id], lp = s.curpred[id];
    same_cur += lc == c;
    same_pred += lc == q;
    pred_pred += lp == q;
    stable += lc == lp;
  }
  const float inv = nv > 0 ? 1.0f / static_cast<float>(nv) : 0.0f;
  const float invL = 1.0f / static_cast<float>(P.L);
  f[0] = same_cur * inv;
  f[1] = same_pred * inv;
  f[2] = pred_pred * inv;
  f[3] = stable * inv;
  f[4] = cnt_cur[c] * invL;
  f[5] = cnt_cur[q] * invL;
  f[6] = progress;
  f[7] = static_cast<float>(nv) / static_cast<float>(P.w);
}

// Census of s.cur into s.aux (per code).
__device__ __forceinline__ void census_cur(const EvolveParams& P, const Smem& s, int C0) {
  for (int c = threadIdx.x; c < C0; c += kThreads) s.aux[c] = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < P.L; r += kThreads) atomicAdd(&s.aux[s.cur[r]], 1);
  __syncthreads();
}

// Gumbel(0, 1) noise of (run seed, cycle, row): a splitmix64 hash of the
// three (Steele, Lea and Flood, "Fast splittable pseudorandom number
// generators", 2014) mapped to u in (0, 1), then -log(-log u).
__device__ __forceinline__ float gumbel_noise(uint64_t seed, int cycle, int row) {
  uint64_t z = seed + 0x9e3779b97f4a7c15ull * (static_cast<uint64_t>(cycle) * 65536ull + static_cast<uint64_t>(row) + 1ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  const float u = (static_cast<float>(z >> 40) + 0.5f) * (1.0f / 16777216.0f);
  return -__logf(-__logf(u));
}

// Relabels to their prediction `take` of the candidates (label != prediction,
// not fixed).  The candidates are compacted into keys whose low 16 bits are
// 65535 - row; each warp scores 32 of them on the tensor pipe
// (mlp_logit_warp) and puts the top 16 bits of the order-preserving image of
// the score (plus Gumbel noise unless P.mlp_greedy: sampling without
// replacement from the network's softmax over the candidates) above the row,
// so all keys are distinct and ties go to the smaller row.  The take-th
// largest key is found by a 4-pass radix select with 8-bit digits.
__device__ __noinline__ void learned_flip(const EvolveParams& P, int prob, int cycle, int take, int C0) {
  const Smem s = carve_smem_any(P);
  Fixed& f = *s.f;
  if (take <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  census_cur(P, s, C0);
  unsigned* key = reinterpret_cast<unsigned*>(s.scratch32);
  if (threadIdx.x == 0) f.sel_count = 0;
  __syncthreads();
  for (int base = warp * 32; base < P.L; base += kThreads) {
    const int r = base + lane;
    const bool c = r < P.L && s.cur[r] != s.curpred[r] && (s.f->fxd == nullptr || s.f->fxd[r] != 1);
    const unsigned b = __ballot_sync(kFull, c);
    int at = 0;
    if (lane == 0 && b != 0u) at = atomicAdd(&f.sel_count, __popc(b));
    at = __shfl_sync(kFull, at, 0);
    if (c) key[at + __popc(b & ((1u << lane) - 1u))] = 0xffffu - static_cast<unsigned>(r);
  }
  __syncthreads();
  const int count = f.sel_count;
  if (take >= count) {
    for (int i = threadIdx.x; i < count; i += kThreads) {
      const int r = 0xffff - static_cast<int>(key[i] & 0xffffu);
      s.cl[r] = s.curpred[r];
    }
    __syncthreads();
    return;
  }
  const float progress = static_cast<float>(cycle) / static_cast<float>(P.T > 0 ? P.T : 1);
  const uint64_t seed = P.seeds[prob];
  for (int base = warp * 32; base < count; base += kThreads) {
    const int i = base + lane;
    uint32_t fw[4] = {0u, 0u, 0u, 0u};
    int r = -1;
    if (i < count) {
      r = 0xffff - static_cast<int>(key[i] & 0xffffu);
      float x[kMlpIn];
      proposal_features(P, s, prob, r, s.aux, progress, x);
      mlp_pack_row(x, fw);
    }
    float z = mlp_logit_warp(P.mlp, fw, min(32, count - base));
    if (i < count) {
      if (!P.mlp_greedy) z += gumbel_noise(seed, cycle, r);
      const unsigned u = __float_as_uint(z);
      const unsigned ord = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
      key[i] = (ord & 0xffff0000u) | (0xffffu - static_cast<unsigned>(r));
    }
  }
  __syncthreads();
  unsigned prefix = 0u;
  int need = take;
  for (int pass = 3; pass >= 0; --pass) {
    const int shift = 8 * pass;
    const unsigned hmask = pass == 3 ? 0u : (0xffffffffu << (shift + 8));
    for (int b = threadIdx.x; b < 256; b += kThreads) f.sel_hist[b] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += kThreads) {
      const unsigned k = key[i];
      if ((k & hmask) == prefix) atomicAdd(&f.sel_hist[(k >> shift) & 255u], 1);
    }
    __syncthreads();
    if (warp == 0) {
      // lane l holds digits 8 l .. 8 l + 7; find the largest digit whose
      // count of keys at or above it reaches `need`
      int c[8], tot = 0;
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        c[d] = f.sel_hist[8 * lane + d];
        tot += c[d];
      }
      int suf = tot;  // keys in lanes >= this lane
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_down_sync(kFull, suf, o);
        if (lane + o < 32) suf += v;
      }
      const unsigned ball = __ballot_sync(kFull, suf >= need);
      if (lane == 31 - __clz(ball)) {
        int above = suf - tot, d = 7;
        while (d > 0 && above + c[d] < need) above += c[d--];
        f.sel_digit = 8 * lane + d;
        f.sel_need = need - above;
      }
    }
    __syncthreads();
    prefix |= static_cast<unsigned>(f.sel_digit) << shift;
    need = f.sel_need;
    __syncthreads();
  }
  for (int i = threadIdx.x; i < count; i += kThreads) {
    if (key[i] >= prefix) {
      const int r = 0xffff - static_cast<int>(key[i] & 0xffffu);
      s.cl[r] = s.curpred[r];
    }
  }
  __syncthreads();
}

// Training snapshot of the current state: features of every row and its
// label / prediction codes.
__device__ __noinline__ void snapshot_state(const EvolveParams& P, int prob, int cycle, int C0) {
  const Smem s = carve_smem_any(P);
  census_cur(P, s, C0);
  const float progress = static_cast<float>(cycle) / static_cast<float>(P.T > 0 ? P.T : 1);
  for (int r = threadIdx.x; r < P.L; r += kThreads) {
    const size_t o = static_cast<size_t>(prob) * P.L + r;
    float x[kMlpIn];
    proposal_features(P, s, prob, r, s.aux, progress, x);
    for (int i = 0; i < kMlpIn; ++i) P.snap_feat[o * kMlpIn + i] = x[i];
    P.snap_cur[o] = s.cur[r];
    P.snap_pred[o] = s.curpred[r];
  }
  __syncthreads();
}

// Points the CTA at problem prob's groups and fixed flags: shared by all
// problems, or one block per problem (per_problem_groups: goff stride L + 1,
// gmem and fixed stride L, group count gcount[prob]).
__device__ __forceinline__ void bind_groups(const EvolveParams& P, const Smem& s, int prob) {
  if (threadIdx.x == 0) {
    const bool per = P.per_problem_groups != 0;
    s.f->goff = P.goff + (per ? static_cast<size_t>(prob) * (P.L + 1) : 0);
    s.f->gmem = P.gmem + (per ? static_cast<size_t>(prob) * P.L : 0);
    s.f->fxd = P.fixed == nullptr ? nullptr : P.fixed + (per ? static_cast<size_t>(prob) * P.L : 0);
    s.f->G = per ? P.gcount[prob] : P.G;
  }
  __syncthreads();
}

// Each of the first ns groups of the shuffle takes its own CV prediction; only
// groups whose prediction differs from their label can change, so just those
// are listed (in s.perm) and walked forward to their final shuffled position:
// walked as they were met, a few lanes of a warp at a time walked while the
// others waited.
__device__ __forceinline__ void flip_sampled(const Smem& s, int G, int ns) {
  Fixed& f = *s.f;
  const int lane = threadIdx.x & 31;
  const int* gmem = f.gmem;
  if (threadIdx.x == 0) f.walk_cnt = 0;
  __syncthreads();
  for (int g0 = threadIdx.x; g0 - lane < G; g0 += 4 * kThreads) {
    int row[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) row[q] = g0 + q * kThreads < G ? gmem[g0 + q * kThreads] : -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool walk = row[q] >= 0 && s.curpred[row[q]] != s.cur[row[q]] && (f.fxd == nullptr || f.fxd[row[q]] != 1);
      const unsigned m = __ballot_sync(kFull, walk);
      if (m == 0u) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&f.walk_cnt, __popc(m));
      at = __shfl_sync(kFull, at, 0);
      if (walk) s.perm[at + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(g0 + q * kThreads);
    }
  }
  __syncthreads();
  const int count = f.walk_cnt;
  for (int i = threadIdx.x; i < count; i += kThreads) {
    const int g = s.perm[i], row = gmem[g];
    if (final_position_of(s, g, ns) < ns) s.cl[row] = s.curpred[row];
  }
}

// u < exp(delta / temperature), delta < 0: in floats where they leave no doubt
// (their quotient is within 3e-7 of itself, so expf of one above -80 within
// 3e-5 of the double), else in doubles, whose exp takes 2000 cycles.
__device__ __forceinline__ int annealed(double u, double delta, double temperature) {
  const float x = static_cast<float>(delta) / static_cast<float>(temperature);
  const float v = static_cast<float>(u);
  if (x > -80.0f) {
    const float e = expf(x);
    if (v > e * 1.0001f) return 0;
    if (v < e * 0.9999f) return 1;
  } else if (x <= -80.0f && v > 1e-30f) {
    return 0;
  }
  return u < exp(__ddiv_rn(delta, temperature));
}

__device__ __forceinline__ void evolve_problem(const EvolveParams& P, const Smem& s, int prob) {
  Fixed& f = *s.f;
  bind_groups(P, s, prob);
  const int L = P.L, T = P.T, G = f.G;
  const int C0 = P.ncodes[prob];
  const uint16_t* init = P.init + static_cast<size_t>(prob) * L;
  uint16_t* gbest = P.clbest + static_cast<size_t>(prob) * L;
  uint16_t* gbestpred = P.cvpredbest + static_cast<size_t>(prob) * L;
  double* vacc = P.vect_acc + static_cast<size_t>(prob) * T;
  double* vscore = P.vect_score + static_cast<size_t>(prob) * T;
  int* psize = P.proposal_size + static_cast<size_t>(prob) * T;
  int* act = P.active + static_cast<size_t>(prob) * T;
  uint8_t* fl = P.flags + static_cast<size_t>(prob) * T * 3;
  const uint16_t* nbp = P.nb + static_cast<size_t>(prob) * L * P.w;

  if (threadIdx.x == 0) {
    mt64_seed(f.rng, P.seeds[prob]);
    f.rev_total = P.rev_off[static_cast<size_t>(prob) * (L + 1) + L];
  }
  int local_empty = 0;
  for (int r = threadIdx.x; r < L; r += kThreads) {
    s.cur[r] = init[r];
    local_empty += nbp[static_cast<size_t>(r) * P.w] == kNoRow;
  }
  __syncthreads();
  const bool has_empty = block_sum(local_empty, f) > 0;

  if (has_empty) count_folds(P, prob, C0);

  // initial evaluation
  vote_block(P, s, prob, s.cur, s.curpred, C0, has_empty);
  int ok = 0;
  for (int r = threadIdx.x; r < L; r += kThreads) {
    ok += s.cur[r] == s.curpred[r];
    gbest[r] = s.cur[r];
    gbestpred[r] = s.curpred[r];
  }
  ok = block_sum(ok, f);
  const int nc0 = label_census(P, s, s.cur, C0);
  objective(P, s, prob, ok, nc0, C0);
  RunState& run = f.run;
  if (threadIdx.x == 0) {
    run = RunState{};
    run.accbest = run.cur_acc = f.acc;
    run.scorebest = run.cur_score = f.score;
    run.nc_cur = run.nc_best = nc0;
  }
  // the size bound of proposal `cycle`
  auto group_bound = [&](int cycle) {
    if (!(P.adaptive && P.pol_adaptive) || T <= 1) return G;
    double progress = __ddiv_rn(static_cast<double>(cycle + 1), static_cast<double>(T + 1));
    progress = progress < 0.0 ? 0.0 : (progress > 1.0 ? 1.0 : progress);
    const double smooth = __dmul_rn(__dmul_rn(progress, progress), __dsub_rn(3.0, __dmul_rn(2.0, progress)));
    double temp = __dsub_rn(1.0, smooth);
    temp = temp < 0.0 ? 0.0 : (temp > 1.0 ? 1.0 : temp);
    const int mc = 1 + static_cast<int>(floor(__dmul_rn(static_cast<double>(G - 1), temp)));
    return mc > 1 ? mc : 1;
  };
  auto cooling = [&](int cycle) {
    return __dsub_rn(1.0, __ddiv_rn(static_cast<double>(cycle + 1), static_cast<double>(T > 1 ? T : 1)));
  };
  if (threadIdx.x == kThreads - 1) {
    f.max_groups = group_bound(0);
    f.cooling[0] = cooling(0);
  }
  // between cycles s.cl equals s.cur: the proposal starts from the current
  // (evolutionary) or best (greedy) state, which s.cur holds
  copy_rows(s.cl, s.cur, L);
  __syncthreads();

  for (int cycle = 0; cycle < T; ++cycle) {
    if (P.snap_feat != nullptr && cycle == P.snap_cycle) snapshot_state(P, prob, cycle, C0);
    if (threadIdx.x == 0) f.ns = G <= 1 ? (G > 0 ? G : 0) : uniform_int_serial(f.rng, 1, f.max_groups);
    __syncthreads();
    shuffle_targets_block(f, s.jarr, G, s.save);
    const int ns = f.ns;
    if (threadIdx.x == 0) psize[cycle] = ns;
    if (ns > 0) {
      bucket_steps_block(s, G, ns);
      if (P.singleton && P.pol_guidance && P.mlp != nullptr) {
        // learned proposal: as many relabellings as the plain draw would make,
        // given to the candidates the network scores highest
        int take = 0;
        for (int g = threadIdx.x; g < G; g += kThreads) {
          const int row = s.f->gmem[g];
          if (s.curpred[row] == s.cur[row]) continue;
          if (s.f->fxd != nullptr && s.f->fxd[row] == 1) continue;
          take += final_position_of(s, g, ns) < ns;
        }
        take = block_sum(take, f);
        learned_flip(P, prob, cycle, take, C0);
      } else if (P.singleton && P.pol_guidance) {
        // Each sampled group takes its own CV prediction; only groups whose
        // prediction differs from their label can change, so walk just those
        // forward to their final shuffled position.
        flip_sampled(s, G, ns);
      } else {
        for (int p = threadIdx.x; p < ns; p += kThreads) s.perm[p] = static_cast<uint16_t>(occupant_of(s, G, p));
        __syncthreads();
        if (threadIdx.x == 0) relabel_serial(P, s.curpred, ns, C0);
      }
    }
    __syncthreads();

    int absorbed = 0;
    if (P.pol_transition && P.absorption) {
      absorbed = absorption_block(P, s, prob, s.curpred, C0);
    }

    const bool cnt_of_cl = P.pol_transition && P.absorption;  // s.cnt holds the counts of s.cl
    {
      const int nd = dirty_rows_block(P, s, prob, has_empty);  // s.pred = s.curpred on return
      vote_block(P, s, prob, s.cl, s.pred, C0, has_empty, nd < 0 ? nullptr : s.jarr, nd);
    }
    const int nc = L < 32768 && C0 < 32768 ? label_census(P, s, s.cl, C0, cnt_of_cl, s.pred, &ok)
                                           : label_census(P, s, s.cl, C0, cnt_of_cl);
    if (L >= 32768 || C0 >= 32768) {
      ok = 0;
      for (int r = threadIdx.x; r < L; r += kThreads) ok += s.cl[r] == s.pred[r];
      ok = block_sum(ok, f);
    }
    objective(P, s, prob, ok, nc, C0);
    // while warp 0 scores: the next cycle's annealing factor and size bound
    if (threadIdx.x == kThreads - 1) {
      f.cooling[(cycle + 1) & 1] = cooling(cycle + 1);
      f.max_groups = group_bound(cycle + 1);
    }
    if (threadIdx.x == 0) {
      const double acc = f.acc, score = f.score;
      const bool improves = score > run.scorebest;
      int acc_cur = improves, impr = improves, st = 0;
      if (P.evolutionary) {
        acc_cur = score >= run.cur_score;
        impr = acc_cur;
        if (!acc_cur && P.pol_stochastic) {
          const double one_minus = __dsub_rn(1.0, run.cur_acc);
          const double clipped = (0.0 < one_minus) ? one_minus : 0.0;
          const double t0 = __dmul_rn(__dmul_rn(0.10, clipped), f.cooling[cycle & 1]);
          const double temperature = (1.0e-9 < t0) ? t0 : 1.0e-9;
          if (temperature > 1.0e-9) {
            st = 2;  // attempted
            acc_cur = annealed(canonical_serial(f.rng), __dsub_rn(score, run.cur_score), temperature);
            if (acc_cur) st = 3;
          }
        }
      }
      if (improves) {
        run.accbest = acc;
        run.scorebest = score;
        run.nc_best = nc;
        ++run.best_updates;
      }
      if (P.evolutionary) {
        if (acc_cur) {
          run.cur_acc = acc;
          run.cur_score = score;
          run.nc_cur = nc;
          ++run.accepts;
        } else {
          ++run.rejections;
        }
        if (st >= 2) ++run.st_att;
        if (st == 3) ++run.st_acc;
      }
      run.absorb_moves += absorbed;
      if (acc_cur && absorbed) ++run.tr_acc;
      if (acc == 1.0 && isfinite(score)) run.success = 1;
      fl[3 * cycle + 0] = acc_cur ? 1 : 0;
      fl[3 * cycle + 1] = (acc_cur && impr) ? 1 : 0;
      fl[3 * cycle + 2] = st == 3 ? 1 : 0;
      act[cycle] = P.evolutionary ? run.nc_cur : run.nc_best;
      vacc[cycle] = run.accbest;
      vscore[cycle] = run.scorebest;
      f.accept = acc_cur | (improves << 1);
    }
    __syncthreads();
    const int code = f.accept;
    const bool accepted = code & 1, improves = (code >> 1) & 1;
    if (improves) {
      for (int r = threadIdx.x; r < L; r += kThreads) {
        gbest[r] = s.cl[r];
        gbestpred[r] = s.pred[r];
      }
    }
    if (P.evolutionary ? accepted : improves) {
      copy_rows(s.cur, s.cl, L);
      copy_rows(s.curpred, s.pred, L);
    } else {
      if (has_empty) {
        for (int r = threadIdx.x; r < L; r += kThreads)
          if (s.cl[r] != s.cur[r]) move_fold(P, prob, r, s.cl[r], s.cur[r]);
        __syncthreads();
      }
      copy_rows(s.cl, s.cur, L);
    }
    __syncthreads();
  }

  if (threadIdx.x == 0) {
    int* c = P.counters + static_cast<size_t>(prob) * 16;
    const int moves = P.pol_transition && P.absorption ? T : 0;  // transitions attempted
    c[0] = T;
    c[1] = T;
    c[2] = run.best_updates;
    c[3] = run.accepts;
    c[4] = run.st_att;
    c[5] = run.st_acc;
    c[6] = run.rejections;
    c[7] = 0;
    c[8] = run.absorb_moves;
    c[9] = moves;
    c[10] = run.tr_acc;
    c[11] = moves;
    c[12] = run.tr_acc;
    c[13] = T + 1;
    c[14] = run.success;
    c[15] = 0;
    P.best[2 * prob] = run.accbest;
    P.best[2 * prob + 1] = run.scorebest;
    P.status[prob] = 0;
  }
  __syncthreads();
}

__device__ __forceinline__ void clear_counters(const Smem& s) {
  for (int i = threadIdx.x; i < s.hist_stride * s.hist_warps; i += kThreads) s.hist[i] = 0;
  __syncthreads();
}

template <bool kRows>
__global__ void __launch_bounds__(kThreads, 1) evolve_kernel(const __grid_constant__ EvolveParams P) {
  const Smem s = carve_smem<kRows>(P);
  clear_counters(s);
  for (int prob = blockIdx.x; prob < P.problems; prob += gridDim.x) evolve_problem(P, s, prob);
}

// ===========================================================================
// PLS-LDA evolution: maximize_core (core.cpp:1269-1549) with PLSLDACV as the
// predictor.  The predictor runs as separate launches over all problems and
// folds (pls.cu), so each cycle is split in two: this kernel accepts the
// previous proposal (its CV predictions are in Q.pred) and builds the next
// one, keeping the engine, the current state and the counters in global
// memory between launches.  PLS adds to the kNN cycle:
//   propose_auto_class_coarsening   core.cpp:995-1108
//   the fragmentation penalty       core.cpp:954-968
// ===========================================================================

// propose_auto_class_coarsening on s.cl.  plogp[k] = (k/L) * log(k/L) as the
// reference rounds it.  The transition entropy is formed as
// log(s) - sum_c c log(c) / s from host tables of k log k and log k: it only
// feeds ceil(temperature * redundant), which an ulp-level difference cannot move
// unless that product lies within an ulp of an integer.  Returns 1 if the labels
// changed.
// A warp per source counts its rows' predictions (for_each_source), takes the
// destination and lists the c log c terms in order; a thread per source adds its
// terms; the candidates are shuffled as the groups are and ranked by counting.
// With a thread per source over the whole class x prediction table and the
// shuffle and the sort in one thread this took 480k to 890k cycles at 7500 rows
// and 100 codes.
__device__ __forceinline__ int coarsening_block(const EvolvePlsParams& Q, const Smem& s, int prob, const uint16_t* pp, int C0) {
  const EvolveParams& P = Q.base;
  Fixed& f = *s.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nc = class_groups(P, s, pp, C0);
  if (nc <= 2) return 0;
  int* dst_of = s.bt;          // per source: destination, -1 = not a candidate
  int* stay_of = s.firstpos;   // per source: rows predicted as itself
  int* terms_of = s.order;     // per source: number of terms
  double* score_of = s.cp;     // per source: candidate score
  double* share_of = s.cp + C0;  // per code: (k/L) log(k/L)
  double* te_of = s.bsur;      // per source: its share of the transition entropy
  // c log c of the counts above 1 (1 log 1 = 0) in ascending code order: a
  // source of n rows has at most n / 2
  double* terms = reinterpret_cast<double*>(s.scratch32);
  for (int c = threadIdx.x; c < C0; c += kThreads) {
    dst_of[c] = -1;
    te_of[c] = 0.0;
    share_of[c] = s.cnt[c] > 0 ? Q.plogp[s.cnt[c]] : 0.0;
  }
  __syncthreads();
  for_each_source(s, C0, [&](int src, int ssize, int items, auto&& each, const int* h) {
    // destination: largest (count, size), smaller code, of the other codes in use
    unsigned key = 0u;
    int dst = 0x7fffffff;
    for (int i = lane; i < items; i += 32) {
      const int d = each(i), size = s.cnt[d];
      if (d == src || size == 0 || h[d] == 0) continue;
      const unsigned k = static_cast<unsigned>(h[d]) << 16 | static_cast<unsigned>(size);
      if (k > key || (k == key && d < dst)) {
        key = k;
        dst = d;
      }
    }
    const unsigned top = __reduce_max_sync(kFull, key);
    dst = __reduce_min_sync(kFull, key == top ? dst : 0x7fffffff);
    double* to = terms + (class_start(s, src) >> 1);
    int k = 0;
    for (int c0 = 0; c0 < C0; c0 += 32) {
      const int v = c0 + lane < C0 ? h[c0 + lane] : 0;
      const unsigned m = __ballot_sync(kFull, v > 1);
      if (v > 1) to[k + __popc(m & ((1u << lane) - 1u))] = Q.klogk[v];
      k += __popc(m);
    }
    if (lane == 0) {
      dst_of[src] = top != 0u ? dst : -1;
      stay_of[src] = h[src];
      terms_of[src] = k;
    }
  });
  __syncthreads();
  for (int src = threadIdx.x; src < C0; src += kThreads) {
    const int ssize = s.cnt[src];
    if (ssize == 0 || s.movable[src] <= 0) continue;
    const double size = static_cast<double>(ssize);
    const double clc = chain_add(0.0, terms + (class_start(s, src) >> 1), terms_of[src]);
    const double te = __dsub_rn(Q.logk[ssize], __ddiv_rn(clc, size));
    te_of[src] = __dmul_rn(__ddiv_rn(size, static_cast<double>(P.L)), te);
    if (dst_of[src] < 0) continue;
    const double stay = __ddiv_rn(static_cast<double>(stay_of[src]), size);
    score_of[src] =
        __dmul_rn(__ddiv_rn(1.0, __dsqrt_rn(static_cast<double>(s.movable[src]))), __dsub_rn(1.0, stay));
  }
  __syncthreads();
  if (warp == 0) {
    // class entropy and mean transition entropy, in source order
    double ce = 0.0, wte = 0.0;
    for (int c0 = 0; c0 < C0; c0 += 8) {
      double a[8], b[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        a[q] = c0 + q < C0 ? share_of[c0 + q] : 0.0;
        b[q] = c0 + q < C0 ? te_of[c0 + q] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        ce = __dsub_rn(ce, a[q]);  // zero for a code not in use
        wte = __dadd_rn(wte, b[q]);
      }
    }
    const double keff = cr_exp(ce);
    const double lr = cr_log(__ddiv_rn(static_cast<double>(nc), 1.0 < keff ? keff : 1.0));
    const double frag = 0.0 < lr ? lr : 0.0;
    const double temperature = __ddiv_rn(frag, __dadd_rn(__dadd_rn(frag, wte), 1.0));
    const double rd = __dsub_rn(static_cast<double>(nc), keff);
    const double redundant = 0.0 < rd ? rd : 0.0;
    int budget = static_cast<int>(ceil(__dmul_rn(temperature, redundant)));
    if (budget < 1 && frag > 0.0) budget = 1;
    if (lane == 0) f.flag = min(budget, nc - 2);
  } else if (warp == 1) {
    // candidates in ascending source order
    int k = 0;
    for (int c0 = 0; c0 < C0; c0 += 32) {
      const int src = c0 + lane;
      const int d = src < C0 ? dst_of[src] : -1;
      const unsigned m = __ballot_sync(kFull, d >= 0);
      if (d >= 0) {
        const int at = k + __popc(m & ((1u << lane) - 1u));
        s.order[at] = src << 16 | d;
        s.weight[at] = score_of[src];
      }
      k += __popc(m);
    }
    if (lane == 0) f.walk_cnt = k;
  }
  __syncthreads();
  const int K = f.walk_cnt, budget = f.flag;
  if (K == 0 || budget <= 0) return 0;
  __syncthreads();
  shuffle_targets_block(f, s.jarr, K, s.save);
  __syncthreads();
  bucket_steps_block(s, K, K);
  for (int q = threadIdx.x; q < K; q += kThreads) {
    const int at = occupant_of(s, K, q);
    s.firstpos[q] = s.order[at];
    s.cp[q] = s.weight[at];
  }
  for (int c = threadIdx.x; c < C0; c += kThreads) s.aux[c] = c;
  __syncthreads();
  // stable order by score, descending; the scores are positive, so their bits
  // compare as they do
  const unsigned long long* bits = reinterpret_cast<const unsigned long long*>(s.cp);
  for (int q = threadIdx.x; q < K; q += kThreads) {
    const unsigned long long mine = bits[q];
    int rank = 0;
    for (int j = 0; j < K; ++j) rank += bits[j] > mine || (bits[j] == mine && j < q);
    s.order[rank] = s.firstpos[q];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int* remap = s.aux;
    int merged = 0;
    for (int q = 0; q < K && merged < budget; ++q) {
      const int src = static_cast<int>(static_cast<unsigned>(s.order[q]) >> 16);
      if (remap[src] != src) continue;
      int d = s.order[q] & 0xffff;
      while (remap[d] != d) d = remap[d];
      if (d == src) continue;
      remap[src] = d;
      ++merged;
    }
    f.flag = merged;
  }
  __syncthreads();
  if (f.flag == 0) return 0;
  int changed = 0;
  const int* remap = s.aux;
  for (int r = threadIdx.x; r < P.L; r += kThreads) {
    if (s.f->fxd != nullptr && s.f->fxd[r] == 1) continue;
    const int a = s.cl[r];
    int d = a;
    while (remap[d] != d) d = remap[d];
    if (d != a) {
      s.cl[r] = static_cast<uint16_t>(d);
      changed = 1;
    }
  }
  return block_sum(changed, f) > 0 ? 1 : 0;
}

// core_objective_score with the PLS fragmentation penalty, in f.acc and f.score
// for thread 0; census current.
__device__ __forceinline__ void objective_pls(const EvolvePlsParams& Q, const Smem& s, int prob, int ok, int nc, int C0) {
  const EvolveParams& P = Q.base;
  Fixed& f = *s.f;
  const bool use_div = P.guarded && P.pol_diversity;
  const bool use_frag = Q.coarsening && Q.pol_frag;
  const bool reject1 = P.guarded && P.pol_reject1;
  if (threadIdx.x == 32) f.acc = __ddiv_rn(static_cast<double>(ok), static_cast<double>(P.L));
  const bool single = reject1 && nc == 1;
  const bool ranked = !single && (use_div || (use_frag && nc > 1));
  // both sums' terms, then the two chains side by side
  double* sq = s.cp;
  double* pl = s.cp + C0;
  if (ranked) {
    map_order(P, s, prob, C0);
    for (int q = threadIdx.x; q < nc; q += kThreads) {
      const int c = s.cnt[s.order[q]];
      sq[q] = use_div ? P.psq[c] : 0.0;
      pl[q] = use_frag ? Q.plogp[c] : 0.0;
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const double acc = f.acc;
  double score = single ? -INFINITY : acc;
  if (ranked) {
    double same = 0.0, entropy = 0.0;
    for (int q0 = 0; q0 < nc; q0 += 8) {
      double a[8], b[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        a[q] = q0 + q < nc ? sq[q0 + q] : 0.0;
        b[q] = q0 + q < nc ? pl[q0 + q] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        same = __dadd_rn(same, a[q]);
        entropy = __dsub_rn(entropy, b[q]);
      }
    }
    if (use_div) {
      const double diff = __dsub_rn(1.0, same);
      score = __dmul_rn(score, __dsqrt_rn(0.0 < diff ? diff : 0.0));
    }
    if (use_frag && nc > 1) {
      const double mse = P.L > 1 ? Q.logn : 0.0;
      double code_cost = 0.0;
      if (mse > 0.0) {
        const double v = __ddiv_rn(entropy, mse);
        code_cost = v < 0.0 ? 0.0 : (1.0 < v ? 1.0 : v);
      }
      const double keff = cr_exp(entropy);
      const double lr = cr_log(__ddiv_rn(static_cast<double>(nc), 1.0 < keff ? keff : 1.0));
      const double frag = 0.0 < lr ? lr : 0.0;
      const double frag_cost = __ddiv_rn(frag, __dadd_rn(1.0, frag));
      const double pc = code_cost < frag_cost ? frag_cost : code_cost;
      score = __dsub_rn(score, __dmul_rn(__dsub_rn(1.0, acc), pc));
    }
  }
  if (threadIdx.x == 0) f.score = score;
}

// Rows of s.cl grouped by code, ascending rows within a code, for the
// cross-product chains of the PLS predictor: a counting sort.  Each of nw warps
// takes a run of rows and has a counter per code; a row's place is its warp's
// first place for the code plus the rows before it.  A warp per code reading all
// rows took 120k to 160k cycles at 7500 rows and 100 codes.
__device__ __forceinline__ void class_lists(const EvolvePlsParams& Q, const Smem& s, int prob, int C0) {
  const int L = Q.base.L, C = Q.base.C0max;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  uint16_t* table = reinterpret_cast<uint16_t*>(s.scratch32);  // nw x C0, of 2 x L rounded up to 8
  const int nw = min(kWarps, 2 * 8 * row_vectors(L) / C0);     // at least 2: C0 <= L
  const int bits = code_bits(C0);
  const int chunk = ((L + nw - 1) / nw + 31) / 32 * 32;
  const int beg = warp < nw ? min(L, warp * chunk) : 0, end = warp < nw ? min(L, beg + chunk) : 0;
  uint16_t* mine = table + min(warp, nw - 1) * C0;
  for (int i = threadIdx.x; i < nw * C0; i += kThreads) table[i] = 0;
  __syncthreads();
  // place(r, at): the row and its place among its warp's rows of the code
  auto walk = [&](auto&& place) {
    for (int b = beg; b < end; b += 32) {
      const bool in = b + lane < end;
      const int code = in ? s.cl[b + lane] : 0;
      const unsigned m = same_code(code, __ballot_sync(kFull, in), bits);
      const int at = in ? mine[code] : 0;
      if (in) place(b + lane, at + __popc(m & below));
      __syncwarp();
      if (in && (m & below) == 0u) mine[code] = static_cast<uint16_t>(at + __popc(m));
      __syncwarp();
    }
  };
  walk([](int, int) {});
  __syncthreads();
  for (int c = threadIdx.x; c < C0; c += kThreads) {
    int run = 0;
    for (int k = 0; k < nw; ++k) {
      const int v = table[k * C0 + c];
      table[k * C0 + c] = static_cast<uint16_t>(run);
      run += v;
    }
    s.cnt[c] = run;
    s.aux[c] = run;
  }
  __syncthreads();
  block_exclusive_scan(s.aux, C0, *s.f);
  int* coff = Q.class_off + static_cast<size_t>(prob) * (C + 1);
  for (int c = threadIdx.x; c <= C; c += kThreads) coff[c] = c < C0 ? s.aux[c] : L;
  for (int i = threadIdx.x; i < nw * C0; i += kThreads) table[i] = static_cast<uint16_t>(table[i] + s.aux[i % C0]);
  __syncthreads();
  uint16_t* rows = Q.class_rows + static_cast<size_t>(prob) * L;
  walk([&](int r, int at) { rows[at] = static_cast<uint16_t>(r); });
  __syncthreads();
}

__device__ __forceinline__ void pls_propose(const EvolvePlsParams& Q, const Smem& s, int prob, int cycle, PlsRunState& st, int C0) {
  const EvolveParams& P = Q.base;
  Fixed& f = *s.f;
  const int L = P.L, T = P.T, G = f.G;
  copy_rows(s.cl, s.cur, L);
  __syncthreads();
  if (threadIdx.x == 0) {
    int ns;
    if (G <= 1) {
      ns = G > 0 ? G : 0;
    } else if (!(P.adaptive && P.pol_adaptive) || T <= 1) {
      ns = uniform_int_serial(f.rng, 1, G);
    } else {
      double progress = __ddiv_rn(static_cast<double>(cycle + 1), static_cast<double>(T + 1));
      progress = progress < 0.0 ? 0.0 : (progress > 1.0 ? 1.0 : progress);
      const double smooth = __dmul_rn(__dmul_rn(progress, progress), __dsub_rn(3.0, __dmul_rn(2.0, progress)));
      double temp = __dsub_rn(1.0, smooth);
      temp = temp < 0.0 ? 0.0 : (temp > 1.0 ? 1.0 : temp);
      const int mc = 1 + static_cast<int>(floor(__dmul_rn(static_cast<double>(G - 1), temp)));
      ns = uniform_int_serial(f.rng, 1, mc > 1 ? mc : 1);
    }
    f.ns = ns;
    P.proposal_size[static_cast<size_t>(prob) * T + cycle] = ns;
  }
  __syncthreads();
  shuffle_targets_block(f, s.jarr, G, s.save);
  const int ns = f.ns;
  if (ns > 0) {
    bucket_steps_block(s, G, ns);
    if (P.singleton && P.pol_guidance) {
      flip_sampled(s, G, ns);
    } else {
      for (int q = threadIdx.x; q < ns; q += kThreads) s.perm[q] = static_cast<uint16_t>(occupant_of(s, G, q));
      __syncthreads();
      if (threadIdx.x == 0) relabel_serial(P, s.curpred, ns, C0);
    }
  }
  __syncthreads();
  const bool attempt_co = P.pol_transition && Q.coarsening && Q.pol_coarsen;
  const bool attempt_ab = P.pol_transition && P.absorption;
  int coarsened = 0, absorbed = 0;
  if (attempt_co) coarsened = coarsening_block(Q, s, prob, s.curpred, C0);
  if (attempt_ab) absorbed = absorption_block(P, s, prob, s.curpred, C0);
  if (threadIdx.x == 0) {
    if (attempt_co || attempt_ab) ++st.tr_att;
    if (attempt_co) {
      ++st.co_att;
      st.co_moves += coarsened;
    }
    if (attempt_ab) {
      ++st.m1_att;
      st.absorb_moves += absorbed;
    }
    st.coarsened = coarsened;
    st.absorbed = absorbed;
  }
  __syncthreads();
  class_lists(Q, s, prob, C0);
}

__device__ __forceinline__ void pls_step(const EvolvePlsParams& Q, const Smem& s, int prob) {
  const EvolveParams& P = Q.base;
  Fixed& f = *s.f;
  bind_groups(P, s, prob);
  const int L = P.L, T = P.T;
  const int C0 = P.ncodes[prob];
  const size_t ro = static_cast<size_t>(prob) * L;
  PlsRunState& gst = Q.state[prob];
  __shared__ PlsRunState st;
  if (Q.phase == 0) {
    if (threadIdx.x == 0) {
      mt64_seed(f.rng, P.seeds[prob]);
      st = PlsRunState{};
    }
    for (int r = threadIdx.x; r < L; r += kThreads) {
      s.cl[r] = P.init[ro + r];
      Q.cl[ro + r] = s.cl[r];
    }
    __syncthreads();
    class_lists(Q, s, prob, C0);
  } else {
    const int cycle = Q.cycle;  // proposal `cycle - 1` was evaluated (cycle 0: the initial labels)
    const Mt64State& g = Q.rng[prob];
    for (int i = threadIdx.x; i < kMtN; i += kThreads) {
      f.rng.mt[i] = g.mt[i];
      f.rng.out[i] = g.out[i];
    }
    if (threadIdx.x == 0) {
      f.rng.pos = g.pos;
      st = gst;
    }
    // four rows of all four arrays in flight (before the first cycle the
    // current state is not read any further)
    for (int r0 = threadIdx.x; r0 < L; r0 += 4 * kThreads) {
      uint16_t v[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const size_t o = ro + min(r0 + q * kThreads, L - 1);
        v[q][0] = Q.cl[o];
        v[q][1] = Q.pred[o];
        v[q][2] = cycle > 0 ? Q.cur[o] : 0;
        v[q][3] = cycle > 0 ? Q.curpred[o] : 0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = r0 + q * kThreads;
        if (r >= L) break;
        s.cl[r] = v[q][0];
        s.pred[r] = v[q][1];
        s.cur[r] = v[q][2];
        s.curpred[r] = v[q][3];
      }
    }
    __syncthreads();
    uint16_t* gbest = P.clbest + ro;
    uint16_t* gbestpred = P.cvpredbest + ro;
    int ok = 0;
    for (int r = threadIdx.x; r < L; r += kThreads) ok += s.cl[r] == s.pred[r];
    ok = block_sum(ok, f);
    const int nc = label_census(P, s, s.cl, C0);
    objective_pls(Q, s, prob, ok, nc, C0);
    if (cycle == 0) {
      for (int r = threadIdx.x; r < L; r += kThreads) {
        s.cur[r] = s.cl[r];
        s.curpred[r] = s.pred[r];
        gbest[r] = s.cl[r];
        gbestpred[r] = s.pred[r];
      }
      if (threadIdx.x == 0) {
        const double acc = f.acc, score = f.score;
        st.accbest = st.cur_acc = acc;
        st.scorebest = st.cur_score = score;
        st.nc_cur = st.nc_best = nc;
      }
      __syncthreads();
    } else {
      const int c = cycle - 1;
      if (threadIdx.x == 0) {
        const double acc = f.acc, score = f.score;
        ++st.proposals;
        const bool improves = score > st.scorebest;
        int accepted = improves, improving = improves, stoch = 0;
        if (P.evolutionary) {
          const double cooling = __dsub_rn(1.0, __ddiv_rn(static_cast<double>(c + 1), static_cast<double>(T > 1 ? T : 1)));
          const double one_minus = __dsub_rn(1.0, st.cur_acc);
          const double clipped = (0.0 < one_minus) ? one_minus : 0.0;
          const double t0 = __dmul_rn(__dmul_rn(0.10, clipped), cooling);
          const double temperature = (1.0e-9 < t0) ? t0 : 1.0e-9;
          int acc_cur = score >= st.cur_score;
          improving = acc_cur;
          if (!acc_cur && P.pol_stochastic && temperature > 1.0e-9) {
            ++st.st_att;
            const double u = canonical_serial(f.rng);
            acc_cur = annealed(u, __dsub_rn(score, st.cur_score), temperature);
            stoch = acc_cur;
          }
          accepted = acc_cur;
        }
        f.accept = accepted | (improves << 1) | (stoch << 2) | (improving << 3);
        if (improves) {
          st.accbest = acc;
          st.scorebest = score;
          ++st.best_updates;
          st.nc_best = nc;
        }
        if (P.evolutionary) {
          if (accepted) {
            st.cur_acc = acc;
            st.cur_score = score;
            st.nc_cur = nc;
            ++st.accepts;
            if (stoch) ++st.st_acc;
          } else {
            ++st.rejections;
          }
        }
        if (accepted && (st.coarsened || st.absorbed)) {
          ++st.tr_acc;
          if (st.coarsened) ++st.co_acc;
          if (st.absorbed) ++st.m1_acc;
        }
        uint8_t* fl = P.flags + (static_cast<size_t>(prob) * T + c) * 3;
        fl[0] = accepted ? 1 : 0;
        fl[1] = (accepted && improving) ? 1 : 0;
        fl[2] = stoch ? 1 : 0;
        P.active[static_cast<size_t>(prob) * T + c] = P.evolutionary ? st.nc_cur : st.nc_best;
        P.vect_acc[static_cast<size_t>(prob) * T + c] = st.accbest;
        P.vect_score[static_cast<size_t>(prob) * T + c] = st.scorebest;
        if (acc == 1.0 && isfinite(score)) st.success = 1;
      }
      __syncthreads();
      const int code = f.accept;
      const bool improves = (code >> 1) & 1;
      const bool take = P.evolutionary ? (code & 1) : improves;
      if (improves) {
        for (int r = threadIdx.x; r < L; r += kThreads) {
          gbest[r] = s.cl[r];
          gbestpred[r] = s.pred[r];
        }
      }
      if (take) {
        copy_rows(s.cur, s.cl, L);
        copy_rows(s.curpred, s.pred, L);
      }
      __syncthreads();
    }
    if (cycle == T) {
      // the rows of the best labels by code, for the projection
      __syncthreads();
      for (int r = threadIdx.x; r < L; r += kThreads) s.cl[r] = gbest[r];
      __syncthreads();
      class_lists(Q, s, prob, C0);
    }
    if (cycle < T) {
      pls_propose(Q, s, prob, cycle, st, C0);
      for (int r = threadIdx.x; r < L; r += kThreads) Q.cl[ro + r] = s.cl[r];
    } else if (threadIdx.x == 0) {
      int* c = P.counters + static_cast<size_t>(prob) * 18;
      c[0] = T;
      c[1] = st.proposals;
      c[2] = st.best_updates;
      c[3] = st.accepts;
      c[4] = st.st_att;
      c[5] = st.st_acc;
      c[6] = st.rejections;
      c[7] = st.co_moves;
      c[8] = st.absorb_moves;
      c[9] = st.tr_att;
      c[10] = st.tr_acc;
      c[11] = st.m1_att;
      c[12] = st.m1_acc;
      c[13] = st.proposals + 1;
      c[14] = st.success;
      c[15] = 0;
      c[16] = st.co_att;
      c[17] = st.co_acc;
      P.best[2 * prob] = st.accbest;
      P.best[2 * prob + 1] = st.scorebest;
      P.status[prob] = 0;
    }
    for (int r = threadIdx.x; r < L; r += kThreads) {
      Q.cur[ro + r] = s.cur[r];
      Q.curpred[ro + r] = s.curpred[r];
    }
  }
  __syncthreads();
  Mt64State& g = Q.rng[prob];
  for (int i = threadIdx.x; i < kMtN; i += kThreads) {
    g.mt[i] = f.rng.mt[i];
    g.out[i] = f.rng.out[i];
  }
  if (threadIdx.x == 0) {
    g.pos = f.rng.pos;
    gst = st;
  }
  __syncthreads();
}

template <bool kRows>
__global__ void __launch_bounds__(kThreads, 1) evolve_pls_kernel(const __grid_constant__ EvolvePlsParams Q) {
  const Smem s = carve_smem<kRows>(Q.base);
  clear_counters(s);
  pls_step(Q, s, Q.first + blockIdx.x);
}

}  // namespace

size_t evolve_smem_bytes(int L, int C0max, bool rows_in_smem, int hist_warps) {
  auto al = [](size_t v) { return (v + 15) / 16 * 16; };
  size_t b = kFixedBytes;
  b += 5 * al(sizeof(int) * C0max) + al(sizeof(int) * (C0max + 1));
  b += 2 * al(sizeof(double) * C0max) + al(sizeof(double) * 2 * C0max);
  b += al(sizeof(int) * C0max) * hist_warps;
  if (rows_in_smem) b += kRowArrays * ((static_cast<size_t>(L) + 7) / 8 * 8) * sizeof(uint16_t);
  return b;
}

bool evolve_place(EvolveParams& p, size_t budget, size_t* smem) {
  // per-row arrays in shared memory first, then counters for as many warps as
  // fit: a source more or less at a time is little beside rows' round trips to L2
  for (const bool rows : {true, false}) {
    for (const int warps : {32, 24, 16, 12, 8, 6, 4, 2, 1}) {
      *smem = evolve_smem_bytes(p.L, p.C0max, rows, warps);
      if (*smem > budget) continue;
      p.smem_rows = rows;
      p.hist_warps = warps;
      return true;
    }
  }
  return false;
}

namespace {

template <class Params>
int launch(void (*kernel)(Params), const Params& p, int grid, size_t smem, void* stream) {
  const cudaError_t e = allow_shared_memory(kernel);
  if (e != cudaSuccess) return static_cast<int>(e);
  kernel<<<grid, kThreads, smem, static_cast<cudaStream_t>(stream)>>>(p);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

int evolve_pls_launch(const EvolvePlsParams& q, int grid, size_t smem, void* stream) {
  return launch(q.base.smem_rows ? evolve_pls_kernel<true> : evolve_pls_kernel<false>, q, grid, smem, stream);
}

int evolve_launch(const EvolveParams& p, int grid, size_t smem, void* stream) {
  return launch(p.smem_rows ? evolve_kernel<true> : evolve_kernel<false>, p, grid, smem, stream);
}

}  // namespace kgb
