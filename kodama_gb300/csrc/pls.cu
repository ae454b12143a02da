// PLS-LDA on the device: the float32 SIMPLS + LDA path of the reference
// (plscv.cpp) restated operation for operation, so that predictions are
// bit-identical to PLSLDACV_CPU / PLSLDAPredict_CPU.
//
//   fold statistics   train_center_scale_float        plscv.cpp:669-698
//   standardisation   subset_scale_float              plscv.cpp:409-424
//   fold Gram         densef_gram                     plscv.cpp:436-447
//   cross-product     centered_label_crossprod_*      plscv.cpp:700-731
//   SIMPLS weights    fit_pls_components_from_crossprod_float  plscv.cpp:816-955
//   LDA               fit_predict_pls_lda_streamed_cpu_float   plscv.cpp:1544-1608
//                     fit_lda_from_score_statistics_float      plscv.cpp:1419-1487
//                     cholesky_solve_float                     plscv.cpp:1379-1412
//
// Every float accumulation of the reference is a sequential chain in a fixed
// order (rows ascending, features ascending, classes ascending); each chain
// runs in one thread (or one warp feeding one accumulator) in that order, and
// the parallelism is across chains: slices x features x classes x rows.
// Double accumulators of the reference (dot_float, mat_vec_float,
// t_mat_vec_float, power_norm2_float) sum exact float products; they are
// reproduced by an exact integer sum with a rounding-safety check, and by
// the sequential double sum only when that check cannot decide
// (warp_exact_dot below).  Built with --fmad=false: no multiply-add is fused
// unless written as one.
#include "pls.cuh"
#include "exact_dot.cuh"
#include "launch_count.cuh"
#include "smem_limit.cuh"

#include <float.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

namespace kgb {

namespace {

constexpr int kFollowRows = 8 * kEvalThreads;  // rows from which a warp follows the scores

// ---------------------------------------------------------------------------
// Preparation (label independent)
// ---------------------------------------------------------------------------

// The values of one column down the rows idx[0..n) of a row-major matrix
// (stride ld), in order: each lane's column, 32 rows' loads in flight while the
// 32 before them are taken.  A column is a serial float chain, so its time is
// the loads' latency: with 8 loads in flight per thread and nothing overlapped
// the two walks over 1800 rows took 287 and 300 us, here 62 each.  Warp-collective;
// lanes with !in read column 0.
template <class Take>
__device__ __forceinline__ void column_walk(const float* __restrict__ X, int ld, const int* __restrict__ idx, int n,
                                            int j, bool in, int lane, Take&& take) {
  if (n <= 0) return;
  const float* xj = X + (in ? j : 0);
  float va[32], vb[32];
  auto rows = [&](int t) { return idx[min(t + lane, n - 1)]; };
  auto fetch = [&](float (&v)[32], int ids) {
#pragma unroll
    for (int q = 0; q < 32; ++q) v[q] = xj[static_cast<size_t>(__shfl_sync(kFull, ids, q)) * ld];
  };
  auto use = [&](const float (&v)[32], int left) {
    if (left >= 32) {
#pragma unroll
      for (int q = 0; q < 32; ++q) take(v[q]);
    } else {
#pragma unroll
      for (int q = 0; q < 32; ++q)
        if (q < left) take(v[q]);
    }
  };
  int ids = rows(0);
  fetch(va, ids);
  ids = rows(32);
  for (int t = 0; t < n; t += 64) {
    const int id2 = rows(t + 64);
    if (t + 32 < n) fetch(vb, ids);
    use(va, n - t);
    ids = rows(t + 96);
    if (t + 64 < n) fetch(va, id2);
    if (t + 32 < n) use(vb, n - t - 32);
  }
}

// train_center_scale_float: a lane per (slice, column).
__global__ void __launch_bounds__(64) stats_kernel(PlsPrepArgs a) {
  const int s = blockIdx.x, r = s / a.F, lane = threadIdx.x & 31;
  const int j = (blockIdx.y * 2 + (threadIdx.x >> 5)) * 32 + lane;
  const bool in = j < a.p;
  const float* X = a.X + static_cast<size_t>(r) * a.L * a.p;
  const int b = a.train_off[s], nt = a.train_off[s + 1] - b;
  const int* rows = a.train_idx + b;
  float m = 0.0f;
  if (a.center) {
    column_walk(X, a.p, rows, nt, j, in, lane, [&](float v) { m = __fadd_rn(m, v); });
    const float inv = nt == 0 ? 0.0f : __fdiv_rn(1.0f, static_cast<float>(nt));
    m = __fmul_rn(m, inv);
  }
  float sd = 1.0f;
  if (a.scale) {
    float acc = 1.0f;  // the reference's scale vector starts at 1
    column_walk(X, a.p, rows, nt, j, in, lane, [&](float v) {
      const float d = __fsub_rn(v, m);
      acc = __fadd_rn(acc, __fmul_rn(d, d));
    });
    // std::max(1.0f, float(rows.size() - 1)) with size_t arithmetic
    const float den1 = static_cast<float>(static_cast<unsigned long long>(nt) - 1ull);
    const float den = 1.0f < den1 ? den1 : 1.0f;
    const float q = __fsqrt_rn(__fdiv_rn(acc, den));
    sd = (q > 0.0f && isfinite(q)) ? q : 1.0f;
  }
  if (!in) return;
  a.mean[static_cast<size_t>(s) * a.p + j] = m;
  a.sdev[static_cast<size_t>(s) * a.p + j] = sd;
}

// subset_scale_float for every row of every slice (and, in predict mode, for
// the rows to predict).
__global__ void standardize_kernel(PlsPrepArgs a) {
  // blockIdx.y strides over slices (problems in predict mode), blockIdx.x over
  // rows, threads over columns: no index division per element
  const int S = a.problems * a.F, p = a.p;
  for (int s = blockIdx.y; s < S; s += gridDim.y) {
    const float* X = a.X + static_cast<size_t>(s / a.F) * a.L * p;
    float* Z = a.Z + static_cast<size_t>(s) * a.L * a.zp;
    const float* mu = a.mean + static_cast<size_t>(s) * p;
    const float* sd = a.sdev + static_cast<size_t>(s) * p;
    for (int i = blockIdx.x; i < a.L; i += gridDim.x)
      for (int j = threadIdx.x; j < p; j += blockDim.x)
        Z[static_cast<size_t>(i) * a.zp + j] = __fdiv_rn(__fsub_rn(X[static_cast<size_t>(i) * p + j], mu[j]), sd[j]);
  }
  if (a.Xv == nullptr) return;
  for (int r = blockIdx.y; r < a.problems; r += gridDim.y) {
    const size_t s = static_cast<size_t>(r) * a.F;
    const float* Xv = a.Xv + static_cast<size_t>(r) * a.NV * p;
    float* Zv = a.Zv + static_cast<size_t>(r) * a.NV * a.zp;
    for (int i = blockIdx.x; i < a.NV; i += gridDim.x)
      for (int j = threadIdx.x; j < p; j += blockDim.x)
        Zv[static_cast<size_t>(i) * a.zp + j] =
            __fdiv_rn(__fsub_rn(Xv[static_cast<size_t>(i) * p + j], a.mean[s * p + j]), a.sdev[s * p + j]);
  }
}

// Column sums of the standardised training rows in row order (the x_sum of
// the cross-product, label independent), and each column's largest biased
// exponent over those rows (the fixed-point bound of block_loading).
__global__ void __launch_bounds__(64) xsum_kernel(PlsPrepArgs a) {
  const int s = blockIdx.x, lane = threadIdx.x & 31;
  const int j = (blockIdx.y * 2 + (threadIdx.x >> 5)) * 32 + lane;
  const bool in = j < a.p;
  const int b = a.train_off[s], e = a.train_off[s + 1];
  float acc = 0.0f;
  int ze = 1;
  column_walk(a.Z + static_cast<size_t>(s) * a.L * a.zp, a.zp, a.train_idx + b, e - b, j, in, lane, [&](float v) {
    acc = __fadd_rn(acc, v);
    ze = max(ze, biased_exp1(v));
  });
  if (!in) return;
  a.xsum[static_cast<size_t>(s) * a.p + j] = acc;
  a.zexp[static_cast<size_t>(s) * a.p + j] = ze;
}

// densef_gram: G(j, k) = sum over training rows (ascending) of z_j * z_k, one
// kGramT x kGramT tile of the lower triangle per CTA (blockIdx.y enumerates
// tiles), written to both triangles.  Each thread keeps a 4 x 4 block of
// entries, every one a float chain over the rows in ascending order; rows are
// staged kGramR at a time (padding rows and columns are never added).
constexpr int kGramT = 64;
constexpr int kGramR = 32;
__global__ void __launch_bounds__(256) gram_kernel(PlsPrepArgs a, const uint8_t* want) {
  const int s = blockIdx.x;
  if (!want[s]) return;
  int tile = blockIdx.y, jb = 0;
  while (tile > jb) {
    tile -= jb + 1;
    ++jb;
  }
  const int kb = tile;
  __shared__ __align__(16) float zj[kGramR][kGramT];
  __shared__ __align__(16) float zk[kGramR][kGramT];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float* Zs = a.Z + static_cast<size_t>(s) * a.L * a.zp;
  const int b = a.train_off[s], e = a.train_off[s + 1];
  float acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.0f;
  for (int t0 = b; t0 < e; t0 += kGramR) {
    for (int i = threadIdx.x; i < kGramR * kGramT; i += 256) {
      const int q = i / kGramT, c = i - q * kGramT;
      const int row = t0 + q < e ? a.train_idx[t0 + q] : -1;
      const int cj = jb * kGramT + c, ck = kb * kGramT + c;
      zj[q][c] = (row >= 0 && cj < a.p) ? Zs[static_cast<size_t>(row) * a.zp + cj] : 0.0f;
      zk[q][c] = (row >= 0 && ck < a.p) ? Zs[static_cast<size_t>(row) * a.zp + ck] : 0.0f;
    }
    __syncthreads();
    // rows of the tile past the last column hold no entry (warp-uniform: a
    // warp is two values of ty)
    const int cnt = jb * kGramT + ty * 4 < a.p ? min(kGramR, e - t0) : 0;
    for (int q = 0; q < cnt; ++q) {
      const float4 vj = *reinterpret_cast<const float4*>(&zj[q][ty * 4]);
      const float4 vk = *reinterpret_cast<const float4*>(&zk[q][tx * 4]);
      const float fj[4] = {vj.x, vj.y, vj.z, vj.w}, fk[4] = {vk.x, vk.y, vk.z, vk.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = __fadd_rn(acc[u][v], __fmul_rn(fj[u], fk[v]));
    }
    __syncthreads();
  }
  float* G = a.gram + static_cast<size_t>(s) * a.p * a.p;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int J = jb * kGramT + ty * 4 + u;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int K = kb * kGramT + tx * 4 + v;
      if (J < a.p && K < a.p && K <= J) {
        G[static_cast<size_t>(J) * a.p + K] = acc[u][v];
        G[static_cast<size_t>(K) * a.p + J] = acc[u][v];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Evaluation: one CTA per slice
// ---------------------------------------------------------------------------

constexpr int kMaxNC = 8;      // components per register pass over the rows
constexpr int kMaxComp = 64;   // components of a fit held per row (local array)
constexpr uint16_t kNoPos = 0xffffu;  // tpos of a validation row
constexpr int kTile = 1024;  // floats per warp: two stages of 64 rows x 8 columns, or four of 32 (stream_scores)

struct EvalShared {
  int m, nt, stop, best, lab, fail, queue;
  float rn, inv;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src));
}

// Scores of all rows of a row-major matrix (zp floats apart, zp a multiple of
// 4, 16-byte aligned) for components q0 .. q0 + NQ - 1: out(row, acc) with
// acc[q] = sum over features in order of z(row, j) * W(j, q0 + q), every product
// and sum rounded on its own.  A warp takes 64 rows, two a lane, so that a weight
// read from shared memory serves two rows; eight columns at a time come in with
// cp.async, the next eight while these are used.  The rows are read in memory
// order, validation rows too: their scores are needed for the predictions anyway,
// and no row waits for an index.  A row's two column chunks swap places every four
// rows, so the lanes' 16-byte reads hit all banks.
// With 128-byte loads of 32 indexed rows into a padded transposing tile, eight
// in flight, this phase was 42% of an evaluation at 6750 x 200 rows, 5
// components (3.4 M cycles a slice).
// The batches are dealt to the first `warps` warps; tick() follows every batch of
// a warp.
// One component alone (the fit's) has little to do per step, so it takes 32 rows
// and keeps three steps in flight instead.
constexpr int kScoreRows = 64;
template <int NQ, class Out, class Tick>
__device__ __forceinline__ void stream_scores(const float* __restrict__ base, int zp, int p, int nrows, const float* W,
                                              int ldw, int q0, float* tile, int lane, int warp, int warps, Out&& out,
                                              Tick&& tick) {
  constexpr int R = NQ == 1 ? 1 : 2, kRows = 32 * R, kStage = kRows * 8, kStages = kTile / kStage;
  const int nblk = (p + 7) / 8, nb = (nrows + kRows - 1) / kRows;
  const int mine = warp < nb ? (nb - warp + warps - 1) / warps : 0;
  const int steps = mine * nblk;
  // the next load: its batch, column block, the batch's first row and this lane's
  // offsets from there (the rows to predict have no limit that keeps row * zp below
  // 2^31; a batch has)
  int lb = warp, lk = 0;
  const float* from = base;
  int src[2 * R];
  const int lr = lane >> 1, lc = (lane & 1) * 4;
  float* const dst = tile + lr * 8 + (lc ^ (((lr >> 2) & 1) << 2));  // 16 rows apart, the swap repeats
  auto load = [&](int step) {
    if (step < steps) {
      if (lk == 0) {
        from = base + static_cast<size_t>(lb * kRows) * zp;
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) src[i] = min(i * 16 + lr, nrows - 1 - lb * kRows) * zp + lc;
      }
      float* to = dst + (step & (kStages - 1)) * kStage;
      if (lk * 8 + lc < zp) {
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) cp_async16(to + i * 128, from + (src[i] + lk * 8));
      }
      if (++lk == nblk) {
        lk = 0;
        lb += warps;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  float acc[R][NQ];
#pragma unroll
  for (int q = 0; q < NQ * R; ++q) acc[q / NQ][q % NQ] = 0.0f;
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) load(i);
  const bool wide = NQ >= 4 && ldw % 4 == 0;  // whole vectors of weights
  int b = warp, k = 0;
  for (int step = 0; step < steps; ++step) {
    load(step + kStages - 1);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 1));
    __syncwarp();
    const float* t = tile + (step & (kStages - 1)) * kStage + lane * 8;
    const int first = ((lane >> 2) & 1) << 2;
    const float* w = W + static_cast<size_t>(k * 8) * ldw + q0;
    float v[R][4];
    auto column = [&](int e) {
      float wq[NQ];
      if (wide) {
#pragma unroll
        for (int q = 0; q < NQ; q += 4) {
          const float4 w4 = *reinterpret_cast<const float4*>(w + q);
          wq[q] = w4.x;
          if (q + 1 < NQ) wq[q + 1] = w4.y;
          if (q + 2 < NQ) wq[q + 2] = w4.z;
          if (q + 3 < NQ) wq[q + 3] = w4.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < NQ; ++q) wq[q] = w[q];
      }
      w += ldw;
      // (packed f32x2 operations are no use here: the assembler contracts
      // a packed product and sum into one rounding)
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
#pragma unroll
        for (int h = 0; h < R; ++h) acc[h][q] = __fadd_rn(acc[h][q], __fmul_rn(v[h][e], wq[q]));
      }
    };
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int h = 0; h < R; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(t + h * 256 + (first ^ (4 * c)));
        v[h][0] = x.x;
        v[h][1] = x.y;
        v[h][2] = x.z;
        v[h][3] = x.w;
      }
      const int left = p - k * 8 - 4 * c;
      if (left >= 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e) column(e);
      } else {
#pragma unroll
        for (int e = 0; e < 3; ++e)
          if (e < left) column(e);
      }
    }
    __syncwarp();
    if (++k == nblk) {
#pragma unroll
      for (int h = 0; h < R; ++h)
        if (b * kRows + 32 * h + lane < nrows) out(b * kRows + 32 * h + lane, acc[h]);
#pragma unroll
      for (int q = 0; q < NQ * R; ++q) acc[q / NQ][q % NQ] = 0.0f;
      k = 0;
      b += warps;
      tick();
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// Calls go(std::integral_constant<int, nc>) for nc of 1 to 8.
template <class Go>
__device__ __forceinline__ void with_components(int nc, Go&& go) {
  switch (nc) {
    case 1: go(std::integral_constant<int, 1>{}); break;
    case 2: go(std::integral_constant<int, 2>{}); break;
    case 3: go(std::integral_constant<int, 3>{}); break;
    case 4: go(std::integral_constant<int, 4>{}); break;
    case 5: go(std::integral_constant<int, 5>{}); break;
    case 6: go(std::integral_constant<int, 6>{}); break;
    case 7: go(std::integral_constant<int, 7>{}); break;
    default: go(std::integral_constant<int, 8>{}); break;
  }
}

// out(row, q, score) for every component q of nc, kMaxNC at a time.
template <class Out, class Tick>
__device__ __forceinline__ void stream_all_scores(const float* __restrict__ base, int zp, int p, int nrows,
                                                  const float* W, int ldw, int nc, float* tile, int lane, int warp,
                                                  int warps, Out&& out, Tick&& tick) {
  for (int q0 = 0; q0 < nc; q0 += kMaxNC) {
    auto go = [&](auto nq) {
      constexpr int NQ = decltype(nq)::value;
      stream_scores<NQ>(base, zp, p, nrows, W, ldw, q0, tile, lane, warp, warps, [&](int row, const float (&acc)[NQ]) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) out(row, q0 + q, acc[q]);
      }, tick);
    };
    with_components(min(kMaxNC, nc - q0), go);
  }
}

// A barrier of the whole evaluation block that the scoring warps and the one that
// follows them meet at from different places of the code, which __syncthreads does
// not allow.
__device__ __forceinline__ void round_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEvalThreads) : "memory"); }

// acc plus the lanes' 32 values in lane order, the same in every lane.  The
// shuffles are issued together, so the chain runs at the speed of its adds; with
// a condition around each add it ran at shuffle latency, 40 cycles a value.
// Values to leave out are passed as +0: a sum that starts at +0 is never -0, so
// adding +0 changes nothing.
__device__ __forceinline__ float warp_add32(float acc, float v) {
  float t[32];
#pragma unroll
  for (int q = 0; q < 32; ++q) t[q] = __shfl_sync(kFull, v, q);
#pragma unroll
  for (int q = 0; q < 32; ++q) acc = __fadd_rn(acc, t[q]);
  return acc;
}

// Sequential float chain over positions b..e-1 of a row-major matrix
// (stride ld, column c) counting only the positions whose flag is set,
// warp-cooperative: each 32-position group is loaded D groups ahead, then
// every lane adds the group's values in position order.
template <int D>
__device__ float warp_masked_chain(const float* __restrict__ m, int ld, int c, const uint8_t* __restrict__ ok, int b,
                                   int e, int lane) {
  float acc = 0.0f;
  if (b >= e) return acc;
  float v[D];
  // flag and value are loaded side by side: a load behind a test of the flag
  // would wait for it
  auto fetch = [&](int i) {
    const int k = min(i, e - 1);
    const float x = m[static_cast<size_t>(k) * ld + c];
    const bool take = ok[k] != 0;
    return i < e && take ? x : 0.0f;
  };
#pragma unroll
  for (int g = 0; g < D; ++g) v[g] = fetch(b + g * 32 + lane);
  for (int base = b; base < e; base += 32 * D) {
#pragma unroll
    for (int g = 0; g < D; ++g) {
      const int gb = base + g * 32;
      if (gb >= e) break;
      const float cur = v[g];
      v[g] = fetch(gb + D * 32 + lane);
      acc = warp_add32(acc, cur);
    }
  }
  return acc;
}

// Per lane, acc and the sequential float chain sum_i t(i, ca) * t(i, cb) over the
// n rows of a row-major matrix of nc columns.  Batches of 256 / nc rows come into
// a ring of four in `buf` (kTile floats), three ahead; the products of the next
// eight rows are formed while those of the last eight are added (+0 past the
// end, as in warp_add32).
__device__ float warp_score_products(float acc, const float* t, int n, int nc, int ca, int cb, float* buf, int lane) {
  static_assert(kTile >= 4 * 256, "batch ring");
  const int rows = 256 / nc;  // nc <= 64: at least 4 rows
  const int nb = (n + rows - 1) / rows;
  auto fetch = [&](int b) {
    if (b < nb) {
      const int total = min(rows, n - b * rows) * nc;
      const float* src = t + static_cast<size_t>(b) * rows * nc;
      float* dst = buf + (b & 3) * 256;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u * 32 + lane < total)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                           static_cast<unsigned>(__cvta_generic_to_shared(dst + u * 32 + lane))),
                       "l"(src + u * 32 + lane));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  for (int b = 0; b < 3; ++b) fetch(b);
  for (int b = 0; b < nb; ++b) {
    asm volatile("cp.async.wait_group 2;\n" ::);
    __syncwarp();
    fetch(b + 3);  // into the slot whose rows were added before the barrier
    const float* r = buf + (b & 3) * 256;
    const int cn = min(rows, n - b * rows);
    float pr[8];
    auto form = [&](int i0) {
      if (i0 + 8 <= cn) {
#pragma unroll
        for (int q = 0; q < 8; ++q) pr[q] = __fmul_rn(r[(i0 + q) * nc + ca], r[(i0 + q) * nc + cb]);
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          pr[q] = i0 + q < cn ? __fmul_rn(r[(i0 + q) * nc + ca], r[(i0 + q) * nc + cb]) : 0.0f;
      }
    };
    form(0);
    for (int i0 = 0; i0 < cn; i0 += 8) {
      float cur[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) cur[q] = pr[q];
      form(i0 + 8);
#pragma unroll
      for (int q = 0; q < 8; ++q) acc = __fadd_rn(acc, cur[q]);
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  return acc;
}

// warp_score_products for up to eight components.  Batches of 32 rows come in by
// columns (of 36 floats, so that the lanes' columns start in different banks) and
// a lane reads eight rows of its two columns in four vectors; missing rows are
// +0.  13 cycles a row, 4.6 of them the sum's chain; with rows of nc floats, a
// length known at run time only and a load per value it was 40, and the scores
// waited for it.
template <int NC>
__device__ __forceinline__ float warp_score_products_by_column(float acc, const float* t, int n, int ca, int cb,
                                                               float* buf, int lane) {
  constexpr int kPitch = 36, kSlot = NC * kPitch, kSlots = 4 * kSlot <= kTile ? 4 : 3;
  static_assert(kSlots * kSlot <= kTile, "batch ring");
  const int nb = (n + 31) / 32;
  int in = 0, out = 0;  // slots
  auto fetch = [&](int b) {
    if (b < nb) {
      const int total = min(32, n - b * 32) * NC;
      const float* src = t + static_cast<size_t>(b) * (32 * NC);
      float* dst = buf + in * kSlot;
#pragma unroll
      for (int u = 0; u < NC; ++u) {
        const int i = u * 32 + lane;
        float* to = dst + (i % NC) * kPitch + i / NC;
        if (i < total)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                           static_cast<unsigned>(__cvta_generic_to_shared(to))),
                       "l"(src + i));
        else
          *to = 0.0f;
      }
      in = in + 1 < kSlots ? in + 1 : 0;
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  for (int b = 0; b < kSlots - 1; ++b) fetch(b);
  for (int b = 0; b < nb; ++b) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kSlots - 2));
    __syncwarp();
    fetch(b + kSlots - 1);  // into the slot whose rows were added before the barrier
    const float4* x = reinterpret_cast<const float4*>(buf + out * kSlot + ca * kPitch);
    const float4* y = reinterpret_cast<const float4*>(buf + out * kSlot + cb * kPitch);
    out = out + 1 < kSlots ? out + 1 : 0;
    float pr[8];
    auto form = [&](int i) {
      const float4 x0 = x[i], x1 = x[i + 1], y0 = y[i], y1 = y[i + 1];
      pr[0] = __fmul_rn(x0.x, y0.x);
      pr[1] = __fmul_rn(x0.y, y0.y);
      pr[2] = __fmul_rn(x0.z, y0.z);
      pr[3] = __fmul_rn(x0.w, y0.w);
      pr[4] = __fmul_rn(x1.x, y1.x);
      pr[5] = __fmul_rn(x1.y, y1.y);
      pr[6] = __fmul_rn(x1.z, y1.z);
      pr[7] = __fmul_rn(x1.w, y1.w);
    };
    form(0);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float cur[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) cur[q] = pr[q];
      if (i + 2 < 8) form(i + 2);
#pragma unroll
      for (int q = 0; q < 8; ++q) acc = __fadd_rn(acc, cur[q]);
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  return acc;
}

__device__ __forceinline__ float score_products(float acc, const float* t, int n, int nc, int ca, int cb, float* buf,
                                                int lane) {
  if (nc > kMaxNC) return warp_score_products(acc, t, n, nc, ca, cb, buf, lane);
  with_components(nc, [&](auto c) {
    acc = warp_score_products_by_column<decltype(c)::value>(acc, t, n, ca, cb, buf, lane);
  });
  return acc;
}

// The sums of positions b..e-1 of a row-major matrix of NC columns whose flag is
// set, in order, every column a chain of its own: lane q < NC returns column q's.
// The lanes bring in a row each (two groups ahead of the one being added) and
// pass them by columns through `buf`; a row left out is +0 (warp_add32).  A
// warp per class and column, and a shuffle a value, took 50 cycles a row and column.
template <int NC>
__device__ __forceinline__ float warp_masked_columns(const float* __restrict__ m, const uint8_t* __restrict__ ok,
                                                     int b, int e, float* buf, int lane) {
  constexpr int kPitch = 36;
  float acc = 0.0f, next[2][NC];
  // flag and values are loaded side by side: loads behind a test of the flag
  // would wait for it
  auto fetch = [&](int i, float (&to)[NC]) {
    const int k = min(i, e - 1);
    const bool take = i < e && ok[k] != 0;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const float x = m[static_cast<size_t>(k) * NC + q];
      to[q] = take ? x : 0.0f;
    }
  };
  if (b >= e) return acc;
  fetch(b + lane, next[0]);
  fetch(b + 32 + lane, next[1]);
  const float4* mine = reinterpret_cast<const float4*>(buf + min(lane, NC - 1) * kPitch);
  for (int g = b; g < e; g += 32) {
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      buf[q * kPitch + lane] = next[0][q];
      next[0][q] = next[1][q];
    }
    __syncwarp();
    if (g + 64 < e) fetch(g + 64 + lane, next[1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 v = mine[i];
      acc = __fadd_rn(acc, v.x);
      acc = __fadd_rn(acc, v.y);
      acc = __fadd_rn(acc, v.z);
      acc = __fadd_rn(acc, v.w);
    }
    __syncwarp();
  }
  return acc;
}

// Label cross-product of every slice: column `code` of s_raw is the sum of the
// class's standardised training rows (ascending) less its share of the column
// sums (centered_label_crossprod, plscv.cpp:700-731).
//
// cross_stream_kernel: a CTA per (slice, 32 features) streams the rows in memory
// order through a ring of 64-row tiles (cp.async, three ahead) and adds each row
// to its class's sums in shared memory.  Warp w owns the codes c & 7 == w, so a
// class's rows are added by one warp in ascending order.  All features of a row
// are read by neighbouring CTAs at about the same time, so the launch runs at
// memory speed (500 slices of 7500 x 200: 3 GB).  The classes' own row lists
// (cross_kernel) read the same lines in random order behind two index loads:
// 2.6 to 2.9 ms a launch there, 0.95 ms here; inside the evaluation kernel
// the lists cost 2.1 M cycles a slice, 60% of it.  The lists remain for more
// classes than shared memory holds sums for.
constexpr int kStreamThreads = 256;
constexpr int kStreamRows = 64;
constexpr int kStreamSlots = 4;

size_t cross_stream_smem(int C) {
  return sizeof(float) * (static_cast<size_t>(C) * 32 + kStreamSlots * kStreamRows * 32) + sizeof(int) * C;
}

__global__ void __launch_bounds__(kStreamThreads) cross_stream_kernel(PlsEvalArgs a) {
  extern __shared__ __align__(16) float xsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = a.p, C = a.C0max, L = a.L;
  const int j0 = blockIdx.x * 32, j = j0 + lane;
  float* ring = xsm;                                          // [slot][row][32]
  float* acc = ring + kStreamSlots * kStreamRows * 32;        // [code][32]
  int* cnt = reinterpret_cast<int*>(acc + static_cast<size_t>(C) * 32);
  const int ntiles = (L + kStreamRows - 1) / kStreamRows;
  for (int s = a.first * a.F + blockIdx.y; s < (a.first + a.problems) * a.F; s += gridDim.y) {
    const int r = s / a.F, f = s % a.F;
    const int* coff = a.class_off + static_cast<size_t>(r) * (C + 1);
    const uint16_t* lab = a.labels + static_cast<size_t>(r) * L;
    const uint8_t* fold = a.predict_mode ? nullptr : a.folds + static_cast<size_t>(r) * L;
    const float* Zs = a.Z + static_cast<size_t>(s) * L * a.zp;
    auto load = [&](int t) {
      if (t < ntiles) {
        float* dst = ring + (t & (kStreamSlots - 1)) * kStreamRows * 32;
#pragma unroll
        for (int i = 0; i < kStreamRows / 32; ++i) {
          const int rr = i * 32 + (threadIdx.x >> 3), c = 4 * (threadIdx.x & 7);
          const int row = min(t * kStreamRows + rr, L - 1);
          if (j0 + c < a.zp) cp_async16(dst + rr * 32 + c, Zs + static_cast<size_t>(row) * a.zp + j0 + c);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    // the codes and folds of a tile's rows, a lane each: fetched two tiles
    // ahead, and looked at only when their tile is added
    constexpr int H = kStreamRows / 32;
    struct RowInfo {
      uint16_t code[H];
      uint8_t fold[H];
    };
    auto fetch_rows = [&](int t, RowInfo& ri) {
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int row = min(t * kStreamRows + h * 32 + lane, L - 1);
        ri.code[h] = lab[row];
        ri.fold[h] = fold != nullptr ? fold[row] : 0;
      }
    };
    for (int t = 0; t < kStreamSlots - 1; ++t) load(t);
    for (int e = threadIdx.x; e < C * 32; e += kStreamThreads) acc[e] = 0.0f;
    for (int c = threadIdx.x; c < C; c += kStreamThreads) cnt[c] = coff[c + 1] - coff[c];
    __syncthreads();
    if (!a.predict_mode) {
      const int* vidx = a.val_idx + a.val_off[s];
      const int nv = a.val_off[s + 1] - a.val_off[s];
      for (int v = threadIdx.x; v < nv; v += kStreamThreads) atomicSub(&cnt[lab[vidx[v]]], 1);
    }
    RowInfo n1, n2;
    fetch_rows(0, n1);
    fetch_rows(1, n2);
    for (int t = 0; t < ntiles; ++t) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kStreamSlots - 2));
      __syncthreads();  // tile t has landed for every thread; tile t - 1 is done with
      load(t + kStreamSlots - 1);
      // this lane's rows: the code if it trains the slice and belongs to this
      // warp, else -1
      int code[H];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int row = t * kStreamRows + h * 32 + lane;
        const bool mine = row < L && (n1.code[h] & 7) == warp && (fold == nullptr || n1.fold[h] != f);
        code[h] = mine ? n1.code[h] : -1;
      }
      n1 = n2;
      fetch_rows(t + 2, n2);
      const float* tile = ring + (t & (kStreamSlots - 1)) * kStreamRows * 32 + lane;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        unsigned m = __ballot_sync(kFull, code[h] >= 0);
        while (m != 0u) {
          // two rows at a time, so that one's loads cover the other's add
          const int q1 = __ffs(m) - 1;
          m &= m - 1u;
          const bool two = m != 0u;
          const int q2 = two ? __ffs(m) - 1 : q1;
          m &= m - 1u;
          const int k1 = __shfl_sync(kFull, code[h], q1), k2 = __shfl_sync(kFull, code[h], q2);
          const float v1 = tile[(h * 32 + q1) * 32], v2 = tile[(h * 32 + q2) * 32];
          float a1 = acc[k1 * 32 + lane], a2 = acc[k2 * 32 + lane];
          a1 = __fadd_rn(a1, v1);
          if (two && k1 == k2) {
            a1 = __fadd_rn(a1, v2);
          } else if (two) {
            a2 = __fadd_rn(a2, v2);
            acc[k2 * 32 + lane] = a2;
          }
          acc[k1 * 32 + lane] = a1;
        }
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    const int nt = a.train_off[s + 1] - a.train_off[s];
    const float inv_n = nt > 0 ? __fdiv_rn(1.0f, static_cast<float>(nt)) : 0.0f;
    const float xs = j < p ? a.xsum[static_cast<size_t>(s) * p + j] : 0.0f;
    for (int c = warp; c < C; c += kStreamThreads / 32) {
      const float y_mean = __fmul_rn(static_cast<float>(cnt[c]), inv_n);
      if (j < p && cnt[c] > 0)
        a.s_raw[(static_cast<size_t>(s) * C + c) * p + j] = __fsub_rn(acc[c * 32 + lane], __fmul_rn(y_mean, xs));
    }
    __syncthreads();
  }
}

// The same from the classes' row lists: a warp per (class, 32 features) with the
// chain in a register and 32 to 64 rows' loads in flight.
constexpr int kCrossThreads = 256;
__global__ void __launch_bounds__(kCrossThreads, 2) cross_kernel(PlsEvalArgs a) {
  const int lane = threadIdx.x & 31, p = a.p, C = a.C0max, JB = (p + 31) / 32;
  for (int s = a.first * a.F + blockIdx.y; s < (a.first + a.problems) * a.F; s += gridDim.y) {
    const int r = s / a.F, f = s % a.F;
    const int* coff = a.class_off + static_cast<size_t>(r) * (C + 1);
    const uint16_t* crow = a.class_rows + static_cast<size_t>(r) * a.L;
    const uint8_t* fold = a.predict_mode ? nullptr : a.folds + static_cast<size_t>(r) * a.L;
    const float* Zs = a.Z + static_cast<size_t>(s) * a.L * a.zp;
    const int nt = a.train_off[s + 1] - a.train_off[s];
    const float inv_n = nt > 0 ? __fdiv_rn(1.0f, static_cast<float>(nt)) : 0.0f;
    const int warps = gridDim.x * (kCrossThreads / 32);
    for (int item = blockIdx.x * (kCrossThreads / 32) + (threadIdx.x >> 5); item < C * JB; item += warps) {
      const int code = item / JB, j = (item - code * JB) * 32 + lane;
      const int b = coff[code], n = coff[code + 1] - b;
      if (n == 0) continue;
      const float* zj = Zs + (j < p ? j : 0);
      float acc = 0.0f, va[32], vb[32];
      int count = 0;
      // rows t .. t + 31 of the class, -1 = past the end or in this fold
      auto rows = [&](int t) {
        int row = t + lane < n ? static_cast<int>(crow[b + t + lane]) : -1;
        if (row >= 0 && fold != nullptr && fold[row] == f) row = -1;
        return row;
      };
      auto fetch = [&](float (&v)[32], int ids) {
  #pragma unroll
        for (int q = 0; q < 32; ++q) {
          const int row = __shfl_sync(kFull, ids, q);
          v[q] = row >= 0 ? zj[static_cast<size_t>(row) * a.zp] : 0.0f;
        }
      };
      auto use = [&](const float (&v)[32], int ids) {
        const unsigned msk = __ballot_sync(kFull, ids >= 0);
        count += __popc(msk);
  #pragma unroll
        for (int q = 0; q < 32; ++q)
          if ((msk >> q) & 1u) acc = __fadd_rn(acc, v[q]);
      };
      int ia = rows(0), ib = rows(32);
      fetch(va, ia);
      for (int t = 0; t < n; t += 64) {
        if (t + 32 < n) fetch(vb, ib);
        const int ic = rows(t + 64), id = rows(t + 96);
        use(va, ia);
        if (t + 64 < n) fetch(va, ic);
        if (t + 32 < n) use(vb, ib);
        ia = ic;
        ib = id;
      }
      if (j < p) {
        const float y_mean = __fmul_rn(static_cast<float>(count), inv_n);
        a.s_raw[(static_cast<size_t>(s) * C + code) * p + j] =
            __fsub_rn(acc, __fmul_rn(y_mean, a.xsum[static_cast<size_t>(s) * p + j]));
      }
    }
  }
}

// kCtas: CTAs an SM, the bound on registers: two hide each other's latencies
// (64 registers, some spilled); where there are no more slices than SMs there is
// only one, with 128.
template <int kCtas>
__global__ void __launch_bounds__(kEvalThreads, kCtas) eval_kernel(PlsEvalArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int s = a.first * a.F + blockIdx.x, r = s / a.F, f = s % a.F;
  const int p = a.p, zp = a.zp, L = a.L, C = a.C0max, NCm = a.requested, ldw = a.ldw;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  EvalShared& sh = *reinterpret_cast<EvalShared*>(smem);
  size_t off = 64;
  auto carve = [&](size_t bytes) {
    unsigned char* q = smem + off;
    off += (bytes + 15) / 16 * 16;
    return q;
  };
  int* cnt = reinterpret_cast<int*>(carve(sizeof(int) * C));
  int* klist = reinterpret_cast<int*>(carve(sizeof(int) * C));
  float* w = reinterpret_cast<float*>(carve(sizeof(float) * p));
  float* ld = reinterpret_cast<float*>(carve(sizeof(float) * p));
  float* pw = reinterpret_cast<float*>(carve(sizeof(float) * p));
  float* tv = reinterpret_cast<float*>(carve(sizeof(float) * C));
  float* Wsm = reinterpret_cast<float*>(carve(sizeof(float) * p * ldw));
  float* Vsm = reinterpret_cast<float*>(carve(sizeof(float) * p * ldw));
  float* cs = reinterpret_cast<float*>(carve(sizeof(float) * C * NCm));
  float* cp = reinterpret_cast<float*>(carve(sizeof(float) * NCm * NCm));
  float* pooled = reinterpret_cast<float*>(carve(sizeof(float) * NCm * NCm));
  float* Lc = reinterpret_cast<float*>(carve(sizeof(float) * NCm * NCm));
  float* sol = reinterpret_cast<float*>(carve(sizeof(float) * NCm * C));
  float* lin = reinterpret_cast<float*>(carve(sizeof(float) * C * NCm));
  float* cst = reinterpret_cast<float*>(carve(sizeof(float) * C));
  double* ssum = reinterpret_cast<double*>(carve(sizeof(double) * NCm));  // PLS-DA score sums
  // shared region: the cross-product (when it fits) and the score tiles,
  // which overlap it unless a slice of the launch computes scores during the
  // fit (no fold Gram)
  float* region = reinterpret_cast<float*>(carve(0));
  // (16-byte copies land in the tiles)
  float* tiles = (a.s_in_smem && a.tiles_after_s) ? region + (static_cast<size_t>(p) * C + 3) / 4 * 4 : region;

  const uint16_t* lab = a.labels + static_cast<size_t>(r) * L;
  const int* coff = a.class_off + static_cast<size_t>(r) * (C + 1);
  const uint16_t* crow = a.class_rows + static_cast<size_t>(r) * L;
  const uint8_t* fold = a.predict_mode ? nullptr : a.folds + static_cast<size_t>(r) * L;
  const float* Zs = a.Z + static_cast<size_t>(s) * L * zp;
  const int tb = a.train_off[s], te = a.train_off[s + 1];
  const int nv = a.predict_mode ? a.NV : a.val_off[s + 1] - a.val_off[s];
  const int* vidx = a.predict_mode ? nullptr : a.val_idx + a.val_off[s];
  uint16_t* pred = a.pred + static_cast<size_t>(r) * (a.predict_mode ? a.NV : L);
  const float* vbase = a.predict_mode ? a.Zv + static_cast<size_t>(r) * a.NV * zp : Zs;

  // --- fold classes: codes with training rows, ascending -------------------
  for (int c = threadIdx.x; c < C; c += kEvalThreads) cnt[c] = coff[c + 1] - coff[c];
  __syncthreads();
  if (!a.predict_mode)
    for (int v = threadIdx.x; v < nv; v += kEvalThreads) atomicSub(&cnt[lab[vidx[v]]], 1);
  __syncthreads();
  if (warp == kEvalWarps - 1) {
    int m = 0;
    for (int c0 = 0; c0 < C; c0 += 32) {
      const bool in = c0 + lane < C && cnt[c0 + lane] > 0;
      const unsigned b = __ballot_sync(kFull, in);
      if (in) klist[m + __popc(b & ((1u << lane) - 1u))] = c0 + lane;
      m += __popc(b);
    }
    if (lane == 0) {
      sh.m = m;
      sh.nt = te - tb;
      sh.queue = 0;
    }
  }
  // class-list position of every row, whether that position trains the slice,
  // and every row's position among the training rows
  uint16_t* posof = a.pos + static_cast<size_t>(s) * L;
  uint8_t* posok = a.posok + static_cast<size_t>(s) * L;
  for (int i0 = threadIdx.x; i0 < L; i0 += 4 * kEvalThreads) {
    int row[4];
    bool train[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) row[q] = crow[min(i0 + q * kEvalThreads, L - 1)];
#pragma unroll
    for (int q = 0; q < 4; ++q) train[q] = fold == nullptr || fold[row[q]] != f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + q * kEvalThreads;
      if (i >= L) break;
      posof[row[q]] = static_cast<uint16_t>(i);
      posok[i] = train[q] ? 1 : 0;
    }
  }
  uint16_t* tpos = a.tpos + static_cast<size_t>(s) * L;
  if (fold != nullptr)
    for (int i = threadIdx.x; i < nv; i += kEvalThreads) tpos[vidx[i]] = kNoPos;
  for (int t0 = threadIdx.x; t0 < te - tb; t0 += 4 * kEvalThreads) {
    int row[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) row[q] = a.train_idx[tb + min(t0 + q * kEvalThreads, te - tb - 1)];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (t0 + q * kEvalThreads < te - tb) tpos[row[q]] = static_cast<uint16_t>(t0 + q * kEvalThreads);
  }
  __syncthreads();
  const int m = sh.m, nt = sh.nt;
  auto predict_all = [&](int code) {
    for (int v = threadIdx.x; v < nv; v += kEvalThreads)
      pred[a.predict_mode ? v : vidx[v]] = static_cast<uint16_t>(code);
  };
  if (m <= 1 || nt == 0) {
    // one training class: it is every prediction (labels.front() without one);
    // a slice without training rows but with classes is padding, with nothing
    // to predict
    predict_all(m >= 1 ? klist[0] : lab[0]);
    if (threadIdx.x == 0) a.eval_comp[s] = 1;
    return;
  }

  // --- label cross-product S (p x m), column k = fold class k, formed by
  // cross_kernel for every code
  float* S = a.s_in_smem ? region : a.s_scr + static_cast<size_t>(s) * p * C;
  for (int k = warp; k < m; k += kEvalWarps) {
    const float* src = a.s_raw + (static_cast<size_t>(s) * C + klist[k]) * p;
    if (a.s_in_smem && p % 4 == 0) {
      for (int j = 4 * lane; j < p; j += 128) cp_async16(S + j + static_cast<size_t>(k) * p, src + j);
    } else {
      for (int j = lane; j < p; j += 32) S[j + static_cast<size_t>(k) * p] = src[j];
    }
  }
  asm volatile("cp.async.wait_all;\n" ::);
  __syncthreads();

  // --- SIMPLS weights ------------------------------------------------------
  const int maxr = min(min(a.max_components, p), max(1, nt - 1));
  const bool gram = a.gram != nullptr && a.use_gram[s];
  const float* G = gram ? a.gram + static_cast<size_t>(s) * p * p : nullptr;
  float* scv = a.sc + static_cast<size_t>(s) * L;
  const int* tix = a.train_idx + tb;
  int fitted = 0;
  for (int comp = 0; comp < maxr; ++comp) {
    for (int j = threadIdx.x; j < p; j += kEvalThreads) w[j] = comp == 0 ? a.w0[j] : pw[j];
    __syncthreads();
    // two power iterations (a second pass only for the strongest-column retry)
    for (int pass = 0; pass < 2; ++pass) {
      for (int it = 0; it < 2; ++it) {
        group_seq_dots(m, p, lane, warp, [&](int c, int k, float& x, float& y) {
          x = S[k + static_cast<size_t>(c) * p];
          y = w[k];
        }, [&](int c, float v) { tv[c] = v; });
        __syncthreads();
        group_seq_dots(p, m, lane, warp, [&](int j, int k, float& x, float& y) {
          x = S[j + static_cast<size_t>(k) * p];
          y = tv[k];
        }, [&](int j, float v) { w[j] = v; });
        __syncthreads();
      }
      if (warp == 0) {
        const float rn = warp_power_norm(w, p, lane);
        if (lane == 0) {
          sh.rn = rn;
          sh.best = -1;
          if (pass == 0 && comp == 0 && !(isfinite(rn) && rn > 1.0e-10f)) {
            // retry on the response column with the largest norm (rare: double sums)
            double bn = 0.0;
            int best = -1;
            for (int k = 0; k < m; ++k) {
              double ns = 0.0;
              for (int j = 0; j < p; ++j) {
                const double v = static_cast<double>(S[j + static_cast<size_t>(k) * p]);
                ns = fma(v, v, ns);
              }
              if (isfinite(ns) && ns > bn) {
                bn = ns;
                best = k;
              }
            }
            if (best >= 0 && bn > 1.0e-20) sh.best = best;
          }
        }
      }
      __syncthreads();
      if (sh.best < 0) break;
      const int best = sh.best;
      for (int j = threadIdx.x; j < p; j += kEvalThreads) w[j] = S[j + static_cast<size_t>(best) * p];
      __syncthreads();
    }
    const float rn = sh.rn;
    if (!(isfinite(rn) && rn > 1.0e-10f)) break;
    for (int j = threadIdx.x; j < p; j += kEvalThreads) w[j] = __fdiv_rn(w[j], rn);
    __syncthreads();
    if (gram) {
      group_seq_dots(p, p, lane, warp, [&](int i, int k, float& x, float& y) {
        x = G[static_cast<size_t>(i) * p + k];
        y = w[k];
      }, [&](int i, float v) { ld[i] = v; });
      __syncthreads();
      if (warp == 0) {
        const float sns = warp_seq_dot(p, [&](int k, float& x, float& y) {
          x = w[k];
          y = ld[k];
        }, lane);
        if (lane == 0) {
          sh.stop = !(isfinite(sns) && sns > 1.0e-20f);
          sh.inv = sh.stop ? 0.0f : __fdiv_rn(1.0f, __fsqrt_rn(sns));
        }
      }
      __syncthreads();
      if (sh.stop) break;
      const float inv = sh.inv;
      for (int j = threadIdx.x; j < p; j += kEvalThreads) {
        w[j] = __fmul_rn(w[j], inv);
        ld[j] = __fmul_rn(ld[j], inv);
      }
      __syncthreads();
    } else {
      // scores of the training rows, their norm, loading = X^T scores
      stream_scores<1>(Zs, zp, p, L, w, 1, 0, tiles + warp * kTile, lane, warp, kEvalWarps,
                       [&](int row, const float (&v)[1]) {
        const int t = tpos[row];
        if (t != kNoPos) scv[t] = v[0];
      }, []() {});
      __syncthreads();
      const float d = block_norm2(scv, nt, tiles, lane, warp);
      if (threadIdx.x == 0) {
        const float sn = __fsqrt_rn(0.0f < d ? d : 0.0f);
        sh.stop = !(isfinite(sn) && sn > 1.0e-10f);
        sh.inv = sh.stop ? 0.0f : __fdiv_rn(1.0f, sn);
      }
      __syncthreads();
      if (sh.stop) break;
      const float inv = sh.inv;
      for (int t = threadIdx.x; t < nt; t += kEvalThreads) scv[t] = __fmul_rn(scv[t], inv);
      for (int j = threadIdx.x; j < p; j += kEvalThreads) w[j] = __fmul_rn(w[j], inv);
      __syncthreads();
      block_loading(Zs, zp, p, tix, nt, scv, a.zexp + static_cast<size_t>(s) * p, ld, tiles, lane, warp);
    }
    for (int j = threadIdx.x; j < p; j += kEvalThreads) pw[j] = w[j];
    // Gram-Schmidt against the previous loadings
    for (int q = 0; q < comp; ++q) {
      if (warp == 0) {
        // one chain over the features: the lanes form 32 products, every lane
        // adds them in order
        float proj = 0.0f;
        for (int j0 = 0; j0 < p; j0 += 32) {
          const int j = j0 + lane;
          const float pr = j < p ? __fmul_rn(Vsm[static_cast<size_t>(j) * ldw + q], ld[j]) : 0.0f;
          proj = warp_add32(proj, pr);
        }
        if (lane == 0) sh.inv = proj;
      }
      __syncthreads();
      const float proj = sh.inv;
      for (int j = threadIdx.x; j < p; j += kEvalThreads)
        ld[j] = __fsub_rn(ld[j], __fmul_rn(proj, Vsm[static_cast<size_t>(j) * ldw + q]));
      __syncthreads();
    }
    if (warp == 0) {
      const float d = warp_seq_dot(p, [&](int k, float& x, float& y) {
        x = ld[k];
        y = ld[k];
      }, lane);
      if (lane == 0) {
        const float ln = __fsqrt_rn(0.0f < d ? d : 0.0f);
        sh.stop = !(isfinite(ln) && ln > 1.0e-10f);
        sh.inv = ln;
      }
    }
    __syncthreads();
    if (sh.stop) break;
    const float ln = sh.inv;
    for (int j = threadIdx.x; j < p; j += kEvalThreads) {
      ld[j] = __fdiv_rn(ld[j], ln);
      Wsm[static_cast<size_t>(j) * ldw + comp] = w[j];
      Vsm[static_cast<size_t>(j) * ldw + comp] = ld[j];
    }
    __syncthreads();
    // deflate the cross-product
    for (int k = threadIdx.x; k < m; k += kEvalThreads) {
      float acc = 0.0f;
      const float* col = S + static_cast<size_t>(k) * p;
#pragma unroll 8
      for (int j = 0; j < p; ++j) acc = __fadd_rn(acc, __fmul_rn(ld[j], col[j]));
      tv[k] = acc;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < p * m; e += kEvalThreads) {
      const int j = e % p, k = e / p;
      S[e] = __fsub_rn(S[e], __fmul_rn(ld[j], tv[k]));
    }
    __syncthreads();
    fitted = comp + 1;
  }

  if (fitted < 1) {
    if (a.predict_mode) {
      // the call ends in an error, but what was queued behind this launch still takes
      // the predictions as codes of classes: they are never left unwritten.  Nor is a
      // status taken back by a later evaluation: the host reads it after the last
      if (threadIdx.x == 0) a.status[s] = 1;
      predict_all(klist[0]);
      return;
    }
    // DegeneratePLSFit: the most frequent training class, smallest on ties
    if (threadIdx.x == 0) {
      int bl = klist[0], bc = -1;
      for (int k = 0; k < m; ++k) {
        if (cnt[klist[k]] > bc) {
          bc = cnt[klist[k]];
          bl = klist[k];
        }
      }
      sh.lab = bl;
      a.eval_comp[s] = 1;
    }
    __syncthreads();
    predict_all(sh.lab);
    return;
  }

  // --- LDA on the first nc score columns -----------------------------------
  const int nc = a.predict_mode ? fitted : min(a.requested, fitted);
  float* Ts = a.T + static_cast<size_t>(s) * L * NCm;   // by class-list position: Ts[pos * nc + q]
  float* Tt = a.Tt + static_cast<size_t>(s) * L * NCm;  // by training position: Tt[t * nc + q]
  float* Tv = a.Tv != nullptr ? a.Tv + static_cast<size_t>(s) * L * NCm : nullptr;  // by validation row: Tv[row * nc + q]
  auto keep_score = [&](int row, int q, float v) {
    const int t = tpos[row];
    if (t != kNoPos) {
      Ts[static_cast<size_t>(posof[row]) * nc + q] = v;
      Tt[static_cast<size_t>(t) * nc + q] = v;
    } else if (Tv != nullptr) {
      Tv[static_cast<size_t>(row) * nc + q] = v;
    }
  };
  // The score cross-products are serial chains over all training rows.  With up
  // to seven components they fit the lanes of one warp, which follows the others
  // a round of batches behind: 50 runs of 7500 x 200 rows, 10 folds, 50 cycles
  // 151.6 -> 149.6 ms.  For 10 and 300 slices of 1500 to 8000 rows, 20 to 200
  // columns and 2 to 7 components the two ways take the same time, so the line at
  // kFollowRows only keeps the rounds' barriers out of short streams.
  const int ncp = nc * (nc + 1) / 2;
  const bool follow = nc < kMaxNC && !a.da_mode && L >= kFollowRows;
  int prr = 0, pcol = min(lane, ncp - 1);
  while (pcol > prr) {
    pcol -= prr + 1;
    ++prr;
  }
  if (!follow) {
    stream_all_scores(Zs, zp, p, L, Wsm, ldw, nc, tiles + warp * kTile, lane, warp, kEvalWarps, keep_score, []() {});
  } else {
    constexpr int kScorers = kEvalWarps - 1;
    const int brows = nc == 1 ? kScoreRows / 2 : kScoreRows;  // of stream_scores
    const int nb = (L + brows - 1) / brows, rounds = (nb + kScorers - 1) / kScorers;
    if (warp < kScorers) {
      int done = 0;
      stream_all_scores(Zs, zp, p, L, Wsm, ldw, nc, tiles + warp * kTile, lane, warp, kScorers, keep_score, [&]() {
        ++done;
        round_sync();
      });
      for (; done < rounds; ++done) round_sync();
    } else {
      float acc = 0.0f;
      int t0 = 0;
      for (int k = 0; k < rounds; ++k) {
        round_sync();  // round k's scores are written
        int cn = 0;
        for (int i = 0; i < kScorers * brows / 32; ++i) {
          const int row = k * kScorers * brows + i * 32 + lane;
          cn += __popc(__ballot_sync(kFull, row < L && tpos[min(row, L - 1)] != kNoPos));
        }
        acc = score_products(acc, Tt + static_cast<size_t>(t0) * nc, cn, nc, prr, pcol, tiles + warp * kTile, lane);
        t0 += cn;
      }
      if (lane < ncp) {
        cp[prr * nc + pcol] = acc;
        cp[pcol * nc + prr] = acc;
      }
    }
  }
  // the rows to predict: scored with the training rows, except the separate
  // ones of predict mode
  float* rowscores = a.predict_mode ? a.Tp + static_cast<size_t>(r) * a.NV * NCm : Tv;
  auto score_rows = [&]() {
    stream_all_scores(vbase, zp, p, nv, Wsm, ldw, nc, tiles + warp * kTile, lane, warp, kEvalWarps,
                      [&](int row, int q, float v) { rowscores[static_cast<size_t>(row) * nc + q] = v; }, []() {});
    __syncthreads();
  };
  __syncthreads();
  // class sums (the training rows of each class in row order, i.e. the
  // flagged class-list positions in order): one warp per chain
  const int ncs = m * nc;
  // largest class first, so that no long chain is begun last
  int* by_size = reinterpret_cast<int*>(cst);  // the constants come later
  if (!a.da_mode) {
    for (int k = threadIdx.x; k < m; k += kEvalThreads) {
      const int mine = cnt[klist[k]];
      int rank = 0;
      for (int j = 0; j < m; ++j) {
        const int other = cnt[klist[j]];
        rank += other > mine || (other == mine && j < k);
      }
      by_size[rank] = k;
    }
    __syncthreads();
  }
  auto class_sums = [&](int at) {
    const int k = by_size[at], code = klist[k];
    with_components(nc, [&](auto c) {
      constexpr int NC = decltype(c)::value;
      const float acc =
          warp_masked_columns<NC>(Ts, posok, coff[code], coff[code + 1], tiles + warp * kTile, lane);
      if (lane < NC) cs[k * NC + lane] = acc;
    });
  };
  auto class_sum = [&](int it) {
    const int k = it / nc, q = it % nc;
    const int code = klist[k];
    const float acc = warp_masked_chain<4>(Ts, nc, q, posok, coff[code], coff[code + 1], lane);
    if (lane == 0) cs[k * nc + q] = acc;
  };
  if (a.da_mode) {
    for (int it = warp; it < ncs; it += kEvalWarps) class_sum(it);
  }
  if (a.da_mode) {
    // --- PLS-DA (the PLS_DA branch of run_plscv_host, plscv.cpp:2428-2443) ---
    // class means of the one-hot labels (label_means_float, plscv.cpp:1210)
    __syncthreads();
    const float inv_n = nt > 0 ? __fdiv_rn(1.0f, static_cast<float>(nt)) : 0.0f;
    for (int k = threadIdx.x; k < m; k += kEvalThreads) cst[k] = __fmul_rn(static_cast<float>(cnt[klist[k]]), inv_n);
    // regression_coefficients_centered_one_hot_float (plscv.cpp:1222-1265):
    // double score sums and double score cross-products over the training rows
    for (int q = warp; q < nc; q += kEvalWarps) {
      const double v = warp_seq_sum_double(nt, [&](int i) { return Tt[static_cast<size_t>(i) * nc + q]; }, lane);
      if (lane == 0) ssum[q] = v;
    }
    for (int it = warp; it < ncp; it += kEvalWarps) {
      int pr = it, rr = 0;
      while (pr > rr) {
        pr -= rr + 1;
        ++rr;
      }
      const int col = pr;
      const float v = warp_seq_dot(nt, [&](int i, float& x, float& y) {
        x = Tt[static_cast<size_t>(i) * nc + col];
        y = Tt[static_cast<size_t>(i) * nc + rr];
      }, lane);
      if (lane == 0) {
        pooled[rr * nc + col] = v;
        pooled[col * nc + rr] = v;
      }
    }
    __syncthreads();
    for (int it = threadIdx.x; it < nc * m; it += kEvalThreads) {
      const int q = it / m, k = it % m;
      sol[q * m + k] = __fsub_rn(cs[k * nc + q], __double2float_rn(__dmul_rn(ssum[q], static_cast<double>(cst[k]))));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // solve_linear_float (plscv.cpp:1346-1377): Gauss-Jordan with partial
      // pivoting on lhs + 1e-9 I
      float* A = pooled;
      for (int i = 0; i < nc; ++i) A[i * nc + i] = __fadd_rn(A[i * nc + i], 1.0e-9f);
      for (int c = 0; c < nc; ++c) {
        int piv = c;
        float best = fabsf(A[c * nc + c]);
        for (int r2 = c + 1; r2 < nc; ++r2) {
          const float val = fabsf(A[r2 * nc + c]);
          if (val > best) {
            best = val;
            piv = r2;
          }
        }
        if (best < 1.0e-12f) continue;
        if (piv != c) {
          for (int j = 0; j < nc; ++j) {
            const float t = A[c * nc + j];
            A[c * nc + j] = A[piv * nc + j];
            A[piv * nc + j] = t;
          }
          for (int j = 0; j < m; ++j) {
            const float t = sol[c * m + j];
            sol[c * m + j] = sol[piv * m + j];
            sol[piv * m + j] = t;
          }
        }
        const float dv = A[c * nc + c];
        for (int j = c; j < nc; ++j) A[c * nc + j] = __fdiv_rn(A[c * nc + j], dv);
        for (int j = 0; j < m; ++j) sol[c * m + j] = __fdiv_rn(sol[c * m + j], dv);
        for (int r2 = 0; r2 < nc; ++r2) {
          if (r2 == c) continue;
          const float fct = A[r2 * nc + c];
          if (fct == 0.0f) continue;
          for (int j = c; j < nc; ++j) A[r2 * nc + j] = __fsub_rn(A[r2 * nc + j], __fmul_rn(fct, A[c * nc + j]));
          for (int j = 0; j < m; ++j) sol[r2 * m + j] = __fsub_rn(sol[r2 * m + j], __fmul_rn(fct, sol[c * m + j]));
        }
      }
      a.eval_comp[s] = nc;
    }
    __syncthreads();
    // predict_pls_da_labels_float (plscv.cpp:1267-1292): first maximum of
    // mean + scores x coefficients
    if (a.predict_mode) score_rows();
    for (int v = threadIdx.x; v < nv; v += kEvalThreads) {
      const int row = a.predict_mode ? v : vidx[v];
      const float* tr = rowscores + static_cast<size_t>(row) * nc;
      float sr[kMaxComp];
      for (int q = 0; q < nc; ++q) sr[q] = tr[q];
      int best = 0;
      float bs = -INFINITY;
      for (int k = 0; k < m; ++k) {
        float sc = cst[k];
        for (int q = 0; q < nc; ++q) sc = __fadd_rn(sc, __fmul_rn(sr[q], sol[q * m + k]));
        if (sc > bs) {
          bs = sc;
          best = k;
        }
      }
      pred[row] = static_cast<uint16_t>(klist[best]);
    }
    return;
  }
  // score cross-products (all training rows in order), where no warp followed
  // the scores: a lane per chain
  for (int c0 = warp * 32; !follow && c0 < ncp; c0 += kEvalWarps * 32) {
    int pr = min(c0 + lane, ncp - 1), rr = 0;
    while (pr > rr) {
      pr -= rr + 1;
      ++rr;
    }
    const int col = pr;
    const float acc = score_products(0.0f, Tt, nt, nc, rr, col, tiles + warp * kTile, lane);
    if (c0 + lane < ncp) {
      cp[rr * nc + col] = acc;
      cp[col * nc + rr] = acc;
    }
  }
  // the class sums go to whichever warp is free
  const bool by_class = nc <= kMaxNC;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(&sh.queue, 1);
    it = __shfl_sync(kFull, it, 0);
    if (it >= (by_class ? m : ncs)) break;
    if (by_class) class_sums(it);
    else class_sum(it);
  }
  __syncthreads();
  // fit_lda_from_score_statistics_float, parallel where the reference's loops
  // are independent of one another
  for (int it = threadIdx.x; it < m * nc; it += kEvalThreads) {
    const int k = it / nc, c = cnt[klist[k]];
    const float inv = c > 0 ? __fdiv_rn(1.0f, static_cast<float>(c)) : 0.0f;
    cs[it] = __fmul_rn(cs[it], inv);
  }
  __syncthreads();
  const float df = static_cast<float>(max(1, nt - m));
  for (int it = threadIdx.x; it < ncp; it += kEvalThreads) {
    int pr = it, rr = 0;
    while (pr > rr) {
      pr -= rr + 1;
      ++rr;
    }
    const int col = pr;
    float between = 0.0f;
    for (int k = 0; k < m; ++k)
      between = __fadd_rn(between, __fmul_rn(__fmul_rn(static_cast<float>(cnt[klist[k]]), cs[k * nc + rr]),
                                             cs[k * nc + col]));
    const float cv = __fdiv_rn(__fsub_rn(cp[rr * nc + col], between), df);
    pooled[rr * nc + col] = cv;
    pooled[col * nc + rr] = cv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // the ridge grid and the Cholesky factor (independent of the right-hand sides)
    float trace = 0.0f;
    for (int rr = 0; rr < nc; ++rr) trace = __fadd_rn(trace, pooled[rr * nc + rr]);
    const float ridge_scale =
        (isfinite(trace) && trace > 0.0f) ? __fdiv_rn(trace, static_cast<float>(max(1, nc))) : 1.0f;
    const float grid[6] = {1e-8f, 1e-6f, 1e-5f, 1e-4f, 1e-3f, 1e-2f};
    bool ok = false;
    for (int g = 0; g < 6 && !ok; ++g) {
      const float lambda = __fmul_rn(grid[g], ridge_scale);
      ok = true;
      for (int row = 0; row < nc && ok; ++row) {
        for (int col = 0; col <= row && ok; ++col) {
          float v = pooled[row * nc + col];
          if (row == col) v = __fadd_rn(v, lambda);
          for (int q = 0; q < col; ++q) v = __fsub_rn(v, __fmul_rn(Lc[row * nc + q], Lc[col * nc + q]));
          if (row == col) {
            if (!isfinite(v) || v <= 0.0f) ok = false;
            else Lc[row * nc + col] = __fsqrt_rn(v);
          } else {
            const float dgl = Lc[col * nc + col];
            if (!isfinite(dgl) || dgl <= 0.0f) ok = false;
            else Lc[row * nc + col] = __fdiv_rn(v, dgl);
          }
        }
      }
    }
    sh.fail = ok ? 0 : 1;
    if (!ok) a.status[s] = 2;
    a.eval_comp[s] = nc;
  }
  __syncthreads();
  if (sh.fail) {
    predict_all(klist[0]);  // valid codes, as above
    return;
  }
  const float* lp = a.logprior + a.lp_off[s];
  for (int k = threadIdx.x; k < m; k += kEvalThreads) {
    // forward and backward substitution for the right-hand side of class k
    for (int row = 0; row < nc; ++row) {
      float v = cs[k * nc + row];
      for (int q = 0; q < row; ++q) v = __fsub_rn(v, __fmul_rn(Lc[row * nc + q], sol[q * m + k]));
      sol[row * m + k] = __fdiv_rn(v, Lc[row * nc + row]);
    }
    for (int row = nc - 1; row >= 0; --row) {
      float v = sol[row * m + k];
      for (int q = row + 1; q < nc; ++q) v = __fsub_rn(v, __fmul_rn(Lc[q * nc + row], sol[q * m + k]));
      sol[row * m + k] = __fdiv_rn(v, Lc[row * nc + row]);
    }
    float dot_mu = 0.0f;
    for (int q = 0; q < nc; ++q) {
      lin[k * nc + q] = sol[q * m + k];
      dot_mu = __fadd_rn(dot_mu, __fmul_rn(cs[k * nc + q], lin[k * nc + q]));
    }
    cst[k] = __fadd_rn(__fmul_rn(-0.5f, dot_mu), lp[cnt[klist[k]]]);
  }
  __syncthreads();
  // --- predictions ---------------------------------------------------------
  {
    if (a.predict_mode) score_rows();
    // NC > 0: the components, in registers (an array of a length known at run
    // time lies in local memory: 116k cycles for 750 rows and 98 classes); 0: nc
    auto predict = [&](auto c) {
      constexpr int NC = decltype(c)::value;
      const int nq = NC > 0 ? NC : nc;
      for (int v = threadIdx.x; v < nv; v += kEvalThreads) {
        const int row = a.predict_mode ? v : vidx[v];
        const float* tr = rowscores + static_cast<size_t>(row) * nq;
        float sr[NC > 0 ? NC : kMaxComp];
#pragma unroll
        for (int q = 0; q < nq; ++q) sr[q] = tr[q];
        int best = 0;
        float bs = -INFINITY;
#pragma unroll 4
        for (int k = 0; k < m; ++k) {
          float sc = cst[k];
#pragma unroll
          for (int q = 0; q < nq; ++q) sc = __fadd_rn(sc, __fmul_rn(sr[q], lin[k * nq + q]));
          if (sc > bs) {
            bs = sc;
            best = k;
          }
        }
        pred[row] = static_cast<uint16_t>(klist[best]);
      }
    };
    if (nc <= kMaxNC) with_components(nc, predict);
    else predict(std::integral_constant<int, 0>{});
  }
}

__global__ void gather_kernel(const float* __restrict__ x, int p, const int* __restrict__ rows, size_t nrows,
                              float* __restrict__ out) {
  const size_t total = nrows * p;
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t i = e / p;
    out[e] = x[static_cast<size_t>(rows[i]) * p + (e - i * p)];
  }
}

__global__ void assemble_kernel(int problems, int n, int L, int NV, const int* land, const int* test_rows,
                                const uint16_t* clbest, const uint16_t* proj, const int* c2l, int C0max, int* res) {
  const size_t per = static_cast<size_t>(L) + NV;
  const size_t total = static_cast<size_t>(problems) * per;
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t r = e / per, i = e - r * per;
    const int* map = c2l + r * C0max;
    if (i < static_cast<size_t>(L)) {
      res[r * n + land[r * L + i]] = map[clbest[r * L + i]];
    } else {
      const size_t t = i - L;
      res[r * n + test_rows[r * NV + t]] = map[proj[r * NV + t]];
    }
  }
}

}  // namespace

int pls_gather_rows(const float* x, int p, const int* rows, size_t nrows, float* out, cudaStream_t st) {
  gather_kernel<<<4 * 152, 256, 0, st>>>(x, p, rows, nrows, out);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int pls_assemble_result(int problems, int n, int L, int NV, const int* land, const int* test_rows,
                        const uint16_t* clbest, const uint16_t* proj, const int* code2label, int C0max, int* res,
                        cudaStream_t st) {
  assemble_kernel<<<2 * 152, 256, 0, st>>>(problems, n, L, NV, land, test_rows, clbest, proj, code2label, C0max,
                                           res);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int pls_prepare(const PlsPrepArgs& a, cudaStream_t st) {
  const int S = a.problems * a.F;
  dim3 g1(S, (a.p + 63) / 64);
  stats_kernel<<<g1, 64, 0, st>>>(a);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  {
    const int ys = std::max(1, std::min(S, 65535));
    const int xs = std::max(1, std::min(std::max(a.L, a.NV), std::max(1, 4096 / ys)));
    standardize_kernel<<<dim3(xs, ys), a.p <= 128 ? 128 : 256, 0, st>>>(a);
  }
  count_launch();
  e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);
  xsum_kernel<<<g1, 64, 0, st>>>(a);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int pls_build_gram(const PlsPrepArgs& a, const uint8_t* want, cudaStream_t st) {
  const int S = a.problems * a.F;
  const int JB = (a.p + kGramT - 1) / kGramT;
  dim3 grid(S, JB * (JB + 1) / 2);
  gram_kernel<<<grid, 256, 0, st>>>(a, want);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

size_t pls_eval_smem(int p, int C0max, int requested, int max_components, bool s_in_smem, bool tiles_after_s) {
  auto al = [](size_t v) { return (v + 15) / 16 * 16; };
  const size_t C = static_cast<size_t>(C0max), N = static_cast<size_t>(requested);
  size_t b = 64;
  b += 2 * al(sizeof(int) * C);
  b += 3 * al(sizeof(float) * p) + al(sizeof(float) * C);
  b += 2 * al(sizeof(float) * p * max_components);
  b += al(sizeof(float) * C * N) + 3 * al(sizeof(float) * N * N) + al(sizeof(float) * N * C);
  b += al(sizeof(float) * C * N) + al(sizeof(float) * C) + al(sizeof(double) * N);
  const size_t cross = s_in_smem ? sizeof(float) * static_cast<size_t>(p) * C : 0;
  const size_t tiles = sizeof(float) * static_cast<size_t>(kEvalWarps) * kTile;
  b += tiles_after_s ? al(cross) + tiles : (cross > tiles ? cross : tiles);
  return b;
}

int pls_evaluate(const PlsEvalArgs& a, cudaStream_t st) {
  const int S = a.problems * a.F;
  if (a.requested > kMaxComp || a.max_components > kMaxComp) return static_cast<int>(cudaErrorInvalidValue);
  // weight rows padded to whole 16-byte vectors, unless that would cost the
  // second CTA of an SM (or not fit at all)
  auto bytes = [&](int ldw) {
    return pls_eval_smem(a.p, a.C0max, a.requested, ldw, a.s_in_smem != 0, a.tiles_after_s != 0);
  };
  const int padded = (a.max_components + 3) / 4 * 4;
  const size_t two_ctas = 112 * 1024, most = 224 * 1024;
  PlsEvalArgs b = a;
  b.ldw = bytes(padded) <= (bytes(a.max_components) <= two_ctas ? two_ctas : most) ? padded : a.max_components;
  const size_t smem = bytes(b.ldw);
  auto* const eval = std::max(S, a.live) <= a.sms ? eval_kernel<1> : eval_kernel<2>;
  if (smem > 48 * 1024) {
    const cudaError_t e = allow_shared_memory(eval);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const size_t stream_smem = cross_stream_smem(a.C0max);
  if (stream_smem <= most) {
    if (stream_smem > 48 * 1024) {
      const cudaError_t e = allow_shared_memory(cross_stream_kernel);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    cross_stream_kernel<<<dim3((a.p + 31) / 32, std::min(S, 65535)), kStreamThreads, stream_smem, st>>>(b);
  } else {
    const int items = a.C0max * ((a.p + 31) / 32), per = kCrossThreads / 32;
    cross_kernel<<<dim3(std::min((items + per - 1) / per, 1024), std::min(S, 65535)), kCrossThreads, 0, st>>>(b);
  }
  eval<<<S, kEvalThreads, smem, st>>>(b);
  count_launch(2);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace kgb
