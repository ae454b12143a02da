// Graph-side kernels of the KODAMA.matrix path.
//
//   graph_minmax / normalize_external: the caller graph as
//     normalize_external_graph (kodama_matrix.cpp:1292-1330) leaves it:
//     one-based detection, invalid / self / non-finite entries dropped,
//     survivors compacted to the left, distances clamped at 0, width K.
//   normalize_indices: normalize_graph_indices (core.cpp:586-622): positions
//     kept, invalid ids -> -1, non-finite or negative distances -> +inf.
//   build_vote_tables: per problem and landmark row, the first k' valid,
//     non-self, out-of-fold neighbours among landmark rows with score -(d*d)
//     (Euclidean metric) or 1 - d (cosine, inner product; core.cpp:672-677):
//     subset_graph_to_rows (kodama_matrix.cpp:1332-1365) followed by
//     precompute_knn_cv_graph (core.cpp:624-692).
//   project_labels: non-landmark label = majority over the first knn.k
//     landmark neighbours of its graph row, ties to the smaller label, none ->
//     label of the first landmark (kodama_matrix.cpp:3221-3261, :169).
//   dissimilarity: co-label proximity (kodama_matrix.cpp:2685-2776):
//     d' = (1 + d) / (same/valid)^2 or +inf, row stably sorted by (d', id).
#include "graph_ops.cuh"
#include "launch_count.cuh"
#include "smem_limit.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <math.h>
#include <stdint.h>

#include <type_traits>

namespace kgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__global__ void minmax_kernel(const int* __restrict__ idx, size_t total, int* mm) {
  int lo = 0x7fffffff, hi = (-0x7fffffff - 1);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int v = idx[i];
    if (v < 0) continue;
    lo = min(lo, v);
    hi = max(hi, v);
  }
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&mm[0], lo);
    atomicMax(&mm[1], hi);
  }
}

__device__ __forceinline__ bool one_based_of(int base, const int* mm, int samples) {
  return base == 1 || (base < 0 && mm[0] >= 1 && mm[1] <= samples);
}

__global__ void normalize_external_kernel(const int* __restrict__ in_idx, const float* __restrict__ in_dist,
                                          int n, int gk, int K, int base, const int* mm,
                                          int* __restrict__ out_idx, float* __restrict__ out_dist) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool ob = one_based_of(base, mm, n);
  int col = 0;
  for (int j = 0; j < gk && col < K; ++j) {
    const size_t src = static_cast<size_t>(i) * gk + j;
    int id = in_idx[src];
    if (ob && id > 0) --id;
    if (id < 0 || id >= n || id == i) continue;
    const float d = in_dist[src];
    if (!isfinite(d)) continue;
    out_idx[static_cast<size_t>(i) * K + col] = id;
    out_dist[static_cast<size_t>(i) * K + col] = (0.0f < d) ? d : 0.0f;  // std::max(0.0f, d)
    ++col;
  }
  for (; col < K; ++col) {
    out_idx[static_cast<size_t>(i) * K + col] = -1;
    out_dist[static_cast<size_t>(i) * K + col] = INFINITY;
  }
}

__global__ void normalize_indices_kernel(const int* __restrict__ in_idx, const float* __restrict__ in_dist,
                                         size_t total, int samples, int base, const int* mm,
                                         int* __restrict__ out_idx, float* __restrict__ out_dist) {
  const bool ob = one_based_of(base, mm, samples);
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    int id = in_idx[i];
    if (ob && id > 0) --id;
    if (id < 0 || id >= samples) {
      out_idx[i] = -1;
      out_dist[i] = INFINITY;
      continue;
    }
    out_idx[i] = id;
    const float d = in_dist[i];
    out_dist[i] = (isfinite(d) && d >= 0.0f) ? d : INFINITY;
  }
}

__global__ void scatter_g2l_kernel(const int* __restrict__ land, int problems, int L, int n, int* __restrict__ g2l) {
  const size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<size_t>(problems) * L) return;
  const int p = static_cast<int>(t / L), i = static_cast<int>(t % L);
  g2l[static_cast<size_t>(p) * n + land[t]] = i;
}

// One thread per (problem, row).
__global__ void vote_table_kernel(VoteTableArgs a) {
  const size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<size_t>(a.problems) * a.L) return;
  const int p = static_cast<int>(t / a.L), i = static_cast<int>(t % a.L);
  const int grow = a.land ? a.land[t] : i;
  const int* g2l = a.g2l ? a.g2l + static_cast<size_t>(p) * a.n : nullptr;
  const uint8_t* fo = a.folds + static_cast<size_t>(p) * a.L;
  const int myfold = fo[i];
  uint16_t* nb = a.nb + t * a.w;
  float* sc = a.sc + t * a.w;
  int col = 0;
  // eight neighbours at a time: their ids and distances, then their local
  // ids, then their folds are each loaded together, so a chunk waits on three
  // rounds of loads instead of three per neighbour
  constexpr int kChunk = 8;
  for (int j0 = 0; j0 < a.K && col < a.w; j0 += kChunk) {
    int gnb[kChunk], loc[kChunk], lf[kChunk];
    float dist[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int j = j0 + u;
      const size_t src = static_cast<size_t>(grow) * a.K + j;
      gnb[u] = j < a.K ? a.gidx[src] : -1;
      dist[u] = j < a.K ? a.gdist[src] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u)
      loc[u] = (gnb[u] >= 0 && gnb[u] < a.n) ? (g2l ? g2l[gnb[u]] : gnb[u]) : -1;
#pragma unroll
    for (int u = 0; u < kChunk; ++u) lf[u] = loc[u] >= 0 ? fo[loc[u]] : -1;
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      if (col >= a.w) break;
      if (loc[u] < 0 || loc[u] == i) continue;
      if (lf[u] == myfold) continue;
      if (!isfinite(dist[u])) continue;
      const float dc = (0.0f < dist[u]) ? dist[u] : 0.0f;
      nb[col] = static_cast<uint16_t>(loc[u]);
      sc[col] = a.score_one_minus ? __fsub_rn(1.0f, dc) : -__fmul_rn(dc, dc);
      ++col;
    }
  }
  for (; col < a.w; ++col) {
    nb[col] = 0xFFFFu;
    sc[col] = -INFINITY;
  }
}

// One thread per (problem, global row).
__global__ void project_kernel(ProjectArgs a) {
  const size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (t >= static_cast<size_t>(a.problems) * a.n) return;
  const int p = static_cast<int>(t / a.n), r = static_cast<int>(t % a.n);
  const int* g2l = a.g2l + static_cast<size_t>(p) * a.n;
  const uint16_t* best = a.clbest + static_cast<size_t>(p) * a.L;
  const int* c2l = a.code2label + static_cast<size_t>(p) * a.C0max;
  const int loc = g2l[r];
  int code;
  if (loc >= 0) {
    code = best[loc];
  } else {
    int votes[kMaxProjectK];
    int nv = 0;
    // eight neighbours at a time, each level of dependent loads issued together
    constexpr int kChunk = 8;
    for (int j0 = 0; j0 < a.K && nv < a.pk; j0 += kChunk) {
      int g[kChunk], l[kChunk], b[kChunk];
#pragma unroll
      for (int u = 0; u < kChunk; ++u) g[u] = j0 + u < a.K ? a.gidx[static_cast<size_t>(r) * a.K + j0 + u] : -1;
#pragma unroll
      for (int u = 0; u < kChunk; ++u) l[u] = (g[u] >= 0 && g[u] < a.n) ? g2l[g[u]] : -1;
#pragma unroll
      for (int u = 0; u < kChunk; ++u) b[u] = l[u] >= 0 ? best[l[u]] : 0;
#pragma unroll
      for (int u = 0; u < kChunk; ++u)
        if (nv < a.pk && l[u] >= 0) votes[nv++] = b[u];
    }
    if (nv == 0) {
      code = best[0];
    } else {
      int bl = 0x7fffffff, bc = 0;
      for (int q = 0; q < nv; ++q) {
        const int v = votes[q];
        int c = 0;
        for (int u = 0; u < nv; ++u) c += votes[u] == v;
        if (c > bc || (c == bc && v < bl)) {
          bl = v;
          bc = c;
        }
      }
      code = bl;
    }
  }
  a.res[t] = c2l[code];
}

// Reverse adjacency of each problem's vote table: rev_idx[rev_off[v] ..
// rev_off[v+1]) lists the rows r whose table contains v.  A CTA per problem and
// range of v: it reads the whole table, counts its own range (and how many entries
// lie below it, where its lists start) and places its own rows.
// What bounds it is the placing, one scattered two-byte store per entry and SM at
// a time, and the two passes' loads, eight a thread in flight: with one CTA for
// all v and a load at a time a table of 5003 x 30 took 221 us.
__global__ void reverse_table_kernel(ReverseArgs a) {
  extern __shared__ int deg[];
  __shared__ int wsum[32];
  __shared__ int below;
  const int p = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nwarps = (blockDim.x + 31) / 32, step = blockDim.x;
  const int width = (a.L + gridDim.y - 1) / gridDim.y;
  const int lo = min(a.L, static_cast<int>(blockIdx.y) * width), hi = min(a.L, lo + width);
  const uint16_t* nb = a.nb + static_cast<size_t>(p) * a.L * a.w;
  int* off = a.rev_off + static_cast<size_t>(p) * (a.L + 1);
  uint16_t* idx = a.rev_idx + static_cast<size_t>(p) * a.L * a.w;
  for (int v = tid; v < hi - lo; v += step) deg[v] = 0;
  if (tid == 0) below = 0;
  __syncthreads();
  const int total = a.L * a.w;  // < 2^22: L < 2^16, w <= 32
  int under = 0;
  for (int e0 = tid; e0 < total; e0 += 8 * step) {
    int v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = e0 + q * step < total ? nb[e0 + q * step] : 0xFFFF;  // 0xFFFF: none
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      under += v[q] < lo;
      if (v[q] >= lo && v[q] < hi) atomicAdd(&deg[v[q] - lo], 1);
    }
  }
  under = __reduce_add_sync(0xffffffffu, under);
  if (lane == 0) atomicAdd(&below, under);
  __syncthreads();
  // exclusive scan of the in-degrees: each thread a contiguous chunk, then
  // the warps' and the block's prefixes
  const int chunk = (hi - lo + step - 1) / step;
  const int b = min(hi - lo, tid * chunk), e = min(hi - lo, b + chunk);
  int local = 0;
  for (int v = b; v < e; ++v) local += deg[v];
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < nwarps ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nwarps) wsum[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  int run = below + (warp > 0 ? wsum[warp - 1] : 0) + incl - local;
  for (int v = b; v < e; ++v) {
    const int c = deg[v];
    deg[v] = run;
    off[lo + v] = run;
    run += c;
  }
  if (hi == a.L && lo < hi && tid == 0) off[a.L] = below + wsum[nwarps - 1];
  __syncthreads();
  for (int e0 = tid; e0 < total; e0 += 8 * step) {
    int v[8], slot[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = e0 + q * step < total ? nb[e0 + q * step] : 0xFFFF;
#pragma unroll
    for (int q = 0; q < 8; ++q) slot[q] = v[q] >= lo && v[q] < hi ? atomicAdd(&deg[v[q] - lo], 1) : -1;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (slot[q] >= 0)
        idx[slot[q]] = static_cast<uint16_t>(static_cast<unsigned>(e0 + q * step) / static_cast<unsigned>(a.w));
  }
}

// Label coding of k-means labels 1..k (one CTA per problem): codes are the
// ranks of the labels present, code2label the labels in ascending order.
__global__ void code_labels_kernel(CodingArgs a) {
  extern __shared__ int cmap[];  // k+1 entries
  const int p = blockIdx.x;
  const int* lab = a.labels + static_cast<size_t>(p) * a.n;
  for (int v = threadIdx.x; v <= a.k; v += blockDim.x) cmap[v] = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < a.n; r += blockDim.x) cmap[lab[r]] = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    int* c2l = a.code2label + static_cast<size_t>(p) * a.C0max;
    for (int v = 0; v <= a.k; ++v) {
      if (cmap[v]) {
        c2l[run] = v;
        cmap[v] = run++;
      }
    }
    a.ncodes[p] = run;
  }
  __syncthreads();
  uint16_t* codes = a.codes + static_cast<size_t>(p) * a.n;
  for (int r = threadIdx.x; r < a.n; r += blockDim.x) codes[r] = static_cast<uint16_t>(cmap[lab[r]]);
}

// FNV-1a over the little-endian bytes of each row of a rows x n int matrix
// (hash_integer_vector, kodama_matrix.cpp:1689-1699); one thread per row.
__global__ void fnv_rows_kernel(const int* __restrict__ data, int rows, int n, uint64_t* __restrict__ out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int* v = data + static_cast<size_t>(r) * n;
  uint64_t h = 1469598103934665603ull;
  for (int i = 0; i < n; ++i) {
    const uint32_t b = static_cast<uint32_t>(v[i]);
#pragma unroll
    for (int s = 0; s < 32; s += 8) {
      h ^= static_cast<uint8_t>((b >> s) & 0xffu);
      h *= 1099511628211ull;
    }
  }
  out[r] = h;
}

// 32 x 32 tiles; a CTA walks the run tiles blockIdx.y, blockIdx.y + gridDim.y,
// ... so any number of runs fits the grid's y limit.  Sample rows of `out` are
// `stride` ints apart; the padding past the runs is written as label 0 (no
// label), so that dissimilarity_kernel can load whole 16-byte vectors.
// idx != nullptr: the CTAs past the last sample tile check a one-based graph
// instead, flagging any stored index outside {negative (missing)} U [1, n].
__global__ void transpose_kernel(const int* __restrict__ res, int runs, int n, int stride, int* __restrict__ out,
                                 const int* __restrict__ idx, size_t total, int* bad) {
  __shared__ int tile[32][33];
  const int sample_tiles = (n + 31) / 32;
  if (static_cast<int>(blockIdx.x) >= sample_tiles) {
    const size_t step = static_cast<size_t>(gridDim.x - sample_tiles) * gridDim.y * 256;
    size_t e = (static_cast<size_t>(blockIdx.x - sample_tiles) * gridDim.y + blockIdx.y) * 256 + threadIdx.y * 32 +
               threadIdx.x;
    for (; e < total; e += step) {
      const int v = idx[e];
      if (v >= 0 && (v < 1 || v > n)) atomicExch(bad, 1);
    }
    return;
  }
  const int s0 = blockIdx.x * 32;
  const int run_tiles = (stride + 31) / 32;
  for (int rt = blockIdx.y; rt < run_tiles; rt += gridDim.y) {
    const int r0 = rt * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
      const int r = r0 + k, s = s0 + threadIdx.x;
      tile[k][threadIdx.x] = r < runs && s < n ? res[static_cast<size_t>(r) * n + s] : 0;
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
      const int s = s0 + k, r = r0 + threadIdx.x;
      if (r < stride && s < n) out[static_cast<size_t>(s) * stride + r] = tile[threadIdx.x][k];
    }
    __syncthreads();
  }
}

// Co-label proximity of one graph row per warp, then a rank sort of the row in
// shared memory.  Eight lanes share a neighbour (four neighbours per step, two
// steps in flight) and read its labels and the row's own as vectors of VEC
// ints.  The counts of 32 neighbours end up one per lane, so the two double
// divisions of each neighbour run on all lanes: double division is a long
// serial sequence here, and one lane forming it for each neighbour in turn was
// most of the earlier kernel's time (20000 rows x 30 neighbours x 100 runs,
// whole in-place call: 879 us; with this split 129 us).  What remains is the
// gather of the neighbours' labels from L2 (rows x neighbours x runs x 4
// bytes).
// A warp reads its whole row before it writes any of it and no other warp
// touches that row, so the outputs may be the inputs.  Nothing is written when
// a.bad is set (an index check in front of the kernel failed).
template <int VEC>
__global__ void __launch_bounds__(256) dissimilarity_kernel(DissimArgs a) {
  using Vec = typename std::conditional<VEC == 4, int4, int>::type;
  extern __shared__ unsigned char dsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  float* kd = reinterpret_cast<float*>(dsm) + static_cast<size_t>(warp) * a.K;
  int* ki = reinterpret_cast<int*>(reinterpret_cast<float*>(dsm) + static_cast<size_t>(wpb) * a.K) +
            static_cast<size_t>(warp) * a.K;
  const int i = blockIdx.x * wpb + warp;
  if (i >= a.n || (a.bad != nullptr && *a.bad != 0)) return;
  const int sub = lane & 7, grp = lane >> 3;
  const int nvec = a.stride / VEC;
  const Vec* lbs = reinterpret_cast<const Vec*>(a.lbs);
  const Vec* li = lbs + static_cast<size_t>(i) * nvec;
  for (int j0 = 0; j0 < a.K; j0 += 32) {
    const int j = j0 + lane;
    const size_t off = static_cast<size_t>(i) * a.K + j;
    const int stored = j < a.K ? a.idx[off] : -1;
    float d = j < a.K ? a.dist[off] : INFINITY;
    const int nb = (stored >= 0 && a.in_one_based) ? stored - 1 : stored;
    const bool live = nb >= 0 && nb < a.n && isfinite(d);
    int my_same = 0, my_valid = 0;
    for (int s = 0; s < 8 && j0 + 4 * s < a.K; s += 2) {
      int same[2] = {0, 0}, valid[2] = {0, 0};
      const Vec* lj[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int q = __shfl_sync(kFull, live ? nb : -1, (4 * (s + u) + grp) & 31);
        lj[u] = q >= 0 ? lbs + static_cast<size_t>(q) * nvec : nullptr;
      }
#pragma unroll 2
      for (int v = sub; v < nvec; v += 8) {
        const Vec x = li[v];
        Vec y[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (lj[u] != nullptr) y[u] = lj[u][v];
          else y[u] = Vec{};
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if constexpr (VEC == 4) {
            const int px = (x.x != 0) & (y[u].x != 0), py = (x.y != 0) & (y[u].y != 0),
                      pz = (x.z != 0) & (y[u].z != 0), pw = (x.w != 0) & (y[u].w != 0);
            valid[u] += px + py + pz + pw;
            same[u] += (px & (x.x == y[u].x)) + (py & (x.y == y[u].y)) + (pz & (x.z == y[u].z)) +
                       (pw & (x.w == y[u].w));
          } else {
            const int p = (x != 0) & (y[u] != 0);
            valid[u] += p;
            same[u] += p & (x == y[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          same[u] += __shfl_xor_sync(kFull, same[u], o);
          valid[u] += __shfl_xor_sync(kFull, valid[u], o);
        }
        // group g holds the counts of neighbour 4 (s + u) + g of this batch
        const int gs = __shfl_sync(kFull, same[u], (lane & 3) * 8), gv = __shfl_sync(kFull, valid[u], (lane & 3) * 8);
        if ((lane >> 2) == s + u) {
          my_same = gs;
          my_valid = gv;
        }
      }
    }
    if (j < a.K) {
      int id = stored;
      if (!live) {
        d = INFINITY;
      } else {
        id = a.out_one_based ? nb + 1 : nb;
        if (my_same == 0 || my_valid == 0) {
          d = INFINITY;
        } else {
          const double agr = __ddiv_rn(static_cast<double>(my_same), static_cast<double>(my_valid));
          d = static_cast<float>(__ddiv_rn(__dadd_rn(1.0, static_cast<double>(d)), __dmul_rn(agr, agr)));
        }
      }
      kd[j] = d;
      ki[j] = id;
    }
  }
  __syncwarp();
  // stable rank sort by (distance, id)
  for (int j = lane; j < a.K; j += 32) {
    const float dj = kd[j];
    const int ij = ki[j];
    int rank = 0;
    for (int q = 0; q < a.K; ++q) {
      const float dq = kd[q];
      const int iq = ki[q];
      const bool less = dq < dj || (!(dj < dq) && iq < ij);
      const bool equal_before = !(dq < dj) && !(dj < dq) && iq == ij && q < j;
      rank += less || equal_before;
    }
    a.out_idx[static_cast<size_t>(i) * a.K + rank] = ij;
    a.out_dist[static_cast<size_t>(i) * a.K + rank] = dj;
  }
}

}  // namespace

int graph_minmax(const int* idx, size_t total, int* mm, cudaStream_t st) {
  const int init[2] = {0x7fffffff, (-0x7fffffff - 1)};
  cudaMemcpyAsync(mm, init, sizeof(init), cudaMemcpyHostToDevice, st);
  const int blocks = static_cast<int>((total + 255) / 256 < 2048 ? (total + 255) / 256 : 2048);
  minmax_kernel<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(idx, total, mm);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int normalize_external(const int* in_idx, const float* in_dist, int n, int gk, int K, int base, const int* mm,
                       int* out_idx, float* out_dist, cudaStream_t st) {
  normalize_external_kernel<<<(n + 255) / 256, 256, 0, st>>>(in_idx, in_dist, n, gk, K, base, mm, out_idx, out_dist);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int normalize_indices(const int* in_idx, const float* in_dist, size_t total, int samples, int base, const int* mm,
                      int* out_idx, float* out_dist, cudaStream_t st) {
  const int blocks = static_cast<int>((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  normalize_indices_kernel<<<blocks > 0 ? blocks : 1, 256, 0, st>>>(in_idx, in_dist, total, samples, base, mm,
                                                                  out_idx, out_dist);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int build_g2l(const int* land, int problems, int L, int n, int* g2l, cudaStream_t st) {
  cudaMemsetAsync(g2l, 0xff, sizeof(int) * static_cast<size_t>(problems) * n, st);
  const size_t total = static_cast<size_t>(problems) * L;
  scatter_g2l_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(land, problems, L, n, g2l);
  return static_cast<int>(cudaGetLastError());
}

int build_vote_tables(const VoteTableArgs& a, cudaStream_t st) {
  const size_t total = static_cast<size_t>(a.problems) * a.L;
  vote_table_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(a);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int build_reverse_tables(const ReverseArgs& a, cudaStream_t st) {
  // two CTAs an SM: ranges until the chip is full, up to 16 of them
  const int parts = std::max(1, std::min(std::min(16, 2 * a.sms / a.problems), a.L));
  const size_t smem = sizeof(int) * (static_cast<size_t>(a.L) / parts + 2);
  if (smem > 48 * 1024) allow_shared_memory(reverse_table_kernel);
  reverse_table_kernel<<<dim3(a.problems, parts), 1024, smem, st>>>(a);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int project_labels(const ProjectArgs& a, cudaStream_t st) {
  const size_t total = static_cast<size_t>(a.problems) * a.n;
  project_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(a);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int code_labels(const CodingArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(int) * (static_cast<size_t>(a.k) + 1);
  if (smem > 48 * 1024) allow_shared_memory(code_labels_kernel);
  code_labels_kernel<<<a.problems, 1024, smem, st>>>(a);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int fnv_rows(const int* data, int rows, int n, uint64_t* out, cudaStream_t st) {
  fnv_rows_kernel<<<(rows + 63) / 64, 64, 0, st>>>(data, rows, n, out);
  count_launch();
  return static_cast<int>(cudaGetLastError());
}

int transpose_runs(const int* res, int runs, int n, int stride, int* out, cudaStream_t st, const int* idx,
                   size_t total, int* bad) {
  const int run_tiles = (stride + 31) / 32, sample_tiles = (n + 31) / 32;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sample_tiles, run_tiles < 65535 ? run_tiles : 65535);
  if (idx != nullptr) {
    // about 1024 CTAs' worth of index checks at most
    const size_t want = (total + 255) / 256;
    cfg.gridDim.x += static_cast<unsigned>(((want < 1024 ? want : 1024) + cfg.gridDim.y - 1) / cfg.gridDim.y);
  }
  cfg.blockDim = dim3(32, 8);
  cfg.stream = st;
  // the launch's own status (not an error left over from earlier work)
  const cudaError_t e = cudaLaunchKernelEx(&cfg, transpose_kernel, res, runs, n, stride, out, idx, total, bad);
  count_launch();
  return static_cast<int>(e);
}

int dissimilarity(const DissimArgs& a, cudaStream_t st) {
  const int wpb = 8;
  // rows of whole 16-byte vectors, or any row length
  const auto kernel = a.stride % 4 == 0 ? dissimilarity_kernel<4> : dissimilarity_kernel<1>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((a.n + wpb - 1) / wpb));
  cfg.blockDim = dim3(wpb * 32);
  cfg.dynamicSmemBytes = static_cast<size_t>(wpb) * a.K * (sizeof(float) + sizeof(int));
  cfg.stream = st;
  if (cfg.dynamicSmemBytes > 48 * 1024) {
    const cudaError_t e = allow_shared_memory(kernel);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
  count_launch();
  return static_cast<int>(e);
}

}  // namespace kgb
