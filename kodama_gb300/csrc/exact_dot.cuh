// Sequential double sums of float products, rounded to float, without double
// arithmetic on the common path: by a warp, by groups of eight lanes and by the
// block of a PLS evaluation (pls.cu).
#pragma once

#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

namespace kgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kEvalThreads = 512;
constexpr int kEvalWarps = kEvalThreads / 32;

__device__ __forceinline__ int biased_exp1(float v) {
  return max(static_cast<int>((__float_as_uint(v) >> 23) & 0xffu), 1);
}

// ---------------------------------------------------------------------------
// float(sum_k double(a_k) * double(b_k)) summed sequentially in double, as the
// reference's dot_float / mat_vec_float / t_mat_vec_float / power_norm2_float
// do, without double arithmetic on the common path.
//
// Each product of two floats is exact in double, so the sequential sum S_seq
// differs from the exact sum S by at most n * 2^-53 * sum|t_k| (recursive
// summation of exact terms; 2^-52 is used below).  A warp forms S exactly as
// a 64-bit fixed-point integer from the 24-bit mantissas (terms below the
// fixed point truncated: at most n units of error), rounds it to float and
// checks that the rounding interval of that float contains S widened by both
// error bounds; then float(S_seq) is that float.  When the check cannot
// decide (S close to a rounding boundary, massive cancellation, non-finite
// or extreme values), lane 0 runs the sequential double sum.  The point:
// this GPU issues a dependent double FMA only every 64-152 cycles.
// ---------------------------------------------------------------------------

__device__ __forceinline__ int clog2i(int n) { return n <= 1 ? 0 : 32 - __clz(n - 1); }

__device__ __forceinline__ float warp_sum_ru(float v) {
  for (int o = 16; o > 0; o >>= 1) v = __fadd_ru(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

__device__ __forceinline__ long long warp_sum_i64(long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// The float nearest to V * 2^LSB, if S_seq provably rounds to it (see above).
__device__ __forceinline__ bool round_check(long long V, int LSB, float A, int n, float& out) {
  if (V == 0) {
    if (A == 0.0f) {
      out = 0.0f;
      return true;
    }
    return false;
  }
  const bool neg = V < 0;
  const unsigned long long mag = neg ? 0ull - static_cast<unsigned long long>(V) : static_cast<unsigned long long>(V);
  const int e = 63 - __clzll(static_cast<long long>(mag));
  const int shift = e - 23;
  if (shift <= 0) return false;
  const float bu = __fadd_ru(__fmul_ru(ldexpf(A, -52 - LSB), static_cast<float>(n)), static_cast<float>(n + 1));
  if (!(bu < 1e30f)) return false;
  const unsigned long long one = 1ull;
  unsigned long long m = mag >> shift;
  const unsigned long long rem = mag & ((one << shift) - 1ull), half = one << (shift - 1);
  const bool up = rem > half || (rem == half && (m & 1ull));
  unsigned long long dlo, dhi;
  if (!up) {
    if (rem == half) return false;
    dhi = half - rem;
    dlo = rem + (m == 0x800000ull ? (half >> 1) : half);
  } else {
    dlo = rem - half;
    dhi = ((one << shift) - rem) + half;
  }
  const float dmin = __ull2float_rz(dlo < dhi ? dlo : dhi);
  if (!(dmin > bu)) return false;
  if (up) ++m;
  int ex = shift + LSB;
  if (m == 0x1000000ull) {
    m >>= 1;
    ++ex;
  }
  if (ex + 23 > 126 || ex + 23 < -126) return false;
  const float fv = ldexpf(static_cast<float>(m), ex);
  out = neg ? -fv : fv;
  return true;
}

// First pass of an exact dot, one term: the largest product exponent (top),
// non-finite operands (bad) and an upward-rounded bound A of sum |x y|.
__device__ __forceinline__ void exact_scan_term(float x, float y, int& top, int& bad, float& A) {
  const unsigned ux = __float_as_uint(x), uy = __float_as_uint(y);
  const int ex = static_cast<int>((ux >> 23) & 0xffu), ey = static_cast<int>((uy >> 23) & 0xffu);
  bad |= (ex == 0xff) | (ey == 0xff);
  if ((ux << 1) != 0u && (uy << 1) != 0u) top = max(top, max(ex, 1) + max(ey, 1) - 252);
  A = __fadd_ru(A, __fmul_ru(fabsf(x), fabsf(y)));
}

// Second pass, one term: x y as a multiple of 2^LSB (truncated below it).
__device__ __forceinline__ long long exact_fixed_term(float x, float y, int LSB) {
  const unsigned ux = __float_as_uint(x), uy = __float_as_uint(y);
  const unsigned bx = (ux >> 23) & 0xffu, by = (uy >> 23) & 0xffu;
  const unsigned mx = (ux & 0x7fffffu) | (bx ? 0x800000u : 0u), my = (uy & 0x7fffffu) | (by ? 0x800000u : 0u);
  const unsigned long long P = static_cast<unsigned long long>(mx) * my;
  if (P == 0ull) return 0;
  const int E = (bx ? static_cast<int>(bx) - 150 : -149) + (by ? static_cast<int>(by) - 150 : -149);
  const int sh = E - LSB;
  unsigned long long v;
  if (sh >= 0) v = P << sh;
  else v = -sh >= 64 ? 0ull : P >> (-sh);
  return ((ux ^ uy) >> 31) ? -static_cast<long long>(v) : static_cast<long long>(v);
}

// Exact fixed-point sum over the warp; returns whether `out` is float(S_seq).
template <class Term>
__device__ bool warp_exact_dot(int n, Term term, int lane, float& out) {
  int top = -100000, bad = 0;
  float A = 0.0f;
  for (int k = lane; k < n; k += 32) {
    float x, y;
    term(k, x, y);
    exact_scan_term(x, y, top, bad, A);
  }
  bad = __reduce_or_sync(kFull, bad);
  top = __reduce_max_sync(kFull, top);
  if (bad) return false;
  A = warp_sum_ru(A);
  if (top == -100000) {  // every term is zero
    out = 0.0f;
    return true;
  }
  const int LSB = top + clog2i(n) - 62;
  long long acc = 0;
  for (int k = lane; k < n; k += 32) {
    float x, y;
    term(k, x, y);
    acc += exact_fixed_term(x, y, LSB);
  }
  acc = warp_sum_i64(acc);
  return round_check(acc, LSB, A, n, out);
}

// The reference's sequential double chains, acc = fma(x_k, y_k, acc) for k
// ascending, by a whole warp.  A product of two floats is exact in double,
// so fma(x, y, acc) is acc + x*y rounded once: the lanes form 32 products at a
// time, every lane adds them in order (the same chain in every lane) and the
// next 32 terms load meanwhile.  n can be a column over the training rows,
// where one lane's loop would wait on every load.
template <class Term>
__device__ double warp_fma_chain(int n, Term term, int lane) {
  double s = 0.0;
  float x = 0.0f, y = 0.0f;
  if (lane < n) term(lane, x, y);
  for (int k0 = 0; k0 < n; k0 += 32) {
    const double prod = __dmul_rn(static_cast<double>(x), static_cast<double>(y));
    x = 0.0f;
    y = 0.0f;
    if (k0 + 32 + lane < n) term(k0 + 32 + lane, x, y);
    const int cnt = min(32, n - k0);
    for (int q = 0; q < cnt; ++q) s = __dadd_rn(s, __shfl_sync(kFull, prod, q));
  }
  return s;
}

// acc = 0.0; acc += double(x_k) for k ascending, the same way.
template <class Term>
__device__ double warp_add_chain(int n, Term term, int lane) {
  double s = 0.0;
  float x = lane < n ? term(lane) : 0.0f;
  for (int k0 = 0; k0 < n; k0 += 32) {
    const double v = static_cast<double>(x);
    x = k0 + 32 + lane < n ? term(k0 + 32 + lane) : 0.0f;
    const int cnt = min(32, n - k0);
    for (int q = 0; q < cnt; ++q) s = __dadd_rn(s, __shfl_sync(kFull, v, q));
  }
  return s;
}

// Sequential double sum of n floats, S_seq (acc = 0.0; acc += double(x_k)
// in order).  All terms are multiples of 2^emin (the smallest ulp); when the
// sum of |x| stays below 2^(emin + 53), every partial sum is exact in double,
// so S_seq is the exact fixed-point sum.  Otherwise lane 0 runs the chain.
template <class Term>
__device__ double warp_seq_sum_double(int n, Term term, int lane) {
  int emin = 1 << 20, emax = -(1 << 20), bad = 0;
  float A = 0.0f;
  for (int k = lane; k < n; k += 32) {
    const float x = term(k);
    const unsigned ux = __float_as_uint(x);
    const int be = static_cast<int>((ux >> 23) & 0xffu);
    bad |= be == 0xff;
    if ((ux << 1) != 0u) {
      const int ue = be ? be - 150 : -149;
      emin = min(emin, ue);
      emax = max(emax, ue);
      A = __fadd_ru(A, fabsf(x));
    }
  }
  bad = __reduce_or_sync(kFull, bad);
  emin = __reduce_min_sync(kFull, emin);
  emax = __reduce_max_sync(kFull, emax);
  A = warp_sum_ru(A);
  bool exact = !bad;
  if (exact && emin == (1 << 20)) return 0.0;  // every term is zero
  if (exact) exact = emax - emin + 24 + clog2i(n) <= 62 && A < ldexpf(1.0f, min(emin + 53, 127));
  if (exact) {
    long long acc = 0;
    for (int k = lane; k < n; k += 32) {
      const float x = term(k);
      const unsigned ux = __float_as_uint(x);
      if ((ux << 1) == 0u) continue;
      const int be = static_cast<int>((ux >> 23) & 0xffu);
      const long long mant = static_cast<long long>((ux & 0x7fffffu) | (be ? 0x800000u : 0u));
      const long long v = mant << ((be ? be - 150 : -149) - emin);
      acc += (ux >> 31) ? -v : v;
    }
    acc = warp_sum_i64(acc);
    // |acc| < 2^53: exact in double; 2^emin is a normal double (emin >= -149)
    return __dmul_rn(__ll2double_rn(acc), __longlong_as_double(static_cast<long long>(emin + 1023) << 52));
  }
  return warp_add_chain(n, term, lane);
}

// dot_float / mat_vec_float / t_mat_vec_float element: float(S_seq).
template <class Term>
__device__ float warp_seq_dot(int n, Term term, int lane) {
  float out = 0.0f;
  if (!warp_exact_dot(n, term, lane, out)) out = __double2float_rn(warp_fma_chain(n, term, lane));
  return out;
}

__device__ __forceinline__ float power_norm2(double sum) {
  if (!isfinite(sum) || sum < 0.0) return INFINITY;
  if (sum <= static_cast<double>(FLT_MAX)) return __fsqrt_rn(__double2float_rn(sum));
  return __double2float_rn(__dsqrt_rn(sum));
}

// power_norm2_float of v[0..n) by one warp.
__device__ float warp_power_norm(const float* v, int n, int lane) {
  float out = 0.0f;
  auto t = [&](int k, float& x, float& y) {
    x = v[k];
    y = v[k];
  };
  if (warp_exact_dot(n, t, lane, out)) return __fsqrt_rn(out);
  return power_norm2(warp_fma_chain(n, t, lane));
}

// One term of a two-float sum: the product and its fma remainder, Knuth's
// two-sum, the remainders into lo; A: upper bound of the sum of magnitudes.
__device__ __forceinline__ void two_float_add(float x, float y, float& hi, float& lo, float& A) {
  const float q = __fmul_rn(x, y);
  const float e = __fmaf_rn(x, y, -q);
  const float t = __fadd_rn(hi, q);
  const float z = __fsub_rn(t, hi);
  const float r = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(q, z));
  lo = __fadd_rn(lo, __fadd_rn(r, e));
  A = __fadd_ru(A, fabsf(q));
  hi = t;
}

// float(S_seq) for many dots at once: groups of eight lanes form a dot each,
// dot it over terms 0..n-1.  S is formed in two floats by error-free steps
// (product: x y and its fma remainder; sum: Knuth's two-sum), s + c with c the
// rounded sum of the remainders.  With A an upper bound of sum |x y|, c holds
// at most (2 nl + 6) roundings of values below u A (nl + 4), nl the terms of a
// lane plus the three joins, and S_seq lies within n 2^-52 A of S (above);
// remainders lost to underflow add n 2^-148.  If both ends of that interval
// round to the same float, float(S_seq) is that float; else the warp forms the
// dot as warp_seq_dot does.  About 12 instructions a term in one pass, where
// the fixed-point form takes 37 in two, and three joins instead of five.
template <class Load, class Put>
__device__ __forceinline__ void group_seq_dots(int dots, int n, int lane, int warp, Load&& load, Put&& put) {
  const int gl = lane & 7, g = lane >> 3;
  const float nl = static_cast<float>((n + 7) / 8 + 3);
  const float unit = 3.5527137e-15f;  // 2^-48
  const float K = (2.0f * nl + 6.0f) * (nl + 4.0f) * 1.1f + static_cast<float>(n) * 0.0625f + 1.0f;
  for (int d0 = warp * 4; d0 < dots; d0 += kEvalWarps * 4) {
    const int d = d0 + g;
    float s = 0.0f, c = 0.0f, A = 0.0f;
    if (d < dots) {
#pragma unroll 8
      for (int k = gl; k < n; k += 8) {
        float x, y;
        load(d, k, x, y);
        two_float_add(x, y, s, c, A);
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const float q = __shfl_xor_sync(kFull, s, o);
      const float t = __fadd_rn(s, q);
      // the two lanes join the same pair in either order: two-sum is exact, so
      // both hold the same value
      const float z = __fsub_rn(t, s);
      const float r = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(q, z));
      c = __fadd_rn(__fadd_rn(c, __shfl_xor_sync(kFull, c, o)), r);
      A = __fadd_ru(A, __shfl_xor_sync(kFull, A, o));
      s = t;
    }
    const float f = __fadd_rn(s, c);
    const float z = __fsub_rn(f, s);
    const float r = __fadd_rn(__fsub_rn(s, __fsub_rn(f, z)), __fsub_rn(c, z));
    const float err = __fadd_ru(__fmul_ru(__fmul_ru(A, 1.0001f), __fmul_ru(K, unit)),
                                __fmul_ru(static_cast<float>(n), 2.8e-45f));
    const bool ok = A > 0.0f && __fadd_rn(f, __fadd_ru(r, err)) == f && __fadd_rn(f, __fadd_rd(r, -err)) == f;
    if (d < dots && gl == 0 && ok) put(d, f);
    unsigned left = __ballot_sync(kFull, d < dots && gl == 0 && !ok);
    while (left != 0u) {
      const int df = d0 + ((__ffs(left) - 1) >> 3);
      left &= left - 1u;
      const float v = warp_seq_dot(n, [&](int k, float& x, float& y) { load(df, k, x, y); }, lane);
      if (lane == 0) put(df, v);
    }
  }
}

constexpr int kLoadChunk = 1024;  // rows of a block_loading chunk

// Fixed points from which a product's remainder lost to underflow (at most 2^-150)
// counts less than a quarter of a unit, within the units round_check is given.
constexpr int kMinLsb = -148;

// v as a multiple of 2^LSB (truncated below it)
__device__ __forceinline__ long long exact_fixed_value(float v, int LSB) {
  const unsigned u = __float_as_uint(v), b = (u >> 23) & 0xffu;
  const long long m = (u & 0x7fffffu) | (b ? 0x800000u : 0u);
  const int sh = (b ? static_cast<int>(b) - 150 : -149) - LSB;
  const long long f = sh >= 0 ? (sh < 63 ? m << sh : 0ll) : (sh > -64 ? m >> -sh : 0ll);
  return (u >> 31) ? -f : f;
}

// float(S_seq) of sum sc[t]^2 over t < n, by the whole block: the sums of
// eight terms as above.  `red` holds 2 kEvalWarps words plus alignment.
__device__ float block_norm2(const float* __restrict__ sc, int n, void* scratch, int lane, int warp) {
  long long* vred = reinterpret_cast<long long*>((reinterpret_cast<uintptr_t>(scratch) + 7) & ~uintptr_t(7));
  float* ared = reinterpret_cast<float*>(vred + kEvalWarps);
  int* mred = reinterpret_cast<int*>(ared + kEvalWarps);
  int mx = 1;
  for (int t = threadIdx.x; t < n; t += kEvalThreads) mx = max(mx, biased_exp1(sc[t]));
  mx = __reduce_max_sync(kFull, mx);
  if (lane == 0) mred[warp] = mx;
  __syncthreads();
  mx = __reduce_max_sync(kFull, mred[lane & (kEvalWarps - 1)]);
  const int LSB = 2 * mx - 252 + clog2i(n) - 62;
  long long acc = 0;
  float A = 0.0f;
  for (int t0 = threadIdx.x; t0 < n; t0 += 8 * kEvalThreads) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = t0 + q * kEvalThreads < n ? sc[t0 + q * kEvalThreads] : 0.0f;
    float hi = 0.0f, lo = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) two_float_add(v[q], v[q], hi, lo, A);
    acc += exact_fixed_value(hi, LSB) + exact_fixed_value(lo, LSB);
  }
  acc = warp_sum_i64(acc);
  A = warp_sum_ru(A);
  if (lane == 0) {
    vred[warp] = acc;
    ared[warp] = A;
  }
  __syncthreads();
  acc = 0;
  A = 0.0f;
  for (int q = 0; q < kEvalWarps; ++q) {
    acc += vred[q];
    A = __fadd_ru(A, ared[q]);
  }
  float out = 0.0f;
  if (!(LSB >= kMinLsb && A > 0.0f && A < 1e37f && round_check(acc, LSB, __fmul_ru(A, 1.0001f), n + 2880, out)))
    out = warp_seq_dot(n, [&](int k, float& x, float& y) {
      x = sc[k];
      y = sc[k];
    }, lane);
  __syncthreads();
  return out;
}

// loading[j] = float(S_seq) of sum over training rows k (ascending) of
// double(Z[tix[k]][j]) * double(sc[k]), for every column j: t_mat_vec_float
// of the scores path (plscv.cpp:884).  A thread per column and row group, so
// the loads of a row are coalesced, and one pass over the rows: the fixed
// point of warp_exact_dot is placed from an upper bound of the largest
// product exponent, zexp[j] (the column's largest exponent, label
// independent) plus the scores' largest exponent, instead of the exact one
// (every term still fits: the bound only lowers the magnitudes).  The row
// indices and scores are staged in shared memory so the loads of Z issue
// back to back.  Partial sums of row groups combine exactly (integers), the
// partial bounds of sum |x y| rounding upward; the check and the sequential
// fallback are those of warp_exact_dot / warp_seq_dot.  `scratch` holds
// 4 * kEvalThreads + 2 * kLoadChunk words plus 8 bytes of alignment; every
// thread of the block calls this.
__device__ void block_loading(const float* __restrict__ Zs, int zp, int p, const int* __restrict__ tix, int nt,
                              const float* __restrict__ sc, const int* __restrict__ zexp, float* ld, float* scratch,
                              int lane, int warp) {
  long long* pacc = reinterpret_cast<long long*>((reinterpret_cast<uintptr_t>(scratch) + 7) & ~uintptr_t(7));
  float* pA = reinterpret_cast<float*>(pacc + kEvalThreads);
  int* pflag = reinterpret_cast<int*>(pA + kEvalThreads);  // non-zero values seen
  // a row's offset and score together
  int2* srow = reinterpret_cast<int2*>((reinterpret_cast<uintptr_t>(pflag + kEvalThreads) + 7) & ~uintptr_t(7));
  int* flist = reinterpret_cast<int*>(pacc);  // undecided columns (after the partials are read)
  __shared__ int fcount, smax;
  const int t = threadIdx.x, lg = clog2i(nt);
  if (t == 0) smax = 1;
  __syncthreads();
  {
    int m = 1;
    for (int k = t; k < nt; k += kEvalThreads) m = max(m, biased_exp1(sc[k]));
    m = __reduce_max_sync(kFull, m);
    if (lane == 0) atomicMax(&smax, m);
  }
  __syncthreads();
  const int se = smax;
  for (int j0 = 0; j0 < p; j0 += kEvalThreads) {
    const int PB = min(p - j0, kEvalThreads), G = kEvalThreads / PB;
    const int g = t / PB, jj = t - g * PB, j = j0 + jj;
    const bool on = g < G;
    const int LSB = (on ? zexp[j] : 1) + se - 252 + lg - 62;
    long long acc = 0;
    float A = 0.0f;
    unsigned nz = 0u;
    for (int k0 = 0; k0 < nt; k0 += kLoadChunk) {
      const int cn = min(kLoadChunk, nt - k0);
      for (int i = t; i < cn; i += kEvalThreads) {
        srow[i] = make_int2(tix[k0 + i] * zp, __float_as_int(sc[k0 + i]));
      }
      __syncthreads();
      if (on) {
        const float* zj = Zs + j;
        // eight terms in two floats (group_seq_dots), then as fixed point
        auto add = [&](const float (&v)[8], const float (&y)[8]) {
          float hi = 0.0f, lo = 0.0f;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            two_float_add(v[q], y[q], hi, lo, A);
            nz |= __float_as_uint(v[q]);
          }
          acc += exact_fixed_value(hi, LSB) + exact_fixed_value(lo, LSB);
        };
        // the next eight rows' values load while these eight are added
        float v[8], y[8], nv[8], ny[8];
        auto fetch = [&](int i0) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int2 r = srow[i0 + q * G];
            nv[q] = zj[r.x];
            ny[q] = __int_as_float(r.y);
          }
        };
        int i0 = g;
        if (i0 + 7 * G < cn) {
          fetch(i0);
          for (; i0 + 15 * G < cn; i0 += 8 * G) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              v[q] = nv[q];
              y[q] = ny[q];
            }
            fetch(i0 + 8 * G);
            add(v, y);
          }
          add(nv, ny);
          i0 += 8 * G;
        }
        if (i0 < cn) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int2 r = i0 + q * G < cn ? srow[i0 + q * G] : make_int2(0, 0);
            v[q] = i0 + q * G < cn ? zj[r.x] : 0.0f;
            y[q] = __int_as_float(r.y);
          }
          add(v, y);
        }
      }
      __syncthreads();
    }
    if (on) {
      pacc[t] = acc;
      pA[t] = A;
      pflag[t] = static_cast<int>(nz << 1);
    }
    __syncthreads();
    float out = 0.0f;
    bool ok = false;
    if (t < PB) {
      int fl = pflag[t];
      for (int q = 1; q < G; ++q) {
        acc += pacc[t + q * PB];
        A = __fadd_ru(A, pA[t + q * PB]);
        fl |= pflag[t + q * PB];
      }
      // a column of zeros; else the check, which counts the roundings of the
      // eight-term sums (below 180 u^2 A) as 16 x 180 terms more; A is not
      // finite where a value is not, and zero where products were lost; a column
      // so small that remainders were lost (kMinLsb) takes the chain
      if (fl == 0) ok = true;
      else if (LSB >= kMinLsb && A > 0.0f && A < 1e37f)
        ok = round_check(acc, LSB, __fmul_ru(A, 1.0001f), nt + 2880, out);
    }
    if (t == 0) fcount = 0;
    __syncthreads();
    if (t < PB) {
      if (ok) ld[j] = out;
      else flist[atomicAdd(&fcount, 1)] = j;
    }
    __syncthreads();
    const int nf = fcount;
    for (int f = warp; f < nf; f += kEvalWarps) {
      const int jf = flist[f];
      const double s = warp_fma_chain(nt, [&](int k, float& x, float& y) {
        x = Zs[static_cast<size_t>(tix[k]) * zp + jf];
        y = sc[k];
      }, lane);
      if (lane == 0) ld[jf] = __double2float_rn(s);
    }
    __syncthreads();
  }
}

}  // namespace

}  // namespace kgb
