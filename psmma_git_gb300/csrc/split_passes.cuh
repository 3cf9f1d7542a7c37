// Device passes shared by the modular paths (split_crt.cu, exact_crt.cu, ntt_th.cu): the statistics of A's
// rows, the generation of H with its column statistics, the integer scaling and the rounding back.
#pragma once

#include <cuda_runtime.h>

#include "psmma_internal.h"
#include "tcgen05_util.cuh"

namespace psmma {

// Device-side parameters of one call (in the workspace).
constexpr int PARAMS_BLOCKS = 32;  // blocks of the single-product parameter pass

struct SplitDevParams {
  unsigned status;
  int PA, PH;                   // bits of the integer-scaled A (per row) and H (per column)
  unsigned long long rho_bits;  // max_j sum_k |H_kj| / max_k |H_kj| (bits of a positive double)
  unsigned done;                // parameter-pass blocks finished
  unsigned hbad;                // block-recursive products: some column of H is not finite
  double part[PARAMS_BLOCKS][6];  // their partial ratio maxima and sums, combined in block order
};

constexpr unsigned long long ABS_MASK = 0x7FFFFFFFFFFFFFFFull;
constexpr unsigned long long INF_BITS = 0x7FF0000000000000ull;
constexpr int NO_SCALE = -100000;

// The bound sums (row sums of squares of A, column sums of |H| and of H^2) are accumulated in
// FP32 on a per-thread power-of-two scale, because GB300 issues FP64 at about one operation
// per SM per cycle.  abs_scaled_up gives |x| * 2^-e as a float that is never below the true
// value (top 23 mantissa bits, rounded up; magnitudes under 2^-126 become 2^-126), from the
// bits of x on the integer pipe, and sets *big when |x| * 2^-e >= 2^56 (then the caller sums
// that thread's values in FP64 instead).  With round-up FP32 adds the sums stay upper bounds.
__device__ __forceinline__ float abs_scaled_up(unsigned long long ab, int e, bool* big) {
  const int fe = (int)(ab >> 52) - 1023 - e + 127;
  *big |= fe >= 127 + 56;
  const int fc = max(1, min(fe, 254));
  unsigned fb = ((unsigned)fc << 23) | ((unsigned)(ab >> 29) & 0x7FFFFFu);
  fb += (fe < 1 || (ab & 0x1FFFFFFFull) != 0ull) ? 1u : 0u;
  return ab ? __uint_as_float(fb) : 0.0f;
}

// Exponent of the lowest set bit of a finite nonzero double, from the bits of its magnitude: the
// value is an integer times 2^lsb_exp.
constexpr int NO_LSB = 0x7FFFFFFF;
__device__ __forceinline__ int lsb_exp(unsigned long long ab) {
  const int ex = (int)(ab >> 52);
  const unsigned long long m = (ab & 0xFFFFFFFFFFFFFull) | (ex ? 1ull << 52 : 0ull);
  return (ex ? ex : 1) - 1075 + __ffsll((long long)m) - 1;
}

// Row max of |A| as the bits of a non-negative double (NaN/Inf compare above all finite) and
// row sums of squares (for the Cauchy-Schwarz bound of the integer product).
// Columns kk >= ka of A come from A2 (ld lda2) at kk - ka (ka = k: A alone).  LSB: also the
// rows' smallest lsb_exp over their nonzero entries (alsb, initialised above every exponent).
__device__ __forceinline__ const double* acol(const double* A, long lda, const double* A2, long lda2, int ka,
                                              int kk) {
  return kk < ka ? A + (long)kk * lda : A2 + (long)(kk - ka) * lda2;
}

template <bool LSB = false>
__device__ __forceinline__ void row_absmax_blk(const double* __restrict__ A, long lda, const double* A2, long lda2,
                                               int ka, int n, int k, int kchunk,
                                               unsigned long long* __restrict__ amax_bits,
                                               double* __restrict__ asq, int bx, int by,
                                               int* __restrict__ alsb = nullptr) {
  int i = bx * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int k0 = by * kchunk, k1 = min(k, k0 + kchunk);
  unsigned long long mb = 0;
  float sq32 = 0.0f;
  int e = NO_SCALE;  // set by the first group with a nonzero entry
  bool big = false;
  int lsb = NO_LSB;
  int kk = k0;
  // eight independent loads in flight per thread (a warp reads 32 consecutive rows)
  for (; kk + 8 <= k1; kk += 8) {
    unsigned long long b[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      b[u] = (unsigned long long)__double_as_longlong(__ldg(acol(A, lda, A2, lda2, ka, kk + u) + i)) & ABS_MASK;
    unsigned long long gm = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) gm = b[u] > gm ? b[u] : gm;
    if constexpr (LSB) {
#pragma unroll
      for (int u = 0; u < 8; ++u) lsb = b[u] ? min(lsb, lsb_exp(b[u])) : lsb;
    }
    mb = gm > mb ? gm : mb;
    if (e == NO_SCALE && gm) e = (int)(gm >> 52) - 1023;
    if (e != NO_SCALE) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float f = abs_scaled_up(b[u], e, &big);
        sq32 = __fmaf_ru(f, f, sq32);
      }
    }
  }
  for (; kk < k1; ++kk) {
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(__ldg(acol(A, lda, A2, lda2, ka, kk) + i)) & ABS_MASK;
    mb = b > mb ? b : mb;
    if constexpr (LSB) lsb = b ? min(lsb, lsb_exp(b)) : lsb;
    if (e == NO_SCALE && b) e = (int)(b >> 52) - 1023;
    if (e != NO_SCALE) {
      const float f = abs_scaled_up(b, e, &big);
      sq32 = __fmaf_ru(f, f, sq32);
    }
  }
  double sq = 0.0;
  if (big) {  // entries 2^56 times the thread's first ones (or Inf/NaN): FP64 sum
    for (kk = k0; kk < k1; ++kk) {
      const double a = __ldg(acol(A, lda, A2, lda2, ka, kk) + i);
      sq = fma(a, a, sq);
    }
  } else if (e != NO_SCALE) {
    sq = ldexp((double)sq32, 2 * e);
  }
  if (mb) atomicMax(amax_bits + i, mb);
  if (sq != 0.0) atomicAdd(asq + i, sq);
  if constexpr (LSB) {
    if (lsb != NO_LSB) atomicMin(alsb + i, lsb);
  }
}

// floor(log2 x) from the bits of a positive finite double, on the integer pipe (GB300's FP64
// pipe is narrow, and the library ilogb goes through it).
__device__ __forceinline__ int ilogb_bits(unsigned long long b) {
  const int ex = (int)(b >> 52);
  return ex ? ex - 1023 : 63 - __clzll((long long)b) - 1074;  // subnormal: b is the mantissa
}

// Exponent s such that |x * 2^s| < 2^P for all |x| <= amax (amax finite, > 0).
__device__ __forceinline__ int scale_exp(unsigned long long amax_bits, int P) {
  return P - 1 - ilogb_bits(amax_bits);
}

// rint(x * 2^e) (round half to even) for finite x with |x * 2^e| < 2^53, computed from the
// bits of x with integer operations only; *neg receives the sign.
__device__ __forceinline__ unsigned long long scaled_int(double x, int e, bool* neg) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  *neg = (b >> 63) != 0;
  const int ex = (int)((b >> 52) & 0x7FF);
  unsigned long long m = b & 0xFFFFFFFFFFFFFull;
  int E = -1074;
  if (ex != 0) {
    m |= 1ull << 52;
    E = ex - 1075;
  }
  const int sh = E + e;
  if (sh >= 0) return m << sh;  // the caller's bound keeps the result below 2^53
  const int k = -sh;
  if (k > 63) return 0;  // below one half
  // round half to even: m / 2^k + 1/2 - 2^-k, plus 2^-k when the last kept bit is odd
  return (m + ((1ull << (k - 1)) - 1) + ((m >> k) & 1)) >> k;
}

// m * 2^x with the sign, for results outside the normal range; out of line, so that its FP64
// instructions are not issued (predicated off) for every element.
static __device__ __noinline__ double scaled_outside_normal(unsigned long long m, int x, bool neg) {
  const double v = ldexp((double)m, x);
  return neg ? -v : v;
}

// (hi:lo) * 2^-e as a double, (hi:lo) a non-negative 128-bit integer in two words, rounded
// to nearest even from the bits; results outside the normal range go through ldexp.
__device__ __forceinline__ double u128w_scaled(unsigned long long hi, unsigned long long lo, bool neg, int e) {
  if ((hi | lo) == 0) return 0.0;
  // normalise so that the leading bit is bit 63 of `top`; `rest` keeps the bits below
  int p;
  unsigned long long top, rest;
  if (hi) {
    const int s = __clzll((long long)hi);
    p = 127 - s;
    top = s ? (hi << s) | (lo >> (64 - s)) : hi;
    rest = s ? (lo << s) : lo;
  } else {
    const int s = __clzll((long long)lo);
    p = 63 - s;
    top = lo << s;
    rest = 0;
  }
  unsigned long long m = top >> 11;  // 53 bits
  const unsigned long long low11 = top & 0x7FFull;
  const bool sticky = (low11 & 0x3FFull) != 0 || rest != 0;
  if ((low11 & 0x400ull) && (sticky || (m & 1))) {
    ++m;
    if (m == (1ull << 53)) {
      m >>= 1;
      ++p;
    }
  }
  const int field = p - e + 1023;
  if (field >= 1 && field <= 2046) {
    unsigned long long bits = ((unsigned long long)field << 52) | (m & 0xFFFFFFFFFFFFFull);
    if (neg) bits |= 1ull << 63;
    return __longlong_as_double((long long)bits);
  }
  return scaled_outside_normal(m, p - 52 - e, neg);
}

// H pass 1: Ht[j][kk] = H(kk, j) in FP64, column max |H| and column sum |H|, and the global
// ratio rho = max_j sum/max over finite columns (prm; nullptr: not kept).  One block per column j.
template <int KIND, bool LSB = false>
// hmax_all != nullptr receives the column maximum over every generated row (with gs.srows the
// statistics cover the first srows rows only).  LSB: also the column's smallest lsb_exp (hlsb).
__device__ __forceinline__ void h_pass1_blk(const GenSpec& gs, int K, int kp, double* __restrict__ Ht,
                                            unsigned long long* __restrict__ hmax_bits, double* __restrict__ hsum,
                                            double* __restrict__ hsq, SplitDevParams* prm, int j,
                                            unsigned long long* __restrict__ hmax_all = nullptr,
                                            int* __restrict__ hlsb = nullptr) {
  double w = 0.0, v = 0.0, w1 = 0.0, dlj = 0.0, drj = 0.0;
  VSplit vs;
  vs.ok = false;
  if (KIND == KIND_CAUCHY || KIND == KIND_CAUCHY_EIG) {
    w = __ldg(gs.Fc + j);   // F(j)
    v = __ldg(gs.Vc + j);   // V(j)
    vs = v_split(v);
  }
  if (KIND == KIND_CAUCHY_EIG) {
    dlj = __ldg(gs.dl + j);  // DIFL(j)
    if (j < gs.fc1_len) {
      w1 = __ldg(gs.Fc1 + j);  // F(j+1)
      drj = __ldg(gs.dr + j);  // DIFR(j)
    }
  }
  unsigned long long mb = 0, mb_all = 0;
  int lsb = NO_LSB;
  float s32 = 0.0f, s2_32 = 0.0f;
  int e = NO_SCALE;  // set by the thread's first nonzero entry
  bool big = false;
  const long srows = gs.srows > 0 ? gs.srows : (long)kp;
  double* row = Ht + (long)j * kp;
  for (int kk = threadIdx.x; kk < kp; kk += blockDim.x) {
    double h = 0.0;
    if (kk < K) {
      if (KIND == KIND_CAUCHY) {
        if (gs.k1 > 0 && kk >= gs.k1) {
          const int t = kk - gs.k1;  // tail rows: dense, or Cauchy with the second row generators
          h = gs.B ? __ldg(gs.B + t + (long)j * gs.ldb) : cauchy_entry(__ldg(gs.Ur2 + t), v, vs, __ldg(gs.Dr2 + t) - w);
        } else {
          double d = __ldg(gs.Dr + kk), u = __ldg(gs.Ur + kk);
          h = cauchy_entry(u, v, vs, d - w);  // U(i)*V(j) / (D(i)-F(j))
        }
      } else if (KIND == KIND_CAUCHY_EIG) {
        if (gs.k1 > 0 && kk >= gs.k1) {
          // tail rows of merged products: dense, or CauchyEig rows in permuted order
          const int t = kk - gs.k1;
          h = gs.B ? __ldg(gs.B + t + (long)j * gs.ldb)
                   : cauchy_entry(__ldg(gs.Ur2 + t), v, vs,
                                  eig_den(__ldg(gs.Dr2 + t), w, w1, dlj, drj, __ldg(gs.rglob2 + t) - 1 <= gs.cg0 + j));
        } else {
          const double fi = __ldg(gs.Dr + kk), u = __ldg(gs.Ur + kk);
          const bool upper = gs.rglob ? (__ldg(gs.rglob + kk) - 1 <= gs.cg0 + j) : (kk - j <= gs.diag_off);
          h = cauchy_entry(u, v, vs, eig_den(fi, w, w1, dlj, drj, upper));
        }
      } else if (KIND == KIND_TOEPLITZ || KIND == KIND_HANKEL) {
        if (gs.k1 > 0 && kk >= gs.k1) {  // dense tail rows (the R P^T factor of a merged product)
          h = __ldg(gs.B + (kk - gs.k1) + (long)j * gs.ldb);
        } else {
          const long idx = KIND == KIND_TOEPLITZ ? (gs.order - 1) + j - kk : (long)kk + j;
          h = (gs.glen <= 0 || (idx >= 0 && idx < gs.glen)) ? __ldg(gs.g + idx) : 0.0;
        }
      } else {  // KIND_DENSE (the split DFT generates F in k_h_pass1_dft3)
        h = __ldg(gs.B + kk + (long)j * gs.ldb);
      }
    }
    row[kk] = h;
    unsigned long long b = (unsigned long long)__double_as_longlong(h) & ABS_MASK;
    mb_all = b > mb_all ? b : mb_all;
    if (kk >= srows) continue;
    mb = b > mb ? b : mb;
    if constexpr (LSB) lsb = b ? min(lsb, lsb_exp(b)) : lsb;
    if (e == NO_SCALE && b) e = (int)(b >> 52) - 1023;
    if (e != NO_SCALE) {
      const float f = abs_scaled_up(b, e, &big);
      s32 = __fadd_ru(s32, f);
      s2_32 = __fmaf_ru(f, f, s2_32);
    }
  }
  double s = 0.0, s2 = 0.0;
  if (big) {  // entries 2^56 times the thread's first one (or Inf/NaN): FP64 sums
    for (int kk = threadIdx.x; kk < srows; kk += blockDim.x) {
      const double h = row[kk];
      s += fabs(h);
      s2 = fma(h, h, s2);
    }
  } else if (e != NO_SCALE) {
    s = ldexp((double)s32, e);
    s2 = ldexp((double)s2_32, 2 * e);
  }
  __shared__ unsigned long long smax[32], smax_all[32];
  __shared__ double ssum[32], ssq[32];
  __shared__ int slsb[32];
  if constexpr (LSB) {
    lsb = __reduce_min_sync(0xffffffffu, lsb);
    if ((threadIdx.x & 31) == 0) slsb[threadIdx.x >> 5] = lsb;
  }
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = ob > mb ? ob : mb;
    ob = __shfl_xor_sync(0xffffffffu, mb_all, o);
    mb_all = ob > mb_all ? ob : mb_all;
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
  if (ln == 0) { smax[wid] = mb; smax_all[wid] = mb_all; ssum[wid] = s; ssq[wid] = s2; }
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    mb = ln < nw ? smax[ln] : 0ull;
    mb_all = ln < nw ? smax_all[ln] : 0ull;
    s = ln < nw ? ssum[ln] : 0.0;
    s2 = ln < nw ? ssq[ln] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
      mb = ob > mb ? ob : mb;
      ob = __shfl_xor_sync(0xffffffffu, mb_all, o);
      mb_all = ob > mb_all ? ob : mb_all;
      s += __shfl_xor_sync(0xffffffffu, s, o);
      s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (ln == 0) {
      if (hmax_all) hmax_all[j] = mb_all;
      hmax_bits[j] = mb;
      hsum[j] = s;
      hsq[j] = s2;
      if constexpr (LSB) {
        for (int w2 = 1; w2 < nw; ++w2) lsb = min(lsb, slsb[w2]);
        hlsb[j] = lsb;
      }
      if (prm != nullptr && mb > 0 && mb < INF_BITS && isfinite(s)) {
        double rho = s / __longlong_as_double((long long)mb);
        atomicMax(&prm->rho_bits, (unsigned long long)__double_as_longlong(rho));
      }
    }
  }
}

}  // namespace psmma
