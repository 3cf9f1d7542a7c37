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
// Columns kk >= ka of A come from A2 (ld lda2) at kk - ka (ka = k: A alone), column kk < ka is column perm[kk] - 1 of A
// where perm is given.  LSB: also the
// rows' smallest lsb_exp over their nonzero entries (alsb, initialised above every exponent).
__device__ __forceinline__ const double* acol(const double* A, long lda, const double* A2, long lda2, int ka,
                                              int kk, const int* perm) {
  return kk < ka ? A + (long)(perm ? __ldg(perm + kk) - 1 : kk) * lda : A2 + (long)(kk - ka) * lda2;
}

// The first of columns [k0, k1) and their distance where they are one run of A or of A2, nullptr otherwise: the choice
// per element is a good part of a pass's instructions (residues of 32 products' A: 955 -> 807 us without it).
__device__ __forceinline__ const double* acol_run(const double* A, long lda, const double* A2, long lda2, int ka, int k0,
                                                  int k1, const int* perm, long* step) {
  if (k0 >= ka) {
    *step = lda2;
    return A2 + (long)(k0 - ka) * lda2;
  }
  *step = lda;
  return k1 <= ka && !perm ? A + (long)k0 * lda : nullptr;
}

template <bool LSB = false>
__device__ __forceinline__ void row_absmax_blk(const double* __restrict__ A, long lda, const double* A2, long lda2,
                                               int ka, int n, int k, int kchunk,
                                               unsigned long long* __restrict__ amax_bits,
                                               double* __restrict__ asq, int bx, int by,
                                               int* __restrict__ alsb = nullptr, const int* perm = nullptr) {
  int i = bx * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int k0 = by * kchunk, k1 = min(k, k0 + kchunk);
  unsigned long long mb = 0;
  float sq32 = 0.0f;
  int e = NO_SCALE;  // set by the first group with a nonzero entry
  bool big = false;
  int lsb = NO_LSB;
  int kk = k0;
  long step;
  const double* run = acol_run(A, lda, A2, lda2, ka, k0, k1, perm, &step);
  const double* p = run + i;
  // eight independent loads in flight per thread (a warp reads 32 consecutive rows)
  for (; kk + 8 <= k1; kk += 8) {
    unsigned long long b[8];
    if (run) {
#pragma unroll
      for (int u = 0; u < 8; ++u, p += step) b[u] = (unsigned long long)__double_as_longlong(__ldg(p)) & ABS_MASK;
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        b[u] = (unsigned long long)__double_as_longlong(__ldg(acol(A, lda, A2, lda2, ka, kk + u, perm) + i)) & ABS_MASK;
    }
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
        (unsigned long long)__double_as_longlong(__ldg(acol(A, lda, A2, lda2, ka, kk, perm) + i)) & ABS_MASK;
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
      const double a = __ldg(acol(A, lda, A2, lda2, ka, kk, perm) + i);
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

// Small operands (M + N at most SMALL_ROWS, K at most SMALL_K): the statistics of A's rows and H's columns are one
// launch, the residues of both another; up to INLINE_ROWS the latter's blocks each evaluate the parameters for
// themselves.  Their passes take a few microseconds each, so that the launches set the time.  Toeplitz, separate
// passes / these, split: n = 256 58.7 / 28.1 us, 1024 108.7 / 81.6, 2048 331 / 305, 3072 the same; FP64: 256 35.8 / 24.2,
// 1024 97.5 / 92.7, 2048 357 / 354, 3072 the same.  Parameters in line / in a launch of their own, split: n = 256
// 28.1 / 29.4, 384 33.0 / 32.3, 512 41.3 / 36.5; FP64: 256 24.2 / 27.7, 384 33.4 / 29.9, 512 47.6 / 38.1.
constexpr int SMALL_ROWS = 4096, SMALL_K = 2048, INLINE_ROWS = 512;
// Rows of A's residue tiles: 16 (one quad a thread) while their blocks do not fill the SMs, 64 otherwise.  FP64
// Toeplitz, 64 / 16: n = 384 34.2 / 29.9 us, 512 40.4 / 38.1, 768 58.9 / 56.7, 1024 92.7 / 92.4, 2048 354 / 366.
constexpr int SMALL_TILE16 = 1536;
inline int small_tile_rows(int M, int N) { return M + N <= SMALL_TILE16 ? 16 : 64; }
static_assert(INLINE_ROWS <= SMALL_TILE16, "the launches with parameters in line have tiles of 16 rows");
inline bool small_operands(int M, int N, int K) { return M + N <= SMALL_ROWS && K <= SMALL_K; }
constexpr int SMALL_RB = 8;  // rows of A a statistics block covers, 256 threads

// Row maxima, squared norms (and lowest bits) of rows 8 b .. 8 b + 7 over all of K, not accumulated into
// what was there: a warp takes 8 rows of 4 columns (64-byte runs), the block 32 columns a step, eight steps in
// flight.  32 rows a block (whole 256-byte runs, a quarter of the blocks) left a chain of 16 such groups of loads at
// K = 1024, the longest of the launch (Toeplitz n = 1024 with 32 rows: FP64 some 20 us more of 93, split 15 of 82).
template <bool LSB>
__device__ __forceinline__ void small_rows_blk(const double* __restrict__ A, long lda, int n, int k, int b,
                                               unsigned long long* __restrict__ amax_bits, double* __restrict__ asq,
                                               int* __restrict__ alsb) {
  __shared__ unsigned long long sm[8][8];
  __shared__ double sq[8][8];
  __shared__ int sl[8][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, row = lane & 7, c0 = 4 * wid + (lane >> 3), i = b * SMALL_RB + row;
  unsigned long long mb = 0;
  float s32 = 0.0f;
  int e = NO_SCALE, lsb = NO_LSB;
  bool big = false;
  for (int k0 = c0; k0 < k; k0 += 256) {
    unsigned long long v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int kk = k0 + 32 * u;
      v[u] = (i < n && kk < k) ? (unsigned long long)__double_as_longlong(__ldg(A + i + (long)kk * lda)) & ABS_MASK : 0ull;
    }
    unsigned long long gm = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) gm = v[u] > gm ? v[u] : gm;
    mb = gm > mb ? gm : mb;
    if constexpr (LSB) {
#pragma unroll
      for (int u = 0; u < 8; ++u) lsb = v[u] ? min(lsb, lsb_exp(v[u])) : lsb;
    }
    if (e == NO_SCALE && gm) e = (int)(gm >> 52) - 1023;
    if (e != NO_SCALE) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float f = abs_scaled_up(v[u], e, &big);
        s32 = __fmaf_ru(f, f, s32);
      }
    }
  }
  double q = 0.0;
  if (big) {  // entries 2^56 times the thread's first ones (or Inf/NaN): FP64 sum
    for (int kk = c0; kk < k; kk += 32) {
      const double x = i < n ? __ldg(A + i + (long)kk * lda) : 0.0;
      q = fma(x, x, q);
    }
  } else if (e != NO_SCALE) {
    q = ldexp((double)s32, 2 * e);
  }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) {
    const unsigned long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = ob > mb ? ob : mb;
    q += __shfl_xor_sync(0xffffffffu, q, o);
    if constexpr (LSB) lsb = min(lsb, __shfl_xor_sync(0xffffffffu, lsb, o));
  }
  if (lane < 8) {
    sm[wid][row] = mb;
    sq[wid][row] = q;
    if constexpr (LSB) sl[wid][row] = lsb;
  }
  __syncthreads();
  if (threadIdx.x < 8 && i < n) {
    for (int w = 1; w < 8; ++w) {
      mb = sm[w][row] > mb ? sm[w][row] : mb;
      q += sq[w][row];
      if constexpr (LSB) lsb = min(lsb, sl[w][row]);
    }
    amax_bits[i] = mb;
    asq[i] = q;
    if constexpr (LSB) alsb[i] = lsb;
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

// Exponents of a row or column that make every product with it zero, or NaN: beyond any sum of two others.
constexpr int EXP_ZERO = 1 << 20, EXP_NAN = 1 << 24;

// i128_scaled's rare results: zero, few bits, outside the normal range, EXP_ZERO and EXP_NAN.  Out of line, so that its
// FP64 instructions are not issued (predicated off) for every element.
static __device__ __noinline__ double i128_scaled_rare(unsigned long long hi, unsigned long long lo, bool neg, int e) {
  if (e >= EXP_ZERO / 2) return e < EXP_NAN / 2 ? 0.0 : __longlong_as_double(0x7FF8000000000000ll);
  if ((hi | lo) == 0) return 0.0;
  const int s = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
  const int p = 127 - s;  // exponent of the leading bit
  const unsigned long long top = s >= 64 ? lo << (s - 64) : s ? (hi << s) | (lo >> (64 - s)) : hi;
  const unsigned long long rest = s >= 64 ? 0 : lo << s;
  unsigned long long m = top >> 11;  // 53 bits
  const bool sticky = (top & 0x3FFull) != 0 || rest != 0;
  if ((top & 0x400ull) && (sticky || (m & 1))) ++m;
  const double v = ldexp((double)m, p - 52 - e);
  return neg ? -v : v;
}

// z * 2^-e as a double, rounded to nearest even from the bits; results outside the normal range go through ldexp.
__device__ __forceinline__ double i128_scaled(__int128 z, int e) {
  const bool neg = z < 0;
  const unsigned __int128 sg = neg ? ~(unsigned __int128)0 : 0, u = ((unsigned __int128)z ^ sg) - sg;
  unsigned w3 = (unsigned)(u >> 96), w2 = (unsigned)(u >> 64), w1 = (unsigned)(u >> 32), w0 = (unsigned)u;
  int x = 127 + 1022 - e;  // biased exponent of bit 31 of w3, less one
  if (w3 == 0) {
    w3 = w2; w2 = w1; w1 = w0; w0 = 0;
    x -= 32;
  }
  const int s = __clz((int)w3);
  x -= s;
  if (w3 == 0 || (unsigned)x >= 2045u) return i128_scaled_rare((unsigned long long)(u >> 64), (unsigned long long)u, neg, e);
  const unsigned t3 = __funnelshift_l(w2, w3, s), t2 = __funnelshift_l(w1, w2, s);
  const unsigned rest = (__funnelshift_l(w0, w1, s) | (w0 << s)) != 0 ? 1u : 0u;
  // the 11 bits below the last kept one, a sticky bit, that last bit
  const unsigned up = (((t2 & 0x7FFu) | rest) + 0x3FFu + ((t2 >> 11) & 1u)) >> 11;
  // the leading bit of t3 >> 11 adds one to the exponent field, a carry out of the mantissa another
  const unsigned head = ((unsigned)x << 20) + (t3 >> 11) + (neg ? 0x80000000u : 0u);
  return __longlong_as_double((long long)((((unsigned long long)head << 32) | ((t3 << 21) | (t2 >> 11))) + up));
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
  // Block maximum first; then every thread's sums on its exponent (round-up FP32: the FP64 pipe's two lanes
  // made the former FP64 reductions and ldexps some 3000 cycles a column).
  __shared__ unsigned long long smax[32], smax_all[32];
  __shared__ float ssum[32], ssq[32];
  __shared__ int slsb[32];
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31, nw = blockDim.x >> 5;
  if constexpr (LSB) {
    lsb = __reduce_min_sync(0xffffffffu, lsb);
    if (ln == 0) slsb[wid] = lsb;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ob = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = ob > mb ? ob : mb;
  }
  if (hmax_all) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ob = __shfl_xor_sync(0xffffffffu, mb_all, o);
      mb_all = ob > mb_all ? ob : mb_all;
    }
  }
  if (ln == 0) {
    smax[wid] = mb;
    smax_all[wid] = mb_all;
  }
  __syncthreads();
  unsigned long long bm = 0;
  for (int w2 = 0; w2 < nw; ++w2) bm = smax[w2] > bm ? smax[w2] : bm;
  const int eb = (int)(bm >> 52) - 1023;
  float fs = 0.0f, fq = 0.0f;  // sums of |h| 2^-eb and h^2 2^-2eb, below 2 k and 4 k
  if (bm < INF_BITS) {
    if (big) {  // entries 2^56 times the thread's first one: FP64 sums
      double s = 0.0, s2 = 0.0;
      for (int kk = threadIdx.x; kk < srows; kk += blockDim.x) {
        const double h = ldexp(row[kk], -eb);
        s += fabs(h);
        s2 = fma(h, h, s2);
      }
      fs = __double2float_ru(s);
      fq = __double2float_ru(s2);
    } else if (e != NO_SCALE) {
      const int d = max(e - eb, -126), d2 = max(2 * (e - eb), -126);  // e <= eb
      fs = __fmul_ru(s32, __uint_as_float((unsigned)(127 + d) << 23));
      fq = __fmul_ru(s2_32, __uint_as_float((unsigned)(127 + d2) << 23));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    fs = __fadd_ru(fs, __shfl_xor_sync(0xffffffffu, fs, o));
    fq = __fadd_ru(fq, __shfl_xor_sync(0xffffffffu, fq, o));
  }
  if (ln == 0) {
    ssum[wid] = fs;
    ssq[wid] = fq;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w2 = 1; w2 < nw; ++w2) {
      fs = __fadd_ru(fs, ssum[w2]);
      fq = __fadd_ru(fq, ssq[w2]);
      mb_all = smax_all[w2] > mb_all ? smax_all[w2] : mb_all;
      if constexpr (LSB) lsb = min(lsb, slsb[w2]);
    }
    if (hmax_all) hmax_all[j] = mb_all;
    hmax_bits[j] = bm;
    const bool finite = bm < INF_BITS;
    hsum[j] = finite ? ldexp((double)fs, eb) : __longlong_as_double((long long)bm);
    hsq[j] = finite ? ldexp((double)fq, 2 * eb) : __longlong_as_double((long long)bm);
    if constexpr (LSB) hlsb[j] = lsb;
    if (prm != nullptr && bm > 0 && finite) {
      const float m = __uint_as_float(0x3F800000u | ((unsigned)(bm >> 29) & 0x7FFFFFu));
      const double rho = bm >> 52 ? (double)__fdiv_ru(fs, m) : (double)srows;
      atomicMax(&prm->rho_bits, (unsigned long long)__double_as_longlong(rho));
    }
  }
}

}  // namespace psmma
