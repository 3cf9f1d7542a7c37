// Low-rank path of the batched merge level: compression of the off-diagonal blocks of Cauchy
// (and CAUCHYEIG) matrices by RRLU or RRQR, of Toeplitz matrices by RRQR, and the products
// that use the factors.
//
// RRLU (rrluCauchy, Cauchylowrank.f90:7-134; pivoting helpers :137-296): structured
// rank-revealing LU in generator space, one thread block per matrix block.  For a block
// T(i,j) = A(i)V(j)/(D(i)-F(j)) (M x N) it gives
//   T ~= X * Y,  X = P^-1 [I; Z'],  Z'(t,j) = U(Rk+t) W(j) / (LD(Rk+t) - LD(j)),
//                Y(j,c) = LU(j) V(c) / (LD(j) - F(c)),  j <= Rk,
// with LD, LU the pivoted row generators, U the Schur-complement row weights, W the
// interpolation weights and PL the row permutation (compress_cauchy, :387-491).  Both
// factors are Cauchy-like, so A*X*Y runs as two structured multiplies.
//
// RRQR (Compress_RRQR, Auxil_2p5D.f90:1063-1189, with MDGEQP3): the explicit tile is
// factorised by Householder QR with column pivoting on the largest partial column norm,
// truncated at the first |R_kk| <= tol |R_11|.  Left-looking form: with F = T^T V Tau
// (T the pivoted tile, V the reflectors) the partially reduced tile is T - V F^T, so one
// step reads the tile once (F(:,k) = tau_k (T^T v_k - F (V^T v_k))) and writes nothing
// but O(M + N) numbers.  Each tile gets a group of co-resident CTAs (cooperative launch)
// in proportion to its size; the groups synchronise with bounded barriers.
#include "psmma_internal.h"
#include "tcgen05_util.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <vector>

namespace psmma {

// ------------------------------------------------------------------------------------------
// RRLU
// ------------------------------------------------------------------------------------------
struct RrluBlock {
  int M, N;           // block size
  const double *gD, *gU, *gF, *gV;  // generator slices: rows (D, U), columns (F, V)
  double *D, *F;      // row / column poles (permuted in place)
  double *A;          // row weights, permuted with D (becomes LU)
  double *U, *V;      // Schur-complement weights (U becomes Z)
  double* W;          // interpolation weights, min(M, N)
  int *PL, *PU;       // 1-based permutations
  int* rank;          // output Rk
  // resumable state: the kernel stops at a step that needs a complete-pivot search, which a
  // grid-wide kernel does for all such blocks at once (cp_i, cp_j), then resumes
  int k_next;         // step to continue from (1-based)
  int phase;          // 0 running, 1 waiting for the search at step k_next, 2 done
  int cp_i, cp_j;     // search result: 1-based row / column offsets from k_next - 1
  double amax;
};

constexpr int RRLU_THREADS = 512;

// Block-wide argmax of |val| with the smallest index on ties (Fortran MAXLOC).
struct ArgMax {
  double v;
  int i;
};

__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ ArgMax block_argmax(ArgMax x, ArgMax* sm) {
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better(x, y);
  }
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) sm[wid] = x;
  __syncthreads();
  if (wid == 0) {
    x = (ln < (int)(blockDim.x >> 5)) ? sm[ln] : ArgMax{-1.0, 0x7fffffff};
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax y;
      y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
      y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
      x = better(x, y);
    }
    if (ln == 0) sm[32] = x;
  }
  __syncthreads();
  ArgMax r = sm[32];
  __syncthreads();
  return r;
}

__device__ double block_sum(double x, double* sm) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31;
  __syncthreads();
  if (ln == 0) sm[wid] = x;
  __syncthreads();
  if (wid == 0) {
    x = (ln < (int)(blockDim.x >> 5)) ? sm[ln] : 0.0;
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (ln == 0) sm[32] = x;
  }
  __syncthreads();
  double r = sm[32];
  __syncthreads();
  return r;
}

// ---- maxima of quotients ---------------------------------------------------------------------
// The pivot searches compare |u / x| in FP64, and a division is some ten instructions on GB300's two-lane FP64
// pipe, one SM per block of the merge level: that pipe bounded the compression.  qkey orders the quotients from
// their exponents and FP32 mantissas with an error of at most two units (2^-19 each); only quotients within
// QK_SLACK units of the largest key are divided and compared in FP64 -- one or two of thousands -- and the result
// is the full search's, ties included.  64 blocks of 2048 x 2048: 4244 us with every quotient divided, 1608 us so.
// QK_EXACT: zero, subnormal or not finite operands and far exponents, always divided.
constexpr int QK_EXACT = -0x70000000, QK_SLACK = 6;
__device__ __forceinline__ int qkey(double u, double x) {
  const unsigned hu = (unsigned)__double2hiint(u), hx = (unsigned)__double2hiint(x);
  const int eu = (int)(hu >> 20) & 0x7FF, ex = (int)(hx >> 20) & 0x7FF;
  if (eu == 0 || eu == 0x7FF || ex == 0 || ex == 0x7FF || abs(eu - ex) > 900) return QK_EXACT;
  const float mu = __uint_as_float(0x3F800000u | ((hu << 3) & 0x7FFFF8u) | ((unsigned)__double2loint(u) >> 29));
  const float mx = __uint_as_float(0x3F800000u | ((hx << 3) & 0x7FFFF8u) | ((unsigned)__double2loint(x) >> 29));
  return ((eu - ex) << 19) + (int)(__float_as_uint(__fdividef(mu, mx)) >> 4);
}
// The key of (a quotient with key k) times |w|; QK_EXACT as above, and where the product may leave the normal range.
__device__ __forceinline__ int qkey_times(int k, double w) {
  const unsigned h = (unsigned)__double2hiint(w);
  const int e = (int)(h >> 20) & 0x7FF;
  const int ep = (k >> 19) - 127 + e - 1023;
  if (k == QK_EXACT || e == 0 || e == 0x7FF || abs(ep) > 1000) return QK_EXACT;
  const float m = __uint_as_float(0x3F800000u | ((unsigned)(k & 0x7FFFF) << 4));
  const float mw = __uint_as_float(0x3F800000u | ((h << 3) & 0x7FFFF8u) | ((unsigned)__double2loint(w) >> 29));
  return (ep << 19) + (int)(__float_as_uint(m * mw) >> 4);
}

// better() on the bits: the values are -1 or |.|, and a NaN (never better) is passed on as -1.
__device__ __forceinline__ ArgMax better_bits(ArgMax a, ArgMax b) {
  const long long x = __double_as_longlong(a.v), y = __double_as_longlong(b.v);
  return (y > x || (y == x && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ ArgMax warp_argmax(ArgMax x) {
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better_bits(x, y);
  }
  return x;
}
__device__ __forceinline__ ArgMax quotient(double u, double x, int i) {
  const double v = fabs(u / x);
  return ArgMax{__double_as_longlong(v) > 0x7FF0000000000000ll ? -1.0 : v, i};
}

// Shared words of a block's searches.  A search writes `key`, synchronises, reads it, writes `best`,
// synchronises, writes best[32], synchronises: the next one's writes are behind every earlier read.
struct SearchSm {
  int key[32];
  ArgMax best[33];
};

// max_i |u(i) / x(i)| over i in [0, len) and its smallest 1-based index; the whole block.
template <class X>
__device__ ArgMax max_quotient(const double* u, X x, int len, SearchSm& sm) {
  const int wid = threadIdx.x >> 5, ln = threadIdx.x & 31, nw = blockDim.x >> 5;
  int km = QK_EXACT;
  ArgMax best{-1.0, 0x7fffffff};
  for (int i = threadIdx.x; i < len; i += blockDim.x) {
    const double xi = x(i);
    const int k = qkey(u[i], xi);
    if (k == QK_EXACT) best = better_bits(best, quotient(u[i], xi, i + 1));
    km = max(km, k);
  }
  km = __reduce_max_sync(0xffffffffu, km);
  if (ln == 0) sm.key[wid] = km;
  __syncthreads();
  km = __reduce_max_sync(0xffffffffu, ln < nw ? sm.key[ln] : QK_EXACT);
  if (km != QK_EXACT)
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      const double xi = x(i);
      const int k = qkey(u[i], xi);
      if (k != QK_EXACT && k >= km - QK_SLACK) best = better_bits(best, quotient(u[i], xi, i + 1));
    }
  best = warp_argmax(best);
  if (ln == 0) sm.best[wid] = best;
  __syncthreads();
  if (wid == 0) {
    best = warp_argmax(ln < nw ? sm.best[ln] : ArgMax{-1.0, 0x7fffffff});
    if (ln == 0) sm.best[32] = best;
  }
  __syncthreads();
  return sm.best[32];
}

// The same by one warp; *key receives the largest key (QK_EXACT if some quotient has none).  Quotients are
// divided only where the key reaches `floor_key` after the product with |w| (a column that cannot win).
template <class X>
__device__ __forceinline__ ArgMax warp_max_quotient(const double* u, X x, int i0, int len, double w, int floor_key, int* key) {
  const int lane = threadIdx.x & 31;
  int km = QK_EXACT;
  bool special = false;
  for (int i = i0 + lane; i < len; i += 32) {
    const int k = qkey(u[i], x(i));
    special |= k == QK_EXACT;
    km = max(km, k);
  }
  km = __reduce_max_sync(0xffffffffu, km);
  special = __any_sync(0xffffffffu, special);
  const int kw = special ? QK_EXACT : qkey_times(km, w);
  *key = kw;
  ArgMax a{-1.0, 0x7fffffff};
  if (kw != QK_EXACT && floor_key != QK_EXACT && kw < floor_key) return a;
  for (int i = i0 + lane; i < len; i += 32) {
    const double xi = x(i);
    const int k = qkey(u[i], xi);
    if (k == QK_EXACT || k >= km - QK_SLACK) a = better_bits(a, quotient(u[i], xi, i - i0 + 1));
  }
  return warp_argmax(a);
}

// CauchyMax (Cauchylowrank.f90:166-188): max_i |u(i) / (D(i) - f)| over i in [0, len) and its
// 1-based index.
__device__ ArgMax cauchy_max(const double* D, double f, const double* u, int len, SearchSm& sm) {
  return max_quotient(u, [=](int i) { return D[i] - f; }, len, sm);
}

__device__ __forceinline__ void swapd(double* a, int i, int j) {
  const double t = a[i];
  a[i] = a[j];
  a[j] = t;
}
__device__ __forceinline__ void swapi(int* a, int i, int j) {
  const int t = a[i];
  a[i] = a[j];
  a[j] = t;
}

// CauchyPivtG (:191-243), 0-based k0 = k - 1.
__device__ void pivt_g(RrluBlock& b, int k0, SearchSm& sm) {
  const int M = b.M, N = b.N;
  ArgMax L = cauchy_max(b.D + k0, b.F[k0], b.U + k0, M - k0, sm);
  ArgMax R = cauchy_max(b.F + k0, b.D[k0], b.V + k0, N - k0, sm);
  double junkL = L.v * fabs(b.V[k0]);
  double junkU = R.v * fabs(b.U[k0]);
  const double piv = fabs(b.U[k0] * b.V[k0] / (b.D[k0] - b.F[k0]));
  if (junkL <= piv && junkU <= piv) return;
  __syncthreads();  // every thread has read the pivot before thread 0 swaps it away
  int flg = junkL > junkU ? 1 : 0;
  int jjL = L.i, jjU = R.i;
  for (int guard = 0; guard < 4 * (M + N); ++guard) {
    if (flg == 1) {
      const int jj = jjL;
      if (threadIdx.x == 0) {
        swapd(b.D, k0, jj + k0 - 1);
        swapd(b.U, k0, jj + k0 - 1);
        swapd(b.A, k0, jj + k0 - 1);
        swapi(b.PL, k0, jj + k0 - 1);
      }
      __syncthreads();
      R = cauchy_max(b.F + k0, b.D[k0], b.V + k0, N - k0, sm);
      jjU = R.i;
      if (jjU == 1) return;
      flg = 0;
    }
    const int jj = jjU;
    if (threadIdx.x == 0) {
      swapd(b.F, k0, jj + k0 - 1);
      swapd(b.V, k0, jj + k0 - 1);
      swapi(b.PU, k0, jj + k0 - 1);
    }
    __syncthreads();
    L = cauchy_max(b.D + k0, b.F[k0], b.U + k0, M - k0, sm);
    jjL = L.i;
    if (jjL == 1) return;
    flg = 1;
  }
}

// Candidate of a multi-column search: value, 1-based column, 1-based row of that column's max.
struct Cand {
  double v;
  int j, i;
};

__device__ __forceinline__ Cand better_c(Cand a, Cand b) {
  if (b.v > a.v || (b.v == a.v && b.j < a.j)) return b;  // earlier column wins ties
  return a;
}

// max over columns j in [0, nc) of |Wt[j]| * max_i |u[i] / (D[i] - P[j])|, i in [0, len);
// one warp per column, then one block reduction.  Ties: earlier column, earlier row
// (the order of the reference's loops with strict '>' and MAXLOC).
__device__ Cand multi_cauchy_max(const double* D, const double* u, int len, const double* P, const double* Wt,
                                 int nc, Cand* smc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cand wb{-1.0, 0x7fffffff, 0};
  int floor_key = QK_EXACT;  // below it a column cannot beat one this warp has seen
  for (int j = warp; j < nc; j += nw) {
    const double pj = P[j];
    int key;
    const ArgMax a = warp_max_quotient(u, [=](int i) { return D[i] - pj; }, 0, len, Wt[j], floor_key, &key);
    if (key != QK_EXACT) {
      if (floor_key != QK_EXACT && key < floor_key) continue;
      floor_key = max(floor_key, key - 2 * QK_SLACK);
    }
    wb = better_c(wb, Cand{a.v * fabs(Wt[j]), j + 1, a.i});
  }
  __syncthreads();
  if (lane == 0) smc[warp] = wb;
  __syncthreads();
  if (threadIdx.x == 0) {
    Cand r = smc[0];
    for (int w = 1; w < nw; ++w) r = better_c(r, smc[w]);
    smc[32] = r;
  }
  __syncthreads();
  Cand r = smc[32];
  __syncthreads();
  return r;
}

// Swaps of CauchyPivtG_CP (:246-296) for the search result (ii, jj) at step k0.
__device__ void apply_cp(RrluBlock& b, int k0, int ii, int jj) {
  if (threadIdx.x == 0) {
    swapd(b.D, k0, ii + k0 - 1);
    swapd(b.U, k0, ii + k0 - 1);
    swapd(b.A, k0, ii + k0 - 1);
    swapi(b.PL, k0, ii + k0 - 1);
    swapd(b.F, k0, jj + k0 - 1);
    swapd(b.V, k0, jj + k0 - 1);
    swapi(b.PU, k0, jj + k0 - 1);
  }
  __syncthreads();
}

// rrluCauchy (:7-134), one block per matrix block, resumable around the complete-pivot
// search (CauchyPivtG_CP): a step whose pivot is below tol * amax saves its state, counts
// itself in *pending and returns; the search runs grid-wide and the next launch resumes.
__global__ void __launch_bounds__(RRLU_THREADS) k_rrlu_cauchy(RrluBlock* blocks, double tol, int* pending) {
  __shared__ SearchSm sm;
  __shared__ Cand smc[33];
  RrluBlock& gb = blocks[blockIdx.x];
  RrluBlock b = gb;
  if (b.phase == 2) return;
  const int M = b.M, N = b.N, mn = min(M, N);
  const double rho = 1.12;
  const int prd = 10;
  bool resume_cp = b.phase == 1;
  if (b.phase == 0 && b.k_next == 1) {
    // D, A from the row generators, F, V from the column generators; U = A, PL = 1..M,
    // PU = 1..N, W = 0 (rrluCauchy :64-71; compress_cauchy zeroes W)
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      b.D[i] = b.gD[i];
      b.A[i] = b.gU[i];
      b.U[i] = b.gU[i];
      b.PL[i] = i + 1;
    }
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      b.F[j] = b.gF[j];
      b.V[j] = b.gV[j];
      b.PU[j] = j + 1;
    }
    for (int j = threadIdx.x; j < mn; j += blockDim.x) b.W[j] = 0.0;
    __syncthreads();
  }
  int Rk = mn;
  double amax = b.amax;
  for (int k = b.k_next; k <= mn; ++k) {
    const int k0 = k - 1;
    double ukk;
    if (resume_cp) {
      resume_cp = false;
      apply_cp(b, k0, b.cp_i, b.cp_j);
      ukk = b.U[k0] * b.V[k0] / (b.D[k0] - b.F[k0]);
      amax = fmax(amax, fabs(ukk));
      if (fabs(ukk) < tol * amax) {
        Rk = k - 1;
        break;
      }
    } else {
      pivt_g(b, k0, sm);
      ukk = b.U[k0] * b.V[k0] / (b.D[k0] - b.F[k0]);
      amax = fmax(amax, fabs(ukk));
      if (fabs(ukk) < tol * amax) {
        if (threadIdx.x == 0) {
          gb.phase = 1;
          gb.k_next = k;
          gb.amax = amax;
          atomicAdd(pending, 1);
        }
        return;
      }
    }
    const double dk = b.D[k0], fk = b.F[k0];
    for (int i = k + threadIdx.x; i < M; i += blockDim.x) b.U[i] = b.U[i] * (b.D[i] - dk) / (b.D[i] - fk);
    for (int j = k + threadIdx.x; j < N; j += blockDim.x) b.V[j] = b.V[j] * (b.F[j] - fk) / (b.F[j] - dk);
    for (int j = threadIdx.x; j < k - 1; j += blockDim.x) b.W[j] = b.W[j] * ((fk - b.D[j]) / (dk - b.D[j]));
    __syncthreads();
    if (threadIdx.x == 0) {
      double wk = (dk - fk) / b.A[k0];
      for (int j = 0; j < k - 1; ++j) wk = wk * (b.F[j] - dk) / (b.D[j] - dk);
      b.W[k0] = wk;
    }
    __syncthreads();
    // swap check every prd steps (searchMax2, :137-163, and the update of :103-129); each
    // swap raises |det| of the leading block by more than rho, so the loop ends -- the guard
    // only bounds it against rounding
    int flgl = k % prd;
    for (int guard = 0; flgl < 1 && guard < 4 * k + 64; ++guard) {
      flgl = 1;
      // max over j < k of |W(j)| * max_i |U(i)/(D(i)-D(j))|, i in [k, M)
      const Cand best = multi_cauchy_max(b.D + k, b.U + k, M - k, b.D, b.W, k, smc);
      if (M - k > 0 && best.v > rho) {
        flgl = 0;
        const int ii = best.j;        // 1-based position among the first k
        const int jj = best.i + k;    // 1-based row beyond k
        const int i0 = ii - 1, j0 = jj - 1;
        const double dii = b.D[i0], djj = b.D[j0];
        for (int j = k + threadIdx.x; j < N; j += blockDim.x) b.V[j] = b.V[j] * ((b.F[j] - dii) / (b.F[j] - djj));
        for (int i = k + threadIdx.x; i < M; i += blockDim.x)
          if (i != j0) b.U[i] = b.U[i] * ((b.D[i] - djj) / (b.D[i] - dii));
        for (int j = threadIdx.x; j < k; j += blockDim.x)
          if (j != i0) b.W[j] = b.W[j] * ((b.D[j] - dii) / (b.D[j] - djj));
        __syncthreads();
        if (threadIdx.x == 0) {
          double ujj = b.A[i0] * ((dii - djj) / (dii - b.F[i0]));
          double wii = (djj - b.F[i0]) / b.A[j0];
          for (int j = 0; j < k; ++j) {
            if (j == i0) continue;
            ujj = ujj * ((dii - b.D[j]) / (dii - b.F[j]));
            wii = wii * ((b.F[j] - djj) / (b.D[j] - djj));
          }
          b.U[j0] = ujj;
          b.W[i0] = wii;
          swapi(b.PL, i0, j0);
          swapd(b.D, i0, j0);
          swapd(b.A, i0, j0);
        }
        __syncthreads();
      }
    }
  }
  if (threadIdx.x == 0) {
    *b.rank = Rk;
    gb.phase = 2;
  }
}

// Complete-pivot search (CauchyPivtG_CP's max over the Schur complement) for the blocks
// waiting in the resumable RRLU: each CTA takes a chunk of columns of one block, one warp
// per column, and leaves its best candidate in cand[blockIdx.x]; the maximum over the
// chunks of a block (ties: earlier column, then earlier row) goes to cp_i, cp_j.
struct CpChunk {
  int blk, c0, c1;  // columns [c0, c1) (absolute) of block blk
};

__global__ void __launch_bounds__(RRLU_THREADS) k_cp_search(const RrluBlock* blocks, const CpChunk* chunks,
                                                             Cand* cand) {
  __shared__ Cand smc[33];
  const CpChunk ch = chunks[blockIdx.x];
  const RrluBlock& b = blocks[ch.blk];
  const int k0 = b.k_next - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cand wb{-1.0, 0x7fffffff, 0};
  int floor_key = QK_EXACT;
  for (int j = ch.c0 + warp; j < ch.c1; j += nw) {
    const double pj = b.F[j];
    int key;
    const ArgMax a = warp_max_quotient(b.U, [&](int i) { return b.D[i] - pj; }, k0, b.M, b.V[j], floor_key, &key);
    if (key != QK_EXACT) {
      if (floor_key != QK_EXACT && key < floor_key) continue;
      floor_key = max(floor_key, key - 2 * QK_SLACK);
    }
    wb = better_c(wb, Cand{a.v * fabs(b.V[j]), j - k0 + 1, a.i});
  }
  if (lane == 0) smc[warp] = wb;
  __syncthreads();
  if (threadIdx.x == 0) {
    Cand r = smc[0];
    for (int w = 1; w < nw; ++w) r = better_c(r, smc[w]);
    cand[blockIdx.x] = r;
  }
}

template <class Block>
__global__ void k_cp_reduce(Block* blocks, const int* __restrict__ blk, const int* __restrict__ first,
                            int count, int total, const Cand* __restrict__ cand) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int e = (t + 1 < count) ? first[t + 1] : total;
  Cand r = cand[first[t]];
  for (int c = first[t] + 1; c < e; ++c) r = better_c(r, cand[c]);
  blocks[blk[t]].cp_i = r.i;
  blocks[blk[t]].cp_j = r.j;
}


// ------------------------------------------------------------------------------------------
// RRLU of accurate-denominator blocks (rrluCauchyEigrow, CauchyHssEig.f90:7-212)
// ------------------------------------------------------------------------------------------
// Rows carry old eigenvalues F = FF(PL) and weights; columns the new eigenvalues D(PU), seen
// only through DIFL/DIFR: every F(i) - D(j) and D(j) - D(k) is formed by computfd / computdd
// (:470-568) from the global arrays with 1-based global indices PL, PU.
struct RrluEigBlock {
  int M, N;
  const double *FF, *DL, *DR;  // global old eigenvalues and distances (n entries)
  int nglob;
  const double *gU, *gV;       // row weights U(r0 + i), column weights V(c0 + j)
  int r0, c0;                  // global 0-based offsets of the block
  double *F, *A, *U, *V, *W;   // row poles (permuted), row weights (becomes LU), Schur weights (Z),
                               // column weights, interpolation weights (min(M, N))
  int *PL, *PU, *PQ;           // global 1-based row / column indices (permuted), local row permutation
  int* rank;
  int k_next, phase, cp_i, cp_j;  // resumable state, as RrluBlock
  double amax;
};

// computfd: F(pl) - D(pu) (CauchyHssEig.f90:519-568)
__device__ __forceinline__ double eig_fd(const RrluEigBlock& b, int pl, int pu) {
  return pl <= pu ? (b.FF[pl - 1] - b.FF[pu - 1]) - b.DL[pu - 1] : (b.FF[pl - 1] - b.FF[pu]) - b.DR[pu - 1];
}
// computdd: D(pj) - D(pk) (CauchyHssEig.f90:470-516), pj != pk
__device__ __forceinline__ double eig_dd(const RrluEigBlock& b, int pj, int pk) {
  return pj < pk ? (b.FF[pj] - b.FF[pk - 1]) + b.DR[pj - 1] - b.DL[pk - 1]
                 : (b.FF[pj - 1] - b.FF[min(pk, b.nglob - 1)]) + b.DL[pj - 1] - b.DR[pk - 1];
}

// CauchyMaxEigmc (:1506-1589): max_i |U(i) / (F(PL(i)) - D(PU(k0)))|, i in [k0, M), 1-based offset
__device__ ArgMax eig_col_max(const RrluEigBlock& b, int k0, SearchSm& sm) {
  const int pu = b.PU[k0];
  return max_quotient(b.U + k0, [&](int i) { return eig_fd(b, b.PL[k0 + i], pu); }, b.M - k0, sm);
}
// CauchyMaxEigm (:1418-1503): max_j |V(j) / (F(PL(k0)) - D(PU(j)))|, j in [k0, N)
__device__ ArgMax eig_row_max(const RrluEigBlock& b, int k0, SearchSm& sm) {
  const int pl = b.PL[k0];
  return max_quotient(b.V + k0, [&](int j) { return eig_fd(b, pl, b.PU[k0 + j]); }, b.N - k0, sm);
}

__device__ __forceinline__ void eig_swap_rows(RrluEigBlock& b, int a, int c) {
  swapd(b.F, a, c);
  swapd(b.U, a, c);
  swapd(b.A, a, c);
  swapi(b.PL, a, c);
  swapi(b.PQ, a, c);
}
__device__ __forceinline__ void eig_swap_cols(RrluEigBlock& b, int a, int c) {
  swapd(b.V, a, c);
  swapi(b.PU, a, c);
}

// CauchyPivtEig (:571-717); the pivot magnitude is |U(k)V(k) / computfd(k, k)|.
__device__ void pivt_eig(RrluEigBlock& b, int k0, SearchSm& sm) {
  ArgMax L = eig_col_max(b, k0, sm);
  ArgMax R = eig_row_max(b, k0, sm);
  const double junkL = L.v * fabs(b.V[k0]);
  const double junkU = R.v * fabs(b.U[k0]);
  const double piv = fabs(b.U[k0] * b.V[k0] / eig_fd(b, b.PL[k0], b.PU[k0]));
  if (junkL <= piv && junkU <= piv) return;
  __syncthreads();  // every thread has read the pivot before thread 0 swaps it away
  int flg = junkL > junkU ? 1 : 0;
  int jjL = L.i, jjU = R.i;
  for (int guard = 0; guard < 4 * (b.M + b.N); ++guard) {
    if (flg == 1) {
      if (threadIdx.x == 0) eig_swap_rows(b, k0, jjL + k0 - 1);
      __syncthreads();
      R = eig_row_max(b, k0, sm);
      jjU = R.i;
      if (jjU == 1) return;
      flg = 0;
    }
    if (threadIdx.x == 0) eig_swap_cols(b, k0, jjU + k0 - 1);
    __syncthreads();
    L = eig_col_max(b, k0, sm);
    jjL = L.i;
    if (jjL == 1) return;
    flg = 1;
  }
}

__global__ void __launch_bounds__(RRLU_THREADS) k_rrlu_eig(RrluEigBlock* blocks, double tol, int* pending) {
  __shared__ SearchSm sm;
  __shared__ Cand smc[33];
  RrluEigBlock& gb = blocks[blockIdx.x];
  RrluEigBlock b = gb;
  if (b.phase == 2) return;
  const int M = b.M, N = b.N, mn = min(M, N);
  const double rho = 1.2;  // rrluCauchyEigrow :49-50
  const int prd = 5;
  bool resume_cp = b.phase == 1;
  if (b.phase == 0 && b.k_next == 1) {
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      b.F[i] = b.FF[b.r0 + i];
      b.A[i] = b.gU[i];
      b.U[i] = b.gU[i];
      b.PL[i] = b.r0 + i + 1;
      b.PQ[i] = i + 1;
    }
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      b.V[j] = b.gV[j];
      b.PU[j] = b.c0 + j + 1;
    }
    for (int j = threadIdx.x; j < mn; j += blockDim.x) b.W[j] = 0.0;
    __syncthreads();
  }
  int Rk = mn;
  double amax = b.amax;
  for (int k = b.k_next; k <= mn; ++k) {
    const int k0 = k - 1;
    double ukk;
    if (resume_cp) {
      resume_cp = false;
      if (threadIdx.x == 0) {  // CauchyPivtEig_CP's swaps (:1004-1134)
        eig_swap_rows(b, k0, b.cp_i + k0 - 1);
        eig_swap_cols(b, k0, b.cp_j + k0 - 1);
      }
      __syncthreads();
      ukk = b.U[k0] * b.V[k0] / eig_fd(b, b.PL[k0], b.PU[k0]);
      amax = fmax(amax, fabs(ukk));
      if (fabs(ukk) < tol * amax) {
        Rk = k - 1;
        break;
      }
    } else {
      pivt_eig(b, k0, sm);
      ukk = b.U[k0] * b.V[k0] / eig_fd(b, b.PL[k0], b.PU[k0]);
      amax = fmax(amax, fabs(ukk));
      if (fabs(ukk) < tol * amax) {
        if (threadIdx.x == 0) {
          gb.phase = 1;
          gb.k_next = k;
          gb.amax = amax;
          atomicAdd(pending, 1);
        }
        return;
      }
    }
    const double fk = b.F[k0];
    const int plk = b.PL[k0], puk = b.PU[k0];
    for (int i = k + threadIdx.x; i < M; i += blockDim.x) b.U[i] = b.U[i] * ((b.F[i] - fk) / eig_fd(b, b.PL[i], puk));
    for (int j = k + threadIdx.x; j < N; j += blockDim.x)
      b.V[j] = b.V[j] * (eig_dd(b, b.PU[j], puk) / (-eig_fd(b, plk, b.PU[j])));
    for (int j = threadIdx.x; j < k - 1; j += blockDim.x)
      b.W[j] = b.W[j] * ((-eig_fd(b, b.PL[j], puk)) / (fk - b.F[j]));
    __syncthreads();
    if (threadIdx.x == 0) {
      double wk = eig_fd(b, plk, puk) / b.A[k0];
      for (int j = 0; j < k - 1; ++j) wk = wk * ((-eig_fd(b, plk, b.PU[j])) / (b.F[j] - fk));
      b.W[k0] = wk;
    }
    __syncthreads();
    // swap check every prd steps (searchMax2Eig, :1137-1203, and the update of :160-205)
    int flgl = k % prd;
    for (int guard = 0; flgl < 1 && guard < 4 * k + 64; ++guard) {
      flgl = 1;
      const Cand best = multi_cauchy_max(b.F + k, b.U + k, M - k, b.F, b.W, k, smc);
      if (M - k > 0 && best.v > rho) {
        flgl = 0;
        const int i0 = best.j - 1, j0 = best.i + k - 1;
        const double fii = b.F[i0], fjj = b.F[j0];
        const int plii = b.PL[i0], pljj = b.PL[j0];
        for (int j = k + threadIdx.x; j < N; j += blockDim.x)
          b.V[j] = b.V[j] * ((-eig_fd(b, plii, b.PU[j])) / (-eig_fd(b, pljj, b.PU[j])));
        for (int i = k + threadIdx.x; i < M; i += blockDim.x)
          if (i != j0) b.U[i] = b.U[i] * ((b.F[i] - fjj) / (b.F[i] - fii));
        for (int j = threadIdx.x; j < k; j += blockDim.x)
          if (j != i0) b.W[j] = b.W[j] * ((b.F[j] - fii) / (b.F[j] - fjj));
        __syncthreads();
        if (threadIdx.x == 0) {
          double ujj = b.A[i0] * ((fii - fjj) / eig_fd(b, plii, b.PU[i0]));
          double wii = eig_fd(b, pljj, b.PU[i0]) / b.A[j0];
          for (int j = 0; j < k; ++j) {
            if (j == i0) continue;
            ujj = ujj * ((fii - b.F[j]) / eig_fd(b, plii, b.PU[j]));
            wii = wii * ((-eig_fd(b, pljj, b.PU[j])) / (b.F[j] - fjj));
          }
          b.U[j0] = ujj;
          b.W[i0] = wii;
          swapi(b.PL, i0, j0);
          swapi(b.PQ, i0, j0);
          swapd(b.F, i0, j0);
          swapd(b.A, i0, j0);
        }
        __syncthreads();
      }
    }
  }
  if (threadIdx.x == 0) {
    *b.rank = Rk;
    gb.phase = 2;
  }
}

// Complete-pivot search for waiting eig blocks (CauchyPivtEig_CP's maximum), as k_cp_search.
__global__ void __launch_bounds__(RRLU_THREADS) k_cp_search_eig(const RrluEigBlock* blocks, const CpChunk* chunks,
                                                                 Cand* cand) {
  __shared__ Cand smc[33];
  const CpChunk ch = chunks[blockIdx.x];
  const RrluEigBlock& b = blocks[ch.blk];
  const int k0 = b.k_next - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  Cand wb{-1.0, 0x7fffffff, 0};
  int floor_key = QK_EXACT;
  for (int j = ch.c0 + warp; j < ch.c1; j += nw) {
    const int pu = b.PU[j];
    int key;
    const ArgMax a =
        warp_max_quotient(b.U, [&](int i) { return eig_fd(b, b.PL[i], pu); }, k0, b.M, b.V[j], floor_key, &key);
    if (key != QK_EXACT) {
      if (floor_key != QK_EXACT && key < floor_key) continue;
      floor_key = max(floor_key, key - 2 * QK_SLACK);
    }
    wb = better_c(wb, Cand{a.v * fabs(b.V[j]), j - k0 + 1, a.i});
  }
  if (lane == 0) smc[warp] = wb;
  __syncthreads();
  if (threadIdx.x == 0) {
    Cand r = smc[0];
    for (int w = 1; w < nw; ++w) r = better_c(r, smc[w]);
    cand[blockIdx.x] = r;
  }
}

// Columns of A(:, R) (n x M, lda) in RRLU pivot order for every compressed block:
// T0(:, j) = A(:, PL(j)) for j < Rk, and on the FP64 path Ar(:, t) = A(:, PL(Rk + t)) for t < M - Rk (PL 1-based).
// One block per column of the batch (columns numbered from c0 per block).
struct GatherDesc {
  const double* A;
  long lda;
  int n, M, Rk, c0;
  const int* PL;
  double *T0, *Ar;  // leading dimension n
};

__global__ void __launch_bounds__(256) k_gather_group(const GatherDesc* __restrict__ d, int count) {
  const int gc = blockIdx.x;
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (d[mid].c0 <= gc) lo = mid; else hi = mid - 1;
  }
  const GatherDesc& e = d[lo];
  const int c = gc - e.c0;
  const double* src = e.A + (long)(e.PL[c] - 1) * e.lda;
  double* dst = (c < e.Rk) ? e.T0 + (long)c * e.n : e.Ar + (long)(c - e.Rk) * e.n;
  for (int i = threadIdx.x; i < e.n; i += blockDim.x) dst[i] = src[i];
}

// ------------------------------------------------------------------------------------------
// RRQR
// ------------------------------------------------------------------------------------------
constexpr int QR_THREADS = 256;
constexpr int QR_WARPS = QR_THREADS / 32;
constexpr int QR_CAP = 256;  // largest rank a tile is factorised to; beyond it the tile is used as is

struct QrTile {
  int M, N, cap;                    // tile size; steps at most cap (<= min(M, N), <= QR_CAP)
  GenSpec gs;                       // generators of the tile (Cauchy or accurate-denominator Cauchy)
  double* T;     // M x N (ld M), columns pivoted; Q(:, 0:r) on exit
  double* V;     // M x cap (ld M): reflectors, V(k,k) = 1, rows < k unused
  double* F;     // F[c*cap + j]; on exit Y = R(0:r,:) P^T (r x N, ld r)
  double* R;     // R[c*cap + i], i <= c
  double* tau;   // cap + 1 (tau[cap] = |R_11|)
  double* s;     // cap: V(k:,0:k)^T v_k
  double *vn1, *vn2;  // partial column norms
  int* jpvt;     // original column of each pivoted column
  int* rank;     // -1 running, -2 verifying; then r (< min(M,N)) or min(M,N) when not compressed
  int* flag;     // k + 1 when step k flagged a partial norm for recomputation
  unsigned* bar; // group barrier counter
  int cta0, ncta;
  long col0;     // first column of this tile in the batch's column numbering
};

// Explicit tiles T(i,c) = U(i)V(c)/(D(i)-F(c)) (ConstCauchy, Auxil_2p5D.f90:138-144), with the
// accurate denominators of CauchylikeEig (ConstCauchyEig, Auxil_2p5D.f90:532-637), or Toeplitz /
// Hankel entries (ConstToeplitzlowrank's tile, Auxil_2p5D.f90:968-1060), their column norms and
// the identity pivot; one block per column of the batch.
__global__ void __launch_bounds__(QR_THREADS) k_qr_tiles(QrTile* tiles, int ntiles) {
  __shared__ double sm[33];
  const long gc = blockIdx.x;
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {  // last tile with col0 <= gc
    const int mid = (lo + hi + 1) >> 1;
    if (tiles[mid].col0 <= gc) lo = mid; else hi = mid - 1;
  }
  const QrTile& t = tiles[lo];
  const int c = (int)(gc - t.col0);
  if (c >= t.N) return;
  const GenSpec& g = t.gs;
  double ss = 0.0;
  if (g.kind == KIND_TOEPLITZ || g.kind == KIND_HANKEL) {
    // ConstToeplitz / ConstHankel (Auxil_2p5D.f90:224-231, 309-316) on the shifted generator
    const bool toep = g.kind == KIND_TOEPLITZ;
    for (int i = threadIdx.x; i < t.M; i += blockDim.x) {
      const double h = toep ? g.g[(g.order - 1) + c - i] : g.g[i + c];
      t.T[i + (long)c * t.M] = h;
      ss = fma(h, h, ss);
    }
  } else {
    // the entries in the double-float form of the split path's H (cauchy_entry: the FP64 pole
    // difference, then u v / x on the FP32 pipe, about 2^-49 relative): the IEEE division
    // would be a dozen instructions on GB300's narrow FP64 pipe, which the QR itself needs
    const bool eig = g.kind == KIND_CAUCHY_EIG;
    const double f = g.Fc[c], v = g.Vc[c];
    const VSplit vs = v_split(v);
    const double f1 = (eig && c < g.fc1_len) ? g.Fc1[c] : 0.0;
    const double dl = eig ? g.dl[c] : 0.0, dr = (eig && c < g.fc1_len) ? g.dr[c] : 0.0;
    for (int i = threadIdx.x; i < t.M; i += blockDim.x) {
      const double h = eig ? cauchy_entry(g.Ur[i], v, vs, eig_den(g.Dr[i], f, f1, dl, dr, i - c <= g.diag_off))
                           : cauchy_entry(g.Ur[i], v, vs, g.Dr[i] - f);
      t.T[i + (long)c * t.M] = h;
      ss = fma(h, h, ss);
    }
  }
  ss = block_sum(ss, sm);
  if (threadIdx.x == 0) {
    const double nrm = sqrt(ss);
    t.vn1[c] = nrm;
    t.vn2[c] = nrm;
    t.jpvt[c] = c;
    if (c == 0) {
      *t.rank = -1;
      *t.flag = 0;
      *t.bar = 0u;
    }
  }
}

// Barrier of the ncta CTAs of one tile (all co-resident: cooperative launch).  The counter
// only grows; the e-th barrier waits for e * ncta arrivals.  Bounded: after WAIT_NS the
// status word gets DEV_ERR_TIMEOUT and every waiter of the launch returns false.
__device__ bool group_sync(unsigned* bar, unsigned target, unsigned* status) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const unsigned long long t0 = globaltimer_ns();
    int good = 1;
    while (true) {
      const unsigned v = *(volatile unsigned*)bar;
      if (v >= target) break;
      if (*(volatile unsigned*)status != 0u) { good = 0; break; }
      if (globaltimer_ns() - t0 > WAIT_NS) {
        atomicOr(status, DEV_ERR_TIMEOUT);
        good = 0;
        break;
      }
      __nanosleep(100);
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Lane part of a warp dot product sum x[i] y[i], i = i0 (mod 32) in [i0, M): four independent
// accumulators keep eight loads in flight.
__device__ __forceinline__ double lane_dot(const double* x, const double* y, int i0, int M) {
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  int i = i0;
  for (; i + 96 < M; i += 128) {
    a0 = fma(__ldcg(x + i), __ldcg(y + i), a0);
    a1 = fma(__ldcg(x + i + 32), __ldcg(y + i + 32), a1);
    a2 = fma(__ldcg(x + i + 64), __ldcg(y + i + 64), a2);
    a3 = fma(__ldcg(x + i + 96), __ldcg(y + i + 96), a3);
  }
  for (; i < M; i += 32) a0 = fma(__ldcg(x + i), __ldcg(y + i), a0);
  return (a0 + a1) + (a2 + a3);
}

// lane_dot for four columns x[0..3] against one y, each column's sum in lane_dot's order; the y
// loads are shared.
__device__ __forceinline__ void lane_dot4(const double* const (&x)[4], const double* y, int i0, int M,
                                          double (&out)[4]) {
  double a[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) a[u][q] = 0.0;
  int i = i0;
  for (; i + 96 < M; i += 128) {
    const double y0 = __ldcg(y + i), y1 = __ldcg(y + i + 32), y2 = __ldcg(y + i + 64), y3 = __ldcg(y + i + 96);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      a[u][0] = fma(__ldcg(x[u] + i), y0, a[u][0]);
      a[u][1] = fma(__ldcg(x[u] + i + 32), y1, a[u][1]);
      a[u][2] = fma(__ldcg(x[u] + i + 64), y2, a[u][2]);
      a[u][3] = fma(__ldcg(x[u] + i + 96), y3, a[u][3]);
    }
  }
  for (; i < M; i += 32) {
    const double y0 = __ldcg(y + i);
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u][0] = fma(__ldcg(x[u] + i), y0, a[u][0]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) out[u] = (a[u][0] + a[u][1]) + (a[u][2] + a[u][3]);
}

// The warp sums of four per-lane values v[0..3], reduced and scattered: lane l ends with the
// total of v[l >> 3].  Every partial sum is one the xor butterfly forms (in commuted order),
// so each total equals the butterfly's.
__device__ __forceinline__ double quad_reduce(const double (&v)[4], int lane) {
  const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0;
  double k0 = b4 ? v[2] : v[0], k1 = b4 ? v[3] : v[1];
  const double s0 = b4 ? v[0] : v[2], s1 = b4 ? v[1] : v[3];
  k0 += __shfl_xor_sync(0xffffffffu, s0, 16);
  k1 += __shfl_xor_sync(0xffffffffu, s1, 16);
  double kk = b3 ? k1 : k0;
  const double ss = b3 ? k0 : k1;
  kk += __shfl_xor_sync(0xffffffffu, ss, 8);
  for (int o = 4; o > 0; o >>= 1) kk += __shfl_xor_sync(0xffffffffu, kk, o);
  return kk;
}

// Step k of the leader CTA: pivot, swap, the current column a = T(k:,k) - V F(k,:)^T over the
// reflectors p0..k-1 of the current panel (earlier ones are applied to T), its Householder
// reflector (beta = -sign(alpha) ||a||, tau = (beta - alpha)/beta, v = a(k+1:)/(alpha - beta)),
// the truncation test and s = V(k:,p0:k)^T v.
__device__ void qr_leader_step(const QrTile& t, int k, int p0, double tol, bool verified, ArgMax* am, double* red,
                               double* fk) {
  const int M = t.M, N = t.N, cap = t.cap;
  ArgMax best{-1.0, 0x7fffffff};
  for (int c = k + threadIdx.x; c < N; c += blockDim.x) best = better(best, ArgMax{__ldcg(t.vn1 + c), c});
  best = block_argmax(best, am);
  const int p = best.i;
  if (p != k) {
    for (int i = k + threadIdx.x; i < M; i += blockDim.x) {
      double* a = t.T + i + (long)k * M;
      double* b = t.T + i + (long)p * M;
      const double x = __ldcg(a), y = __ldcg(b);
      *a = y;
      *b = x;
    }
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
      double x, y;
      if (j >= p0) {
        x = __ldcg(t.F + (long)k * cap + j);
        y = __ldcg(t.F + (long)p * cap + j);
        t.F[(long)k * cap + j] = y;
        t.F[(long)p * cap + j] = x;
      }
      x = __ldcg(t.R + (long)k * cap + j);
      y = __ldcg(t.R + (long)p * cap + j);
      t.R[(long)k * cap + j] = y;
      t.R[(long)p * cap + j] = x;
    }
    if (threadIdx.x == 0) {
      double x = __ldcg(t.vn1 + k);
      t.vn1[k] = __ldcg(t.vn1 + p);
      t.vn1[p] = x;
      x = __ldcg(t.vn2 + k);
      t.vn2[k] = __ldcg(t.vn2 + p);
      t.vn2[p] = x;
      const int q = __ldcg(t.jpvt + k);
      t.jpvt[k] = __ldcg(t.jpvt + p);
      t.jpvt[p] = q;
    }
    __syncthreads();
  }
  for (int j = p0 + threadIdx.x; j < k; j += blockDim.x) fk[j - p0] = __ldcg(t.F + (long)k * cap + j);
  __syncthreads();
  double* vk = t.V + (long)k * M;
  double xsq = 0.0;
  for (int i = k + threadIdx.x; i < M; i += blockDim.x) {
    double a = __ldcg(t.T + i + (long)k * M);
    int j = p0;
    for (; j + 4 <= k; j += 4) {  // four loads in flight, the same FMA order
      double vv[4];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) vv[jj] = __ldcg(t.V + i + (long)(j + jj) * M);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) a = fma(-vv[jj], fk[j + jj - p0], a);
    }
    for (; j < k; ++j) a = fma(-__ldcg(t.V + i + (long)j * M), fk[j - p0], a);
    vk[i] = a;
    if (i > k) xsq = fma(a, a, xsq);
  }
  xsq = block_sum(xsq, red);  // contains the barrier that publishes vk within the CTA
  const double alpha = __ldcg(vk + k);
  const double xnorm = sqrt(xsq);
  double beta = alpha, tau = 0.0;
  if (xnorm != 0.0) {
    beta = -copysign(hypot(alpha, xnorm), alpha);
    tau = (beta - alpha) / beta;
    const double scal = 1.0 / (alpha - beta);
    for (int i = k + 1 + threadIdx.x; i < M; i += blockDim.x) vk[i] = __ldcg(vk + i) * scal;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    vk[k] = 1.0;
    t.R[(long)k * cap + k] = beta;
    t.tau[k] = tau;
    const double r11 = (k == 0) ? fabs(beta) : __ldcg(t.tau + cap);
    if (k == 0) t.tau[cap] = r11;
    // Compress_RRQR's scan (:1150-1156).  The pivot came from downdated norms, which drift
    // at this level; the first time the test passes, the group recomputes every partial
    // norm exactly (rank = -2) and the step is redone, so truncation means that no column
    // of the reduced tile is larger than tol |R_11|.
    if (fabs(beta) <= tol * r11) *t.rank = verified ? k : -2;
  }
  __syncthreads();
  // s(j) = sum_{i >= k} V(i,j) v(i), p0 <= j < k: one warp per j
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j = p0 + warp; j < k; j += QR_WARPS) {
    double a = lane_dot(t.V + (long)j * M, vk, k + lane, M);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) t.s[j] = a;
  }
}

// Panel restart (the trailing update of DLAQPS): T(r0:, c) -= V(r0:, p0:k1) F(c, p0:k1)^T for
// every column c >= c0, written back, and the exact partial norms ||T(r0:, c)||.  One warp
// per column, the columns shared by the CTAs of the group.
__device__ void qr_restart(const QrTile& t, int p0, int k1, int r0, int c0, int local, double (*fw)[QR_CAP]) {
  const int M = t.M, N = t.N, cap = t.cap;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nj = k1 - p0;
  for (int c = c0 + local * QR_WARPS + warp; c < N; c += t.ncta * QR_WARPS) {
    double* tc = t.T + (long)c * M;
    for (int j = lane; j < nj; j += 32) fw[warp][j] = __ldcg(t.F + (long)c * cap + p0 + j);
    __syncwarp();
    double ss = 0.0;
    for (int i = r0 + lane; i < M; i += 128) {  // four rows per lane in flight
      double a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = (i + 32 * u < M) ? __ldcg(tc + i + 32 * u) : 0.0;
      // four reflectors per pass with their 16 loads issued first (the loads of one
      // reflector alone leave the lane waiting on L2 between FMAs); same FMA order
      int j = 0;
      for (; j + 4 <= nj; j += 4) {
        double vv[4][4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const double* vj = t.V + (long)(p0 + j + jj) * M;
#pragma unroll
          for (int u = 0; u < 4; ++u) vv[jj][u] = (i + 32 * u < M) ? __ldcg(vj + i + 32 * u) : 0.0;
        }
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const double w = fw[warp][j + jj];
#pragma unroll
          for (int u = 0; u < 4; ++u) a[u] = fma(-vv[jj][u], w, a[u]);
        }
      }
      for (; j < nj; ++j) {
        const double* vj = t.V + (long)(p0 + j) * M;
        const double w = fw[warp][j];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + 32 * u < M) a[u] = fma(-__ldcg(vj + i + 32 * u), w, a[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + 32 * u < M) {
          if (nj > 0) tc[i + 32 * u] = a[u];
          ss = fma(a[u], a[u], ss);
        }
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) {
      t.vn1[c] = sqrt(ss);
      t.vn2[c] = sqrt(ss);
    }
    __syncwarp();
  }
}

struct QrSmem {
  ArgMax am[33];
  double red[33];
  double fk[QR_CAP + 1];
  double sv[QR_CAP + 1];
  double vrow[QR_CAP + 1];
  double fw[QR_WARPS][QR_CAP];
};

// The factorisation of one tile by CTA `local` of its group; false when a barrier gave up.
__device__ bool qr_tile(const QrTile& t, int local, double tol, unsigned* status, QrSmem& sm) {
  ArgMax* am = sm.am;
  double* red = sm.red;
  double* fk = sm.fk;
  double* sv = sm.sv;
  double* vrow = sm.vrow;
  double(*fw)[QR_CAP] = sm.fw;
  const int M = t.M, N = t.N, cap = t.cap;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double tol3z = 1.0536712127723509e-08;  // sqrt(2^-53), LAPACK dgeqp3's recompute threshold
  unsigned epoch = 0;
  bool truncated = false;
  int p0 = 0;  // first reflector not yet applied to T (the current panel)
  for (int k = 0; k < cap; ++k) {
    if (local == 0) qr_leader_step(t, k, p0, tol, false, am, red, fk);
    if (!group_sync(t.bar, (++epoch) * t.ncta, status)) return false;
    int state = __ldcg(t.rank);
    if (state == -2) {
      // apply the panel to the trailing tile (rows and columns >= k), exact norms, redo step k
      qr_restart(t, p0, k, k, k, local, fw);
      p0 = k;
      if (!group_sync(t.bar, (++epoch) * t.ncta, status)) return false;
      if (local == 0) {
        if (threadIdx.x == 0) *t.rank = -1;
        __syncthreads();
        qr_leader_step(t, k, p0, tol, true, am, red, fk);
      }
      if (!group_sync(t.bar, (++epoch) * t.ncta, status)) return false;
      state = __ldcg(t.rank);
    }
    if (state >= 0) {
      truncated = true;
      break;
    }
    // every other column c > k: F(c,k), R(k,c) and the norm downdate (dgeqp3/dlaqps); a
    // column whose norm needs recomputing flags a panel restart after this step (DLAQPS
    // ends its panel there: the pending reflectors are applied to T, norms recomputed)
    const double tk = __ldcg(t.tau + k);
    for (int j = p0 + threadIdx.x; j < k; j += blockDim.x) {
      sv[j - p0] = __ldcg(t.s + j);
      vrow[j - p0] = __ldcg(t.V + k + (long)j * M);
    }
    __syncthreads();
    const double* vk = t.V + (long)k * M;
    bool flagged = false;
    // The warp's columns in turn: the dot products over the rows (lanes split the rows), then
    // the scalar tail -- F(c,k), R(k,c) and the norm downdate, some 36 FP64 instructions with
    // two divisions and a square root -- once per 32 columns, lane j taking the warp's j-th
    // column: GB300's FP64 pipe costs a warp instruction whatever the lanes, so a tail run by
    // the whole warp for each column cost a third of the step at M = 2048.
    int slot = 0, sc = -1;
    double sd = 0.0, sf = 0.0, sr = 0.0;
    auto tail = [&]() {
      if (sc >= 0) {
        const double f = tk * (sd - sf);
        const double rkc = __ldcg(t.T + (long)sc * M + k) - sr - f;  // V(k,k) = 1
        const double v1 = __ldcg(t.vn1 + sc), v2 = __ldcg(t.vn2 + sc);
        double nv1 = v1;
        if (v1 != 0.0) {
          double temp = fabs(rkc) / v1;
          temp = fmax(0.0, 1.0 - temp * temp);
          const double q = v1 / v2;
          const double temp2 = temp * q * q;
          if (temp2 <= tol3z) flagged = true;
          else nv1 = v1 * sqrt(temp);
        }
        t.F[(long)sc * cap + k] = f;
        t.R[(long)sc * cap + k] = rkc;
        t.vn1[sc] = nv1;
      }
      sc = -1;
      slot = 0;
    };
    // Four columns at a time: one pass over v_k for their dot products (each column's sum in
    // lane_dot's order), then a reduce-scatter of the three sums of the four columns (levels
    // 16 and 8 split the lanes between the columns, 4, 2, 1 finish each column in its eight
    // lanes): 18 FP64 adds for four columns where a butterfly per column takes 60, with the
    // same partial sums (FP64 addition commutes), so the totals are the butterfly's.
    const int stride = t.ncta * QR_WARPS;
    const int u_me = lane >> 3;  // the column of the quad whose totals this lane ends with
    for (int c = k + 1 + local * QR_WARPS + warp; c < N; c += 4 * stride) {
      double dot[4], fs[4], rs[4];
      const double* tc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) tc[u] = t.T + (long)min(c + u * stride, N - 1) * M;
      lane_dot4(tc, vk, k + lane, M, dot);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double* fc = t.F + (long)min(c + u * stride, N - 1) * cap;
        fs[u] = 0.0;
        rs[u] = 0.0;
        for (int j = p0 + lane; j < k; j += 32) {
          const double fj = __ldcg(fc + j);
          fs[u] = fma(fj, sv[j - p0], fs[u]);
          rs[u] = fma(vrow[j - p0], fj, rs[u]);
        }
      }
      const double td = quad_reduce(dot, lane), tf = quad_reduce(fs, lane), tr = quad_reduce(rs, lane);
      // lane 8 u + slot holds column u's totals: stash them for the tail
      const int cu = c + u_me * stride;
      if ((lane & 7) == slot && cu < N) {
        sd = td;
        sf = tf;
        sr = tr;
        sc = cu;
      }
      if (++slot == 8) tail();
    }
    if (slot > 0) tail();
    flagged = __any_sync(0xffffffffu, flagged);
    if (flagged && lane == 0) atomicMax(t.flag, k + 1);
    if (!group_sync(t.bar, (++epoch) * t.ncta, status)) return false;
    if (__ldcg(t.flag) == k + 1 && k + 1 < cap) {
      // panel restart: apply reflectors p0..k to rows and columns > k, exact norms
      qr_restart(t, p0, k + 1, k + 1, k + 1, local, fw);
      p0 = k + 1;
      if (!group_sync(t.bar, (++epoch) * t.ncta, status)) return false;
    }
  }
  if (!truncated) {
    // not truncated within cap steps: the tile is used as is
    if (local == 0 && threadIdx.x == 0) *t.rank = min(M, N);
    return true;
  }
  const int r = __ldcg(t.rank);
  if (r == 0) return true;
  // Q(:, j) = H_0 ... H_j e_j for j < r (warp per column, in place in T), and
  // Y(i, jpvt(c)) = R(i, c) for c >= i (R P^T, DLAPMT) into F's storage
  for (int j = local * QR_WARPS + warp; j < r; j += t.ncta * QR_WARPS) {
    double* x = t.T + (long)j * M;
    const double tj = __ldcg(t.tau + j);
    const double* vj = t.V + (long)j * M;
    for (int i = lane; i < M; i += 32) x[i] = (i < j) ? 0.0 : (i == j ? 1.0 - tj : -tj * __ldcg(vj + i));
    __syncwarp();
    for (int h = j - 1; h >= 0; --h) {
      const double* vh = t.V + (long)h * M;
      double d = lane_dot(vh, x, h + lane, M);  // V(h,h) = 1
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      d *= __ldcg(t.tau + h);
      __syncwarp();
      for (int i = h + lane; i < M; i += 32) x[i] -= d * __ldcg(vh + i);
      __syncwarp();
    }
  }
  const long total = (long)r * N;
  for (long e = (long)local * blockDim.x + threadIdx.x; e < total; e += (long)t.ncta * blockDim.x) {
    const int c = (int)(e / r), i = (int)(e % r);
    const double y = (c >= i) ? __ldcg(t.R + (long)c * cap + i) : 0.0;
    t.F[(long)__ldcg(t.jpvt + c) * r + i] = y;
  }
  return true;
}

// Grouped column-pivoted QR: CTA b factorises the tiles list[start[b] .. start[b+1]) in turn
// (a large tile has a group of CTAs, small tiles share one CTA).  Cooperative launch.
__global__ void __launch_bounds__(QR_THREADS, 2) k_rrqr_grouped(QrTile* tiles, const int* __restrict__ start,
                                                              const int* __restrict__ list, double tol,
                                                              unsigned* status) {
  __shared__ QrSmem sm;
  for (int e = start[blockIdx.x]; e < start[blockIdx.x + 1]; ++e) {
    const QrTile t = tiles[list[e]];
    if (!qr_tile(t, blockIdx.x - t.cta0, tol, status, sm)) return;
  }
}

}  // namespace psmma

// ------------------------------------------------------------------------------------------
// Batched merge level: Q_i = alpha * A_i * H_i + beta * Q_i for a batch of Cauchy products,
// the off-diagonal blocks of each H_i (2 x 2 split at n_i / 2) compressed.  After the
// compression the products run in two grouped rounds (one launch per phase for all
// products of a round), recorded in one CUDA graph:
//   round 1: diagonal blocks (beta applied) and the first factor products,
//   round 2: the second factor products and uncompressed off-diagonal blocks (beta = 1).
// ------------------------------------------------------------------------------------------
using namespace psmma;

namespace {

struct OffBlock {
  int item, r0, M, c0, N;  // rows [r0, r0+M), columns [c0, c0+N) of H_item
};

// Bump allocation over one workspace; with base 0 it only measures.
struct Bump {
  uintptr_t base, off = 0;
  explicit Bump(void* b) : base((uintptr_t)b) {}
  template <class T>
  T* take(size_t count, size_t align = 256) {
    off = (off + align - 1) & ~(uintptr_t)(align - 1);
    T* p = (T*)(base + off);
    off += count * sizeof(T);
    return p;
  }
};

// Part A of the workspace: compression state, gather buffers, descriptors, status words.
struct Plan {
  std::vector<OffBlock> blocks;
  std::vector<RrluBlock> lu;
  std::vector<RrluEigBlock> lue;  // RRLU of accurate-denominator blocks
  std::vector<QrTile> qr;
  RrluBlock* d_lu = nullptr;
  RrluEigBlock* d_lue = nullptr;
  QrTile* d_qr = nullptr;
  int* d_ranks = nullptr;        // RRLU ranks
  int* d_pending = nullptr;      // RRLU blocks waiting for a complete-pivot search
  CpChunk* d_chunks = nullptr;   // column chunks of the search
  Cand* d_cand = nullptr;
  int *d_cpblk = nullptr, *d_cpfirst = nullptr;
  int chunk_cap = 0;
  static constexpr int CP_COLS = 64;
  std::vector<double*> gather;   // per block: RRLU n x M, RRQR n x cap
  GatherDesc* d_gather = nullptr;
  unsigned* d_status = nullptr;  // [0..7] product rounds, [8] QR
  int* d_map = nullptr;          // CTA work lists of the grouped QR launch
  long qr_cols = 0;
  static constexpr int MAP_MAX = 8192;
  static constexpr int N_STATUS = 16;
};

// Generators of the sub-block H(r0:, c0:) of an item's n x n matrix.  Cauchy: gen = [D|F|U|V]
// (ldgen); accurate-denominator Cauchy: gen = [F|U|V|DIFL|DIFR]; Toeplitz / Hankel: gen = G
// (2n - 1), H(i, j) = G(n + j - i) / G(i + j - 1) (1-based), so a sub-block is the same formula
// on G shifted by c0 - r0 / r0 + c0.
GenSpec sub_gens(int kind, const double* gen, long ldgen, int n, int r0, int c0) {
  GenSpec g;
  g.kind = kind;
  if (kind == KIND_TOEPLITZ) {
    g.g = gen + (c0 - r0);
    g.order = n;
    return g;
  }
  if (kind == KIND_HANKEL) {
    g.g = gen + (r0 + c0);
    g.order = n;
    return g;
  }
  if (kind == KIND_CAUCHY_EIG) {
    const double *F = gen, *U = gen + ldgen, *V = gen + 2 * ldgen, *DL = gen + 3 * ldgen, *DR = gen + 4 * ldgen;
    g.Dr = F + r0;
    g.Ur = U + r0;
    g.Fc = F + c0;
    g.Fc1 = F + c0 + 1;
    g.Vc = V + c0;
    g.dl = DL + c0;
    g.dr = DR + c0;
    g.fc1_len = n - 1 - c0;
    g.diag_off = c0 - r0;
    return g;
  }
  g.Dr = gen + r0;
  g.Fc = gen + ldgen + c0;
  g.Ur = gen + 2 * ldgen + r0;
  g.Vc = gen + 3 * ldgen + c0;
  return g;
}

// What the products need from the RRLU of block b: the poles and weights of
// Z'(t, j) = Z(Rk+t) W(j) / (P(Rk+t) - P(j)) (plain Cauchy in the pivoted row poles), the
// generators of Y = the rows PL(1:Rk) of the block with the unpermuted columns, and the
// local row permutation for the gather.
struct LuParts {
  const double *pole, *z, *w;
  GenSpec y;
  const int* perm;
};

LuParts lu_parts(const Plan& P, int kind, int b, const psmma_batch_item* items) {
  const OffBlock& ob = P.blocks[b];
  const psmma_batch_item& it = items[ob.item];
  LuParts lp;
  if (kind == KIND_CAUCHY_EIG) {
    const RrluEigBlock& r = P.lue[b];
    lp.pole = r.F;
    lp.z = r.U;
    lp.w = r.W;
    lp.y = sub_gens(kind, it.gen, it.ldgen, it.n, ob.r0, ob.c0);  // the columns C
    lp.y.Dr = r.F;      // F(PL(i))
    lp.y.Ur = r.A;      // LU
    lp.y.rglob = r.PL;  // global rows, for the branch of the denominator
    lp.y.cg0 = ob.c0;
    lp.perm = r.PQ;
  } else {
    const RrluBlock& r = P.lu[b];
    lp.pole = r.D;
    lp.z = r.U;
    lp.w = r.W;
    lp.y.kind = KIND_CAUCHY;
    lp.y.Dr = r.D;  // LD
    lp.y.Ur = r.A;  // LU
    lp.y.Fc = r.gF;
    lp.y.Vc = r.gV;
    lp.perm = r.PL;
  }
  return lp;
}

void make_plan(Plan& P, Bump& bump, const psmma_batch_item* items, int count, int compressor, int kind) {
  P.blocks.clear();
  for (int i = 0; i < count; ++i) {
    const int n = items[i].n, h = n / 2;
    if (h == 0) continue;
    P.blocks.push_back(OffBlock{i, 0, h, h, n - h});  // H(R1, C2)
    P.blocks.push_back(OffBlock{i, h, n - h, 0, h});  // H(R2, C1)
  }
  const int nb = (int)P.blocks.size();
  P.gather.assign(nb, nullptr);
  if (compressor == PSMMA_COMPRESS_RRLU && kind == KIND_CAUCHY_EIG) {
    P.lue.resize(nb);
    for (int b = 0; b < nb; ++b) {
      const OffBlock& ob = P.blocks[b];
      const psmma_batch_item& it = items[ob.item];
      RrluEigBlock& r = P.lue[b];
      r.M = ob.M;
      r.N = ob.N;
      r.FF = it.gen;                       // [F|U|V|DIFL|DIFR]
      r.DL = it.gen + 3 * (long)it.ldgen;
      r.DR = it.gen + 4 * (long)it.ldgen;
      r.nglob = it.n;
      r.gU = it.gen + (long)it.ldgen + ob.r0;
      r.gV = it.gen + 2 * (long)it.ldgen + ob.c0;
      r.r0 = ob.r0;
      r.c0 = ob.c0;
      r.F = bump.take<double>(ob.M);
      r.A = bump.take<double>(ob.M);
      r.U = bump.take<double>(ob.M);
      r.V = bump.take<double>(ob.N);
      r.W = bump.take<double>(std::min(ob.M, ob.N));
      r.PL = bump.take<int>(ob.M);
      r.PU = bump.take<int>(ob.N);
      r.PQ = bump.take<int>(ob.M);
      r.k_next = 1;
      r.phase = 0;
      r.cp_i = r.cp_j = 0;
      r.amax = 0.0;
      P.gather[b] = bump.take<double>((size_t)it.n * ob.M);
    }
    P.d_lue = bump.take<RrluEigBlock>(std::max(1, nb));
    P.d_ranks = bump.take<int>(std::max(1, nb));
    P.chunk_cap = nb;
    for (int b = 0; b < nb; ++b) P.chunk_cap += (P.blocks[b].N + Plan::CP_COLS - 1) / Plan::CP_COLS;
    P.d_pending = bump.take<int>(1);
    P.d_chunks = bump.take<CpChunk>(P.chunk_cap);
    P.d_cand = bump.take<Cand>(P.chunk_cap);
    P.d_cpblk = bump.take<int>(std::max(1, nb));
    P.d_cpfirst = bump.take<int>(std::max(1, nb));
    P.d_gather = bump.take<GatherDesc>(std::max(1, nb));
    for (int b = 0; b < nb; ++b) P.lue[b].rank = P.d_ranks + b;
  } else if (compressor == PSMMA_COMPRESS_RRLU) {
    P.lu.resize(nb);
    for (int b = 0; b < nb; ++b) {
      const OffBlock& ob = P.blocks[b];
      const psmma_batch_item& it = items[ob.item];
      RrluBlock& r = P.lu[b];
      r.M = ob.M;
      r.N = ob.N;
      r.gD = it.gen + ob.r0;
      r.gU = it.gen + 2 * (long)it.ldgen + ob.r0;
      r.gF = it.gen + it.ldgen + ob.c0;
      r.gV = it.gen + 3 * (long)it.ldgen + ob.c0;
      r.D = bump.take<double>(ob.M);
      r.A = bump.take<double>(ob.M);
      r.U = bump.take<double>(ob.M);
      r.F = bump.take<double>(ob.N);
      r.V = bump.take<double>(ob.N);
      r.W = bump.take<double>(std::min(ob.M, ob.N));
      r.PL = bump.take<int>(ob.M);
      r.PU = bump.take<int>(ob.N);
      r.k_next = 1;
      r.phase = 0;
      r.cp_i = r.cp_j = 0;
      r.amax = 0.0;
      P.gather[b] = bump.take<double>((size_t)it.n * ob.M);
    }
    P.d_lu = bump.take<RrluBlock>(std::max(1, nb));
    P.d_ranks = bump.take<int>(std::max(1, nb));
    P.chunk_cap = nb;
    for (int b = 0; b < nb; ++b) P.chunk_cap += (P.blocks[b].N + Plan::CP_COLS - 1) / Plan::CP_COLS;
    P.d_pending = bump.take<int>(1);
    P.d_chunks = bump.take<CpChunk>(P.chunk_cap);
    P.d_cand = bump.take<Cand>(P.chunk_cap);
    P.d_cpblk = bump.take<int>(std::max(1, nb));
    P.d_cpfirst = bump.take<int>(std::max(1, nb));
    P.d_gather = bump.take<GatherDesc>(std::max(1, nb));
    for (int b = 0; b < nb; ++b) P.lu[b].rank = P.d_ranks + b;
  } else {
    P.qr.resize(nb);
    long col0 = 0;
    for (int b = 0; b < nb; ++b) {
      const OffBlock& ob = P.blocks[b];
      const psmma_batch_item& it = items[ob.item];
      QrTile& q = P.qr[b];
      q.M = ob.M;
      q.N = ob.N;
      q.cap = std::min(std::min(ob.M, ob.N), QR_CAP);
      q.gs = sub_gens(kind, it.gen, it.ldgen, it.n, ob.r0, ob.c0);
      q.T = bump.take<double>((size_t)ob.M * ob.N);
      q.V = bump.take<double>((size_t)ob.M * q.cap);
      q.F = bump.take<double>((size_t)ob.N * q.cap);
      q.R = bump.take<double>((size_t)ob.N * q.cap);
      q.tau = bump.take<double>(q.cap + 1);
      q.s = bump.take<double>(q.cap);
      q.vn1 = bump.take<double>(ob.N);
      q.vn2 = bump.take<double>(ob.N);
      q.jpvt = bump.take<int>(ob.N);
      q.rank = bump.take<int>(1);
      q.flag = bump.take<int>(1);
      q.bar = bump.take<unsigned>(1);
      q.col0 = col0;
      col0 += ob.N;
      P.gather[b] = bump.take<double>((size_t)it.n * q.cap);
    }
    P.qr_cols = col0;
    P.d_qr = bump.take<QrTile>(std::max(1, nb));
    P.d_map = bump.take<int>(Plan::MAP_MAX + nb);
  }
  P.d_status = bump.take<unsigned>(Plan::N_STATUS);
}

// Products of the two rounds for the given ranks (rank >= min(M, N): block not compressed).
struct Rounds {
  std::vector<SplitProblem> r1, r2;
  double executed = 0.0;
  int max_rank = 0, full_blocks = 0;
};

void build_rounds(const Plan& P, const psmma_batch_item* items, int count, int compressor, int kind,
                  const int* ranks, double alpha, double beta, Rounds& R) {
  for (int i = 0; i < count; ++i) {
    const psmma_batch_item& it = items[i];
    const int n = it.n, h = n / 2;
    if (n == 0) continue;
    // diagonal blocks: Q(:, C1) = alpha A(:, R1) H(R1, C1) + beta Q(:, C1), and for R2, C2
    if (h > 0)
      R.r1.push_back(SplitProblem{n, h, h, alpha, beta, it.A, it.lda, sub_gens(kind, it.gen, it.ldgen, n, 0, 0), it.Q,
                                  it.ldq});
    R.r1.push_back(SplitProblem{n, n - h, n - h, alpha, beta, it.A + (long)h * it.lda, it.lda,
                                sub_gens(kind, it.gen, it.ldgen, n, h, h), it.Q + (long)h * it.ldq, it.ldq});
    R.executed += 2.0 * n * ((double)h * h + (double)(n - h) * (n - h));
  }
  const int nb = (int)P.blocks.size();
  for (int b = 0; b < nb; ++b) {
    const OffBlock& ob = P.blocks[b];
    const psmma_batch_item& it = items[ob.item];
    const int n = it.n, mn = std::min(ob.M, ob.N), Rk = ranks[b];
    const double* Ablk = it.A + (long)ob.r0 * it.lda;  // A(:, R)
    double* Qblk = it.Q + (long)ob.c0 * it.ldq;        // Q(:, C)
    if (Rk >= mn) {
      // not compressed: the generated tile (the reference would reuse a stale buffer here)
      ++R.full_blocks;
      R.r2.push_back(SplitProblem{n, ob.N, ob.M, alpha, 1.0, Ablk, it.lda, sub_gens(kind, it.gen, it.ldgen, n, ob.r0, ob.c0),
                                  Qblk, it.ldq});
      R.executed += 2.0 * n * (double)ob.M * ob.N;
      continue;
    }
    R.max_rank = std::max(R.max_rank, Rk);
    if (Rk == 0) continue;
    double* T = P.gather[b];
    if (compressor == PSMMA_COMPRESS_RRLU) {
      const LuParts lp = lu_parts(P, kind, b, items);
      // T0 += Ar * Z',  Z'(t, j) = Z(Rk+t) W(j) / (P(Rk+t) - P(j))  (T0, Ar gathered)
      GenSpec gz;
      gz.kind = KIND_CAUCHY;
      gz.Dr = lp.pole + Rk;
      gz.Ur = lp.z + Rk;
      gz.Fc = lp.pole;
      gz.Vc = lp.w;
      if (ob.M - Rk > 0)
        R.r1.push_back(SplitProblem{n, Rk, ob.M - Rk, 1.0, 1.0, T + (size_t)n * Rk, n, gz, T, n});
      // Q(:, C) += alpha * T0 * Y, Y = rows PL(1:Rk) of the block with the unpermuted columns
      R.r2.push_back(SplitProblem{n, ob.N, Rk, alpha, 1.0, T, n, lp.y, Qblk, it.ldq});
      R.executed += 2.0 * n * (double)(ob.M - Rk) * Rk + 2.0 * n * (double)Rk * ob.N;
    } else {
      const QrTile& q = P.qr[b];
      // T = A(:, R) * Q(:, 1:Rk), then Q(:, C) += alpha * T * (R P^T)
      GenSpec gq;
      gq.kind = KIND_DENSE;
      gq.B = q.T;
      gq.ldb = ob.M;
      R.r1.push_back(SplitProblem{n, Rk, ob.M, 1.0, 0.0, Ablk, it.lda, gq, T, n});
      GenSpec gyy;
      gyy.kind = KIND_DENSE;
      gyy.B = q.F;
      gyy.ldb = Rk;
      R.r2.push_back(SplitProblem{n, ob.N, Rk, alpha, 1.0, T, n, gyy, Qblk, it.ldq});
      R.executed += 2.0 * n * (double)ob.M * Rk + 2.0 * n * (double)Rk * ob.N;
    }
  }
}

// Split path: round 1 holds only the first factor products; round 2 has one product per
// output column block C, its diagonal block and the factor of the off-diagonal block (R_o, C)
// concatenated along K, so each output is recombined (CRT) once:
//   Q(:, C) = alpha * [A(:, R_d) | T] * [H(R_d, C); Y] + beta * Q(:, C),
// with Y the rows of H(PL(1:Rk), C) (RRLU, Cauchy with the pivoted row generators) or
// R P^T (RRQR, dense); an uncompressed block gives the whole column block A * H(:, C).
void build_rounds_split(const Plan& P, const psmma_batch_item* items, int count, int compressor, int kind,
                        const int* ranks, double alpha, double beta, Rounds& R) {
  // the off-diagonal block whose columns are C1 (rows R2) and C2 (rows R1), per item
  std::vector<int> blk_c1(count, -1), blk_c2(count, -1);
  for (int b = 0; b < (int)P.blocks.size(); ++b) {
    const OffBlock& ob = P.blocks[b];
    (ob.c0 == 0 ? blk_c1 : blk_c2)[ob.item] = b;
  }
  for (int b = 0; b < (int)P.blocks.size(); ++b) {
    const OffBlock& ob = P.blocks[b];
    const psmma_batch_item& it = items[ob.item];
    const int n = it.n, mn = std::min(ob.M, ob.N), Rk = ranks[b];
    if (Rk >= mn) {
      ++R.full_blocks;
      continue;
    }
    R.max_rank = std::max(R.max_rank, Rk);
    if (Rk == 0) continue;
    double* T = P.gather[b];
    if (compressor == PSMMA_COMPRESS_RRLU) {
      const LuParts lp = lu_parts(P, kind, b, items);
      GenSpec gz;  // Z'(t, j) = Z(Rk+t) W(j) / (P(Rk+t) - P(j)): T0 += A(:, PL(Rk+1:)) * Z'
      gz.kind = KIND_CAUCHY;
      gz.Dr = lp.pole + Rk;
      gz.Ur = lp.z + Rk;
      gz.Fc = lp.pole;
      gz.Vc = lp.w;
      if (ob.M - Rk > 0) {
        // A's columns are read through the pivots (gathered first: a copy of half of A, 363 of 11000 us at 32 problems)
        SplitProblem q{n, Rk, ob.M - Rk, 1.0, 1.0, it.A + (long)ob.r0 * it.lda, it.lda, gz, T, n};
        q.perm = lp.perm + Rk;
        R.r1.push_back(q);
        R.executed += 2.0 * n * (double)(ob.M - Rk) * Rk;
      }
    } else {
      GenSpec gq;  // T = A(:, R) * Q(:, 1:Rk)
      gq.kind = KIND_DENSE;
      gq.B = P.qr[b].T;
      gq.ldb = ob.M;
      R.r1.push_back(SplitProblem{n, Rk, ob.M, 1.0, 0.0, it.A + (long)ob.r0 * it.lda, it.lda, gq, T, n});
      R.executed += 2.0 * n * (double)ob.M * Rk;
    }
  }
  for (int i = 0; i < count; ++i) {
    const psmma_batch_item& it = items[i];
    const int n = it.n, h = n / 2;
    if (n == 0) continue;
    for (int half = 0; half < 2; ++half) {
      const int d0 = half == 0 ? 0 : h, dn = half == 0 ? h : n - h;  // R_d = C = [d0, d0 + dn)
      if (dn == 0) continue;
      double* Qc = it.Q + (long)d0 * it.ldq;
      const int b = half == 0 ? blk_c1[i] : blk_c2[i];
      const int Rk = b >= 0 ? ranks[b] : 0;
      const int mn = b >= 0 ? std::min(P.blocks[b].M, P.blocks[b].N) : 0;
      if (b >= 0 && Rk >= mn) {
        // uncompressed: the whole column block A * H(:, C)
        R.r2.push_back(SplitProblem{n, dn, n, alpha, beta, it.A, it.lda, sub_gens(kind, it.gen, it.ldgen, n, 0, d0), Qc,
                                    it.ldq});
        R.executed += 2.0 * n * (double)n * dn;
        continue;
      }
      SplitProblem q{n, dn, dn + Rk, alpha, beta, it.A + (long)d0 * it.lda, it.lda,
                     sub_gens(kind, it.gen, it.ldgen, n, d0, d0), Qc, it.ldq};
      if (Rk > 0) {
        q.A2 = P.gather[b];
        q.lda2 = n;
        q.ka = dn;
        q.gs.k1 = dn;
        if (compressor == PSMMA_COMPRESS_RRLU) {
          const LuParts lp = lu_parts(P, kind, b, items);
          q.gs.Dr2 = lp.y.Dr;        // pivoted row poles (1:Rk)
          q.gs.Ur2 = lp.y.Ur;        // LU(1:Rk)
          q.gs.rglob2 = lp.y.rglob;  // CauchyEig: global rows of the tail
          q.gs.cg0 = d0;
        } else {
          q.gs.B = P.qr[b].F;  // R P^T (Rk x N, ld Rk)
          q.gs.ldb = Rk;
        }
      }
      R.r2.push_back(q);
      R.executed += 2.0 * n * (double)dn * (dn + Rk);
    }
  }
}

// Workspace of the product rounds (part B).
struct RoundGroups {
  SplitGroup s1, s2;
  F64Group f[2 * 5];  // per round: Cauchy, accurate-denominator Cauchy, Toeplitz, Hankel, dense
};

// dense last: within a round the beta-scaled product of an output block comes first
constexpr int kNF64Kinds = 5;
constexpr int kF64Kinds[kNF64Kinds] = {KIND_CAUCHY, KIND_CAUCHY_EIG, KIND_TOEPLITZ, KIND_HANKEL, KIND_DENSE};

std::vector<F64Prob> f64_of(const std::vector<SplitProblem>& v, int kind) {
  std::vector<F64Prob> out;
  for (const SplitProblem& q : v)
    if (q.gs.kind == kind) out.push_back(F64Prob{q.M, q.N, q.K, q.alpha, q.beta, q.A, q.lda, q.gs, q.Q, q.ldq});
  return out;
}

size_t rounds_bytes(const Rounds& R, int precision, int n_moduli) {
  if (precision == PSMMA_PREC_SPLIT)
    return split_group_bytes(R.r1.data(), (int)R.r1.size(), n_moduli) + 4096 +
           split_group_bytes(R.r2.data(), (int)R.r2.size(), n_moduli) + 4096;
  return f64_group_bytes((int)R.r1.size()) * kNF64Kinds + f64_group_bytes((int)R.r2.size()) * kNF64Kinds + 4096;
}

int prepare_rounds(const Rounds& R, int precision, int n_moduli, const SplitTune& tune, void* work,
                   size_t lwork, cudaStream_t st, RoundGroups& G) {
  Bump b(work);
  if (precision == PSMMA_PREC_SPLIT) {
    const size_t b1 = split_group_bytes(R.r1.data(), (int)R.r1.size(), n_moduli);
    const size_t b2 = split_group_bytes(R.r2.data(), (int)R.r2.size(), n_moduli);
    char* w1 = b.take<char>(b1, 4096);
    char* w2 = b.take<char>(b2, 4096);
    if (b.off > lwork) return PSMMA_EWORKSPACE;
    int rc = split_group_prepare(R.r1.data(), (int)R.r1.size(), n_moduli, tune, w1, b1, st, &G.s1);
    if (!rc) rc = split_group_prepare(R.r2.data(), (int)R.r2.size(), n_moduli, tune, w2, b2, st, &G.s2);
    return rc;
  }
  const std::vector<SplitProblem>* rs[2] = {&R.r1, &R.r2};
  for (int r = 0; r < 2; ++r)
    for (int k = 0; k < kNF64Kinds; ++k) {
      const std::vector<F64Prob> v = f64_of(*rs[r], kF64Kinds[k]);
      char* w = b.take<char>(f64_group_bytes((int)v.size()), 256);
      if (b.off > lwork) return PSMMA_EWORKSPACE;
      const int rc = f64_group_prepare(v.data(), (int)v.size(), w, st, &G.f[kNF64Kinds * r + k]);
      if (rc) return rc;
    }
  return PSMMA_OK;
}

int enqueue_rounds(const RoundGroups& G, int precision, unsigned* status, cudaStream_t st) {
  int rc = PSMMA_OK;
  if (precision == PSMMA_PREC_SPLIT) {
    rc = split_group_enqueue(G.s1, st, status + 0);
    if (!rc) rc = split_group_enqueue(G.s2, st, status + 1);
    return rc;
  }
  for (int i = 0; i < 2 * kNF64Kinds && !rc; ++i) rc = f64_group_enqueue(G.f[i], st);
  return rc;
}

// Worst-case part B for a batch (every block at its largest rank and also uncompressed).
size_t rounds_bound(const Plan& P, const psmma_batch_item* items, int count, int compressor, int kind,
                    int precision, int n_moduli) {
  const int nb = (int)P.blocks.size();
  std::vector<int> rk(nb), full(nb);
  for (int b = 0; b < nb; ++b) {
    const int mn = std::min(P.blocks[b].M, P.blocks[b].N);
    rk[b] = compressor == PSMMA_COMPRESS_RRLU ? std::max(0, mn - 1) : std::min(std::max(0, mn - 1), QR_CAP);
    full[b] = mn;
  }
  Rounds a, f;
  auto build = precision == PSMMA_PREC_SPLIT ? build_rounds_split : build_rounds;
  build(P, items, count, compressor, kind, rk.data(), 1.0, 0.0, a);
  build(P, items, count, compressor, kind, full.data(), 1.0, 0.0, f);
  return rounds_bytes(a, precision, n_moduli) + rounds_bytes(f, precision, n_moduli);
}

// Work assignment of the grouped QR over `grid` co-resident CTAs: a tile of work w = M N gets
// a group of round(w / W) CTAs (W = total / grid) when that is >= 2; the other tiles are
// packed onto the remaining CTAs, largest first onto the least loaded (each alone on its CTA).
int launch_rrqr(Plan& P, int grid, double tol, unsigned* status, cudaStream_t st) {
  const int nb = (int)P.qr.size();
  double wsum = 0.0;
  for (const QrTile& q : P.qr) wsum += (double)q.M * q.N;
  const double W = wsum / grid;
  std::vector<int> ncta(nb, 0);
  int dedicated = 0;
  for (int b = 0; b < nb; ++b) {
    const QrTile& q = P.qr[b];
    int c = (int)std::lround((double)q.M * q.N / W);
    c = std::min(c, std::max(1, q.N / QR_WARPS));  // at least a column per warp
    ncta[b] = c >= 2 ? c : 0;
    dedicated += ncta[b];
  }
  int packable = 0;
  for (int b = 0; b < nb; ++b) packable += ncta[b] == 0;
  // leave at least one CTA per eight packed tiles (and one at all)
  const int reserve = packable ? std::max(1, std::min(packable, grid / 8)) : 0;
  while (dedicated > grid - reserve) {
    int big = -1;
    for (int b = 0; b < nb; ++b)
      if (ncta[b] > 2 && (big < 0 || ncta[b] > ncta[big])) big = b;
    if (big < 0) break;
    --ncta[big];
    --dedicated;
  }
  if (dedicated > grid - reserve) {  // too many groups: every tile alone
    for (int b = 0; b < nb; ++b) ncta[b] = 0;
    dedicated = 0;
  }
  std::vector<std::vector<int>> lists(grid);
  int next = 0;
  for (int b = 0; b < nb; ++b)
    if (ncta[b] >= 2) {
      P.qr[b].cta0 = next;
      P.qr[b].ncta = ncta[b];
      for (int c = 0; c < ncta[b]; ++c) lists[next + c].push_back(b);
      next += ncta[b];
    }
  const int free0 = next, nfree = grid - next;
  std::vector<int> small;
  for (int b = 0; b < nb; ++b)
    if (ncta[b] < 2) small.push_back(b);
  std::sort(small.begin(), small.end(), [&](int a, int b) {
    return (double)P.qr[a].M * P.qr[a].N > (double)P.qr[b].M * P.qr[b].N;
  });
  std::vector<double> load(std::max(1, nfree), 0.0);
  for (int b : small) {
    int c = (int)(std::min_element(load.begin(), load.end()) - load.begin());
    load[c] += (double)P.qr[b].M * P.qr[b].N;
    P.qr[b].cta0 = free0 + c;
    P.qr[b].ncta = 1;
    lists[free0 + c].push_back(b);
  }
  std::vector<int> h_start(grid + 1, 0), h_list;
  for (int c = 0; c < grid; ++c) {
    h_start[c] = (int)h_list.size();
    for (int b : lists[c]) h_list.push_back(b);
  }
  h_start[grid] = (int)h_list.size();
  // a tile of a group appears once per CTA of the group: at most grid + nb entries
  if (grid + 1 + (int)h_list.size() > Plan::MAP_MAX + nb) return PSMMA_EUNSUPPORTED;
  int* d_start = P.d_map;
  int* d_list = P.d_map + grid + 1;
  if (cudaMemcpyAsync(P.d_qr, P.qr.data(), sizeof(QrTile) * nb, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_start, h_start.data(), sizeof(int) * (grid + 1), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(d_list, h_list.data(), sizeof(int) * h_list.size(), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return PSMMA_EDEVICE;
  QrTile* tiles = P.d_qr;
  const int* ps = d_start;
  const int* pl = d_list;
  void* args[] = {(void*)&tiles, (void*)&ps, (void*)&pl, (void*)&tol, (void*)&status};
  if (cudaLaunchCooperativeKernel((const void*)k_rrqr_grouped, dim3(grid), dim3(QR_THREADS), args, 0, st) !=
      cudaSuccess)
    return PSMMA_EDEVICE;
  return PSMMA_OK;
}

int check_batch(int count, const psmma_batch_item* items, int precision, int n_moduli, int compressor,
                double tol, int kind = KIND_CAUCHY) {
  const bool vec = kind == KIND_TOEPLITZ || kind == KIND_HANKEL;  // gen = G (2n - 1), ldgen = its length
  if (vec && compressor != PSMMA_COMPRESS_RRQR) return PSMMA_EUNSUPPORTED;
  if (count < 0 || (count > 0 && !items)) return PSMMA_ENULL;
  if (precision != PSMMA_PREC_FP64 && precision != PSMMA_PREC_SPLIT) return PSMMA_EUNSUPPORTED;
  if (precision == PSMMA_PREC_SPLIT && n_moduli != 0 && (n_moduli < 8 || n_moduli > 16)) return PSMMA_EUNSUPPORTED;
  if (compressor != PSMMA_COMPRESS_RRQR && compressor != PSMMA_COMPRESS_RRLU) return PSMMA_EUNSUPPORTED;
  if (!(tol > 0.0) || !(tol < 1.0)) return PSMMA_EUNSUPPORTED;
  for (int i = 0; i < count; ++i) {
    const psmma_batch_item& it = items[i];
    if (it.n < 0) return -2;
    if (it.lda < std::max(1, it.n)) return -9;
    if (it.ldq < std::max(1, it.n)) return -14;
    if (it.n > 0 && (!it.A || !it.Q)) return PSMMA_ENULL;
    if (it.n > 0 && (!it.gen || it.ldgen < (vec ? 2 * it.n - 1 : it.n))) return PSMMA_EGEN;
  }
  return PSMMA_OK;
}

size_t part_a_bytes(Plan& P, const psmma_batch_item* items, int count, int compressor, int kind) {
  Bump m(nullptr);
  make_plan(P, m, items, count, compressor, kind);
  return m.off + 4096;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// Autotuner of the grouped split GEMM (tile widths, raster group): configurations are timed
// on a whole batch and the best is kept per batch signature (and, with PSMMA_TUNE_CACHE set
// to a file, across processes: one "signature narrow_max mid_max group_m" line each).
// ------------------------------------------------------------------------------------------
namespace {

std::mutex g_tune_mu;
std::map<unsigned long long, SplitTune> g_tune;
bool g_tune_loaded = false;
thread_local const SplitTune* t_force = nullptr;  // set while the tuner runs a candidate

// FNV-1a of the batch shape: count, precision, moduli, compressor and the sizes binned at
// 1/8 octave (batches of the same size distribution share a configuration).
unsigned long long batch_signature(int count, const psmma_batch_item* items, int compressor, int precision,
                                   int n_moduli) {
  std::vector<int> bins;
  for (int i = 0; i < count; ++i)
    bins.push_back(items[i].n > 0 ? (int)std::lround(8.0 * std::log2((double)items[i].n)) : -1);
  std::sort(bins.begin(), bins.end());
  unsigned long long h = 1469598103934665603ull;
  auto mix = [&](long long v) {
    for (int b = 0; b < 8; ++b) {
      h ^= (unsigned long long)((v >> (8 * b)) & 0xff);
      h *= 1099511628211ull;
    }
  };
  mix(count);
  mix(precision);
  mix(n_moduli);
  mix(compressor);
  for (int b : bins) mix(b);
  return h;
}

void tune_load_locked() {
  if (g_tune_loaded) return;
  g_tune_loaded = true;
  const char* path = std::getenv("PSMMA_TUNE_CACHE");
  if (!path || !*path) return;
  FILE* f = std::fopen(path, "r");
  if (!f) return;
  unsigned long long sig;
  SplitTune t;
  while (std::fscanf(f, "%llx %d %d %d", &sig, &t.narrow_max, &t.mid_max, &t.group_m) == 4) g_tune[sig] = t;
  std::fclose(f);
}

SplitTune tune_for(unsigned long long sig) {
  if (t_force) return *t_force;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_load_locked();
  auto it = g_tune.find(sig);
  return it == g_tune.end() ? SplitTune() : it->second;
}

void tune_store(unsigned long long sig, const SplitTune& t) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_load_locked();
  g_tune[sig] = t;
  const char* path = std::getenv("PSMMA_TUNE_CACHE");
  if (!path || !*path) return;
  if (FILE* f = std::fopen(path, "a")) {
    std::fprintf(f, "%llx %d %d %d\n", sig, t.narrow_max, t.mid_max, t.group_m);
    std::fclose(f);
  }
}

// The resumable RRLU of all blocks: launch, then while blocks wait for a complete-pivot
// search run it grid-wide and resume them.  Every resume advances some block by a step, so
// the loop is bounded by the largest min(M, N).
template <class Block>
int run_rrlu(Plan& P, std::vector<Block>& hb, Block* d_blocks, void (*krrlu)(Block*, double, int*),
             void (*ksearch)(const Block*, const CpChunk*, Cand*), double tol, std::vector<int>& ranks,
             cudaStream_t st) {
  const int nb = (int)hb.size();
  if (cudaMemcpyAsync(d_blocks, hb.data(), sizeof(Block) * nb, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemsetAsync(P.d_pending, 0, sizeof(int), st) != cudaSuccess)
    return PSMMA_EDEVICE;
  krrlu<<<nb, RRLU_THREADS, 0, st>>>(d_blocks, tol, P.d_pending);
  if (cudaGetLastError() != cudaSuccess) return PSMMA_EDEVICE;
  int max_iter = 2;
  for (const OffBlock& ob : P.blocks) max_iter = std::max(max_iter, std::min(ob.M, ob.N) + 2);
  std::vector<Block> cur(nb);
  std::vector<CpChunk> chunks;
  std::vector<int> cpblk, cpfirst;
  int iter = 0;
  for (; iter < max_iter; ++iter) {
    int pend = 0;
    if (cudaMemcpyAsync(&pend, P.d_pending, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(cur.data(), d_blocks, sizeof(Block) * nb, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return PSMMA_EDEVICE;
    if (pend == 0) break;
    chunks.clear();
    cpblk.clear();
    cpfirst.clear();
    for (int b = 0; b < nb; ++b) {
      if (cur[b].phase != 1) continue;
      cpblk.push_back(b);
      cpfirst.push_back((int)chunks.size());
      for (int c = cur[b].k_next - 1; c < cur[b].N; c += Plan::CP_COLS)
        chunks.push_back(CpChunk{b, c, std::min(cur[b].N, c + Plan::CP_COLS)});
    }
    if (chunks.empty() || (int)chunks.size() > P.chunk_cap) return PSMMA_EDEVICE;
    if (cudaMemcpyAsync(P.d_chunks, chunks.data(), sizeof(CpChunk) * chunks.size(), cudaMemcpyHostToDevice, st) !=
            cudaSuccess ||
        cudaMemcpyAsync(P.d_cpblk, cpblk.data(), sizeof(int) * cpblk.size(), cudaMemcpyHostToDevice, st) !=
            cudaSuccess ||
        cudaMemcpyAsync(P.d_cpfirst, cpfirst.data(), sizeof(int) * cpfirst.size(), cudaMemcpyHostToDevice, st) !=
            cudaSuccess ||
        cudaMemsetAsync(P.d_pending, 0, sizeof(int), st) != cudaSuccess)
      return PSMMA_EDEVICE;
    ksearch<<<(unsigned)chunks.size(), RRLU_THREADS, 0, st>>>(d_blocks, P.d_chunks, P.d_cand);
    k_cp_reduce<Block><<<((int)cpblk.size() + 127) / 128, 128, 0, st>>>(d_blocks, P.d_cpblk, P.d_cpfirst,
                                                                        (int)cpblk.size(), (int)chunks.size(),
                                                                        P.d_cand);
    krrlu<<<nb, RRLU_THREADS, 0, st>>>(d_blocks, tol, P.d_pending);
    if (cudaGetLastError() != cudaSuccess) return PSMMA_EDEVICE;
  }
  if (iter == max_iter) return PSMMA_EDEVICE;
  if (cudaMemcpyAsync(ranks.data(), P.d_ranks, sizeof(int) * nb, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return PSMMA_EDEVICE;
  return PSMMA_OK;
}

// ------------------------------------------------------------------------------------------
// The product rounds' CUDA graph, kept per (device, stream): each call captures its launches
// (cheap, host only) and, when an executable graph exists for the stream, updates it in place
// with cudaGraphExecUpdate (new pointers, ranks, alpha/beta); only a change of topology (other
// launch count or kernels) instantiates a new one.  The capture stream and its event persist
// with the entry.
// ------------------------------------------------------------------------------------------
struct GraphSlot {
  std::mutex mu;  // one call at a time uses a slot
  cudaStream_t cap = nullptr;
  cudaEvent_t ev = nullptr;
  cudaGraphExec_t exec = nullptr;
};

std::mutex g_graph_mu;
std::map<std::pair<int, cudaStream_t>, GraphSlot*> g_graphs;

GraphSlot* graph_slot(cudaStream_t stream) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(g_graph_mu);
  GraphSlot*& g = g_graphs[{dev, stream}];
  if (!g) {
    GraphSlot* n = new GraphSlot;
    if (cudaStreamCreateWithFlags(&n->cap, cudaStreamNonBlocking) != cudaSuccess) {
      delete n;
      return nullptr;
    }
    if (cudaEventCreateWithFlags(&n->ev, cudaEventDisableTiming) != cudaSuccess) {
      cudaStreamDestroy(n->cap);
      delete n;
      return nullptr;
    }
    g = n;
  }
  return g;
}

// Updates the slot's executable graph to `graph`, or instantiates it when the slot has none or
// the update is refused (topology changed).  *reused = 1 when the existing executable was kept.
int graph_exec_for(GraphSlot* gs, cudaGraph_t graph, int* reused) {
  *reused = 0;
  if (gs->exec) {
    cudaGraphExecUpdateResultInfo info;
    if (cudaGraphExecUpdate(gs->exec, graph, &info) == cudaSuccess) {
      *reused = 1;
      return PSMMA_OK;
    }
    cudaGetLastError();
    cudaGraphExecDestroy(gs->exec);
    gs->exec = nullptr;
  }
  if (cudaGraphInstantiate(&gs->exec, graph, 0) != cudaSuccess) {
    gs->exec = nullptr;
    return PSMMA_EDEVICE;
  }
  return PSMMA_OK;
}

}  // namespace

static size_t batch_workspace(int kind, int count, const psmma_batch_item* items, int compressor,
                              const psmma_opts* opts) {
  const int precision = opts ? opts->precision : PSMMA_PREC_FP64;
  const int n_moduli = opts ? opts->n_moduli : 0;
  if (count <= 0 || !items || check_batch(count, items, precision, n_moduli, compressor, 0.5, kind)) return 0;
  Plan P;
  const size_t a = part_a_bytes(P, items, count, compressor, kind);
  return a + rounds_bound(P, items, count, compressor, kind, precision, n_moduli) + 4096;
}

extern "C" size_t psmma_batch_workspace_size(int count, const psmma_batch_item* items, int compressor,
                                             const psmma_opts* opts) {
  return batch_workspace(KIND_CAUCHY, count, items, compressor, opts);
}

extern "C" size_t psmma_cauchyeig_batch_workspace_size(int count, const psmma_batch_item* items, int compressor,
                                                       const psmma_opts* opts) {
  return batch_workspace(KIND_CAUCHY_EIG, count, items, compressor, opts);
}

extern "C" size_t psmma_toeplitz_batch_workspace_size(int count, const psmma_batch_item* items,
                                                      const psmma_opts* opts) {
  return batch_workspace(KIND_TOEPLITZ, count, items, PSMMA_COMPRESS_RRQR, opts);
}

static int batch_run(int kind, int count, const psmma_batch_item* items, double alpha, double beta, int compressor,
                     double tol, const psmma_opts* opts, int* ranks_out, psmma_batch_stats* stats, void* stream) {
  const int precision = opts ? opts->precision : PSMMA_PREC_FP64;
  const int n_moduli = opts ? opts->n_moduli : 0;
  int rc = check_batch(count, items, precision, n_moduli, compressor, tol, kind);
  if (rc) return rc;
  if (stats) *stats = psmma_batch_stats{0.0, 0.0, 0.0, 0, 0, 0, 0};
  if (count == 0) return PSMMA_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const StreamCall call(st, !(opts && opts->work));

  Plan P;
  const size_t need_a = part_a_bytes(P, items, count, compressor, kind);
  char* work_a = nullptr;
  char* work_b = nullptr;
  size_t lwork_b = 0;
  if (opts && opts->work) {
    const size_t bound = need_a + rounds_bound(P, items, count, compressor, kind, precision, n_moduli) + 4096;
    if (opts->lwork < bound) return PSMMA_EWORKSPACE;
    work_a = (char*)opts->work;
    work_b = (char*)((((uintptr_t)work_a + need_a) + 4095) & ~(uintptr_t)4095);
    lwork_b = (size_t)(work_a + opts->lwork - work_b);
  } else {
    work_a = (char*)pool_get(need_a, st, &rc, 0);
    if (rc) return rc;
  }
  Bump bump((void*)(((uintptr_t)work_a + 255) & ~(uintptr_t)255));
  make_plan(P, bump, items, count, compressor, kind);
  const int nb = (int)P.blocks.size();
  if (cudaMemsetAsync(P.d_status, 0, sizeof(unsigned) * Plan::N_STATUS, st) != cudaSuccess) return PSMMA_EDEVICE;
  unsigned* qr_status = P.d_status + 8;
  prof_begin(st);

  // ---- phase 1: compression of every off-diagonal block
  std::vector<int> ranks(nb, 0);
  double compress_flops = 0.0;
  if (nb && compressor == PSMMA_COMPRESS_RRLU) {
    rc = (kind == KIND_CAUCHY_EIG) ? run_rrlu(P, P.lue, P.d_lue, k_rrlu_eig, k_cp_search_eig, tol, ranks, st)
                                   : run_rrlu(P, P.lu, P.d_lu, k_rrlu_cauchy, k_cp_search, tol, ranks, st);
    if (rc) return rc;
    for (int b = 0; b < nb; ++b) compress_flops += 12.0 * (ranks[b] + 1) * (P.blocks[b].M + P.blocks[b].N);
  } else if (nb) {
    if (cudaMemcpyAsync(P.d_qr, P.qr.data(), sizeof(QrTile) * nb, cudaMemcpyHostToDevice, st) != cudaSuccess)
      return PSMMA_EDEVICE;
    if (P.qr_cols > 0x7fffffffL) return PSMMA_EUNSUPPORTED;
    k_qr_tiles<<<(unsigned)P.qr_cols, QR_THREADS, 0, st>>>(P.d_qr, nb);
    if (cudaGetLastError() != cudaSuccess) return PSMMA_EDEVICE;
    int dev = 0, sms = 0, occ = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_rrqr_grouped, QR_THREADS, 0) != cudaSuccess || occ < 1)
      return PSMMA_EDEVICE;
    const int grid = std::min(sms * std::min(occ, 4), Plan::MAP_MAX - 1);
    rc = launch_rrqr(P, grid, tol, qr_status, st);
    if (rc) return rc;
    unsigned qs = 0;
    if (cudaMemcpyAsync(&qs, qr_status, sizeof(unsigned), cudaMemcpyDeviceToHost, st) != cudaSuccess)
      return PSMMA_EDEVICE;
    for (int b = 0; b < nb; ++b)
      if (cudaMemcpyAsync(&ranks[b], P.qr[b].rank, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return PSMMA_EDEVICE;
    if (cudaStreamSynchronize(st) != cudaSuccess) return PSMMA_EDEVICE;
    if (qs & DEV_ERR_TIMEOUT) return PSMMA_ETIMEDOUT;
    for (int b = 0; b < nb; ++b) {
      const double M = P.blocks[b].M, N = P.blocks[b].N, r = std::min(ranks[b], P.qr[b].cap);
      compress_flops += 4.0 * M * N * (r + 1) + 4.0 * M * r * r;
    }
  }
  if (ranks_out)
    for (int b = 0; b < nb; ++b) ranks_out[b] = ranks[b];
  prof_mark(st, compressor == PSMMA_COMPRESS_RRLU ? "compress_rrlu" : "compress_rrqr");

  // ---- phase 2: the product rounds, one CUDA graph
  Rounds R;
  (precision == PSMMA_PREC_SPLIT ? build_rounds_split : build_rounds)(P, items, count, compressor, kind,
                                                                      ranks.data(), alpha, beta, R);
  const size_t need_b = rounds_bytes(R, precision, n_moduli);
  if (!work_b) {
    work_b = (char*)pool_get(need_b, st, &rc, 1);
    if (rc) return rc;
    lwork_b = need_b;
  }
  RoundGroups G;
  const SplitTune tune = tune_for(batch_signature(count, items, compressor + 4 * kind, precision, n_moduli));
  rc = prepare_rounds(R, precision, n_moduli, tune, work_b, lwork_b, st, G);
  if (rc) return rc;
  std::vector<GatherDesc> gd;
  int gather_cols = 0;
  if (compressor == PSMMA_COMPRESS_RRLU) {
    for (int b = 0; b < nb; ++b) {
      const OffBlock& ob = P.blocks[b];
      const psmma_batch_item& it = items[ob.item];
      if (ranks[b] <= 0 || ranks[b] >= std::min(ob.M, ob.N)) continue;
      GatherDesc g;
      g.A = it.A + (long)ob.r0 * it.lda;
      g.lda = it.lda;
      g.n = it.n;
      g.M = ob.M;
      g.Rk = ranks[b];
      g.c0 = gather_cols;
      g.PL = lu_parts(P, kind, b, items).perm;
      g.T0 = P.gather[b];
      g.Ar = P.gather[b] + (size_t)it.n * ranks[b];
      gd.push_back(g);
      gather_cols += precision == PSMMA_PREC_SPLIT ? ranks[b] : ob.M;  // the split passes read the rest in place
    }
    if (!gd.empty() && cudaMemcpyAsync(P.d_gather, gd.data(), sizeof(GatherDesc) * gd.size(),
                                       cudaMemcpyHostToDevice, st) != cudaSuccess)
      return PSMMA_EDEVICE;
  }
  prof_mark(st, "prepare_rounds");
  if (prof_enabled()) {
    // traced run: the same launches directly on the stream, one event per phase
    if (!gd.empty()) k_gather_group<<<gather_cols, 256, 0, st>>>(P.d_gather, (int)gd.size());
    prof_mark(st, "gather");
    rc = enqueue_rounds(G, precision, P.d_status, st);
    unsigned sts[Plan::N_STATUS] = {0};
    if (!rc && (cudaMemcpyAsync(sts, P.d_status, sizeof(sts), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess))
      rc = PSMMA_EDEVICE;
    for (unsigned v : sts)
      if (!rc && (v & DEV_ERR_TIMEOUT)) rc = PSMMA_ETIMEDOUT;
    if (stats) {
      double eff = 0.0;
      for (int i = 0; i < count; ++i) eff += 2.0 * items[i].n * (double)items[i].n * items[i].n;
      *stats = psmma_batch_stats{eff, R.executed, compress_flops, nb, R.max_rank, R.full_blocks, 0};
    }
    return rc;
  }
  GraphSlot* gsl = graph_slot(st);
  if (!gsl) return PSMMA_EDEVICE;
  std::lock_guard<std::mutex> glk(gsl->mu);
  cudaStream_t cap = gsl->cap;
  cudaEvent_t ev = gsl->ev;
  cudaEventRecord(ev, st);
  cudaStreamWaitEvent(cap, ev, 0);  // the graph follows the compression and the copies above
  cudaGraph_t graph = nullptr;
  int reused = 0;
  if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = PSMMA_EDEVICE;
  if (!rc && !gd.empty()) {
    k_gather_group<<<gather_cols, 256, 0, cap>>>(P.d_gather, (int)gd.size());
    if (cudaGetLastError() != cudaSuccess) rc = PSMMA_EDEVICE;
  }
  if (!rc) rc = enqueue_rounds(G, precision, P.d_status, cap);
  cudaError_t ce = cudaStreamEndCapture(cap, &graph);
  if (!rc && ce != cudaSuccess) rc = PSMMA_EDEVICE;
  if (!rc) rc = graph_exec_for(gsl, graph, &reused);
  if (!rc && cudaGraphLaunch(gsl->exec, cap) != cudaSuccess) rc = PSMMA_EDEVICE;
  cudaEventRecord(ev, cap);
  cudaStreamWaitEvent(st, ev, 0);  // later work on `stream` follows the graph
  unsigned sts[Plan::N_STATUS] = {0};
  if (!rc && (cudaMemcpyAsync(sts, P.d_status, sizeof(sts), cudaMemcpyDeviceToHost, cap) != cudaSuccess ||
              cudaStreamSynchronize(cap) != cudaSuccess))
    rc = PSMMA_EDEVICE;
  if (graph) cudaGraphDestroy(graph);
  for (unsigned v : sts)
    if (!rc && (v & DEV_ERR_TIMEOUT)) rc = PSMMA_ETIMEDOUT;
  if (stats) {
    double eff = 0.0;
    for (int i = 0; i < count; ++i) eff += 2.0 * items[i].n * (double)items[i].n * items[i].n;
    stats->effective_flops = eff;
    stats->executed_flops = R.executed;
    stats->compress_flops = compress_flops;
    stats->n_blocks = nb;
    stats->max_rank = R.max_rank;
    stats->full_rank_blocks = R.full_blocks;
    stats->graph_reused = reused;
  }
  return rc;
}

extern "C" int psmma_cauchy_batch_lowrank(int count, const psmma_batch_item* items, double alpha, double beta,
                                          int compressor, double tol, const psmma_opts* opts, int* ranks_out,
                                          psmma_batch_stats* stats, void* stream) {
  return batch_run(KIND_CAUCHY, count, items, alpha, beta, compressor, tol, opts, ranks_out, stats, stream);
}

extern "C" int psmma_cauchyeig_batch_lowrank(int count, const psmma_batch_item* items, double alpha, double beta,
                                             int compressor, double tol, const psmma_opts* opts, int* ranks_out,
                                             psmma_batch_stats* stats, void* stream) {
  return batch_run(KIND_CAUCHY_EIG, count, items, alpha, beta, compressor, tol, opts, ranks_out, stats, stream);
}

extern "C" int psmma_toeplitz_batch_lowrank(int count, const psmma_batch_item* items, double alpha, double beta,
                                            double tol, const psmma_opts* opts, int* ranks_out,
                                            psmma_batch_stats* stats, void* stream) {
  return batch_run(KIND_TOEPLITZ, count, items, alpha, beta, PSMMA_COMPRESS_RRQR, tol, opts, ranks_out, stats, stream);
}

extern "C" int psmma_tune_batch(int count, const psmma_batch_item* items, double alpha, double beta, int compressor,
                                double tol, const psmma_opts* opts, psmma_tune_result* out, void* stream) {
  const int precision = opts ? opts->precision : PSMMA_PREC_FP64;
  const int n_moduli = opts ? opts->n_moduli : 0;
  int rc = check_batch(count, items, precision, n_moduli, compressor, tol);
  if (rc) return rc;
  if (out) *out = psmma_tune_result{64, 128, 12, 0, 0.0f, 0.0f};
  if (count == 0 || precision != PSMMA_PREC_SPLIT) return PSMMA_OK;  // FP64 path: one tile shape
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return PSMMA_EDEVICE;
  const SplitTune dflt;
  const int widths[4][2] = {{0, 0}, {64, 0}, {64, 128}, {64, 256}};
  const int groups[3] = {4, 8, 16};
  std::vector<SplitTune> cands{dflt};
  for (auto& w : widths)
    for (int gm : groups) cands.push_back(SplitTune{w[0], w[1], gm});
  float best = 0.0f, first = 0.0f;
  SplitTune best_t = dflt;
  for (size_t c = 0; c < cands.size() && !rc; ++c) {
    t_force = &cands[c];
    rc = batch_run(KIND_CAUCHY, count, items, alpha, beta, compressor, tol, opts, nullptr, nullptr, stream);
    float ms = 0.0f;
    for (int rep = 0; rep < 2 && !rc; ++rep) {  // the faster of two timed runs (the first warmed up)
      cudaEventRecord(e0, st);
      rc = batch_run(KIND_CAUCHY, count, items, alpha, beta, compressor, tol, opts, nullptr, nullptr, stream);
      cudaEventRecord(e1, st);
      float t = 0.0f;
      if (!rc && (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&t, e0, e1) != cudaSuccess))
        rc = PSMMA_EDEVICE;
      ms = rep == 0 ? t : std::min(ms, t);
    }
    t_force = nullptr;
    if (rc) break;
    if (c == 0) first = ms;
    if (c == 0 || ms < best) {
      best = ms;
      best_t = cands[c];
    }
  }
  t_force = nullptr;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  // a candidate replaces the default only when it is clearly faster: differences within 2 %
  // are run-to-run noise of a power-capped GPU, and the default is the configuration tested most
  if (best > 0.98f * first) {
    best = first;
    best_t = dflt;
  }
  tune_store(batch_signature(count, items, compressor, precision, n_moduli), best_t);
  if (out) *out = psmma_tune_result{best_t.narrow_max, best_t.mid_max, best_t.group_m, (int)cands.size(), best, first};
  return PSMMA_OK;
}
