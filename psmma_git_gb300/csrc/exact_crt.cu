// The FP64 precision's fast route: the structured product Q = alpha*A*H + beta*Q with A*H formed
// EXACTLY on the BF16 tensor cores and rounded once.
//
// GB300 issues about two FP64 multiply-adds per SM per cycle, on the scalar and on the tensor
// form alike (0.6e12 a second), so a product of 2 n^3 FP64 flops is bound by that pipe.  The
// modular GEMM of split_crt.cu runs BF16 at 1700 times that rate, and unlike the split precision,
// which rounds A and H to the bits its moduli cover, this route takes as many moduli as the
// operands need:
//   1. a_max, the lowest set bit and the 2-norm of every row of A; the same of every column of H,
//      generated in FP64 by the entry formulas of the DMMA kernel (fp64_structured.cu).
//   2. Row i times 2^-lsb_i and column j times 2^-lsb_j are integers without any rounding.  A bound
//      of |Z_ij| = |(A'H')_ij| from the norms gives the number of moduli whose product exceeds
//      2 |Z| (8 to 32 in steps of 4, up to 241 bits), on the device.
//   3. One BF16 GEMM per modulus, the Chinese remainder theorem on 32-bit words, and one rounding
//      of Z 2^(lsb_i + lsb_j) to FP64; then alpha and beta.
// The rounded sum of exact products is at least as accurate as any order of FP64 additions.  Where
// a row or column spans more than 112 bits, the bound exceeds the moduli, an entry is not finite or
// a device wait gave up, the flag `nmod` is 0 and the DMMA kernel, enqueued behind this route and
// gated on that flag, computes the product as it would alone.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "psmma_internal.h"
#include "split_passes.cuh"
#include "tcgen05_util.cuh"

namespace psmma {

int launch_modular_gemm(__nv_bfloat16* RA, __nv_bfloat16* RH, int8_t* R, int M, int N, int kp, int kr, int planes,
                        const int* moduli, const int* nmod_dev, unsigned* status, int sms, cudaStream_t stream);

namespace {

// ------------------------------------------------------------------------------------------
// Moduli and CRT constants (compile time)
// ------------------------------------------------------------------------------------------
// Pairwise coprime, at most 256: 2^8, 3*5*17, 11*23, 13*19, 7*31 and primes.
constexpr int EX_MAX = 32, EX_GROUPS = EX_MAX / 4, EX_WORDS = 8, EX_PARTS = 10, EX_CHUNKS = 8;
constexpr int kExModuli[EX_MAX] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193, 191,
                                   217, 181, 179, 173, 167, 163, 157, 151, 149, 139, 137, 131, 127, 113, 109, 107};

// The CRT for the first 4 G moduli.  They form parts of three and then, where 4 G is not a multiple of three, one or two
// of four (8 moduli: 3, 3, 2), each of a product P_g < 2^32; a part's moduli are first combined in 32-bit arithmetic:
//   X_g = b_g + sum_i r_i c_i (mod P_g),  X_g = Z W_g^-1 mod P_g,  W_g = M / P_g,
// and Z = sum_g X_g W_g - q M with q the nearest integer to sum_g X_g / P_g.  The parts of four have the smallest
// moduli: sum_g X_g W_g[s] stays below 2^63 for every 32-bit word s, so that the sums are the words of Z.
__host__ __device__ constexpr int ex_fours(int G) { return G == 2 ? 0 : 4 * G % 3; }
__host__ __device__ constexpr int ex_parts(int G) { return G == 2 ? 3 : (4 * G - 4 * ex_fours(G)) / 3 + ex_fours(G); }
__host__ __device__ constexpr int ex_first(int G, int g) {  // first modulus of part g
  const int threes = G == 2 ? 3 : ex_parts(G) - ex_fours(G);
  return g < threes ? 3 * g : 3 * threes + 4 * (g - threes);
}
__host__ __device__ constexpr int ex_size(int G, int g) { return (g + 1 < ex_parts(G) ? ex_first(G, g + 1) : 4 * G) - ex_first(G, g); }
__host__ __device__ constexpr int ex_shift(int G) { return G == 2 ? 47 : 52; }  // fixed point of 1 / P_g: P_g >= 2^15.7, 2^20 above
__host__ __device__ constexpr int ex_words(int G) { return G; }                 // log2 M = 63.6, 94.8, 125.2, 155.4, 184.6, 213.1, 240.4
struct ExCrt {
  unsigned c[EX_MAX], f[EX_MAX];      // c_i, floor(2^20 c_i / P_g)
  // the starts of both sums, so that they are those of r + 128 in [0, 255]; P_g, floor(2^ex_shift / P_g)
  unsigned b[EX_PARTS], fb[EX_PARTS], P[EX_PARTS], G[EX_PARTS];
  unsigned W[EX_PARTS][EX_WORDS];     // W_g
  unsigned Mneg[EX_WORDS];            // 2^256 - M
};
struct ExTables {
  ExCrt crt[EX_GROUPS + 1];           // by group count (2..8)
  float g[EX_MAX][EX_CHUNKS];         // 2^(14 t) mod m, symmetric; [0] = 1 / m
  float m[EX_MAX];
};

constexpr unsigned long long ex_inv(unsigned long long a, unsigned long long m) {
  for (unsigned long long x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 0;
}

constexpr ExTables make_tables() {
  ExTables T{};
  for (int l = 0; l < EX_MAX; ++l) {
    const int m = kExModuli[l];
    T.m[l] = (float)m;
    long long p = 1;
    for (int t = 0; t < EX_CHUNKS; ++t) {
      const long long s = p > m / 2 ? p - m : p;
      T.g[l][t] = t == 0 ? 1.0f / (float)m : (float)s;
      p = p * (1 << 14) % m;
    }
  }
  for (int G = 2; G <= EX_GROUPS; ++G) {
    ExCrt& C = T.crt[G];
    for (int g = 0; g < ex_parts(G); ++g) {
      const int first = ex_first(G, g), size = ex_size(G, g);
      unsigned long long P = 1;
      for (int i = 0; i < size; ++i) P *= (unsigned long long)kExModuli[first + i];
      C.P[g] = (unsigned)P;
      C.G[g] = (unsigned)((1ull << ex_shift(G)) / P);
      C.W[g][0] = 1;
      for (int l = 0; l < 4 * G; ++l) {
        if (l >= first && l < first + size) continue;
        unsigned long long carry = 0;
        for (int t = 0; t < EX_WORDS; ++t) {
          const unsigned long long v = (unsigned long long)C.W[g][t] * kExModuli[l] + carry;
          C.W[g][t] = (unsigned)v;
          carry = v >> 32;
        }
      }
      unsigned long long bias = 0, fbias = 0;
      for (int i = 0; i < size; ++i) {
        const unsigned long long m = kExModuli[first + i], Q = P / m;
        unsigned long long w = 0;  // W_g mod m
        for (int t = EX_WORDS - 1; t >= 0; --t) w = ((w << 32) + C.W[g][t]) % m;
        const unsigned long long y = ex_inv(w, m) * ex_inv(Q % m, m) % m;
        C.c[first + i] = (unsigned)(Q * y);
        C.f[first + i] = (unsigned)((Q * y << 20) / P);
        bias += 128 * (Q * y);
        fbias += 128ull * C.f[first + i];
      }
      const unsigned long long b = (P - bias % P) % P;  // takes the 128s out of X again
      C.b[g] = (unsigned)(b + bias);
      C.fb[g] = (unsigned)((b << 20) / P + fbias);
    }
    unsigned M[EX_WORDS] = {1, 0, 0, 0, 0, 0, 0, 0};
    for (int l = 0; l < 4 * G; ++l) {
      unsigned long long carry = 0;
      for (int t = 0; t < EX_WORDS; ++t) {
        const unsigned long long v = (unsigned long long)M[t] * kExModuli[l] + carry;
        M[t] = (unsigned)v;
        carry = v >> 32;
      }
    }
    unsigned long long carry = 1;
    for (int t = 0; t < EX_WORDS; ++t) {
      carry += (unsigned)~M[t];
      C.Mneg[t] = (unsigned)carry;
      carry >>= 32;
    }
  }
  return T;
}

__constant__ ExTables kEx = make_tables();

struct ExLog2 {
  float v[EX_GROUPS + 1];  // log2 of the product of the first 4 G moduli, rounded down
};

// ------------------------------------------------------------------------------------------
// Device parameters and workspace
// ------------------------------------------------------------------------------------------
struct ExParams {
  unsigned status;
  int nmod;      // moduli of this call; 0: the DMMA route
  int ncA, ncH;  // 14-bit chunks of A' and H'
  unsigned run_dmma;
};

size_t al1k(size_t x) { return (x + 1023) & ~(size_t)1023; }

struct ExLayout {
  int kp, kr;
  size_t off_amax, off_asq, off_alsb, off_hmax, off_hsum, off_hsq, off_hlsb, off_ht, off_ra, off_rh, off_r, total;
};

ExLayout ex_layout(int M, int N, int K, int planes) {
  ExLayout L;
  L.kp = (K + 63) / 64 * 64;
  L.kr = (N + 255) / 256 * 256;
  size_t o = 1024;
  L.off_amax = o; o += al1k((size_t)M * 8);
  L.off_asq = o;  o += al1k((size_t)M * 8);
  L.off_alsb = o; o += al1k((size_t)M * 4);
  L.off_hmax = o; o += al1k((size_t)N * 8);
  L.off_hsum = o; o += al1k((size_t)N * 8);
  L.off_hsq = o;  o += al1k((size_t)N * 8);
  L.off_hlsb = o; o += al1k((size_t)N * 4);
  L.off_ht = o;   o += al1k((size_t)N * L.kp * 8);
  L.off_ra = o;   o += al1k((size_t)planes * M * L.kp * 2);
  L.off_rh = o;   o += al1k((size_t)planes * N * L.kp * 2);
  L.off_r = o;    o += al1k((size_t)planes * M * L.kr);
  L.total = o;
  return L;
}

// ------------------------------------------------------------------------------------------
// Passes
// ------------------------------------------------------------------------------------------
__global__ void k_ex_init(ExParams* prm, unsigned long long* amax, double* asq, int* alsb, int M) {
  grid_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *prm = ExParams{0u, 0, 0, 0, 1u};
  if (i < M) {
    amax[i] = 0ull;
    asq[i] = 0.0;
    alsb[i] = NO_LSB;
  }
}

__global__ void k_ex_row_stats(const double* __restrict__ A, long lda, int n, int k, int kchunk,
                               unsigned long long* __restrict__ amax, double* __restrict__ asq,
                               int* __restrict__ alsb) {
  grid_wait();
  row_absmax_blk<true>(A, lda, nullptr, 0, k, n, k, kchunk, amax, asq, blockIdx.x, blockIdx.y, alsb);
}

template <int KIND>
__global__ void k_ex_h(GenSpec gs, int K, int kp, double* __restrict__ Ht, unsigned long long* __restrict__ hmax,
                       double* __restrict__ hsum, double* __restrict__ hsq, int* __restrict__ hlsb) {
  grid_wait();
  h_pass1_blk<KIND, true>(gs, K, kp, Ht, hmax, hsum, hsq, nullptr, blockIdx.x, nullptr, hlsb);
}

// Both, for small operands: the first blocks SMALL_RB rows of A each, then a column of H each.
template <int KIND>
__global__ void __launch_bounds__(256) k_ex_stats(GenSpec gs, int M, int N, int K, int kp, const double* __restrict__ A,
                                                  long lda, unsigned long long* __restrict__ amax,
                                                  double* __restrict__ asq, int* __restrict__ alsb,
                                                  double* __restrict__ Ht, unsigned long long* __restrict__ hmax,
                                                  double* __restrict__ hsum, double* __restrict__ hsq,
                                                  int* __restrict__ hlsb) {
  grid_wait();
  const int rb = (M + SMALL_RB - 1) / SMALL_RB, b = blockIdx.x;
  if (b < rb)
    small_rows_blk<true>(A, lda, M, K, b, amax, asq, alsb);
  else
    h_pass1_blk<KIND, true>(gs, K, kp, Ht, hmax, hsum, hsq, nullptr, b - rb, nullptr, hlsb);
}

// An upper bound of log2 of the mantissa (in [1, 2)) of the normal double with bits b.
__device__ __forceinline__ float log2_mant_up(unsigned long long b) {
  const float f = __uint_as_float(0x3F800000u | ((unsigned)(b >> 29) & 0x7FFFFFu));
  return log2f(f) + 1e-5f;
}

// Number of moduli and chunk counts from the statistics.  With a'_i = row i of A' = A 2^-alsb_i and
// h'_j likewise, |Z_ij| <= max|a'| max sum|h'| and <= max ||a'||_2 max ||h'||_2; the CRT needs
// |Z| < 0.497 M.  Norms whose squares leave the range of FP64 count max * sqrt(k).
// One block; thread 0 returns them.
struct ExStats {
  const unsigned long long* amax;
  const double* asq;
  const int* alsb;
  const unsigned long long* hmax;
  const double *hsum, *hsq;
  const int* hlsb;
};
__device__ __forceinline__ ExParams ex_params(const ExStats& st, const ExLog2& lg, int max_groups, int M, int N, int K) {
  const unsigned long long *amax = st.amax, *hmax = st.hmax;
  const double *asq = st.asq, *hsum = st.hsum, *hsq = st.hsq;
  const int *alsb = st.alsb, *hlsb = st.hlsb;
  ExParams prm{0u, 0, 0, 0, 1u};
  float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // bits A, log2 max A, log2 ||A||, bits H, log2 sum H, log2 ||H||
  int bad = 0;
  const float lk = log2f((float)K) + 1e-3f;
  for (int r = threadIdx.x; r < M + N; r += blockDim.x) {
    const bool h = r >= M;
    const int i = h ? r - M : r;
    const unsigned long long b = h ? hmax[i] : amax[i];
    if (b == 0) continue;
    if (b >= INF_BITS) { bad = 1; continue; }
    const int lsb = h ? hlsb[i] : alsb[i], top = ilogb_bits(b);
    const float bits = (float)(top + 1 - lsb);
    const bool safe = top > -450 && top < 450;
    const unsigned long long q = (unsigned long long)__double_as_longlong(h ? hsq[i] : asq[i]);
    const int eq = (int)(q >> 52) - 1023;
    const float two = safe && q < INF_BITS && eq > -1000 && q != 0
                          ? 0.5f * ((float)(eq - 2 * lsb) + log2_mant_up(q)) + 0.01f
                          : bits + 0.5f * lk;
    float one = bits;
    if (h) {
      const unsigned long long sb = (unsigned long long)__double_as_longlong(hsum[i]);
      const int es = (int)(sb >> 52) - 1023;
      one = safe && sb < INF_BITS && sb != 0 ? (float)(es - lsb) + log2_mant_up(sb) + 0.01f : bits + lk;
    }
    const int o = h ? 3 : 0;
    v[o] = fmaxf(v[o], bits);
    v[o + 1] = fmaxf(v[o + 1], one);
    v[o + 2] = fmaxf(v[o + 2], two);
  }
  __shared__ float sv[32][6];
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int t = 0; t < 6; ++t) v[t] = fmaxf(v[t], __shfl_xor_sync(0xffffffffu, v[t], o));
  if ((threadIdx.x & 31) == 0)
    for (int t = 0; t < 6; ++t) sv[threadIdx.x >> 5][t] = v[t];
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)blockDim.x / 32; ++w)
      for (int t = 0; t < 6; ++t) v[t] = fmaxf(v[t], sv[w][t]);
    const float need = fminf(v[1] + v[4], v[2] + v[5]) + 1.05f;
    int g = 2;
    while (g <= max_groups && lg.v[g] < need) ++g;
    const bool fits = !bad && g <= max_groups && v[0] <= 14.f * EX_CHUNKS && v[3] <= 14.f * EX_CHUNKS;
    prm.ncA = ((int)v[0] + 13) / 14;
    prm.ncH = ((int)v[3] + 13) / 14;
    prm.nmod = fits ? 4 * g : 0;
    prm.run_dmma = fits ? 0u : 1u;
  }
  return prm;
}

__global__ void __launch_bounds__(1024) k_ex_params(ExParams* prm, ExLog2 lg, int max_groups, int M, int N, int K,
                                                    ExStats st) {
  grid_wait();
  const ExParams p = ex_params(st, lg, max_groups, M, N, K);
  if (threadIdx.x == 0) *prm = p;
}

// ------------------------------------------------------------------------------------------
// Residues.  x * 2^-lsb is cut into NC 14-bit chunks (exact floats, signed); with
// g_t = 2^(14 t) mod m symmetric, sum_t g_t c_t is congruent to it and below 2^14 (1 + 7 * 128) <
// 2^24, so the FMAs are exact; quotient and remainder as in split_crt.cu's residue_f (|r| <= 128).
// ------------------------------------------------------------------------------------------
template <int NC>
struct ExChunks {
  float c[NC];
};

template <int NC>
__device__ __forceinline__ ExChunks<NC> ex_chunks(double x, int lsb) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF);
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | (ex ? 1ull << 52 : 0ull);
  int sh = (ex ? ex : 1) - 1075 - lsb;  // >= -52: the bits shifted out are zero
  unsigned long long lo, hi = 0;
  if (sh <= 0) {
    lo = m == 0 ? 0 : m >> min(63, -sh);
  } else if (sh < 64) {
    lo = m << sh;
    hi = m >> (64 - sh);
  } else {
    lo = 0;
    hi = m << min(63, sh - 64);
  }
  const bool neg = (b >> 63) != 0;
  const float s = neg ? -1.0f : 1.0f, o = neg ? 8388608.0f : -8388608.0f;
  ExChunks<NC> r;
#pragma unroll
  for (int t = 0; t < NC; ++t) {
    const unsigned long long w = t < 4 ? lo >> (14 * t) : (t == 4 ? (lo >> 56) | (hi << 8) : hi >> (14 * t - 64));
    r.c[t] = fmaf(__uint_as_float(0x4B000000u | ((unsigned)w & 0x3FFFu)), s, o);
  }
  return r;
}

// Four neighbouring integers, moduli l0 .. l1 - 1: one 8-byte store per plane.
template <int NC>
__device__ __forceinline__ void ex_write_quad(const double (&x)[4], int lsb, bool ok, int l0, int l1, uint2* dst,
                                              size_t plane_u2) {
  ExChunks<NC> c[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) c[q] = ex_chunks<NC>(ok ? x[q] : 0.0, lsb);
  dst += (size_t)l0 * plane_u2;
#pragma unroll 4
  for (int l = l0; l < l1; ++l) {
    const float inv = kEx.g[l][0], mf = kEx.m[l];
    unsigned f[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float t = c[q].c[0];
#pragma unroll
      for (int e = 1; e < NC; ++e) t = fmaf(c[q].c[e], kEx.g[l][e], t);
      const float qq = fmaf(t, inv, 12582912.0f) - 12582912.0f;
      f[q] = __float_as_uint(fmaf(-qq, mf, t));
    }
    *dst = make_uint2(__byte_perm(f[0], f[1], 0x7632), __byte_perm(f[2], f[3], 0x7632));
    dst += plane_u2;
  }
}

__device__ __forceinline__ void ex_write_quad_nc(int nc, const double (&x)[4], int lsb, bool ok, int l0, int l1, uint2* dst,
                                                 size_t plane_u2) {
  if (nc <= 4)
    ex_write_quad<4>(x, lsb, ok, l0, l1, dst, plane_u2);
  else if (nc <= 6)
    ex_write_quad<6>(x, lsb, ok, l0, l1, dst, plane_u2);
  else
    ex_write_quad<8>(x, lsb, ok, l0, l1, dst, plane_u2);
}

// RA[l][i][kk], rows i, K-major: tiles of TR rows x 64 columns of A transposed through shared memory (element
// (k, r) at column (r + k/4) mod TR of row k: conflict-free both ways).  64 rows read whole 512-byte runs;
// 16 rows leave one quad a thread instead of a chain of four.
template <int TR>
__device__ __forceinline__ void ex_residues_A_blk(const double* __restrict__ A, long lda, int n, int k, int kp,
                                                  const int* __restrict__ alsb, int l0, int l1, int nc,
                                                  __nv_bfloat16* __restrict__ RA, int bx, int by) {
  __shared__ double tile[64][TR];
  constexpr int TX = TR < 32 ? TR : 32;
  const int i0 = bx * TR, k0 = by * 64;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  for (int kk = ty; kk < 64; kk += 256 / TX) {
    const int gk = k0 + kk;
#pragma unroll
    for (int rr = tx; rr < TR; rr += TX) {
      const int gi = i0 + rr;
      tile[kk][(rr + (kk >> 2)) & (TR - 1)] = (gi < n && gk < k) ? __ldg(A + gi + (long)gk * lda) : 0.0;
    }
  }
  __syncthreads();
  const size_t plane = (size_t)n * kp;
  const int tq = threadIdx.x & 15, tr = threadIdx.x >> 4;
  for (int r = tr; r < TR; r += 16) {
    const int gi = i0 + r;
    if (gi >= n) continue;
    const int lsb = alsb[gi], kk = 4 * tq;
    double x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = tile[kk + q][(r + tq) & (TR - 1)];
    ex_write_quad_nc(nc, x, lsb, lsb != NO_LSB, l0, l1, (uint2*)(RA + (size_t)gi * kp + k0 + kk), plane / 4);
  }
}

__global__ void __launch_bounds__(256) k_ex_residues_A(const double* __restrict__ A, long lda, int n, int k, int kp,
                                                       const int* __restrict__ alsb, const ExParams* prm,
                                                       __nv_bfloat16* __restrict__ RA) {
  grid_wait();
  const int nmod = prm->nmod;
  if (nmod == 0) return;
  ex_residues_A_blk<64>(A, lda, n, k, kp, alsb, 0, nmod, prm->ncA, RA, blockIdx.x, blockIdx.y);
}

// Entries kk .. kk + 3 of column j.
__device__ __forceinline__ void ex_residues_H_quad(const double* __restrict__ Ht, int ncols, int kp,
                                                   const int* __restrict__ hlsb, int l0, int l1, int nc,
                                                   __nv_bfloat16* __restrict__ RH, int j, int kk) {
  const int lsb = hlsb[j];
  const double2 h01 = *(const double2*)(Ht + (size_t)j * kp + kk);
  const double2 h23 = *(const double2*)(Ht + (size_t)j * kp + kk + 2);
  const double x[4] = {h01.x, h01.y, h23.x, h23.y};
  const size_t plane = (size_t)ncols * kp;
  ex_write_quad_nc(nc, x, lsb, lsb != NO_LSB, l0, l1, (uint2*)(RH + (size_t)j * kp + kk), plane / 4);
}

__global__ void __launch_bounds__(128) k_ex_residues_H(const double* __restrict__ Ht, int ncols, int kp,
                                                       const int* __restrict__ hlsb, const ExParams* prm,
                                                       __nv_bfloat16* __restrict__ RH) {
  grid_wait();
  const int nmod = prm->nmod;
  if (nmod == 0) return;
  const int j = blockIdx.x, kk = 4 * (blockIdx.y * blockDim.x + threadIdx.x);
  if (kk >= kp) return;  // kp is a multiple of 64
  ex_residues_H_quad(Ht, ncols, kp, hlsb, 0, nmod, prm->ncH, RH, j, kk);
}

// Both, for small operands: blocks 0 .. a_blocks - 1 are the tiles of A, the others 256 quads of H each.
// INLINE: every block evaluates the parameters, block 0 publishes them; these launches do not fill the SMs, and
// blockIdx.y takes half of the moduli (an integer's 28 to 32 residues are a serial chain): with that and tiles of 16 rows
// a call of n = 256 is some 3 us of 24 shorter.
template <bool INLINE, int TR>
__global__ void __launch_bounds__(256) k_ex_residues(const double* __restrict__ A, long lda, int M, int N, int K, int kp,
                                                     ExStats st, ExLog2 lg, int max_groups, int a_blocks,
                                                     const double* __restrict__ Ht, __nv_bfloat16* __restrict__ RA,
                                                     __nv_bfloat16* __restrict__ RH, ExParams* prm) {
  __shared__ ExParams sp;
  grid_wait();
  if (INLINE) {
    const ExParams p = ex_params(st, lg, max_groups, M, N, K);
    if (threadIdx.x == 0) {
      sp = p;
      if (blockIdx.x == 0 && blockIdx.y == 0) *prm = p;
    }
  } else if (threadIdx.x == 0) {
    sp = *prm;
  }
  __syncthreads();
  if (sp.nmod == 0) return;
  const int b = blockIdx.x, half = sp.nmod / 2;  // nmod is a multiple of four
  const int l0 = INLINE ? blockIdx.y * half : 0, l1 = INLINE ? l0 + half : sp.nmod;
  if (b < a_blocks) {
    const int tm = (M + TR - 1) / TR;
    ex_residues_A_blk<TR>(A, lda, M, K, kp, st.alsb, l0, l1, sp.ncA, RA, b % tm, b / tm);
  } else {
    const int q = (b - a_blocks) * 256 + threadIdx.x, per = kp / 4, j = q / per;
    if (j < N) ex_residues_H_quad(Ht, N, kp, st.hlsb, l0, l1, sp.ncH, RH, j, 4 * (q - j * per));
  }
}

// ------------------------------------------------------------------------------------------
// CRT
// ------------------------------------------------------------------------------------------
// (t3:t2) the 64 bits from the leading one, of exponent p + e, `rest` whether any bit is set below: results that are not
// normal, one rounding at their own precision (ldexp rounds a double exactly scaled; 53 bits would be
// rounded twice).
__device__ __noinline__ double ex_outside_normal(unsigned t3, unsigned t2, bool rest, bool neg, int field) {
  const unsigned long long top = ((unsigned long long)t3 << 32) | t2;
  if (field > 2045) {
    unsigned long long m = top >> 11;
    m += (top & 0x400ull) && ((top & 0x3FFull) != 0 || rest || (m & 1));
    const double v = ldexp((double)m, field - 1023 - 52);
    return neg ? -v : v;
  }
  const int drop = 1 - field + 11;  // bits of `top` below the subnormal's last place
  if (drop > 64) return neg ? -0.0 : 0.0;
  const unsigned long long keep = drop < 64 ? top >> drop : 0;
  const unsigned long long half = 1ull << (drop - 1);
  const bool st2 = (top & (half - 1)) != 0 || rest;
  unsigned long long bits = keep + (((top & half) && (st2 || (keep & 1))) ? 1 : 0);
  if (neg) bits |= 1ull << 63;
  return __longlong_as_double((long long)bits);
}

// The element of the 4 G residues r(l), times 2^e, rounded to nearest even.
// Instruction issue bounds it; sums that are the words of Z need no repacking (28-bit limbs of four-moduli parts: the
// Toeplitz multiply of n = 2048 14 us longer, 1024 3 us).
template <int G, class Residue>
__device__ __forceinline__ double ex_crt(Residue r, int e) {
  constexpr int NW = ex_words(G);
  const ExCrt& C = kEx.crt[G];
  unsigned long long acc[NW - 1];
  unsigned top = 0, qs = 1u << (ex_shift(G) - 33);
#pragma unroll
  for (int t = 0; t < NW - 1; ++t) acc[t] = 0;
#pragma unroll
  for (int g = 0; g < ex_parts(G); ++g) {
    unsigned t = C.b[g], f = C.fb[g];
#pragma unroll
    for (int i = 0; i < ex_size(G, g); ++i) {
      const unsigned u = (unsigned)r(ex_first(G, g) + i);
      t += u * C.c[ex_first(G, g) + i];
      f += u * C.f[ex_first(G, g) + i];
    }
    const unsigned X = t - (f >> 20) * C.P[g];  // in [0, 1.002 P_g)
    qs += __umulhi(X, C.G[g]);                  // X / P_g
#pragma unroll
    for (int s = 0; s < NW - 1; ++s) acc[s] += (unsigned long long)X * C.W[g][s];
    if (G < 7) top += X * C.W[g][NW - 1];  // 28 and 32 moduli: W_g < 2^192, 2^224
  }
  const unsigned q = qs >> (ex_shift(G) - 32);
  unsigned w[NW];
  unsigned long long carry = 0;
#pragma unroll
  for (int s = 0; s < NW - 1; ++s) {
    carry += acc[s] + (unsigned long long)q * C.Mneg[s];
    w[s] = (unsigned)carry;
    carry >>= 32;
  }
  w[NW - 1] = top + q * C.Mneg[NW - 1] + (unsigned)carry;
  const bool neg = (int)w[NW - 1] < 0;
  const unsigned sg = neg ? 0xFFFFFFFFu : 0u;
  carry = sg & 1u;
#pragma unroll
  for (int s = 0; s < NW; ++s) {
    carry += w[s] ^ sg;
    w[s] = (unsigned)carry;
    carry >>= 32;
  }
  // the three words from the leading nonzero one, and whether anything is below
  unsigned below[NW];
  below[0] = w[0];
#pragma unroll
  for (int s = 1; s < NW; ++s) below[s] = below[s - 1] | w[s];
  unsigned h = w[NW - 1], m = w[NW - 2], l = NW > 2 ? w[NW > 2 ? NW - 3 : 0] : 0, rest = NW > 3 ? below[NW > 3 ? NW - 4 : 0] : 0;
  int field = 32 * NW - 1 + e + 1023;
#pragma unroll
  for (int s = 1; s < NW; ++s)
    if (h == 0) {
      h = m;
      m = l;
      l = NW - 3 - s >= 0 ? w[NW - 3 - s >= 0 ? NW - 3 - s : 0] : 0;
      rest = NW - 4 - s >= 0 ? below[NW - 4 - s >= 0 ? NW - 4 - s : 0] : 0;
      field -= 32;
    }
  if (h == 0) return 0.0;
  const int s = __clz((int)h);
  field -= s;
  const unsigned t3 = __funnelshift_l(m, h, s), t2 = __funnelshift_l(l, m, s);
  rest = (rest | (l << s)) != 0 ? 1u : 0u;
  if (field < 1 || field > 2045) return ex_outside_normal(t3, t2, rest != 0, neg, field);
  const unsigned up = (((t2 & 0x7FFu) | rest) + 0x3FFu + ((t2 >> 11) & 1u)) >> 11;  // as i128_scaled
  const unsigned head = ((unsigned)(field - 1) << 20) + (t3 >> 11) + (neg ? 0x80000000u : 0u);
  return __longlong_as_double((long long)((((unsigned long long)head << 32) | ((t3 << 21) | (t2 >> 11))) + up));
}

// TI rows x 128 columns a block (32 x 8 threads), four neighbouring columns of a row per thread,
// transposed through shared memory as in crt_combine_blk.  TI = 32 writes whole 256-byte runs of
// Q's columns; smaller outputs take TI = 8, four times the blocks, each with a quarter of the serial
// recombinations.
template <int G, int TI>
__device__ __forceinline__ void ex_combine(const int8_t* __restrict__ R, int n, int k, int kr,
                                           const int* __restrict__ alsb, const int* __restrict__ hlsb, double alpha,
                                           double beta, double* __restrict__ Q, long ldq, double (&tile)[32][4 * TI + 1]) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i0 = blockIdx.y * TI, j0 = blockIdx.x * 128, jb = j0 + 4 * tx;
  const size_t plane = (size_t)n * kr;
  for (int a = 0; a < TI / 8; ++a) {
    const int il = ty + 8 * a, i = i0 + il;
    double val[4] = {0.0, 0.0, 0.0, 0.0};
    if (i < n && jb < k) {
      unsigned w[4 * G];
      const int8_t* rp = R + (size_t)i * kr + jb;
#pragma unroll
      for (int l = 0; l < 4 * G; ++l) w[l] = __ldg((const unsigned*)(rp + (size_t)l * plane));
      const int ea = alsb[i];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int eh = jb + c < k ? hlsb[jb + c] : NO_LSB;
        if (ea != NO_LSB && eh != NO_LSB)
          val[c] = ex_crt<G>([&](int l) { return (int)(int8_t)(w[l] >> (8 * c)); }, ea + eh);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) tile[tx][c * TI + il] = val[c];
  }
  __syncthreads();
  const bool scale = alpha != 1.0, accumulate = beta != 0.0;
  const int t = ty * 32 + tx, ir = t % TI, i = i0 + ir, left = i < n ? k - j0 : 0;
  double* qp = Q + i + (long)(j0 + t / TI) * ldq;
#pragma unroll
  for (int u0 = 0; u0 < TI / 2; u0 += 4) {
    double q[4];
    const double* ql = qp;
#pragma unroll
    for (int u = 0; u < 4; ++u, ql += ldq * (256 / TI)) q[u] = accumulate && t / TI + (u0 + u) * (256 / TI) < left ? *ql : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u, qp += ldq * (256 / TI)) {
      const int jl = t / TI + (u0 + u) * (256 / TI);
      if (jl < left) {
        double v = tile[jl >> 2][(jl & 3) * TI + ir];
        if (scale || accumulate) {
          v *= alpha;
          if (accumulate) v = fma(beta, q[u], v);
        }
        *qp = v;
      }
    }
  }
}

// One element a thread, 8 rows x 32 columns a block, for the smallest outputs: the four serial recombinations of a
// thread are most of the pass there.
template <int G>
__device__ __forceinline__ void ex_combine_one(const int8_t* __restrict__ R, int n, int k, int kr,
                                               const int* __restrict__ alsb, const int* __restrict__ hlsb, double alpha,
                                               double beta, double* __restrict__ Q, long ldq) {
  const int i = blockIdx.y * 8 + threadIdx.y, j = blockIdx.x * 32 + threadIdx.x;
  if (i >= n || j >= k) return;
  const size_t plane = (size_t)n * kr;
  const int8_t* rp = R + (size_t)i * kr + j;
  int8_t b[4 * G];
#pragma unroll
  for (int l = 0; l < 4 * G; ++l) b[l] = __ldg(rp + (size_t)l * plane);
  const int ea = alsb[i], eh = hlsb[j];
  double* qp = Q + i + (long)j * ldq;
  double v = 0.0;
  if (ea != NO_LSB && eh != NO_LSB) v = ex_crt<G>([&](int l) { return (int)b[l]; }, ea + eh);
  if (alpha != 1.0 || beta != 0.0) {
    v *= alpha;
    if (beta != 0.0) v = fma(beta, *qp, v);
  }
  *qp = v;
}

// TI = 1: ex_combine_one.
template <int TI>
__global__ void __launch_bounds__(256, 2) k_ex_combine(const int8_t* __restrict__ R, int n, int k, int kr, ExParams* prm,
                                                    const int* __restrict__ alsb, const int* __restrict__ hlsb,
                                                    double alpha, double beta, double* __restrict__ Q, long ldq) {
  __shared__ double tile[32][4 * TI + 1];
  grid_wait();
  const int nmod = prm->nmod;
  if (nmod == 0) return;
  if (prm->status != 0) {  // a wait of the GEMM gave up: the DMMA kernel computes the product
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) prm->run_dmma = 1u;
    return;
  }
  switch (nmod / 4) {
#define PSMMA_COMBINE(G)                                                       \
  case G:                                                                      \
    if constexpr (TI == 1)                                                     \
      ex_combine_one<G>(R, n, k, kr, alsb, hlsb, alpha, beta, Q, ldq);         \
    else                                                                       \
      ex_combine<G, TI>(R, n, k, kr, alsb, hlsb, alpha, beta, Q, ldq, tile);   \
    break;
    PSMMA_COMBINE(2)
    PSMMA_COMBINE(3)
    PSMMA_COMBINE(4)
    PSMMA_COMBINE(5)
    PSMMA_COMBINE(6)
    PSMMA_COMBINE(7)
    PSMMA_COMBINE(8)
#undef PSMMA_COMBINE
  }
}

ExLog2 ex_log2() {
  ExLog2 r;
  double l = 0.0;
  r.v[0] = r.v[1] = 0.0f;
  for (int i = 0; i < EX_MAX; ++i) {
    l += std::log2((double)kExModuli[i]);
    if (i % 4 == 3) r.v[(i + 1) / 4] = (float)(l - 1e-3);
  }
  return r;
}

constexpr size_t EX_WORK_CAP = (size_t)40 << 30;

// Planes the workspace cap allows (a multiple of 4, at most 32).
int ex_planes(int M, int N, int K) {
  int planes = EX_MAX;
  while (planes > 0 && ex_layout(M, N, K, planes).total > EX_WORK_CAP) planes -= 4;
  return planes;
}

}  // namespace

size_t exact_workspace(int M, int N, int K) {
  const int planes = ex_planes(M, N, K);
  return planes >= 16 ? ex_layout(M, N, K, planes).total : 0;
}

// Whether the route is faster than the DMMA kernel, whose time is that of whole 128 x 128 x 16 tile steps, some 75 us each
// (2 FP64 FMAs per SM and cycle): one wave of them costs more than the route's passes at every size (Toeplitz n = 32: 166
// us against 22; n = 256: 610 / 24; n = 2048: 16.0 ms / 0.354; n = 4096: 129 / 1.83) but where H has two steps of rows and A
// so many rows that its passes, whose planes hold 64 columns of A and 256 of Q whatever K and N are, take longer
// (500000 x 5: 3.9 ms against 2.0; 50000 x 5 0.42 / 0.24, 5000 x 5 0.069 / 0.083; 19456 x 32 0.180 / 0.156, 150000 x 32
// 1.20 / 1.22).  Sizes are those the passes' grids cover.
bool exact_route(int M, int N, int K, int sms) {
  if (K >= (1 << 21) || M > 8 * 65535 || N > 8 * 65535) return false;
  if (K > 32 || N > 128) return true;
  const int waves = ((M + 127) / 128 + sms - 1) / sms;
  return 30.0 + 0.0078 * M < waves * (6.0 + 72.0 * ((K + 15) / 16));
}

// Enqueues the exact route of Q (M x N) = alpha A (M x K) H (K x N) + beta Q; *gate receives the
// device word that tells the DMMA kernel behind it to run.
int launch_exact(int M, int N, int K, double alpha, const double* A, long lda, const GenSpec& gs, double beta,
                 double* Q, long ldq, void* work, size_t lwork, cudaStream_t stream, const unsigned** gate) {
  const int planes = ex_planes(M, N, K);
  const ExLayout L = ex_layout(M, N, K, planes);
  if (planes < 16 || !work || lwork < L.total) return PSMMA_EWORKSPACE;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return PSMMA_EDEVICE;
  static const ExLog2 lg = ex_log2();
  char* w = (char*)work;
  ExParams* prm = (ExParams*)w;
  auto* amax = (unsigned long long*)(w + L.off_amax);
  auto* hmax = (unsigned long long*)(w + L.off_hmax);
  double *asq = (double*)(w + L.off_asq), *hsum = (double*)(w + L.off_hsum), *hsq = (double*)(w + L.off_hsq);
  int *alsb = (int*)(w + L.off_alsb), *hlsb = (int*)(w + L.off_hlsb);
  double* Ht = (double*)(w + L.off_ht);
  auto* RA = (__nv_bfloat16*)(w + L.off_ra);
  auto* RH = (__nv_bfloat16*)(w + L.off_rh);
  int8_t* R = (int8_t*)(w + L.off_r);
  *gate = &prm->run_dmma;

  const ExStats xs{amax, asq, alsb, hmax, hsum, hsq, hlsb};
  prof_begin(stream);
  if (small_operands(M, N, K)) {
    const int blocks = N + (M + SMALL_RB - 1) / SMALL_RB;
    switch (gs.kind) {
#define PSMMA_STATS(KD) \
  case KD: k_ex_stats<KD><<<blocks, 256, 0, stream>>>(gs, M, N, K, L.kp, A, lda, amax, asq, alsb, Ht, hmax, hsum, hsq, hlsb); break;
      PSMMA_STATS(KIND_CAUCHY)
      PSMMA_STATS(KIND_TOEPLITZ)
      PSMMA_STATS(KIND_HANKEL)
      PSMMA_STATS(KIND_CAUCHY_EIG)
#undef PSMMA_STATS
      default: return PSMMA_EUNSUPPORTED;
    }
    prof_mark(stream, "statistics");
    const int tr = small_tile_rows(M, N), a_blocks = ((M + tr - 1) / tr) * (L.kp / 64), h_blocks = (N * (L.kp / 4) + 255) / 256;
    if (M + N <= INLINE_ROWS) {
      launch_behind(true, k_ex_residues<true, 16>, dim3(a_blocks + h_blocks, 2), 256, 0, stream, A, lda, M, N, K, L.kp, xs, lg, planes / 4,
                    a_blocks, Ht, RA, RH, prm);
    } else {
      launch_behind(true, k_ex_params, 1, 1024, 0, stream, prm, lg, planes / 4, M, N, K, xs);
      launch_behind(true, tr == 16 ? k_ex_residues<false, 16> : k_ex_residues<false, 64>, a_blocks + h_blocks, 256, 0, stream, A, lda, M, N, K, L.kp, xs, lg, planes / 4,
                    a_blocks, Ht, RA, RH, prm);
    }
    prof_mark(stream, "residues");
  } else {
    k_ex_init<<<(M + 255) / 256, 256, 0, stream>>>(prm, amax, asq, alsb, M);
    // enough blocks for some eight waves, so that the loads of a chunk (eight in flight a thread) are
    // not a serial chain: the Toeplitz multiply of n = 3072 at 1024-column chunks 1052 us, so 900
    int kchunk = 1024;
    while (kchunk > 16 && (long)((M + 127) / 128) * ((K + kchunk - 1) / kchunk) < 8L * sms) kchunk >>= 1;
    launch_behind(true, k_ex_row_stats, dim3((M + 127) / 128, (K + kchunk - 1) / kchunk), 128, 0, stream, A, lda, M, K, kchunk,
                  amax, asq, alsb);
    prof_mark(stream, "row_scale");
    switch (gs.kind) {
#define PSMMA_H(KD) \
  case KD: launch_behind(true, k_ex_h<KD>, N, 256, 0, stream, gs, K, L.kp, Ht, hmax, hsum, hsq, hlsb); break;
      PSMMA_H(KIND_CAUCHY)
      PSMMA_H(KIND_TOEPLITZ)
      PSMMA_H(KIND_HANKEL)
      PSMMA_H(KIND_CAUCHY_EIG)
#undef PSMMA_H
      default: return PSMMA_EUNSUPPORTED;
    }
    prof_mark(stream, "h_generate");
    launch_behind(true, k_ex_params, 1, 1024, 0, stream, prm, lg, planes / 4, M, N, K, xs);
    prof_mark(stream, "params");
    launch_behind(true, k_ex_residues_A, dim3((M + 63) / 64, L.kp / 64), 256, 0, stream, A, lda, M, K, L.kp, alsb, prm, RA);
    prof_mark(stream, "residues_A");
    launch_behind(true, k_ex_residues_H, dim3(N, (L.kp / 4 + 127) / 128), 128, 0, stream, Ht, N, L.kp, hlsb, prm, RH);
    prof_mark(stream, "residues_H");
  }
  // the whole chain overlaps its launches: the route is never captured
  const int st = launch_modular_gemm(RA, RH, R, M, N, L.kp, L.kr, planes, kExModuli, &prm->nmod, &prm->status, sms, stream);
  if (st) return st;
  prof_mark(stream, "modular_gemm");
  const int cols = (N + 127) / 128;
  if ((long)cols * ((M + 7) / 8) < 2L * sms)
    launch_behind(true, k_ex_combine<1>, dim3((N + 31) / 32, (M + 7) / 8), dim3(32, 8), 0, stream, R, M, N, L.kr, prm, alsb, hlsb,
                  alpha, beta, Q, ldq);
  else if ((long)cols * ((M + 31) / 32) >= 4L * sms)
    launch_behind(true, k_ex_combine<32>, dim3(cols, (M + 31) / 32), dim3(32, 8), 0, stream, R, M, N, L.kr, prm, alsb, hlsb,
                  alpha, beta, Q, ldq);
  else
    launch_behind(true, k_ex_combine<8>, dim3(cols, (M + 7) / 8), dim3(32, 8), 0, stream, R, M, N, L.kr, prm, alsb, hlsb, alpha,
                  beta, Q, ldq);
  prof_mark(stream, "crt_combine");
  return cudaGetLastError() == cudaSuccess ? PSMMA_OK : PSMMA_EDEVICE;
}

}  // namespace psmma
