// The Toeplitz and Hankel multiplies of the split precision by number-theoretic transforms.
//
// Row r of A H is a convolution of row r of A (reversed for Hankel) with the generator, its outputs
// k - 1 .. 2 k - 2.  The modular GEMMs of split_crt.cu form the integer product Z = A'H' of the
// scaled operands in 3^L n (k / 2^L)^2 multiply-adds per modulus; here the same integer Z comes from
// cyclic convolutions of length L = 2^m >= 2 k - 1 modulo four (or five) primes below 2^30, in
// n L log2 L butterflies per prime, and the Chinese remainder theorem.  All arithmetic is exact, so
// Q is the GEMM path's bit for bit where that path scales every column alike.
//
// Scaling: row i of A to PA bits as in split_crt.cu; the generator by one power of two, the finest that
// any column would take (a column whose largest entry is 2^s below the generator's keeps its PH bits,
// the others carry up to s more).  The primes' product exceeds that of the caller's moduli by the bits
// this needs (9 for the default 14 moduli, 17 for 13); a generator of wider columns, or one that is not
// finite, is left to the GEMM path, enqueued behind this one and gated on the device.
//
// Transform of X^L - 1 by recursive splitting, (X^(N/2) - z)(X^(N/2) + z): butterflies (u + z v, u - z v)
// whose z depends on the block alone, sixteen points a thread and pass (four levels between two
// exchanges through shared memory), products by Shoup's method (z and floor(2^32 z / p): three 32-bit
// multiplications), values kept below 4 p < 2^32.  The last levels, the product with the generator's
// transform and the first inverse levels stay in registers.  ncu at L = 2^14: the 32-bit multiply pipe
// 73 % busy (81 issue slots a point of 58 the butterflies need), issue 68 %, DRAM 5 %.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "psmma_internal.h"
#include "split_passes.cuh"

namespace psmma {
namespace {

typedef unsigned u32;
typedef unsigned long long u64;

constexpr int NT_MAXP = 5;
constexpr u32 kPrimes[NT_MAXP] = {1073479681u, 1072496641u, 1071513601u, 1070727169u, 1068564481u};  // 1 mod 2^16
constexpr u32 kGens[NT_MAXP] = {11, 11, 23, 11, 7};  // primitive roots
constexpr int NT_MIN_LOG = 13, NT_MAX_LOG = 15;  // shorter: the GEMMs are faster; 2^15: 128 KB of shared memory

constexpr u32 mulp(u64 a, u64 b, u32 p) { return (u32)(a * b % p); }
constexpr u32 powp(u64 a, u64 e, u32 p) {
  u64 r = 1;
  for (a %= p; e; e >>= 1, a = a * a % p)
    if (e & 1) r = r * a % p;
  return (u32)r;
}
constexpr u32 shoup(u32 w, u32 p) { return (u32)(((u64)w << 32) / p); }

// Constants of the transforms of length 2^lg: per prime the powers w^(2^i) of a primitive L-th root and
// of its inverse, and the factor folded into the generator's transform: 1 / L and the CRT's
// (M / p)^-1 mod p.
struct NttConsts {
  int np, lg;
  u32 p[NT_MAXP];
  uint2 two32[NT_MAXP];                 // 2^32 mod p
  uint2 w[NT_MAXP][16], wi[NT_MAXP][16];
  uint2 fold[NT_MAXP];
  u64 inv64[NT_MAXP];                   // floor(2^64 / p)
  // CRT: Z = sum_q X_q W_q - q M, W_q = M / p_q, limbs of 32 bits; G = floor(2^52 / p)
  u32 W[NT_MAXP][NT_MAXP], Mneg[4], G[NT_MAXP];
};

NttConsts make_ntt(int np, int lg) {
  NttConsts c;
  memset(&c, 0, sizeof(c));
  c.np = np;
  c.lg = lg;
  for (int q = 0; q < np; ++q) {
    const u32 p = kPrimes[q];
    c.p[q] = p;
    const u32 t = (u32)((1ull << 32) % p);
    c.two32[q] = make_uint2(t, shoup(t, p));
    u32 w = powp(kGens[q], (p - 1) >> lg, p), wi = powp(w, p - 2, p);
    for (int i = 0; i < 16; ++i) {
      c.w[q][i] = make_uint2(w, shoup(w, p));
      c.wi[q][i] = make_uint2(wi, shoup(wi, p));
      w = mulp(w, w, p);
      wi = mulp(wi, wi, p);
    }
    u64 other = 1;  // M / p mod p
    for (int r = 0; r < np; ++r)
      if (r != q) other = other * (kPrimes[r] % p) % p;
    const u32 f = mulp(powp(other, p - 2, p), powp(powp(2, (u64)lg, p), p - 2, p), p);
    c.fold[q] = make_uint2(f, shoup(f, p));
    c.inv64[q] = ~0ull / p;  // p is odd: floor((2^64 - 1) / p) = floor(2^64 / p)
    c.G[q] = (u32)((1ull << 52) / p);
    for (int r = -1; r < 1; ++r) {  // W_q and (once) M as products in 32-bit limbs
      u32 limb[NT_MAXP] = {1, 0, 0, 0, 0};
      for (int s = 0; s < np; ++s) {
        if (r < 0 && s == q) continue;
        u64 carry = 0;
        for (int l = 0; l < NT_MAXP; ++l) {
          const u64 v = (u64)limb[l] * kPrimes[s] + carry;
          limb[l] = (u32)v;
          carry = v >> 32;
        }
      }
      if (r < 0) {
        memcpy(c.W[q], limb, sizeof(limb));
      } else {  // 2^128 - M (mod 2^128)
        u64 carry = 1;
        for (int l = 0; l < 4; ++l) {
          carry += (u32)~limb[l];
          c.Mneg[l] = (u32)carry;
          carry >>= 32;
        }
      }
    }
  }
  return c;
}

double ntt_log2(int np) {
  double l = 0.0;
  for (int q = 0; q < np; ++q) l += std::log2((double)kPrimes[q]);
  return l - 1e-6;
}

// ------------------------------------------------------------------------------------------
// Workspace: inside the split path's (its A and H residue planes and outputs, which only the gated
// fallback writes), the flag words in the part the fallback does not clear.
// ------------------------------------------------------------------------------------------
struct NttParams {
  u32 fallback;      // read by the gated kernels
  int emin, emax;    // exponents of the smallest and largest nonzero column maxima
  u32 bad;           // the generator holds a NaN or an infinity
};

__device__ __forceinline__ bool ntt_ok(const NttParams* t, const SplitDevParams* prm, int slack) {
  return t->bad == 0u && t->emax - t->emin <= slack && prm->PH + (t->emax - t->emin) <= 62;
}
// The generator's exponent: entries times 2^gen_exp are rounded to integers.
__device__ __forceinline__ int gen_exp(const NttParams* t, const SplitDevParams* prm) {
  return prm->PH - 1 - t->emin;
}

// ------------------------------------------------------------------------------------------
// Column statistics.  Column j of either matrix holds the generator's entries j .. j + k - 1 (in one
// order or the other): a suffix of the first k entries and a prefix of the last k - 1.  Maxima, and
// sums of |g| and g^2 in FP32 rounded up on the scale of the largest entry, as in h_pass1_blk.
// ------------------------------------------------------------------------------------------
struct Stat {
  u64 m;
  float s, q;
};
__device__ __forceinline__ Stat join(Stat a, Stat b) {
  return {a.m > b.m ? a.m : b.m, __fadd_ru(a.s, b.s), __fadd_ru(a.q, b.q)};
}
__device__ __forceinline__ Stat shfl_up(Stat a, int o) {
  return {__shfl_up_sync(0xffffffffu, a.m, o), __shfl_up_sync(0xffffffffu, a.s, o), __shfl_up_sync(0xffffffffu, a.q, o)};
}

__global__ void __launch_bounds__(1024) k_ntt_colstats(const double* __restrict__ g, int k, u64* __restrict__ hmax,
                                                       double* __restrict__ hsq, SplitDevParams* prm, NttParams* t) {
  __shared__ u64 gm[32];
  __shared__ Stat ws[2][32];
  __shared__ u64 s_all;
  __shared__ int s_min, s_max;
  __shared__ float s_rho;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  u64 m = 0;
  for (int i = tid; i < 2 * k - 1; i += 1024) {
    const u64 b = (u64)__double_as_longlong(__ldg(g + i)) & ABS_MASK;
    m = b > m ? b : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const u64 x = __shfl_xor_sync(0xffffffffu, m, o);
    m = x > m ? x : m;
  }
  if (lane == 0) gm[wid] = m;
  if (tid == 0) { s_min = 0x7FFFFFFF; s_max = -0x7FFFFFFF; s_rho = 0.0f; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 32; ++w) m = gm[w] > m ? gm[w] : m;
    s_all = m;
  }
  __syncthreads();
  const u64 all = s_all;
  const int e0 = (int)(all >> 52) - 1023;
  // thread tid: entries [tid c, (tid + 1) c) of the reversed first part (suffixes become prefixes), and
  // of the second part shifted by one (column j takes k .. k + j - 1)
  const int c = (k + 1023) / 1024;
  auto entry = [&](int part, int i) -> Stat {  // i in [0, k)
    const int idx = part == 0 ? k - 1 - i : k - 1 + i;
    if (i >= k || (part == 1 && i == 0)) return {0ull, 0.0f, 0.0f};
    const u64 b = (u64)__double_as_longlong(__ldg(g + idx)) & ABS_MASK;
    bool big = false;
    const float f = abs_scaled_up(b, e0, &big);
    return {b, f, __fmul_ru(f, f)};
  };
  Stat pre[2];
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    Stat a{0ull, 0.0f, 0.0f};
    for (int i = tid * c; i < min(k, (tid + 1) * c); ++i) a = join(a, entry(part, i));
    Stat inc = a;
    for (int o = 1; o < 32; o <<= 1) {
      const Stat x = shfl_up(inc, o);
      if (lane >= o) inc = join(x, inc);
    }
    if (lane == 31) ws[part][wid] = inc;
    Stat ex = shfl_up(inc, 1);
    pre[part] = lane == 0 ? Stat{0ull, 0.0f, 0.0f} : ex;
  }
  __syncthreads();
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    Stat b{0ull, 0.0f, 0.0f};
    for (int w = 0; w < wid; ++w) b = join(b, ws[part][w]);
    pre[part] = join(b, pre[part]);
  }
  // the suffix of column j covers reversed entries 0 .. k - 1 - j; store it, then join the prefix
  for (int i = tid * c; i < min(k, (tid + 1) * c); ++i) {
    pre[0] = join(pre[0], entry(0, i));
    const int j = k - 1 - i;
    hmax[j] = pre[0].m;
    hsq[j] = __hiloint2double(__float_as_int(pre[0].s), __float_as_int(pre[0].q));
  }
  __syncthreads();
  int emin = 0x7FFFFFFF, emax = -0x7FFFFFFF;
  float rho = 0.0f;
  for (int i = tid * c; i < min(k, (tid + 1) * c); ++i) {
    pre[1] = join(pre[1], entry(1, i));
    const u64 b = hmax[i];
    const double sq = hsq[i];
    const Stat s = join(Stat{b, __int_as_float(__double2hiint(sq)), __int_as_float(__double2loint(sq))}, pre[1]);
    hmax[i] = s.m;
    hsq[i] = ldexp((double)s.q, 2 * e0);
    if (s.m != 0) {
      const int e = ilogb_bits(s.m);
      emin = min(emin, e);
      emax = max(emax, e);
      bool big = false;
      rho = fmaxf(rho, __fdiv_ru(s.s, abs_scaled_up(s.m, e0, &big)) * 1.000001f);
    }
  }
  atomicMin(&s_min, emin);
  atomicMax(&s_max, emax);
  atomicMax((int*)&s_rho, __float_as_int(rho));
  __syncthreads();
  if (tid == 0) {
    t->emin = s_min == 0x7FFFFFFF ? 0 : s_min;
    t->emax = s_min == 0x7FFFFFFF ? 0 : s_max;
    t->bad = all >= INF_BITS ? 1u : 0u;
    t->fallback = 0u;
    prm->rho_bits = (u64)__double_as_longlong((double)s_rho);
  }
}

// ------------------------------------------------------------------------------------------
// A' as 64-bit integers, row-major (reversed within the row for Hankel), zero rows for rows that are
// zero or not finite; block (0, 0) also publishes the fallback flag.
// ------------------------------------------------------------------------------------------
template <bool REV>
__global__ void __launch_bounds__(256) k_ntt_scale(const double* __restrict__ A, long lda, int n, int k, int kp,
                                                   const u64* __restrict__ amax, const SplitDevParams* prm, NttParams* t,
                                                   int slack, long long* __restrict__ Ai) {
  __shared__ double tile[64][65];
  const bool ok = ntt_ok(t, prm, slack);
  if (!ok) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) t->fallback = 1u;
    return;
  }
  const int i0 = blockIdx.x * 64, k0 = blockIdx.y * 64;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  for (int kk = ty; kk < 64; kk += 4) {
    const int gi = i0 + tx, gk = k0 + kk;
    tile[kk][tx] = (gi < n && gk < k) ? __ldg(A + gi + (long)gk * lda) : 0.0;
  }
  __syncthreads();
  const int PA = prm->PA;
  for (int r = ty; r < 64; r += 4) {
    const int gi = i0 + r, gk = k0 + tx;
    if (gi >= n || gk >= k) continue;
    const u64 ab = amax[gi];
    long long v = 0;
    if (ab > 0 && ab < INF_BITS) {
      bool neg;
      v = (long long)scaled_int(tile[tx][r], scale_exp(ab, PA), &neg);
      if (neg) v = -v;
    }
    Ai[(size_t)gi * kp + (REV ? k - 1 - gk : gk)] = v;
  }
}

// ------------------------------------------------------------------------------------------
// Modular arithmetic
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ u32 smul(u32 x, uint2 w, u32 p) { return x * w.x - __umulhi(x, w.y) * p; }  // [0, 2p)
__device__ __forceinline__ u32 red(u32 x, u32 p) { return min(x, x - p); }  // one conditional subtraction

// A signed 63-bit integer modulo p, in [0, 2p].
__device__ __forceinline__ u32 mod_i64(long long v, uint2 t32, u32 p) {
  const u64 a = (u64)(v < 0 ? -v : v);
  const u32 lo = red(red((u32)a, 2 * p), 2 * p);       // 2^32 < 4 p + 2 p
  const u32 r = red(smul((u32)(a >> 32), t32, p) + lo, 2 * p);  // [0, 2p)
  return v < 0 ? 2 * p - r : r;
}

// Twiddle table of a prime.  Block b of level s has z = w^(L brv_s(b) / 2^(s+1)).  A pass that starts at
// level 4 ps on blocks b < 16^ps uses, at its level l, blocks (b << l) + i, i < 2^l: that entry stands at
// (f << 4 ps) + b with f = 2^l + i (1 <= f < 16, in the last levels' pass < 2^LB), so that threads of
// neighbouring blocks read neighbouring entries.
__device__ __forceinline__ uint2 table_entry(u32 idx, int np16, int lg, const uint2* pw, u32 p, u64 inv64) {
  int ps = 0;
  while (ps < np16 && (idx >> (4 * ps + 4)) != 0) ++ps;
  const u32 f = idx >> (4 * ps), blk = idx & ((1u << (4 * ps)) - 1);
  const int l = 31 - __clz((int)f), s = 4 * ps + l;
  const u32 b = (blk << l) + (f - (1u << l));
  // exponent bits: brv_s(b) << (lg - s - 1); bit i of b is exponent bit lg - 2 - i
  u32 x = 1;
  for (int i = 0; i < s; ++i)
    if ((b >> i) & 1) x = smul(x, pw[lg - 2 - i], p);
  x = red(x, p);
  const u64 y = (u64)x << 32;
  u64 q = __umul64hi(y, inv64);
  if (y - q * p >= p) ++q;
  return make_uint2(x, (u32)q);
}

__global__ void k_ntt_tables(const __grid_constant__ NttConsts c, int np16, uint2* __restrict__ tab) {
  const int L = 1 << c.lg, q = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * L; i += gridDim.x * blockDim.x) {
    const int idx = i & (L - 1);
    if (idx == 0) continue;
    tab[(size_t)q * 2 * L + i] =
        table_entry((u32)idx, np16, c.lg, i < L ? c.w[q] : c.wi[q], c.p[q], c.inv64[q]);
  }
}

// ------------------------------------------------------------------------------------------
// Passes over a transform in shared memory.  L = 16^NP 2^LB: NP passes of four levels, then LB levels.
// ------------------------------------------------------------------------------------------
// Bits 4 + LB .. 8 of an index XORed onto bits LB .. 4 and bits 5 .. 4 + LB onto bits 0 .. LB - 1: the 32
// threads of a warp hit 32 banks at the strides of every pass and at stride 2^LB (the last levels).
template <int LB>
__device__ __forceinline__ int sw(int p) {
  return p ^ (((p >> (4 + LB)) & ((1 << (5 - LB)) - 1)) << LB) ^ ((p >> 5) & ((1 << LB) - 1));
}

// Levels l0 .. 3 of a sixteen-point group of the pass that starts at level s4 = 4 ps; tab points at the
// entry of the group's block.
__device__ __forceinline__ void fwd16(u32 (&x)[16], const uint2* __restrict__ tab, int s4, u32 p, int l0) {
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    if (l < l0) continue;
    const int h = 8 >> l;
#pragma unroll
    for (int i = 0; i < (1 << l); ++i) {
      const uint2 w = __ldg(tab + (((1 << l) + i) << s4));
#pragma unroll
      for (int j = 0; j < h; ++j) {
        u32 &u = x[2 * h * i + j], &v = x[2 * h * i + j + h];
        const u32 a = red(u, 2 * p), t = smul(v, w, p);
        u = a + t;
        v = a - t + 2 * p;
      }
    }
  }
}
__device__ __forceinline__ void inv16(u32 (&x)[16], const uint2* __restrict__ tab, int s4, u32 p, int l0) {
#pragma unroll
  for (int l = 3; l >= 0; --l) {
    if (l < l0) continue;
    const int h = 8 >> l;
#pragma unroll
    for (int i = 0; i < (1 << l); ++i) {
      const uint2 w = __ldg(tab + (((1 << l) + i) << s4));
#pragma unroll
      for (int j = 0; j < h; ++j) {
        u32 &u = x[2 * h * i + j], &v = x[2 * h * i + j + h];
        const u32 a = u, b = v;
        u = red(a + b, 2 * p);
        v = smul(a - b + 2 * p, w, p);
      }
    }
  }
}

// Passes P0 .. NP - 1.  Unrolled, so that shared addresses are an XOR with a constant and the table's
// entries stand at constant offsets from the block's.
template <int LB, int NP, int P0>
__device__ __forceinline__ void fwd_mid(u32* s, const uint2* __restrict__ tab, u32 p) {
  constexpr int LG = 4 * NP + LB;
#pragma unroll
  for (int ps = P0; ps < NP; ++ps) {
    const int lm = LG - 4 * ps - 4;  // log2 of the points' stride M
    for (int u = threadIdx.x; u < (1 << (LG - 4)); u += blockDim.x) {
      const int b = u >> lm, m = u & ((1 << lm) - 1);
      const int a = sw<LB>((b << (lm + 4)) + m);
      u32 x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = s[a ^ sw<LB>(r << lm)];
      fwd16(x, tab + b, 4 * ps, p, 0);
#pragma unroll
      for (int r = 0; r < 16; ++r) s[a ^ sw<LB>(r << lm)] = x[r];
    }
    __syncthreads();
  }
}

// The last LB levels of a contiguous group of R = 2^LB points, forward.
template <int R>
__device__ __forceinline__ void fwd_last(u32 (&x)[R], const uint2* __restrict__ tab, int s4, u32 p) {
#pragma unroll
  for (int l = 0; (1 << l) < R; ++l) {
    const int h = R >> (l + 1);
#pragma unroll
    for (int i = 0; i < (1 << l); ++i) {
      const uint2 w = __ldg(tab + (((1 << l) + i) << s4));
#pragma unroll
      for (int j = 0; j < h; ++j) {
        u32 &u = x[2 * h * i + j], &v = x[2 * h * i + j + h];
        const u32 a = red(u, 2 * p), t = smul(v, w, p);
        u = a + t;
        v = a - t + 2 * p;
      }
    }
  }
}
template <int R>
__device__ __forceinline__ void inv_first(u32 (&x)[R], const uint2* __restrict__ tab, int s4, u32 p) {
#pragma unroll
  for (int h = 1; h < R; h <<= 1) {
    const int blocks = R / (2 * h);
#pragma unroll
    for (int i = 0; i < blocks; ++i) {
      const uint2 w = __ldg(tab + ((blocks + i) << s4));
#pragma unroll
      for (int j = 0; j < h; ++j) {
        u32 &u = x[2 * h * i + j], &v = x[2 * h * i + j + h];
        const u32 a = u, b = v;
        u = red(a + b, 2 * p);
        v = smul(a - b + 2 * p, w, p);
      }
    }
  }
}

// The generator's transform times 1 / L and the CRT's factor, with Shoup quotients: place r of group u of
// the last levels at ghat[q][r L / 2^LB + u].
template <int LB, int NP>
__global__ void __launch_bounds__(512) k_ntt_gen(const __grid_constant__ NttConsts c, const double* __restrict__ g, int k,
                                                 const SplitDevParams* prm, const NttParams* t, int slack,
                                                 const uint2* __restrict__ tab, uint2* __restrict__ ghat) {
  extern __shared__ u32 ntt_smem[];
  constexpr int LG = 4 * NP + LB, L = 1 << LG, R = 1 << LB;
  if (!ntt_ok(t, prm, slack)) return;
  const int q = blockIdx.x;
  const u32 p = c.p[q];
  const uint2* tb = tab + (size_t)q * 2 * L;
  const int e = gen_exp(t, prm);
  const int rot = L / 2 - (k - 1);  // output k - 1 of the convolution to L / 2
  for (int i = threadIdx.x; i < L; i += blockDim.x) {
    u32 x = 0;
    const int src = (i - rot) & (L - 1);
    if (src < 2 * k - 1) {
      bool neg;
      long long v = (long long)scaled_int(__ldg(g + src), e, &neg);
      x = mod_i64(neg ? -v : v, c.two32[q], p);
    }
    ntt_smem[sw<LB>(i)] = x;
  }
  __syncthreads();
  fwd_mid<LB, NP, 0>(ntt_smem, tb, p);
  for (int u = threadIdx.x; u < (L >> LB); u += blockDim.x) {
    u32 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = ntt_smem[sw<LB>((u << LB) + r)];
    fwd_last<R>(x, tb + u, 4 * NP, p);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const u32 y = red(smul(x[r], c.fold[q], p), p);
      const u64 z = (u64)y << 32;
      u64 d = __umul64hi(z, c.inv64[q]);
      if (z - d * p >= p) ++d;
      ghat[(size_t)q * L + r * (L >> LB) + u] = make_uint2(y, (u32)d);
    }
  }
}

// Row blockIdx.x / np of A', prime blockIdx.x % np: out[q][row][j] = (Z_(row, j) (M/p)^-1) mod p.
template <int LB, int NP>
__global__ void __launch_bounds__(512, 2) k_ntt_rows(const __grid_constant__ NttConsts c, int n, int k, int kp, int kr,
                                                     const SplitDevParams* prm, const NttParams* t, int slack,
                                                     const uint2* __restrict__ tab, const uint2* __restrict__ ghat,
                                                     const long long* __restrict__ Ai, u32* __restrict__ out) {
  extern __shared__ u32 ntt_smem[];
  constexpr int LG = 4 * NP + LB, L = 1 << LG, R = 1 << LB, M1 = L / 16;
  if (!ntt_ok(t, prm, slack)) return;
  const int row = blockIdx.x / c.np, q = blockIdx.x - row * c.np;
  const u32 p = c.p[q];
  const uint2 t32 = c.two32[q];
  const uint2* tf = tab + (size_t)q * 2 * L;
  const uint2* ti = tf + L;
  u32* s = ntt_smem;
  // first pass: the row fills the lower half (2 k - 1 <= L), so the first level copies it
  const long long* src = Ai + (size_t)row * kp;
  for (int m = threadIdx.x; m < M1; m += blockDim.x) {
    u32 x[16];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = m + r * M1;
      x[r] = i < k ? mod_i64(__ldg(src + i), t32, p) : 0u;
      x[r + 8] = x[r];
    }
    fwd16(x, tf, 0, p, 1);
    const int a = sw<LB>(m);
#pragma unroll
    for (int r = 0; r < 16; ++r) s[a ^ sw<LB>(r * M1)] = x[r];
  }
  __syncthreads();
  fwd_mid<LB, NP, 1>(s, tf, p);
  // last levels, product, first inverse levels
  const uint2* gh = ghat + (size_t)q * L;
  for (int u = threadIdx.x; u < (L >> LB); u += blockDim.x) {
    u32 x[R];
    const int a = sw<LB>(u << LB);
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = s[a ^ r];
    fwd_last<R>(x, tf + u, 4 * NP, p);
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = smul(x[r], __ldg(gh + r * (L >> LB) + u), p);
    inv_first<R>(x, ti + u, 4 * NP, p);
#pragma unroll
    for (int r = 0; r < R; ++r) s[a ^ r] = x[r];
  }
  __syncthreads();
#pragma unroll
  for (int ps = NP - 1; ps >= 1; --ps) {
    const int lm = LG - 4 * ps - 4;
    for (int u = threadIdx.x; u < M1; u += blockDim.x) {
      const int b = u >> lm, m = u & ((1 << lm) - 1);
      const int a = sw<LB>((b << (lm + 4)) + m);
      u32 x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = s[a ^ sw<LB>(r << lm)];
      inv16(x, ti + b, 4 * ps, p, 0);
#pragma unroll
      for (int r = 0; r < 16; ++r) s[a ^ sw<LB>(r << lm)] = x[r];
    }
    __syncthreads();
  }
  // last inverse pass: the generator is rotated so that the outputs wanted start at L / 2; of the last
  // level, whose z is 1, only the differences are formed
  u32* dst = out + ((size_t)q * n + row) * kr;
  for (int m = threadIdx.x; m < M1; m += blockDim.x) {
    u32 x[16];
    const int a = sw<LB>(m);
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = s[a ^ sw<LB>(r * M1)];
    inv16(x, ti, 0, p, 1);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int j = m + r * M1;
      if (j < k) dst[j] = red(red(x[r] - x[r + 8] + 2 * p, 2 * p), p);
    }
  }
}

// ------------------------------------------------------------------------------------------
// CRT: Z = sum_q X_q W_q - round(sum_q X_q / p_q) M in 32-bit limbs (|Z| < 2^126), scaled and rounded as in
// split_crt.cu; 32 x 128 tiles transposed through shared memory.  8192^2, four primes: 443 -> 329 us with the limbs'
// sums as the words of Z and four elements of Q in flight.
// ------------------------------------------------------------------------------------------
template <int NPR>
__global__ void __launch_bounds__(256) k_ntt_crt(const __grid_constant__ NttConsts c, const u32* __restrict__ X, int n, int k,
                                                 int kr, const u64* __restrict__ amax, const SplitDevParams* prm,
                                                 const NttParams* t, int slack, double alpha, double beta,
                                                 double* __restrict__ Q, long ldq) {
  __shared__ double tile[32][129];  // as crt_combine_blk's
  if (!ntt_ok(t, prm, slack)) return;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 128, jb = j0 + 4 * tx;
  const int PA = prm->PA, ge = gen_exp(t, prm);
  for (int a = 0; a < 4; ++a) {
    const int il = ty + 8 * a, i = i0 + il;
    double val[4] = {0.0, 0.0, 0.0, 0.0};
    if (i < n && jb < k) {
      const u64 ab = amax[i];
      uint4 w[NPR];
#pragma unroll
      for (int q = 0; q < NPR; ++q) w[q] = __ldg((const uint4*)(X + ((size_t)q * n + i) * kr + jb));
      const int e = ge + (ab >= INF_BITS ? EXP_NAN : ab == 0 ? EXP_ZERO : scale_exp(ab, PA));
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        u64 acc[3] = {0, 0, 0};
        u32 top = 0, qs = 1u << 19;
#pragma unroll
        for (int q = 0; q < NPR; ++q) {
          const u32 x = v == 0 ? w[q].x : v == 1 ? w[q].y : v == 2 ? w[q].z : w[q].w;
          qs += __umulhi(x, c.G[q]);
#pragma unroll
          for (int l = 0; l < 3; ++l) acc[l] += (u64)x * c.W[q][l];
          if (NPR > 4) top += x * c.W[q][3];  // four primes: W_q < 2^90
          if (NPR > 4 && q == 3) {  // four terms x W[l] stay below 2^64, the fifth would not
            acc[1] += acc[0] >> 32;
            acc[0] = (u32)acc[0];
            top += (u32)(acc[2] >> 32);
            acc[2] = (u32)acc[2];
          }
        }
        const u32 qq = qs >> 20;
        const u64 z0 = acc[0] + (u64)qq * c.Mneg[0];
        const u64 z1 = acc[1] + (u64)qq * c.Mneg[1] + (z0 >> 32);
        const u64 z2 = acc[2] + (u64)qq * c.Mneg[2] + (z1 >> 32);
        const u32 z3 = top + qq * c.Mneg[3] + (u32)(z2 >> 32);
        // |Z| < 2^126: the low 128 bits in two's complement are Z
        const unsigned __int128 z = ((unsigned __int128)(((u64)z3 << 32) | (u32)z2) << 64) | ((z1 << 32) | (u32)z0);
        val[v] = i128_scaled((__int128)z, e);
      }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) tile[tx][v * 32 + il] = val[v];
  }
  __syncthreads();
  const bool scale = alpha != 1.0, accumulate = beta != 0.0;
  const int i = i0 + tx, left = i < n ? k - j0 : 0;
  double* qp = Q + i + (long)(j0 + ty) * ldq;
#pragma unroll
  for (int b0 = 0; b0 < 16; b0 += 4) {
    double qv[4];
    const double* ql = qp;
#pragma unroll
    for (int b = 0; b < 4; ++b, ql += 8 * ldq) qv[b] = accumulate && ty + 8 * (b0 + b) < left ? *ql : 0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b, qp += 8 * ldq) {
      const int jl = ty + 8 * (b0 + b);
      if (jl < left) {
        double v = tile[jl >> 2][(jl & 3) * 32 + tx];
        if (scale) v *= alpha;
        if (accumulate) v = fma(beta, qv[b], v);
        *qp = v;
      }
    }
  }
}

template <int LB, int NP>
int launch_lg(const NttConsts& c, const double* g, int n, int k, int kp, int kr, const SplitDevParams* prm,
              const NttParams* t, int slack, uint2* tab, uint2* ghat, const long long* Ai, u32* out, cudaStream_t s) {
  constexpr int L = 1 << (4 * NP + LB);
  constexpr int smem = L * 4;
  if (set_smem_attr(k_ntt_gen<LB, NP>, smem) != cudaSuccess || set_smem_attr(k_ntt_rows<LB, NP>, smem) != cudaSuccess)
    return PSMMA_EDEVICE;
  k_ntt_gen<LB, NP><<<c.np, std::max(32, std::min(512, L / 16)), smem, s>>>(c, g, k, prm, t, slack, tab, ghat);
  prof_mark(s, "ntt_generator");
  k_ntt_rows<LB, NP><<<n * c.np, std::max(32, std::min(512, L / 16)), smem, s>>>(c, n, k, kp, kr, prm, t, slack, tab, ghat,
                                                                                Ai, out);
  prof_mark(s, "ntt_rows");
  return PSMMA_OK;
}

}  // namespace

// log2 of the transform length for order k, or 0 where the route does not cover it (orders that fit a
// transform of 2^(NT_MIN_LOG - 1) among them).
int ntt_log(int k) {
  if ((1L << (NT_MIN_LOG - 1)) >= 2L * k - 1) return 0;
  int lg = NT_MIN_LOG;
  while (lg <= NT_MAX_LOG && (1L << lg) < 2L * k - 1) ++lg;
  return lg <= NT_MAX_LOG ? lg : 0;
}

// Bytes of the route's buffers (tables, the generator's transform, A', residues).
size_t ntt_bytes(int n, int k) {
  const int lg = ntt_log(k);
  if (!lg) return 0;
  const size_t L = (size_t)1 << lg, kp = (size_t)(k + 63) / 64 * 64;
  return NT_MAXP * L * 24 + (size_t)n * kp * 8 + (size_t)NT_MAXP * n * kp * 4 + 4096;
}

// Enqueues the route.  prm, amax, asq, hmax, hsq as split_core lays them out (params, maxima and sums
// cleared); flag_mem: 256 bytes that the fallback does not touch before its kernels have read the flag;
// buf: ntt_bytes; *gate receives the word that makes the fallback run.  log2M: of the caller's moduli.
int launch_ntt(bool hankel, int n, int k, double alpha, const double* A, long lda, const double* g, double beta, double* Q,
               long ldq, double log2M, SplitDevParams* prm, u64* amax, double* asq, u64* hmax, double* hsq, void* flag_mem,
               void* buf, cudaStream_t stream, const unsigned** gate) {
  const int lg = ntt_log(k);
  if (!lg || (long)n * NT_MAXP >= 0x7FFFFFFFL) return PSMMA_EUNSUPPORTED;
  // four primes where they leave four bits for unequal columns
  const int np = ntt_log2(4) - log2M >= 4.0 ? 4 : 5;
  const int slack = (int)std::floor(std::min(ntt_log2(np), 127.0) - log2M - 0.01);
  const NttConsts c = make_ntt(np, lg);
  const size_t L = (size_t)1 << lg;
  const int kp = (k + 63) / 64 * 64, kr = kp;
  NttParams* t = (NttParams*)flag_mem;
  *gate = &t->fallback;
  char* w = (char*)buf;
  uint2* tab = (uint2*)w;              w += NT_MAXP * L * 16;
  uint2* ghat = (uint2*)w;             w += NT_MAXP * L * 8;
  long long* Ai = (long long*)w;       w += (size_t)n * kp * 8;
  u32* out = (u32*)w;

  prof_begin(stream);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return PSMMA_EDEVICE;
  int st = launch_row_stats(A, lda, n, k, amax, asq, sms, stream);
  if (st) return st;
  prof_mark(stream, "row_scale");
  k_ntt_colstats<<<1, 1024, 0, stream>>>(g, k, hmax, hsq, prm, t);
  k_ntt_tables<<<dim3((unsigned)std::min<size_t>(256, 2 * L / 128), np), 128, 0, stream>>>(c, lg >= 14 ? 3 : 2, tab);
  prof_mark(stream, "generator_stats");
  st = launch_split_params(prm, log2M, n, k, k, amax, asq, hmax, hsq, stream);
  if (st) return st;
  prof_mark(stream, "params");
  const dim3 gs((n + 63) / 64, kp / 64);
  if (hankel)
    k_ntt_scale<true><<<gs, 256, 0, stream>>>(A, lda, n, k, kp, amax, prm, t, slack, Ai);
  else
    k_ntt_scale<false><<<gs, 256, 0, stream>>>(A, lda, n, k, kp, amax, prm, t, slack, Ai);
  prof_mark(stream, "scale_A");
#define PSMMA_NTT(lgv, lb, np16) \
  case lgv: st = launch_lg<lb, np16>(c, g, n, k, kp, kr, prm, t, slack, tab, ghat, Ai, out, stream); break;
  switch (lg) {
    PSMMA_NTT(13, 5, 2)
    PSMMA_NTT(14, 2, 3)
    PSMMA_NTT(15, 3, 3)
    default: return PSMMA_EUNSUPPORTED;
  }
#undef PSMMA_NTT
  if (st) return st;
  const dim3 gc((k + 127) / 128, (n + 31) / 32);
  if (np == 4)
    k_ntt_crt<4><<<gc, dim3(32, 8), 0, stream>>>(c, out, n, k, kr, amax, prm, t, slack, alpha, beta, Q, ldq);
  else
    k_ntt_crt<5><<<gc, dim3(32, 8), 0, stream>>>(c, out, n, k, kr, amax, prm, t, slack, alpha, beta, Q, ldq);
  prof_mark(stream, "crt_combine");
  return cudaGetLastError() == cudaSuccess ? PSMMA_OK : PSMMA_EDEVICE;
}

}  // namespace psmma
