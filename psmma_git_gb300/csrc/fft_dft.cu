// The DFT multiply C = alpha F B + beta C (PZMDFTL, pzmdftL.f90:1-2) as a fast Fourier transform of
// every column of B in 64-bit fixed point on the integer pipes.
//
// GB300 issues two FP64 operations per SM and cycle but 64 integer adds and 24-32 widening 32-bit
// multiply-adds, so an FFT in FP64 would be bound by the FP64 pipe at some 25 times its memory
// traffic.  Here a column lives in shared memory as complex 64-bit integers with one exponent per
// column (block floating point): a butterfly add is two integer instructions, a twiddle product
// twelve widening multiply-adds.  Before every pass the column is shifted up to 59 bits from its
// actual largest entry, so that each pass rounds at 2^-59 of it or better; twiddles are exact to
// 2^-61.  Outputs are rounded to FP64 once.  The error, some 2^-57 of the column's norm plus that
// rounding, is below that of FP64 additions in any order.
//
//   direct      n with no prime factor above 5, n <= 14400: in-place decimation in frequency, the last
//               pass reading in digit-reversed order and writing C's column in order.
//   Bluestein   other n with 2 n - 1 <= 14400: F(j, l) = c_j c_l conj(c_(j-l)) with the chirp c_j =
//               exp(-pi i j^2 / n), a cyclic convolution of length L >= 2 n - 1 (L with no prime factor
//               above 5): decimation in frequency, the product with the chirp's transform in the
//               digit-reversed order, decimation in time back.
//   two levels  larger n = R n': one radix-R pass through global memory, then transforms of length n' of
//               one of the two forms.
// Sizes none of the three covers keep the dense products (split_crt.cu, fp64_structured.cu).
//
// Measured (n = k, against the dense products it replaces): split precision n = 4096 0.29 ms (2.64),
// 8192 1.37 (7.17), 16384 8.9 (43.0); FP64 n = 4800 0.69 ms (209).  ncu at n = 8192, before the first pass
// took its entries from registers (1.73 ms): 510 instructions a point with the conversions, the integer
// pipe 51 % and the wide multiply-adds 37 % busy, issue 45 %, DRAM 12 %: bound by the passes' instructions
// and by the latencies that 16 warps (128 registers each thread) leave uncovered.
#include <algorithm>
#include <cstring>

#include "psmma_internal.h"

namespace psmma {
namespace {

typedef long long i64;
typedef unsigned long long u64;

constexpr int FFT_MAX = 14400;    // 16 B a point: 225 of the 227 KB of shared memory
constexpr int FFT_MAX_PASSES = 12;
constexpr int FFT_TOP = 59;       // entries are below 2^59 at the start of a pass

// ------------------------------------------------------------------------------------------
// Sines and cosines of 2 pi t / n to about 2^-62, in integers
// ------------------------------------------------------------------------------------------
__host__ __device__ constexpr u64 mulhi64(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  if (!__builtin_is_constant_evaluated()) return __umul64hi(a, b);
#endif
  const u64 a0 = a & 0xFFFFFFFFull, a1 = a >> 32, b0 = b & 0xFFFFFFFFull, b1 = b >> 32;
  const u64 m0 = a1 * b0 + ((a0 * b0) >> 32), m1 = a0 * b1 + (m0 & 0xFFFFFFFFull);
  return a1 * b1 + (m0 >> 32) + (m1 >> 32);
}

struct CosSin {
  i64 c, s;  // Q62
};

// Taylor series of cos and sin at x = (pi / 4) f, f in [0, 1] as Q64 (2^64 - 1 for 1), with
// Horner steps t <- 1 - x^2 t / (k (k + 1)) in Q63: the first term left out is below
// 2^-64 (0.785^22 / 22!).
__host__ __device__ constexpr CosSin octant(u64 f) {
  const u64 one = 1ull << 63;
  const u64 x = mulhi64(f, 0xC90FDAA22168C235ull);
  const u64 x2 = mulhi64(x, x);
  u64 c = one, s = one;
  // the steps written out: divisions by constants
#define PSMMA_STEP(k)                                  \
  s = one - mulhi64(x2, s) / (u64)((k) * ((k) + 1));   \
  c = one - mulhi64(x2, c) / (u64)(((k) - 1) * (k));
  PSMMA_STEP(20) PSMMA_STEP(18) PSMMA_STEP(16) PSMMA_STEP(14) PSMMA_STEP(12)
  PSMMA_STEP(10) PSMMA_STEP(8) PSMMA_STEP(6) PSMMA_STEP(4) PSMMA_STEP(2)
#undef PSMMA_STEP
  s = mulhi64(x, s);  // Q64 * Q63 -> Q63
  CosSin r{};
  r.c = (i64)((c + 1) >> 1);
  r.s = (i64)((s + 1) >> 1);
  return r;
}

// exp(-2 pi i t / n) = c + i s (Q62), 0 <= t < n < 2^29.
__host__ __device__ constexpr CosSin root(u64 t, u64 n) {
  const u64 e = 8 * t, o = e / n;
  u64 r = e - o * n;
  if (o & 1) r = n - r;
  u64 f = ~0ull;
  if (r < n) {
    const u64 q1 = (r << 32) / n, rem = (r << 32) - q1 * n;
    f = (q1 << 32) | ((rem << 32) / n);
  }
  const CosSin v = octant(f);
  CosSin w{};
  switch ((int)o) {
    case 0: w.c = v.c; w.s = -v.s; break;
    case 1: w.c = v.s; w.s = -v.c; break;
    case 2: w.c = -v.s; w.s = -v.c; break;
    case 3: w.c = -v.c; w.s = -v.s; break;
    case 4: w.c = -v.c; w.s = v.s; break;
    case 5: w.c = -v.s; w.s = v.c; break;
    case 6: w.c = v.s; w.s = v.c; break;
    default: w.c = v.c; w.s = v.s; break;
  }
  return w;
}

// A twiddle as signed halves: c = x 2^32 + y, s = z 2^32 + w, y and w in [-2^31, 2^31).
struct Tw {
  int x, y, z, w;
};
__host__ __device__ constexpr Tw halves(i64 c, i64 s) {
  Tw t{};
  t.x = (int)((c + 0x80000000ll) >> 32);
  t.y = (int)(c - (i64)t.x * (1ll << 32));
  t.z = (int)((s + 0x80000000ll) >> 32);
  t.w = (int)(s - (i64)t.z * (1ll << 32));
  return t;
}

// The roots inside the composite butterflies, w_R^t for t < R <= 16 (Q62).
struct SmallTw {
  Tw w[17][16];
  Tw c3, c5a, c5b;  // sin(60); cos(72), sin(72); cos(144), sin(144)
};
constexpr SmallTw make_small() {
  SmallTw S{};
  for (int R = 2; R <= 16; ++R)
    for (int t = 0; t < R; ++t) {
      const CosSin v = root((u64)t, (u64)R);
      S.w[R][t] = halves(v.c, v.s);
    }
  const CosSin a = root(1, 3), b = root(1, 5), d = root(2, 5);
  S.c3 = halves(-a.s, 0);
  S.c5a = halves(b.c, -b.s);
  S.c5b = halves(d.c, -d.s);
  return S;
}
__constant__ SmallTw kSmall = make_small();

// ------------------------------------------------------------------------------------------
// Complex fixed-point arithmetic
// ------------------------------------------------------------------------------------------
struct Cx {
  i64 r, i;
};
__device__ __forceinline__ Cx operator+(Cx a, Cx b) { return {a.r + b.r, a.i + b.i}; }
__device__ __forceinline__ Cx operator-(Cx a, Cx b) { return {a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ Cx sar(Cx a, int s) { return {a.r >> s, a.i >> s}; }
// a b + c as one instruction (left to itself the compiler forms the product and adds it in two more:
// 680 instead of 510 instructions a point at n = 8192, 2.13 instead of 1.73 ms).
__device__ __forceinline__ i64 wmad(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
  i64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (i64)a * b + c;
#endif
}

// (x w) 2^-64 rounded, w = c + i s in halves: with w in Q62 the product over 4.  The halves of x
// are taken signed, the product of the low halves (below one unit) left out.  |x| <= 2.6 * 2^61:
// the middle sums stay below 0.71 |x| + 1.42 * 2^61 + 2^31 < 2^63.
__device__ __forceinline__ Cx cmul(Cx x, Tw t) {
  const int al = (int)x.r, ah = (int)((x.r + 0x80000000ll) >> 32);
  const int bl = (int)x.i, bh = (int)((x.i + 0x80000000ll) >> 32);
  const int nz = -t.z, nw = -t.w;
  const i64 hr = wmad(bh, nz, wmad(ah, t.x, 0)), hi = wmad(bh, t.x, wmad(ah, t.z, 0));
  const i64 mr = wmad(bl, nz, wmad(bh, nw, wmad(al, t.x, wmad(ah, t.y, 0x80000000ll))));
  const i64 mi = wmad(bl, t.x, wmad(bh, t.y, wmad(al, t.z, wmad(ah, t.w, 0x80000000ll))));
  return {hr + (mr >> 32), hi + (mi >> 32)};
}

// x c for a real c in Q62 (halves h, l), at full scale.
__device__ __forceinline__ i64 rmul(i64 x, int h, int l) {
  const int xl = (int)x, xh = (int)((x + 0x80000000ll) >> 32);
  const i64 m = wmad(xl, h, wmad(xh, l, 1ll << 29));
  return ((i64)xh * h) * 4 + (m >> 30);
}
__device__ __forceinline__ Cx rmul(Cx x, int h, int l) { return {rmul(x.r, h, l), rmul(x.i, h, l)}; }

// R-point transforms in registers, growing by at most R.
template <int R>
__device__ __forceinline__ void bf(Cx (&x)[R]);
template <>
__device__ __forceinline__ void bf<2>(Cx (&x)[2]) {
  const Cx a = x[0];
  x[0] = a + x[1];
  x[1] = a - x[1];
}
template <>
__device__ __forceinline__ void bf<3>(Cx (&x)[3]) {
  const Cx t = x[1] + x[2], u = rmul(x[1] - x[2], kSmall.c3.x, kSmall.c3.y), m = x[0] - sar(t, 1);
  x[0] = x[0] + t;
  x[1] = {m.r + u.i, m.i - u.r};
  x[2] = {m.r - u.i, m.i + u.r};
}
template <>
__device__ __forceinline__ void bf<4>(Cx (&x)[4]) {
  const Cx a = x[0] + x[2], b = x[0] - x[2], c = x[1] + x[3], d = x[1] - x[3];
  x[0] = a + c;
  x[2] = a - c;
  x[1] = {b.r + d.i, b.i - d.r};
  x[3] = {b.r - d.i, b.i + d.r};
}
template <>
__device__ __forceinline__ void bf<5>(Cx (&x)[5]) {
  const Tw A = kSmall.c5a, B = kSmall.c5b;
  const Cx t1 = x[1] + x[4], t2 = x[2] + x[3], t3 = x[1] - x[4], t4 = x[2] - x[3];
  const Cx a1 = x[0] + rmul(t1, A.x, A.y) + rmul(t2, B.x, B.y);
  const Cx a2 = x[0] + rmul(t1, B.x, B.y) + rmul(t2, A.x, A.y);
  const Cx b1 = rmul(t3, A.z, A.w) + rmul(t4, B.z, B.w);
  const Cx b2 = rmul(t3, B.z, B.w) - rmul(t4, A.z, A.w);
  x[0] = x[0] + t1 + t2;
  x[1] = {a1.r + b1.i, a1.i - b1.r};
  x[4] = {a1.r - b1.i, a1.i + b1.r};
  x[2] = {a2.r + b2.i, a2.i - b2.r};
  x[3] = {a2.r - b2.i, a2.i + b2.r};
}

// R = R1 R2: R2 transforms of R1 points, the products with w_R^(n2 k1) over 4, R1 transforms of R2
// points.  Entries below 2^60 in modulus stay below 2^62.4 throughout; the result is over 4.
template <int R1, int R2>
__device__ __forceinline__ void bf_comp(Cx (&x)[R1 * R2]) {
  constexpr int R = R1 * R2;
  Cx y[R1][R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) {
    Cx t[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) t[n1] = x[R2 * n1 + n2];
    bf<R1>(t);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      const int e = n2 * k1;
      if (e == 0)
        y[k1][n2] = sar(t[k1], 2);
      else if (4 * e == R)
        y[k1][n2] = sar(Cx{t[k1].i, -t[k1].r}, 2);
      else
        y[k1][n2] = cmul(t[k1], kSmall.w[R][e]);
    }
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) {
    bf<R2>(y[k1]);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) x[k1 + R1 * k2] = y[k1][k2];
  }
}
template <> __device__ __forceinline__ void bf<6>(Cx (&x)[6]) { bf_comp<2, 3>(x); }
template <> __device__ __forceinline__ void bf<8>(Cx (&x)[8]) { bf_comp<2, 4>(x); }
template <> __device__ __forceinline__ void bf<9>(Cx (&x)[9]) { bf_comp<3, 3>(x); }
template <> __device__ __forceinline__ void bf<10>(Cx (&x)[10]) { bf_comp<2, 5>(x); }
template <> __device__ __forceinline__ void bf<12>(Cx (&x)[12]) { bf_comp<4, 3>(x); }
template <> __device__ __forceinline__ void bf<15>(Cx (&x)[15]) { bf_comp<3, 5>(x); }
template <> __device__ __forceinline__ void bf<16>(Cx (&x)[16]) { bf_comp<4, 4>(x); }

// Bits the butterfly itself gives up (composite: the inner product's 2) and the external twiddle
// product's (2, or 3 where the last factor is 5, so that a pass never grows).
__host__ __device__ constexpr int inner_shift(int R) { return R > 5 ? 2 : 0; }
__host__ __device__ constexpr int outer_shift(int R) { return (R == 5 || R == 10 || R == 15) ? 3 : 2; }

// ------------------------------------------------------------------------------------------
// Plans
// ------------------------------------------------------------------------------------------
struct Pass {
  int R, N, M, tw;  // radix, block length, N / R, first entry in the twiddle table
};
struct Plan {
  int n, np, entries;  // length, passes, twiddle entries
  Pass p[FFT_MAX_PASSES];
};

// Radices of the passes.  Powers of two take 16; in the general passes, whose addresses are not an XOR
// with a constant, 16 and 15 points and their addresses do not fit 128 registers (n = 4800 as
// 2 * 10 * 15 * 16 0.81 ms, its spills gone with 5 * 8 * 10 * 12).
const int kRadices[] = {16, 12, 10, 9, 8, 6, 5, 4, 3, 2};

// Depth first over the radices, the largest first, for exactly `left` passes.
bool factor(int n, int left, int* r, int at, int from) {
  if (n == 1) return left == 0;
  if (left == 0) return false;
  for (int i = from; i < 10; ++i)
    if (n % kRadices[i] == 0) {
      r[at] = kRadices[i];
      if (factor(n / kRadices[i], left - 1, r, at + 1, i)) return true;
    }
  return false;
}

bool make_plan(int n, Plan* P) {
  memset(P, 0, sizeof(*P));
  P->n = n;
  int r[FFT_MAX_PASSES];
  for (int np = 1; np <= 8; ++np)
    if (n == 1 || factor(n, np, r, 0, (n & (n - 1)) ? 1 : 0)) {
      P->np = n == 1 ? 0 : np;
      std::reverse(r, r + P->np);  // the largest radix last: the last pass of the direct form finds
                                   // each butterfly's place by np - 1 divisions
      // powers of two also begin with a radix of 16 (the first pass then takes its entries from global memory)
      if ((n & (n - 1)) == 0 && P->np > 2) std::swap(r[0], r[1]);
      int N = n;
      for (int i = 0; i < P->np; ++i) {
        P->p[i] = {r[i], N, N / r[i], P->entries};
        if (N > r[i]) P->entries += N - N / r[i];
        N /= r[i];
      }
      return true;
    }
  return false;
}

bool smooth(int n) {
  for (int f : {2, 3, 5})
    while (n % f == 0) n /= f;
  return n == 1;
}

enum { FORM_DIRECT = 0, FORM_BLUESTEIN = 1 };

struct Route {
  int R0;    // radix of the pass through global memory (1: none)
  int form;  // of the transforms of length n1 = n / R0
  int n1;
  Plan plan;  // of length n1, or L for Bluestein
};

// The transform length of Bluestein's form: the 5-smooth L >= 2 n - 1 with the least L * passes.
bool bluestein(int n, Plan* P) {
  double best = 1e300;
  for (int L = 2 * n - 1; L <= FFT_MAX && L <= 3 * n + 16; ++L) {
    if (!smooth(L)) continue;
    Plan q;
    if (!make_plan(L, &q)) continue;
    const double cost = (double)L * (q.np + 2);
    if (cost < best) {
      best = cost;
      *P = q;
    }
  }
  return best < 1e300;
}

bool one_level(int n, Route* r) {
  r->R0 = 1;
  r->n1 = n;
  if (n <= FFT_MAX && smooth(n) && make_plan(n, &r->plan)) {
    r->form = FORM_DIRECT;
    return true;
  }
  r->form = FORM_BLUESTEIN;
  return 2 * n - 1 <= FFT_MAX && bluestein(n, &r->plan);
}

bool make_route(int n, Route* r) {
  if (n < 1) return false;
  if (one_level(n, r)) return true;
  for (int want = 0; want < 2; ++want)  // a direct second level before a convolution
    for (int R : {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16})
      if (n % R == 0 && one_level(n / R, r) && r->form == want) {
        r->R0 = R;
        return true;
      }
  return false;
}

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

struct Layout {
  size_t off_tw, off_c1, off_c2, off_bh, off_eb, off_tw0, off_ce, off_x, total;
};
Layout layout(const Route& r, int k) {
  Layout L{};
  size_t o = 0;
  L.off_tw = o; o += al256((size_t)r.plan.entries * 16 + 16);
  if (r.form == FORM_BLUESTEIN) {
    L.off_c1 = o; o += al256((size_t)r.n1 * 16);
    L.off_c2 = o; o += al256((size_t)r.n1 * 16);
    L.off_bh = o; o += al256((size_t)r.plan.n * 16);
    L.off_eb = o; o += 256;
  }
  if (r.R0 > 1) {
    L.off_tw0 = o; o += al256((size_t)(r.R0 - 1) * r.n1 * 16);
    L.off_ce = o;  o += al256((size_t)k * 4);
    L.off_x = o;   o += al256((size_t)r.R0 * r.n1 * k * 16);
  }
  L.total = o;
  return L;
}

// ------------------------------------------------------------------------------------------
// Tables
// ------------------------------------------------------------------------------------------
// Twiddles of every pass, entry (s - 1) M + m = w_N^(m s) over 2^(outer_shift - 2) (the product with
// it is then over 2^outer_shift); the chirp c_j and c_j times 2^(lg - 1) / L in (1/2, 1], the
// inverse transform's 1 / L up to its exponent; the pass through global memory's twiddles.
__global__ void k_fft_tables(Plan P, Tw* __restrict__ tw, int n1, Tw* __restrict__ c1, Tw* __restrict__ c2, int R0,
                             Tw* __restrict__ tw0) {
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int e = t0; e < P.entries; e += stride) {
    int p = 0;
    while (p + 1 < P.np && P.p[p + 1].N > P.p[p + 1].R && P.p[p + 1].tw <= e) ++p;
    const int q = e - P.p[p].tw, M = P.p[p].M, s = q / M + 1, m = q % M;
    CosSin v = root((u64)m * s, (u64)P.p[p].N);
    const int sh = outer_shift(P.p[p].R) - 2;
    if (sh) {
      v.c = (v.c + (1ll << (sh - 1))) >> sh;
      v.s = (v.s + (1ll << (sh - 1))) >> sh;
    }
    tw[e] = halves(v.c, v.s);
  }
  if (c1) {
    const u64 n2 = 2 * (u64)n1;
    int lg = 0;
    while ((1 << lg) < P.n) ++lg;
    // 2^(lg - 1) / L as Q64, at most 1
    const u64 num = 1ull << (lg - 1), q1 = (num << 32) / (u64)P.n, rem = (num << 32) - q1 * (u64)P.n;
    const u64 rho = (q1 << 32) | ((rem << 32) / (u64)P.n);  // lg - 1 <= 13; L > num: below 2^64
    for (int j = t0; j < n1; j += stride) {
      const CosSin v = root((u64)j * j % n2, n2);
      c1[j] = halves(v.c, v.s);
      const bool whole = (1 << lg) == P.n;  // L a power of two: 1/2
      const u64 ac = (u64)(v.c < 0 ? -v.c : v.c), as = (u64)(v.s < 0 ? -v.s : v.s);
      const i64 pc = whole ? (i64)(ac >> 1) : (i64)mulhi64(ac, rho), ps = whole ? (i64)(as >> 1) : (i64)mulhi64(as, rho);
      c2[j] = halves(v.c < 0 ? -pc : pc, v.s < 0 ? -ps : ps);
    }
  }
  if (tw0) {
    const int sh = outer_shift(R0) - 2;
    for (int e = t0; e < (R0 - 1) * n1; e += stride) {
      const int s = e / n1 + 1, m = e % n1;
      CosSin v = root((u64)m * s, (u64)n1 * R0);
      if (sh) {
        v.c = (v.c + (1ll << (sh - 1))) >> sh;
        v.s = (v.s + (1ll << (sh - 1))) >> sh;
      }
      tw0[e] = halves(v.c, v.s);
    }
  }
}

// ------------------------------------------------------------------------------------------
// A column in shared memory
// ------------------------------------------------------------------------------------------
// 16-byte entries; an entry's low three index bits are XORed with its higher digits, so that the
// eight threads of a 128-byte phase hit eight bank groups at every power-of-two stride.
__device__ __forceinline__ int sw(int p) { return p ^ (((p >> 3) ^ (p >> 6) ^ (p >> 9) ^ (p >> 12)) & 7); }
__device__ __forceinline__ Cx ld(const longlong2* s, int p) {
  const longlong2 v = s[sw(p)];
  return {v.x, v.y};
}
__device__ __forceinline__ void st(longlong2* s, int p, Cx v) { s[sw(p)] = make_longlong2(v.r, v.i); }

// The largest and smallest high words of the entries a thread writes; published as the largest
// magnitude (one's complement for negative values).
struct Range {
  int hi = 0, lo = 0;
  __device__ __forceinline__ void add(Cx v) {
    const int a = (int)(v.r >> 32), b = (int)(v.i >> 32);
    hi = max(hi, max(a, b));
    lo = min(lo, min(a, b));
  }
};
__device__ __forceinline__ void publish(Range r, unsigned* word) {
  const unsigned m = __reduce_max_sync(0xffffffffu, (unsigned)max(r.hi, ~r.lo));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(word, m);
}
// The left shift that brings the largest entry just below 2^top (a zero high word: 32 bits at most
// are taken, the next pass takes the rest).
__device__ __forceinline__ int headroom(unsigned m, int top) { return max(0, __clz((int)m) - (64 - top)); }

// Loads R entries base + M r, shifted up by d.  P2: lengths are powers of two, base and M r share no
// bit and sw is linear over XOR, so that an address is one XOR with a value all threads share.
template <int R, bool P2>
__device__ __forceinline__ void load_r(const longlong2* s, int base, int M, int d, Cx (&x)[R]) {
  const int b0 = P2 ? sw(base) : base;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const longlong2 v = P2 ? s[b0 ^ sw(M * r)] : s[sw(b0 + M * r)];
    x[r] = {v.x, v.y};
  }
  if (d) {
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = {x[r].r << d, x[r].i << d};
  }
}

// One in-place pass.  DIF: butterfly, then twiddles; DIT: twiddles, then butterfly.  Entries are
// shifted up by d as they are loaded.  Returns the range of the entries written.
template <int R, bool DIT, bool P2>
__device__ __forceinline__ Range pass_r(longlong2* s, const Pass& P, int n, int d, const Tw* __restrict__ tw) {
  Range range;
  const int M = P.M, cnt = n / R;
  for (int u = threadIdx.x; u < cnt; u += blockDim.x) {
    const int b = u / M, m = u - b * M, base = b * P.N + m;
    const int4* t = (const int4*)(tw + P.tw) + m;
    Cx x[R];
    load_r<R, P2>(s, base, M, d, x);
    if (DIT) {
      if (M > 1) {
        x[0] = sar(x[0], outer_shift(R));
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const int4 w = __ldg(t + (r - 1) * M);
          x[r] = cmul(x[r], Tw{w.x, w.y, w.z, w.w});
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = sar(x[r], outer_shift(R));
      }
    }
    bf<R>(x);
    if (!DIT && M > 1) {
      x[0] = sar(x[0], outer_shift(R));
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const int4 w = __ldg(t + (r - 1) * M);
        x[r] = cmul(x[r], Tw{w.x, w.y, w.z, w.w});
      }
    }
    const int b0 = P2 ? sw(base) : base;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s[P2 ? b0 ^ sw(M * r) : sw(b0 + M * r)] = make_longlong2(x[r].r, x[r].i);
      range.add(x[r]);
    }
  }
  return range;
}

// P2: powers of two alone.
template <bool DIT, bool P2>
__device__ __forceinline__ Range pass(longlong2* s, const Pass& P, int n, int d, const Tw* tw) {
  if (P2 || (n & (n - 1)) == 0) switch (P.R) {
      case 16: return pass_r<16, DIT, true>(s, P, n, d, tw);
      case 8: return pass_r<8, DIT, true>(s, P, n, d, tw);
      case 4: return pass_r<4, DIT, true>(s, P, n, d, tw);
      default: return pass_r<2, DIT, true>(s, P, n, d, tw);
    }
  if constexpr (P2) return Range{};
  switch (P.R) {
    case 12: return pass_r<12, DIT, false>(s, P, n, d, tw);
    case 10: return pass_r<10, DIT, false>(s, P, n, d, tw);
    case 9: return pass_r<9, DIT, false>(s, P, n, d, tw);
    case 8: return pass_r<8, DIT, false>(s, P, n, d, tw);
    case 6: return pass_r<6, DIT, false>(s, P, n, d, tw);
    case 5: return pass_r<5, DIT, false>(s, P, n, d, tw);
    case 4: return pass_r<4, DIT, false>(s, P, n, d, tw);
    case 3: return pass_r<3, DIT, false>(s, P, n, d, tw);
    default: return pass_r<2, DIT, false>(s, P, n, d, tw);
  }
}

// v 2^e as a double, rounded to nearest even.
__device__ __noinline__ double fx_slow(u64 m, int e, bool neg) {
  const double v = ldexp((double)m, e);
  return neg ? -v : v;
}
__device__ __forceinline__ double fx_double(i64 v, int e) {
  if (v == 0) return 0.0;
  const bool neg = v < 0;
  const u64 a = neg ? (u64)(-v) : (u64)v;
  const int z = __clzll((i64)a);
  const u64 t = a << z;
  const int field = 63 - z + e + 1023;
  if (field < 1 || field > 2045) return fx_slow(a, e, neg);
  const u64 up = ((t & 0x7FFull) + ((t >> 11) & 1)) > 0x400ull ? 1 : 0;
  u64 bits = (((u64)field << 52) | ((t >> 11) & 0xFFFFFFFFFFFFFull)) + up;
  if (neg) bits |= 1ull << 63;
  return __longlong_as_double((i64)bits);
}

// The exponent e of a column from its largest high word (sign removed, finite): every entry is below
// 2^(e + 1).  Subnormal columns take the leading bit of that word, or of the 32 bits under it.
__device__ __forceinline__ int col_exponent(unsigned h) {
  const int ex = (int)(h >> 20);
  return ex ? ex - 1023 : (h ? 63 - __clz((int)h) - 1074 : 31 - 1074);
}

// x 2^(58 - emax) rounded, for |x| < 2^(emax + 1).
__device__ __forceinline__ i64 fx_from(double x, int emax) {
  const u64 b = (u64)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF);
  const u64 m = (b & 0xFFFFFFFFFFFFFull) | (ex ? 1ull << 52 : 0ull);
  const int sh = (ex ? ex : 1) - 1075 + (FFT_TOP - 1) - emax;  // at most 6 (27 in a subnormal column)
  u64 v;
  if (sh >= 0)
    v = m << sh;
  else
    v = sh < -62 ? 0 : (m + (1ull << (-sh - 1))) >> -sh;
  return (b >> 63) ? -(i64)v : (i64)v;
}

__device__ __forceinline__ double2 load_c(const double* p, bool aligned) {
  if (aligned) return __ldg((const double2*)p);
  return make_double2(__ldg(p), __ldg(p + 1));
}

struct FftArgs {
  const double* B;
  long ldb;  // in complex elements
  double* C;
  long ldc;
  int n, k, n1, R0, form;
  double alpha, beta;
  int b16, c16;    // B, C 16-byte aligned
  int ahead;       // columns in flight on the GPU
  int ieee;        // non-finite columns as FP64 sums give them (else NaN)
  const Tw *tw, *c1, *c2, *bh;
  const int* eb;   // exponent of the chirp's transform
  const longlong2* X;  // two levels: columns after the first pass, [column][s][m]
  const int* ce;       // their exponents (NO_EXP: not finite)
};
constexpr int NO_EXP = 0x7FFFFFFF;

__device__ __forceinline__ void put(const FftArgs& a, int col, int j, Cx v, int e) {
  double re = fx_double(v.r, e), im = fx_double(v.i, e);
  double* p = a.C + 2 * ((long)col * a.ldc + j);
  if (a.alpha != 1.0 || a.beta != 0.0) {
    re *= a.alpha;
    im *= a.alpha;
    if (a.beta != 0.0) {
      re = fma(a.beta, p[0], re);
      im = fma(a.beta, p[1], im);
    }
  }
  if (a.c16) {
    *(double2*)p = make_double2(re, im);
  } else {
    p[0] = re;
    p[1] = im;
  }
}

// Signs of cos and sin of 2 pi t / n, 0 <= t < n: 0, 1 or -1.
__device__ __forceinline__ int cos_sign(int t, int n) {
  const int q = 4 * t;
  return q < n || q > 3 * n ? 1 : q > n && q < 3 * n ? -1 : 0;
}
__device__ __forceinline__ int sin_sign(int t, int n) { return t == 0 || 2 * t == n ? 0 : 2 * t < n ? 1 : -1; }

// Class of a sum, a set of bits: a term +inf, a term -inf.  Both (a NaN from inf * 0 counts as both): NaN.
constexpr unsigned POS_INF = 1u, NEG_INF = 2u, IS_NAN = 3u;
__device__ __forceinline__ unsigned inf_class(int sign) { return sign > 0 ? POS_INF : sign < 0 ? NEG_INF : IS_NAN; }

// A column with a NaN or an infinity: NaN, or (ieee) the class of the dense product's FP64 sums.  A NaN reaches every
// output, and so does an infinity, as an infinity of the sign of its cosine or sine or, where that is zero, a NaN;
// finite terms decide nothing.  So only the infinities are summed, by their classes: they are listed in the column's
// shared memory (`bytes`; a part of the column at a time where their number might not fit), after which each output is
// as many steps as it takes to become NaN or to end the list.  (FP64 sums over all entries took n divisions and
// sincospi an output on one SM: 265 ms a column of 4800.)
__device__ __noinline__ void nonfinite_column(const FftArgs& a, int col, int s, unsigned char* smem, int bytes) {
  const double* src = a.B + 2 * (long)col * a.ldb;
  unsigned char* cls = smem;  // of output s + R0 q: the real part's two bits, then the imaginary part's
  int* list = (int*)(smem + (a.n1 + 3) / 4 * 4);
  const int room = (bytes - (a.n1 + 3) / 4 * 4) / 4;
  __shared__ int count, nan;
  for (int q = threadIdx.x; q < a.n1; q += blockDim.x) cls[q] = 0;
  if (threadIdx.x == 0) nan = a.ieee ? 0 : 1;
  __syncthreads();
  for (int l0 = 0; l0 < a.n && nan == 0; l0 += room) {
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    for (int l = l0 + threadIdx.x; l < min(a.n, l0 + room); l += blockDim.x) {
      const double2 b = load_c(src + 2 * (long)l, a.b16);
      if (isnan(b.x) || isnan(b.y)) nan = 1;
      // index, and a sign each for the real and the imaginary part: 0 finite, 1 +inf, 2 -inf
      const int code = (isinf(b.x) ? (b.x > 0 ? 1 : 2) : 0) | (isinf(b.y) ? (b.y > 0 ? 4 : 8) : 0);
      if (code) list[atomicAdd(&count, 1)] = l << 4 | code;
    }
    __syncthreads();
    if (nan == 0)
      for (int q = threadIdx.x; q < a.n1; q += blockDim.x) {
        const int j = s + a.R0 * q;
        unsigned re = cls[q] & 3u, im = cls[q] >> 2;
        for (int i = 0; i < count && (re & im) != IS_NAN; ++i) {
          const int l = list[i] >> 4, t = (int)((u64)j * l % (u64)a.n), cs = cos_sign(t, a.n), sn = sin_sign(t, a.n);
          if (list[i] & 3) {
            const int g = list[i] & 1 ? 1 : -1;
            re |= inf_class(g * cs);
            im |= inf_class(-g * sn);
          }
          if (list[i] & 12) {
            const int g = list[i] & 4 ? 1 : -1;
            re |= inf_class(g * sn);
            im |= inf_class(g * cs);
          }
        }
        cls[q] = (unsigned char)(re | im << 2);
      }
    __syncthreads();  // the list is filled again
  }
  const double value[4] = {0.0, __longlong_as_double((i64)0x7FF0000000000000ll), __longlong_as_double((i64)0xFFF0000000000000ull),
                           __longlong_as_double(0x7FF8000000000000ll)};
  for (int q = threadIdx.x; q < a.n1; q += blockDim.x) {
    double re = value[nan ? IS_NAN : cls[q] & 3u], im = value[nan ? IS_NAN : cls[q] >> 2];
    double* p = a.C + 2 * ((long)col * a.ldc + s + a.R0 * q);
    re *= a.alpha;
    im *= a.alpha;
    if (a.beta != 0.0) {
      re = fma(a.beta, p[0], re);
      im = fma(a.beta, p[1], im);
    }
    p[0] = re;
    p[1] = im;
  }
}

// The last pass of the direct form: butterfly tau of radix R reads its block at the digit-reversed
// position of tau and writes outputs tau + q n1 / R.
template <int R, bool P2>
__device__ __forceinline__ void last_r(longlong2* s, const Plan& P, const FftArgs& a, int col, int s0, int d, int e) {
  const int cnt = P.n / R;
  for (int u = threadIdx.x; u < cnt; u += blockDim.x) {
    int rest = u, base = 0;
    for (int p = 0; p + 1 < P.np; ++p) {
      const int q = rest / P.p[p].R;
      base += (rest - q * P.p[p].R) * P.p[p].M;
      rest = q;
    }
    Cx x[R];
    load_r<R, P2>(s, base, 1, d, x);
    bf<R>(x);
#pragma unroll
    for (int r = 0; r < R; ++r) put(a, col, s0 + a.R0 * (u + r * cnt), x[r], e + inner_shift(R));
  }
}

// Passes p0 .. np - 1 of one column's transform, in place; words[p] holds the magnitude before pass p, `e` the
// exponent of the entries, kept by every thread.
template <bool P2 = false>
__device__ __forceinline__ int forward(longlong2* s, const Plan& P, const Tw* tw, unsigned* words, int p0, int np, int& e) {
  for (int p = p0; p < np; ++p) {
    const int d = headroom(words[p], FFT_TOP);
    publish(pass<false, P2>(s, P.p[p], P.n, d, tw), &words[p + 1]);
    e += inner_shift(P.p[p].R) + (P.p[p].M > 1 ? outer_shift(P.p[p].R) : 0) - d;
    __syncthreads();
  }
  return np;
}

// FIRST16: direct form, a power of two of at least 512 points, a thread per radix-16 butterfly.
template <bool FIRST16>
__global__ void __launch_bounds__(512, 1) k_fft(const __grid_constant__ Plan P, const __grid_constant__ FftArgs a) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  longlong2* s = (longlong2*)fft_smem;
  __shared__ unsigned words[2 * FFT_MAX_PASSES + 4];
  __shared__ unsigned hmax;
  const int col = blockIdx.x / a.R0, s0 = blockIdx.x - col * a.R0;
  const bool blue = !FIRST16 && a.form == FORM_BLUESTEIN;
  if (threadIdx.x < 2 * FFT_MAX_PASSES + 4) words[threadIdx.x] = 0u;
  if (threadIdx.x == 0) hmax = 0u;
  __syncthreads();
  int e, p0 = 0;
  if (!FIRST16 && a.R0 > 1) {
    e = a.ce[col];
    if (e == NO_EXP) {
      nonfinite_column(a, col, s0, fft_smem, (P.n + 7) / 8 * 128);
      return;
    }
    const longlong2* src = a.X + ((long)col * a.R0 + s0) * a.n1;
    Range m;
    for (int l = threadIdx.x; l < a.n1; l += blockDim.x) {
      const longlong2 v = src[l];
      Cx x{v.x, v.y};
      if (blue) {
        const int4 w = __ldg((const int4*)a.c1 + l);
        x = cmul(x, Tw{w.x, w.y, w.z, w.w});
      }
      st(s, l, x);
      m.add(x);
    }
    publish(m, &words[0]);
    if (blue) e += 2;
  } else if (FIRST16) {
    // a thread's sixteen entries stay in registers from global memory through the first pass
    const double* src = a.B + 2 * (long)col * a.ldb;
    const int M = P.n / 16, m0 = threadIdx.x;
    double2 v[16];
    unsigned hm = 0;
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = load_c(src + 2 * (m0 + M * r), a.b16);
#pragma unroll
    for (int r = 0; r < 16; ++r)
      hm = max(hm, max((unsigned)__double2hiint(v[r].x) & 0x7FFFFFFFu, (unsigned)__double2hiint(v[r].y) & 0x7FFFFFFFu));
    hm = __reduce_max_sync(0xffffffffu, hm);
    if ((threadIdx.x & 31) == 0) atomicMax(&hmax, hm);
    __syncthreads();
    const unsigned hmx = hmax;
    if (hmx >= 0x7FF00000u) {
      nonfinite_column(a, col, 0, fft_smem, (P.n + 7) / 8 * 128);
      return;
    }
    const int emax = col_exponent(hmx);
    Cx x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = {fx_from(v[r].x, emax), fx_from(v[r].y, emax)};
    bf<16>(x);
    x[0] = sar(x[0], outer_shift(16));
    const int4* t = (const int4*)(a.tw + P.p[0].tw) + m0;
    const int b0 = sw(m0);
    Range m;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (r > 0) {
        const int4 w = __ldg(t + (r - 1) * M);
        x[r] = cmul(x[r], Tw{w.x, w.y, w.z, w.w});
      }
      s[b0 ^ sw(M * r)] = make_longlong2(x[r].r, x[r].i);
      m.add(x[r]);
    }
    publish(m, &words[1]);
    e = emax - (FFT_TOP - 1) + inner_shift(16) + outer_shift(16);
    p0 = 1;
  } else {
    const double* src = a.B + 2 * (long)col * a.ldb;
    unsigned hm = 0;
    for (int l = threadIdx.x; l < a.n1; l += blockDim.x) {
      const double2 v = load_c(src + 2 * l, a.b16);
      s[sw(l)] = make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y));
      hm = max(hm, max((unsigned)__double2hiint(v.x) & 0x7FFFFFFFu, (unsigned)__double2hiint(v.y) & 0x7FFFFFFFu));
    }
    hm = __reduce_max_sync(0xffffffffu, hm);
    if ((threadIdx.x & 31) == 0) atomicMax(&hmax, hm);
    __syncthreads();
    const unsigned hmx = hmax;
    if (hmx >= 0x7FF00000u) {
      nonfinite_column(a, col, 0, fft_smem, (P.n + 7) / 8 * 128);
      return;
    }
    const int emax = col_exponent(hmx);
    Range m;
    for (int l = threadIdx.x; l < a.n1; l += blockDim.x) {
      const longlong2 v = s[sw(l)];
      Cx x{fx_from(__longlong_as_double(v.x), emax), fx_from(__longlong_as_double(v.y), emax)};
      if (blue) {
        const int4 w = __ldg((const int4*)a.c1 + l);
        x = cmul(x, Tw{w.x, w.y, w.z, w.w});
      }
      st(s, l, x);
      m.add(x);
    }
    publish(m, &words[0]);
    e = emax - (FFT_TOP - 1) + (blue ? 2 : 0);
  }
  // the column that follows on this SM, into L2
  if (a.R0 == 1 && col + a.ahead < a.k) {
    const char* next = (const char*)(a.B + 2 * (long)(col + a.ahead) * a.ldb);
    for (int l = threadIdx.x * 128; l < a.n1 * 16; l += blockDim.x * 128)
      asm volatile("prefetch.global.L2 [%0];\n" ::"l"(next + l));
  }
  if (blue)
    for (int l = a.n1 + threadIdx.x; l < P.n; l += blockDim.x) st(s, l, Cx{0, 0});
  __syncthreads();

  if (!blue) {
    if (P.np == 0) {  // n1 = 1
      if (threadIdx.x == 0) put(a, col, s0, ld(s, 0), e);
      return;
    }
    const int w = forward<FIRST16>(s, P, a.tw, words, p0, P.np - 1, e);
    const int d = headroom(words[w], FFT_TOP);
    e -= d;
    const int R = P.p[P.np - 1].R;
    if (FIRST16 || (P.n & (P.n - 1)) == 0) {
      switch (R) {
        case 16: last_r<16, true>(s, P, a, col, s0, d, e); break;
        case 8: last_r<8, true>(s, P, a, col, s0, d, e); break;
        case 4: last_r<4, true>(s, P, a, col, s0, d, e); break;
        default: last_r<2, true>(s, P, a, col, s0, d, e); break;
      }
      return;
    }
    switch (R) {
      case 12: last_r<12, false>(s, P, a, col, s0, d, e); break;
      case 10: last_r<10, false>(s, P, a, col, s0, d, e); break;
      case 9: last_r<9, false>(s, P, a, col, s0, d, e); break;
      case 8: last_r<8, false>(s, P, a, col, s0, d, e); break;
      case 6: last_r<6, false>(s, P, a, col, s0, d, e); break;
      case 5: last_r<5, false>(s, P, a, col, s0, d, e); break;
      case 4: last_r<4, false>(s, P, a, col, s0, d, e); break;
      case 3: last_r<3, false>(s, P, a, col, s0, d, e); break;
      default: last_r<2, false>(s, P, a, col, s0, d, e); break;
    }
    return;
  }
  if constexpr (FIRST16) return;

  // ---- Bluestein: transform, product with the chirp's, inverse transform (of the swapped parts)
  int w = forward(s, P, a.tw, words, 0, P.np, e);
  {
    const int d = headroom(words[w], 61);
    Range m;
    for (int l = threadIdx.x; l < P.n; l += blockDim.x) {
      const Cx v = ld(s, l);
      const int4 q = __ldg((const int4*)a.bh + l);
      const Cx x = cmul(Cx{v.r << d, v.i << d}, Tw{q.x, q.y, q.z, q.w});
      st(s, l, Cx{x.i, x.r});
      m.add(x);
    }
    publish(m, &words[++w]);
    e += 2 - d + *a.eb;
    __syncthreads();
  }
  for (int p = P.np - 1; p >= 0; --p) {
    const int d = headroom(words[w], 61);
    publish(pass<true, false>(s, P.p[p], P.n, d, a.tw), &words[++w]);
    e += inner_shift(P.p[p].R) + outer_shift(P.p[p].R) - d;
    __syncthreads();
  }
  {
    const int d = headroom(words[w], 61);
    int lg = 0;
    while ((1 << lg) < P.n) ++lg;
    e += 2 - d - (lg - 1);  // c2 carries 2^(lg - 1) / L
    for (int j = threadIdx.x; j < a.n1; j += blockDim.x) {
      const Cx v = ld(s, j);
      const int4 q = __ldg((const int4*)a.c2 + j);
      put(a, col, s0 + a.R0 * j, cmul(Cx{v.i << d, v.r << d}, Tw{q.x, q.y, q.z, q.w}), e);
    }
  }
}

// The transform of the conjugate chirp b_m = exp(+pi i m^2 / n), m = -(n - 1) .. n - 1 wrapped modulo
// L, in the passes' output order, its entries in [-1, 1] as Q62 halves times 2^*eb.
__global__ void __launch_bounds__(512, 1) k_fft_chirp(const __grid_constant__ Plan P, int n1, const Tw* __restrict__ tw,
                                                      const Tw* __restrict__ c1, Tw* __restrict__ bh, int* __restrict__ eb) {
  extern __shared__ __align__(16) unsigned char fft_smem[];
  longlong2* s = (longlong2*)fft_smem;
  __shared__ unsigned words[FFT_MAX_PASSES + 4];
  if (threadIdx.x < FFT_MAX_PASSES + 4) words[threadIdx.x] = 0u;
  __syncthreads();
  Range m;
  for (int l = threadIdx.x; l < P.n; l += blockDim.x) {
    const int q = l < n1 ? l : (P.n - l < n1 ? P.n - l : -1);
    Cx x{0, 0};
    if (q >= 0) {
      const int4 t = __ldg((const int4*)c1 + q);
      const i64 c = (i64)t.x * (1ll << 32) + t.y, sn = (i64)t.z * (1ll << 32) + t.w;
      x = {c >> 4, -(sn >> 4)};  // Q58
    }
    st(s, l, x);
    m.add(x);
  }
  publish(m, &words[0]);
  __syncthreads();
  int e = -58;
  const int w = forward(s, P, tw, words, 0, P.np, e);
  const int d = headroom(words[w], 62);
  for (int l = threadIdx.x; l < P.n; l += blockDim.x) {
    const Cx v = ld(s, l);
    bh[l] = halves(v.r << d, v.i << d);
  }
  if (threadIdx.x == 0) *eb = e - d + 62;  // entries below 2^62: Q62 values in (-1, 1)
}

// Two levels: the columns' exponents, then the radix-R0 pass, X[col][s][m] = w_n^(m s) times the
// butterfly's output s of the R0 entries m + n1 r.
__global__ void __launch_bounds__(256) k_fft_colexp(FftArgs a, int* __restrict__ ce) {
  __shared__ unsigned hmax;
  if (threadIdx.x == 0) hmax = 0u;
  __syncthreads();
  const double* src = a.B + 2 * (long)blockIdx.x * a.ldb;
  unsigned hm = 0;
  for (int l = threadIdx.x; l < a.n; l += blockDim.x) {
    const double2 v = load_c(src + 2 * l, a.b16);
    hm = max(hm, max((unsigned)__double2hiint(v.x) & 0x7FFFFFFFu, (unsigned)__double2hiint(v.y) & 0x7FFFFFFFu));
  }
  hm = __reduce_max_sync(0xffffffffu, hm);
  if ((threadIdx.x & 31) == 0) atomicMax(&hmax, hm);
  __syncthreads();
  if (threadIdx.x == 0)
    ce[blockIdx.x] = hmax >= 0x7FF00000u ? NO_EXP
                                         : col_exponent(hmax) - (FFT_TOP - 1) + inner_shift(a.R0) + outer_shift(a.R0);
}

template <int R>
__global__ void __launch_bounds__(256) k_fft_pass0(FftArgs a, const Tw* __restrict__ tw0, longlong2* __restrict__ X) {
  const int col = blockIdx.x;
  const int ce = a.ce[col];
  if (ce == NO_EXP) return;
  const int emax = ce + (FFT_TOP - 1) - inner_shift(R) - outer_shift(R);
  const double* src = a.B + 2 * (long)col * a.ldb;
  for (int m = blockIdx.y * blockDim.x + threadIdx.x; m < a.n1; m += gridDim.y * blockDim.x) {
    Cx x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double2 v = load_c(src + 2 * ((long)m + (long)a.n1 * r), a.b16);
      x[r] = {fx_from(v.x, emax), fx_from(v.y, emax)};
    }
    bf<R>(x);
    longlong2* dst = X + (long)col * R * a.n1 + m;
    x[0] = sar(x[0], outer_shift(R));
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r > 0) {
        const int4 w = __ldg((const int4*)tw0 + (long)(r - 1) * a.n1 + m);
        x[r] = cmul(x[r], Tw{w.x, w.y, w.z, w.w});
      }
      dst[(long)r * a.n1] = make_longlong2(x[r].r, x[r].i);
    }
  }
}

void launch_pass0(int R, dim3 grid, cudaStream_t s, const FftArgs& a, const Tw* tw0, longlong2* X) {
  switch (R) {
    case 16: k_fft_pass0<16><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 15: k_fft_pass0<15><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 12: k_fft_pass0<12><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 10: k_fft_pass0<10><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 9: k_fft_pass0<9><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 8: k_fft_pass0<8><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 6: k_fft_pass0<6><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 5: k_fft_pass0<5><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 4: k_fft_pass0<4><<<grid, 256, 0, s>>>(a, tw0, X); break;
    case 3: k_fft_pass0<3><<<grid, 256, 0, s>>>(a, tw0, X); break;
    default: k_fft_pass0<2><<<grid, 256, 0, s>>>(a, tw0, X); break;
  }
}

}  // namespace

// Bytes of workspace of the transform route for an n x k DFT, 0 where it does not cover n.
size_t fft_workspace(int n, int k) {
  Route r;
  if (n <= 0 || k <= 0 || !make_route(n, &r) || (long)k * r.R0 >= 0x7FFFFFFFL) return 0;
  return layout(r, k).total;
}

int launch_fft(int n, int k, double alpha, const double* B, long ldb, double beta, double* C, long ldc, bool ieee,
               void* work, size_t lwork, cudaStream_t stream) {
  Route r;
  if (!make_route(n, &r)) return PSMMA_EUNSUPPORTED;
  const Layout L = layout(r, k);
  if (!work || lwork < L.total) return PSMMA_EWORKSPACE;
  char* w = (char*)work;
  Tw* tw = (Tw*)(w + L.off_tw);
  const bool blue = r.form == FORM_BLUESTEIN;
  Tw *c1 = blue ? (Tw*)(w + L.off_c1) : nullptr, *c2 = blue ? (Tw*)(w + L.off_c2) : nullptr;
  Tw* bh = blue ? (Tw*)(w + L.off_bh) : nullptr;
  int* eb = blue ? (int*)(w + L.off_eb) : nullptr;
  Tw* tw0 = r.R0 > 1 ? (Tw*)(w + L.off_tw0) : nullptr;
  FftArgs a;
  memset(&a, 0, sizeof(a));
  a.B = B; a.ldb = ldb; a.C = C; a.ldc = ldc;
  a.n = n; a.k = k; a.n1 = r.n1; a.R0 = r.R0; a.form = r.form;
  a.alpha = alpha; a.beta = beta;
  a.b16 = ((uintptr_t)B & 15) == 0;
  a.c16 = ((uintptr_t)C & 15) == 0;
  a.ieee = ieee;
  a.tw = tw; a.c1 = c1; a.c2 = c2; a.bh = bh; a.eb = eb;
  a.X = r.R0 > 1 ? (const longlong2*)(w + L.off_x) : nullptr;
  a.ce = r.R0 > 1 ? (const int*)(w + L.off_ce) : nullptr;
  const int N = r.plan.n;
  const size_t smem = (size_t)((N + 7) / 8 * 8) * 16;
  // 128 registers a thread: 512 threads fill an SM.  They are shared by the columns whose entries fit
  // its shared memory (8 at most), so that one column's loads and stores overlap another's passes.
  const bool first16 = r.R0 == 1 && !blue && (N & (N - 1)) == 0 && N >= 512 && N <= 8192 && r.plan.p[0].R == 16;
  int cols = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)227 * 1024 / (smem + 2048)));
  int threads = std::max(64, 512 / cols / 32 * 32);
  if (first16) {
    threads = N / 16;
    cols = std::min(cols, 512 / threads);
  }

  prof_begin(stream);
  const int entries = std::max(r.plan.entries, std::max(r.n1, r.R0 > 1 ? (r.R0 - 1) * r.n1 : 0));
  k_fft_tables<<<std::max(1, std::min((entries + 127) / 128, 2048)), 128, 0, stream>>>(r.plan, tw, r.n1, c1, c2, r.R0,
                                                                                     tw0);
  if (blue) {
    if (set_smem_attr(k_fft_chirp, FFT_MAX * 16) != cudaSuccess) return PSMMA_EDEVICE;
    k_fft_chirp<<<1, 512, smem, stream>>>(r.plan, r.n1, tw, c1, bh, eb);
  }
  prof_mark(stream, "dft_tables");
  if (r.R0 > 1) {
    k_fft_colexp<<<k, 256, 0, stream>>>(a, (int*)(w + L.off_ce));
    launch_pass0(r.R0, dim3(k, std::max(1, std::min(64, (r.n1 + 255) / 256))), stream, a, tw0, (longlong2*)(w + L.off_x));
    prof_mark(stream, "dft_first_pass");
  }
  // the attribute is the kernel's, shared by every thread that launches it: one value for all
  if (set_smem_attr(k_fft<true>, FFT_MAX * 16) != cudaSuccess || set_smem_attr(k_fft<false>, FFT_MAX * 16) != cudaSuccess)
    return PSMMA_EDEVICE;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return PSMMA_EDEVICE;
  a.ahead = sms * cols;
  (first16 ? k_fft<true> : k_fft<false>)<<<k * r.R0, threads, smem, stream>>>(r.plan, a);
  prof_mark(stream, "dft_transform");
  return cudaGetLastError() == cudaSuccess ? PSMMA_OK : PSMMA_EDEVICE;
}

}  // namespace psmma
