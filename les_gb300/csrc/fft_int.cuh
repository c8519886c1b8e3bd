// FP64 plane transforms on the integer pipe.
//
// GB300 retires about 1.7 FP64 operations per clock per SM (measured; 108 for
// FP32), so a radix-16 FP64 butterfly costs 5.9 clocks per element and SM.
// These transforms keep every value as a 64-bit integer with one binary
// exponent per row (x pass) or column (y pass): additions are two 32-bit adds
// (58 per clock per SM measured), a product with a twiddle is three
// 32 x 32 -> 64-bit multiply-adds per real product (27 per clock), and the
// same butterfly costs 0.4 clocks.  The FP64 pipe only converts: one
// instruction per value on the way out (1.9 per clock).
//
// Measured against the FP64 kernels (256^2 planes): field and derivatives of
// 64 planes (les_filt_da) 1122 -> 174 us, FP64 step at 256^3 89.0 -> 19.3 ms.
// What bounds them is latency at the warps that fit, not a pipe: of the three
// launches of that les_filt_da the x pass has 14 to 15 warps an SM (128 registers;
// 80 to 96 and 20 warps on other lengths) and issues in 42 and 51 % of the cycles,
// the y pass 27 warps (64 registers, 24 to 476 bytes spilled) and 51 %; the
// integer pipe is 46 to 55 % busy, the FP64 pipe 31 to 42 %, DRAM 15 to 20 %.  The
// x pass in three steps of at most eight values (64 registers, 32 warps) was no
// faster at any length.
//
// Precision.  A value is a multiple of 2^ex with |value / 2^ex| < 2^61, so a
// row's largest elements carry 55 to 60 bits (an FP64 number: 53) and
// all others the same absolute resolution; a transform's error is set by its
// largest inputs in FP64 arithmetic as well.  The scale is chosen from the
// data: from the row's largest exponent at the load, for an inverse from the
// sums of moduli of its first butterflies (a spectrum that one mode dominates
// keeps its full width), and from the largest value between the steps (the
// inverse x pass instead takes the sum of all moduli, which bounds all of it; at
// 384 points the first step's, see RowShape).  Each choice leaves the headroom
// that the following step can need, so nothing overflows.
// Twiddles are rounded to 62 fractional bits, halves in a direction of each row
// and column (FixShift).  Against extended precision, as a share of the FP64
// kernels' relative error, 16 x 64 to 64 x 256, 256^2 and 384 x 32 with their 3/2
// grids: 0.07 to 0.83 in the plane transforms, the field, its derivatives and the
// 3/2 round trip for noise, a mean wind of 130 and of 12000 times the noise,
// smooth fields and fields that fall off along x or along y; a single point 0.17
// to 1.03, its filtered field in rows of 64 by 24 rows 1.34 (2.2 x 2^-53).  The
// largest error of a plane stays within 8 of its rms.
//
// Not-a-number and infinity in a row or column make all of it NaN, as the
// butterflies of an FP64 transform do.  Values below 2^-1042 count as zero.
#pragma once
#include <type_traits>
#include "fft.cuh"

namespace les {

typedef long long i64;
struct cfix {
  i64 x, y;
};

// ---- products ---------------------------------------------------------------
__device__ __forceinline__ i64 mad_w(int a, int b, i64 c) {
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ i64 mad_wu(unsigned a, unsigned b, i64 c) {
  i64 r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
// a = h 2^32 + l with l signed, so that all partial products are signed
struct fsplit {
  int h, l;
  __device__ __forceinline__ explicit fsplit(i64 a)
      : h((int)(a >> 32) + (int)((unsigned)(int)a >> 31)), l((int)a) {}
};
constexpr i64 FIX_ONE = 1ll << 62;   // 1.0 of a multiplier
constexpr i64 FIX_RND = 1ll << 29;   // half of the last kept bit of the cross terms
__host__ __device__ constexpr int fix_lo(i64 c) { return (int)(unsigned)((unsigned long long)c & 0xffffffffull); }
__host__ __device__ constexpr int fix_hi(i64 c) { return (int)((c - (i64)fix_lo(c)) >> 32); }

// a c / 2^62 for |a| < 2^61, |c| <= 2^62: the two high products, rounded
// (the dropped low x low product is below one unit of the result)
__device__ __forceinline__ i64 fmul(i64 a, int ch, int cl) {
  const fsplit p(a);
  const i64 m = mad_w(p.l, ch, mad_w(p.h, cl, FIX_RND));
  return mad_w(p.h << 2, ch, m >> 30);
}
// complex a (w.x + i w.y), |a| < 2^61 in modulus
__device__ __forceinline__ cfix fcmul(cfix a, int rh, int rl, int ih, int il) {
  const fsplit p(a.x), q(a.y);
  const int nh = -ih, nl = -il;
  const i64 m = mad_w(q.l, nh, mad_w(q.h, nl, mad_w(p.l, rh, mad_w(p.h, rl, FIX_RND))));
  const i64 n = mad_w(q.l, rh, mad_w(q.h, rl, mad_w(p.l, ih, mad_w(p.h, il, FIX_RND))));
  const int p4 = p.h << 2, q4 = q.h << 2;
  cfix r;
  r.x = mad_w(q4, nh, mad_w(p4, rh, m >> 30));
  r.y = mad_w(q4, rh, mad_w(p4, ih, n >> 30));
  return r;
}
// twiddle table entry: (re hi, re lo, im hi, im lo)
__device__ __forceinline__ cfix ftw(cfix a, int4 w) { return fcmul(a, w.x, w.y, w.z, w.w); }
__device__ __forceinline__ cfix ftwc(cfix a, int4 w) { return fcmul(a, w.x, w.y, -w.z, -w.w); }

__device__ __forceinline__ cfix fadd(cfix a, cfix b) { a.x += b.x; a.y += b.y; return a; }
__device__ __forceinline__ cfix fsub(cfix a, cfix b) { a.x -= b.x; a.y -= b.y; return a; }
// a / 2, halves to the even neighbour (see FixShift)
__device__ __forceinline__ i64 fhalf(i64 a) { return (a + (i64)(((unsigned)a >> 1) & 1u)) >> 1; }

// ---- constants: cos(2 pi k / 144) in 62 fractional bits -----------------------
__host__ __device__ constexpr i64 fix_cos144(int k) {
  constexpr i64 t[144] = {
    4611686018427387904ll, 4607296715203800411ll, 4594137160821195716ll, 4572232405239281286ll,
    4541624145405292212ll, 4502370645881482257ll, 4454546627935218059ll, 4398243127302799819ll,
    4333567320897763126ll, 4260642322793532497ll, 4179606949868785275ll, 4090615457561633222ll,
    3993837246235628775ll, 3889456538716544935ll, 3777672029613755863ll, 3658696507093754878ll,
    3532756447825785444ll, 3400091585870629178ll, 3260954456333195553ll, 3115609914647596549ll,
    2964334632409774423ll, 2807416570717393844ll, 2645154432019525852ll, 2477857091519558913ll,
    2305843009213693952ll, 2129439623684241497ll, 1948982728801669864ll, 1764815834521887442ll,
    1577289512995517789ll, 1386760731233885708ll, 1193592171602022505ll, 998151541432170641ll,
    800810873071977681ll, 601945815699777620ll, 401934920255029411ll, 201158918845088287ll,
    0ll, -201158918845088287ll, -401934920255029411ll, -601945815699777620ll,
    -800810873071977681ll, -998151541432170641ll, -1193592171602022505ll, -1386760731233885708ll,
    -1577289512995517789ll, -1764815834521887442ll, -1948982728801669864ll, -2129439623684241497ll,
    -2305843009213693952ll, -2477857091519558913ll, -2645154432019525852ll, -2807416570717393844ll,
    -2964334632409774423ll, -3115609914647596549ll, -3260954456333195553ll, -3400091585870629178ll,
    -3532756447825785444ll, -3658696507093754878ll, -3777672029613755863ll, -3889456538716544935ll,
    -3993837246235628775ll, -4090615457561633222ll, -4179606949868785275ll, -4260642322793532497ll,
    -4333567320897763126ll, -4398243127302799819ll, -4454546627935218059ll, -4502370645881482257ll,
    -4541624145405292212ll, -4572232405239281286ll, -4594137160821195716ll, -4607296715203800411ll,
    -4611686018427387904ll, -4607296715203800411ll, -4594137160821195716ll, -4572232405239281286ll,
    -4541624145405292212ll, -4502370645881482257ll, -4454546627935218059ll, -4398243127302799819ll,
    -4333567320897763126ll, -4260642322793532497ll, -4179606949868785275ll, -4090615457561633222ll,
    -3993837246235628775ll, -3889456538716544935ll, -3777672029613755863ll, -3658696507093754878ll,
    -3532756447825785444ll, -3400091585870629178ll, -3260954456333195553ll, -3115609914647596549ll,
    -2964334632409774423ll, -2807416570717393844ll, -2645154432019525852ll, -2477857091519558913ll,
    -2305843009213693952ll, -2129439623684241497ll, -1948982728801669864ll, -1764815834521887442ll,
    -1577289512995517789ll, -1386760731233885708ll, -1193592171602022505ll, -998151541432170641ll,
    -800810873071977681ll, -601945815699777620ll, -401934920255029411ll, -201158918845088287ll,
    0ll, 201158918845088287ll, 401934920255029411ll, 601945815699777620ll,
    800810873071977681ll, 998151541432170641ll, 1193592171602022505ll, 1386760731233885708ll,
    1577289512995517789ll, 1764815834521887442ll, 1948982728801669864ll, 2129439623684241497ll,
    2305843009213693952ll, 2477857091519558913ll, 2645154432019525852ll, 2807416570717393844ll,
    2964334632409774423ll, 3115609914647596549ll, 3260954456333195553ll, 3400091585870629178ll,
    3532756447825785444ll, 3658696507093754878ll, 3777672029613755863ll, 3889456538716544935ll,
    3993837246235628775ll, 4090615457561633222ll, 4179606949868785275ll, 4260642322793532497ll,
    4333567320897763126ll, 4398243127302799819ll, 4454546627935218059ll, 4502370645881482257ll,
    4541624145405292212ll, 4572232405239281286ll, 4594137160821195716ll, 4607296715203800411ll,
  };
  return t[((k % 144) + 144) % 144];
}
template <int K> struct FixCos { static constexpr i64 v = fix_cos144(K); };
template <int K> struct FixSin { static constexpr i64 v = fix_cos144(K - 36); };

template <int I, int N, class F> __device__ __forceinline__ void sfor(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    sfor<I + 1, N>(static_cast<F&&>(f));
  }
}
// a exp(SIGN 2 pi i K / N)
template <int K, int N, int SIGN> __device__ __forceinline__ cfix frot(cfix a) {
  static_assert(144 % N == 0, "table");
  constexpr int k = K * (144 / N);
  constexpr i64 R = FixCos<k>::v, I = SIGN * FixSin<k>::v;
  cfix r;
  if constexpr (R == FIX_ONE) {
    r = a;
  } else if constexpr (R == -FIX_ONE) {
    r.x = -a.x; r.y = -a.y;
  } else if constexpr (I == FIX_ONE) {
    r.x = -a.y; r.y = a.x;
  } else if constexpr (I == -FIX_ONE) {
    r.x = a.y; r.y = -a.x;
  } else if constexpr (R == I) {  // an eighth turn: two real products
    r.x = fmul(a.x - a.y, fix_hi(R), fix_lo(R));
    r.y = fmul(a.x + a.y, fix_hi(R), fix_lo(R));
  } else if constexpr (R == -I) {
    r.x = fmul(a.x + a.y, fix_hi(R), fix_lo(R));
    r.y = fmul(a.y - a.x, fix_hi(R), fix_lo(R));
  } else {
    r = fcmul(a, fix_hi(R), fix_lo(R), fix_hi(I), fix_lo(I));
  }
  return r;
}

// ---- butterflies: natural-order DFT of N values in registers -------------------
template <int N> struct FixSplit;  // N = A * B
template <> struct FixSplit<6> { static constexpr int a = 2, b = 3; };
template <> struct FixSplit<8> { static constexpr int a = 2, b = 4; };
template <> struct FixSplit<9> { static constexpr int a = 3, b = 3; };
template <> struct FixSplit<12> { static constexpr int a = 4, b = 3; };
template <> struct FixSplit<16> { static constexpr int a = 4, b = 4; };
template <> struct FixSplit<24> { static constexpr int a = 8, b = 3; };

template <int N, int SIGN> __device__ __forceinline__ void fdft(cfix* v) {
  if constexpr (N == 2) {
    const cfix a = v[0], b = v[1];
    v[0] = fadd(a, b);
    v[1] = fsub(a, b);
  } else if constexpr (N == 3) {
    const cfix a = v[0], s = fadd(v[1], v[2]), d = fsub(v[1], v[2]);
    constexpr i64 S3 = FixSin<48>::v;  // sin(2 pi / 3)
    cfix m, r;
    m.x = a.x - fhalf(s.x);
    m.y = a.y - fhalf(s.y);
    const i64 rx = fmul(d.x, fix_hi(S3), fix_lo(S3)), ry = fmul(d.y, fix_hi(S3), fix_lo(S3));
    r.x = SIGN < 0 ? ry : -ry;   // SIGN i sin(..) d
    r.y = SIGN < 0 ? -rx : rx;
    v[0] = fadd(a, s);
    v[1] = fadd(m, r);
    v[2] = fsub(m, r);
  } else if constexpr (N == 4) {
    const cfix t0 = fadd(v[0], v[2]), t1 = fsub(v[0], v[2]), t2 = fadd(v[1], v[3]), d = fsub(v[1], v[3]);
    cfix p, m;  // t1 + i d, t1 - i d
    p.x = t1.x - d.y; p.y = t1.y + d.x;
    m.x = t1.x + d.y; m.y = t1.y - d.x;
    v[0] = fadd(t0, t2);
    v[2] = fsub(t0, t2);
    v[1] = SIGN < 0 ? m : p;
    v[3] = SIGN < 0 ? p : m;
  } else {
    constexpr int A = FixSplit<N>::a, B = FixSplit<N>::b;  // n = a + A b, k = c + B d
    cfix t[A][B];
    sfor<0, A>([&](auto ia) {
      constexpr int a = decltype(ia)::value;
#pragma unroll
      for (int b = 0; b < B; ++b) t[a][b] = v[a + A * b];
      fdft<B, SIGN>(t[a]);
      sfor<1, B>([&](auto ic) {
        constexpr int c = decltype(ic)::value;
        t[a][c] = frot<a * c, N, SIGN>(t[a][c]);
      });
    });
    sfor<0, B>([&](auto ic) {
      constexpr int c = decltype(ic)::value;
      cfix u[A];
#pragma unroll
      for (int a = 0; a < A; ++a) u[a] = t[a][c];
      fdft<A, SIGN>(u);
#pragma unroll
      for (int d = 0; d < A; ++d) v[c + B * d] = u[d];
    });
  }
}
// components below 2^fix_in(N) keep an N-point DFT's values below 2^61 in
// modulus: N sqrt(2) 2^bits < 2^61
__host__ __device__ constexpr int fix_in(int n) {
  int b = 60;
  // 2 n^2 < 4^(61 - b)
  while (2ll * n * n >= (1ll << (2 * (61 - b)))) --b;
  return b;
}

// ---- conversions ---------------------------------------------------------------
constexpr int FIX_TINY = 61 << 20;      // high word of the smallest exponent the direct scaling takes
constexpr int FIX_PRE = 800;            // exponent added to rows below it
__device__ __forceinline__ unsigned fix_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// exponent of the scale that brings values of high-word magnitude up to m
// below 2^bits (0 for a zero row, which stays zero)
__device__ __forceinline__ int fix_shift(unsigned m, int bits) { return m ? bits + 1022 - (int)(m >> 20) : 0; }
// x 2^s, truncated, on the integer pipe (the FP64 pipe's conversion would
// bound these kernels: 81 % busy with it).  c = 1082 - s; the scale keeps the
// result below 2^60, and zeros and subnormals fall to zero by their exponent.
__device__ __forceinline__ i64 fix_of(double x, int c) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int d = min(c - (int)((hi >> 20) & 0x7ffu), 63);
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  m = (m << 7) >> d;
  const i64 sg = (i64)((int)hi >> 31);
  return ((i64)m ^ sg) - sg;
}
// x k 2^s for an integer k < 2^8 (the product is exact before the
// truncation); e1 = 1078 - s, the result below 2^57
__device__ __forceinline__ i64 fix_times(double x, unsigned k, int e1) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int d = min(e1 - (int)((hi >> 20) & 0x7ffu), 63);
  unsigned long long m = (unsigned long long)mad_wu(lo, k, 0) +
                         ((unsigned long long)(((hi & 0xfffffu) | 0x100000u) * k) << 32);
  m = (m << 3) >> d;
  const i64 sg = (i64)((int)hi >> 31);
  return ((i64)m ^ sg) - sg;
}
__device__ __forceinline__ double fix_pow2(int e) {  // 2^e, -1022 <= e <= 1023
  return __hiloint2double((e + 1023) << 20, 0);
}
// v 2^ex factor for N pairs, in place of the integers.  A power of two joins
// the exponent, so that the FP64 pipe has the conversion alone; any other
// factor costs one product more (two near the ends of the FP64 range).
template <int N, int NV>
__device__ __forceinline__ void fix_out(const cfix (&v)[NV], double2 (&o)[N], int ex, double factor) {
  const int fh = __double2hiint(factor);
  if (__double2loint(factor) == 0 && (fh & 0x800fffff) == 0 && fh >= (1 << 20)) {
    ex += (fh >> 20) - 1023;
    factor = 1.0;
  }
  const int e1 = min(max(ex, -960), 900);
  if (factor == 1.0 && e1 == ex) {
    const int e20 = ex * (1 << 20);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      o[i].x = __ll2double_rn(v[i].x);
      o[i].y = __ll2double_rn(v[i].y);
      const int hx = __double2hiint(o[i].x), hy = __double2hiint(o[i].y);
      o[i].x = __hiloint2double(hx ? hx + e20 : 0, __double2loint(o[i].x));
      o[i].y = __hiloint2double(hy ? hy + e20 : 0, __double2loint(o[i].y));
    }
  } else {
    const double f1 = factor * fix_pow2(e1);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      o[i].x = __ll2double_rn(v[i].x) * f1;
      o[i].y = __ll2double_rn(v[i].y) * f1;
    }
    if (e1 != ex) {
      const double f2 = fix_pow2(min(max(ex - e1, -1022), 1023));
#pragma unroll
      for (int i = 0; i < N; ++i) { o[i].x *= f2; o[i].y *= f2; }
    }
  }
}
__device__ __forceinline__ double nan_if(bool bad, double f) {
  return bad ? __longlong_as_double(0x7ff8000000000000ll) : f;
}
// A right shift (0 <= s < 31) with rounding, halves up or, where `down`, down.  The
// values often end in zeros (53 bits of 60), so halves are frequent, and rounded
// the same way throughout they add up in one place: forward in the modes that
// all rows share (a mean wind's ky = 0: 1.2e-13 of the pressure at 96 x 64
// instead of 2.6e-14), inverse at x = y = 0 (50 eps of the field's rms in planes of
// 288 x 384 instead of 8; the FP64 kernels 12).  So each row, column and, where
// the loss is largest, element has its own direction, which costs no operation
// per element; to the even neighbour takes two (the 3/2 round trip 2.8 % slower).
__device__ __forceinline__ bool fix_coin(unsigned x) {
  x *= 0x9e3779b1u;
  x ^= x >> 15;
  return (int)(x * 0x9e3779b1u) < 0;
}
struct FixShift {
  int s;
  unsigned rnd;
  __device__ __forceinline__ FixShift(int s_, bool down) : s(s_), rnd((1u << s_) >> 1) {
    if (down && s_ > 0) --rnd;
  }
  __device__ __forceinline__ i64 operator()(i64 v) const { return (v + (i64)(unsigned long long)rnd) >> s; }
};
__device__ __forceinline__ unsigned fix_top(i64 v) {  // magnitude of the high word (one's complement)
  const int h = (int)(v >> 32);
  return (unsigned)(h ^ (h >> 31));
}
// right shift that brings values of high-word magnitude m below 2^bits
__device__ __forceinline__ int fix_down(unsigned m, int bits) { return max(64 - __clz((int)m) - bits, 0); }
// the same for a sum of moduli below sum 2^unit, to below 2^60
__device__ __forceinline__ int fix_down_sum(unsigned sum, int unit) { return max(32 - __clz((int)sum) + unit - 60, 0); }
// a bound on |x| + |y| in units of 2^(32 + SH)
template <int SH> __device__ __forceinline__ unsigned fix_l1(cfix v) {
  return ((fix_top(v.x) + fix_top(v.y) + 2u) >> SH) + 1u;
}

}  // namespace les
