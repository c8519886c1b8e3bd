// FP64 y pass (cols) on the integer pipe; see fft_int.cuh.
//
// TX columns per block, a column of N = R1 R2 R3 rows served by TT threads.  Rows
// n = n1 + (N / R1) n2: the thread of job n1 holds the R1 rows over n2 and makes
// the first butterflies; then R1 transforms of N / R1 points are left, done in
// one step (R3 = 1) or two (R2, then R3), with an exchange through shared memory
// before each step (the middle step reads and writes its own slots).  The
// spectral side holds k = j + J k1 the same way.  The inverse runs the steps
// backwards.  With steps of at most 8 values a thread makes do with 64 registers,
// so that 32 warps fit an SM to hide the latency that bounds the pass, at the
// price of spills: 24 to 476 bytes a thread at 256 rows, up to 512 at 192 and 384
// (both directions) and 20 to 544 in the 3/2 passes.  Two steps of 16 (128
// registers, 16 warps) against three, when the shapes were chosen: les_filt_da on
// 64 planes of 256^2 189 against 172 us, 3/2 round trip of 32 planes of 192^2 165
// against 145 us, FP64 step at 256^3 20.0 against 19.5 ms; 24 warps instead of 32
// (no spills) 20.6 ms.  Columns are numbered through all levels, so that only the
// last block of a launch has idle ones.
//
// Outputs that only drop the Nyquist row (filt_da's field) or multiply by
// the column's kx need no transform at all in y: the field less its
// alternating sum, sum_y (-1)^y f / ny, is what the round trip gives.  They are
// written last, from the input again (cached), so that no register holds it.
#include <algorithm>
#include "fft_int.cuh"
#include "les_internal.h"

namespace les {
namespace {

constexpr int ICOL_TX = 8;
constexpr int ICOL_SLOTS = 4 + 2 * COL_MAXO;

// largest m of the column (all threads of the block take part)
template <int TX> __device__ __forceinline__ unsigned col_max(unsigned m, unsigned* slot, int b) {
#pragma unroll
  for (int o = TX; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) < TX) atomicMax(slot + b, m);
  __syncthreads();
  return slot[b];
}
// sum over the column's threads of a pair of integers
template <int TX> __device__ __forceinline__ void col_sum(i64& sx, i64& sy, i64* slot, int b) {
#pragma unroll
  for (int o = TX; o < 32; o <<= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
  }
  if ((threadIdx.x & 31) < TX) {
    atomicAdd(reinterpret_cast<unsigned long long*>(slot + 2 * b), (unsigned long long)sx);
    atomicAdd(reinterpret_cast<unsigned long long*>(slot + 2 * b + 1), (unsigned long long)sy);
  }
  __syncthreads();
  sx = slot[2 * b];
  sy = slot[2 * b + 1];
}
// the column's scale: x to integers below 2^bits; returns the exponent of one
// unit.  slots: two rows of TX words.
template <int TX, int CNT, int NV>
__device__ __forceinline__ int col_fix(double2 (&x)[NV], cfix (&v)[NV], unsigned* slots, int b, int bits, bool& bad) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < CNT; ++i) m = max(m, max(fix_mag(x[i].x), fix_mag(x[i].y)));
  const unsigned lm = m;
#pragma unroll
  for (int o = TX; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) < TX) atomicMax(slots + b, m);
  const int tiny = __syncthreads_or(lm != 0u && lm < (unsigned)FIX_TINY);
  m = slots[b];
  int pre = 0;
  if (tiny) {  // some value is near the smallest FP64 exponents
    if (m != 0u && m < (unsigned)FIX_TINY) {
      pre = FIX_PRE;
      const double f = fix_pow2(FIX_PRE);
#pragma unroll
      for (int i = 0; i < CNT; ++i) { x[i].x *= f; x[i].y *= f; }
    }
    m = 0;
#pragma unroll
    for (int i = 0; i < CNT; ++i) m = max(m, max(fix_mag(x[i].x), fix_mag(x[i].y)));
    m = col_max<TX>(m, slots + TX, b);
  }
  const int s = fix_shift(m, bits), c = 1082 - s;
  bad = bad || m >= 0x7ff00000u;
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    v[i].x = fix_of(x[i].x, c);
    v[i].y = fix_of(x[i].y, c);
  }
  return -s - pre;
}

constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }
constexpr int clog2(int n) { int b = 0; while ((1 << b) < n) ++b; return b; }
constexpr int cmax(int a, int b) { return a > b ? a : b; }
template <int R1_, int R2_, int R3_, int TT_> struct ColShape {
  static constexpr int R1 = R1_, R2 = R2_, R3 = R3_, TT = TT_, N = R1 * R2 * R3;
  static constexpr int N1 = N / R1, JA = cdiv(N1, TT);                     // physical side: jobs, jobs a thread
  static constexpr int NB = R1 * R3, JB = cdiv(NB, TT);                    // middle (or, R3 = 1, last) step
  static constexpr int SJ = R3 > 1 ? R1 * R2 : R1, SR = R3 > 1 ? R3 : R2;  // spectral side: k = job + SJ i, i < SR
  static constexpr int JS = cdiv(SJ, TT);
  static constexpr int PE = JA * R1, SE = JS * SR, E = cmax(PE, cmax(SE, JB * R2));
  static_assert(N1 % 2 == 0 && TT % 2 == 0 && SR % 2 == 0, "row parity by thread, sign of ky by element");
  // shift of the alternating sum's terms: N of them below 2^fix_in(R1) (strictly:
  // multiples of 2^(fix_in(R1) - 53)) stay below 2^63.  3 for 288 and 384 rows, else 2.
  static constexpr int ALT = cmax(2, clog2(N) + fix_in(R1) - 63);
  static_assert(clog2(N) + fix_in(R1) - ALT <= 63, "alternating sum");
};
// slot of element p of the sub-transform k2
template <class P, int TX> __device__ __forceinline__ int col_at(int k2, int p, int b) { return (k2 * P::N1 + p) * TX + b; }

// forward: v[j R1 + i] = x[(q + TT j) + N1 i], components below 2^fix_in(R1),
// to v[j SR + i] = X[(q + TT j) + SJ i].  The scale is taken again before each
// step: headroom for 64 points at once would cost a column that one row
// dominates three bits.  slot: two rows of TX words.
template <class P, int TX, int NV>
__device__ __forceinline__ void col_fwd(cfix (&v)[NV], cfix* S, unsigned* slot, const int4* __restrict__ tw, int q, int b, bool coin,
                                        int& ex) {
  constexpr int R1 = P::R1, R2 = P::R2, R3 = P::R3, TT = P::TT;
  unsigned top = 0;
#pragma unroll
  for (int j = 0; j < P::JA; ++j) {
    const int n1 = q + TT * j;
    if (n1 < P::N1) {
      fdft<R1, -1>(v + j * R1);
#pragma unroll
      for (int i = 0; i < R1; ++i) {
        cfix a = v[j * R1 + i];
        if (i > 0) a = ftw(a, __ldg(&tw[n1 * i]));
        top = max(top, max(fix_top(a.x), fix_top(a.y)));
        S[col_at<P, TX>(i, n1, b)] = a;
      }
    }
  }
  if constexpr (R3 > 1) {
    const FixShift s1(fix_down(col_max<TX>(top, slot, b), fix_in(R2)), coin);
    ex += s1.s;
    slot += TX;
    top = 0;
#pragma unroll
    for (int j = 0; j < P::JB; ++j) {
      const int t = q + TT * j, k2 = t / R3, m1 = t - k2 * R3;
      if (t < P::NB) {
        cfix w[R2];
#pragma unroll
        for (int i = 0; i < R2; ++i) {
          const cfix a = S[col_at<P, TX>(k2, m1 + R3 * i, b)];
          w[i].x = s1(a.x);
          w[i].y = s1(a.y);
        }
        fdft<R2, -1>(w);
#pragma unroll
        for (int i = 0; i < R2; ++i) {
          if (i > 0) w[i] = ftw(w[i], __ldg(&tw[m1 * i * R1]));
          top = max(top, max(fix_top(w[i].x), fix_top(w[i].y)));
          S[col_at<P, TX>(k2, m1 + R3 * i, b)] = w[i];
        }
      }
    }
  }
  const FixShift s(fix_down(col_max<TX>(top, slot, b), fix_in(P::SR)), coin);
  ex += s.s;
#pragma unroll
  for (int j = 0; j < P::JS; ++j) {
    const int t = q + TT * j;
    if (t < P::SJ) {
      const int k2 = R3 > 1 ? t % R1 : t, l2 = R3 > 1 ? t / R1 : 0;
#pragma unroll
      for (int i = 0; i < P::SR; ++i) {
        const cfix a = S[col_at<P, TX>(k2, R3 * l2 + i, b)];
        v[j * P::SR + i].x = s(a.x);
        v[j * P::SR + i].y = s(a.y);
      }
      fdft<P::SR, -1>(v + j * P::SR);
    }
  }
}
// inverse: from v[j SR + i] = X[(q + TT j) + SJ i] with sums of moduli that stay
// below 2^60 up to the last step (col_weigh), to v[j R1 + i] = x[(q + TT j) + N1 i]
template <class P, int TX, int NV>
__device__ __forceinline__ void col_inv(cfix (&v)[NV], cfix* S, unsigned* slot, const int4* __restrict__ tw, int q, int b, bool coin,
                                        int& ex) {
  constexpr int R1 = P::R1, R2 = P::R2, R3 = P::R3, TT = P::TT;
  unsigned top = 0;
#pragma unroll
  for (int j = 0; j < P::JS; ++j) {
    const int t = q + TT * j;
    if (t < P::SJ) {
      const int k2 = R3 > 1 ? t % R1 : t, l2 = R3 > 1 ? t / R1 : 0;
      fdft<P::SR, 1>(v + j * P::SR);
#pragma unroll
      for (int i = 0; i < P::SR; ++i) {
        cfix a = v[j * P::SR + i];
        if (i > 0) a = ftwc(a, __ldg(&tw[R3 > 1 ? i * l2 * R1 : i * k2]));
        if (R3 == 1) top = max(top, max(fix_top(a.x), fix_top(a.y)));
        S[col_at<P, TX>(k2, R3 * l2 + i, b)] = a;
      }
    }
  }
  if constexpr (R3 > 1) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < P::JB; ++j) {
      const int t = q + TT * j, k2 = t / R3, m1 = t - k2 * R3;
      if (t < P::NB) {
        cfix w[R2];
#pragma unroll
        for (int i = 0; i < R2; ++i) w[i] = S[col_at<P, TX>(k2, m1 + R3 * i, b)];
        fdft<R2, 1>(w);
#pragma unroll
        for (int i = 0; i < R2; ++i) {
          w[i] = ftwc(w[i], __ldg(&tw[(m1 + R3 * i) * k2]));
          top = max(top, max(fix_top(w[i].x), fix_top(w[i].y)));
          S[col_at<P, TX>(k2, m1 + R3 * i, b)] = w[i];
        }
      }
    }
  }
  const FixShift s(fix_down(col_max<TX>(top, slot, b), fix_in(R1)), coin);
  ex += s.s;
#pragma unroll
  for (int j = 0; j < P::JA; ++j) {
    const int n1 = q + TT * j;
    if (n1 < P::N1) {
#pragma unroll
      for (int i = 0; i < R1; ++i) {
        const cfix a = S[col_at<P, TX>(i, n1, b)];
        v[j * R1 + i].x = s(a.x);
        v[j * R1 + i].y = s(a.y);
      }
      fdft<R1, 1>(v + j * R1);
    }
  }
}
// w(k) v with integer weights, 0 or 1, or (sgn) |ky| as an integer, negative
// wavenumbers (i >= SR/2) changing sign, scaled so that the sums of moduli of
// col_inv's steps before its own scaling stay below 2^60: a job's sum (SR values of
// at most 2^18 units of 2^44, weights up to N/2: below 2^31 units), times R2 where
// a second step follows.  The products are exact 96-bit integers before the shift.
// coin: the direction of halves (FixShift).
template <class P, int TX, int NV>
__device__ __forceinline__ void col_weigh(cfix (&v)[NV], const unsigned (&w)[P::SE], bool sgn, unsigned* slot, int b, bool coin,
                                          int& ex) {
  static_assert(P::SR * (P::N / 2) < 1 << 13, "a job's sum of moduli");
  unsigned sum = 0;
#pragma unroll
  for (int j = 0; j < P::JS; ++j) {
    unsigned t = 0;
#pragma unroll
    for (int i = 0; i < P::SR; ++i)
      if (w[j * P::SR + i]) t += fix_l1<12>(v[j * P::SR + i]) * w[j * P::SR + i];
    sum = max(sum, t);
  }
  const int s = fix_down_sum(col_max<TX>(sum, slot, b), 44 + (P::R3 > 1 ? clog2(P::R2) : 0));
  const FixShift f[2] = {FixShift(s, coin), FixShift(s, !coin)};  // of the elements: 0 1 1 0 1 0 0 1 ...
  const i64 flip = sgn ? -1 : 0;
  ex += s;
#pragma unroll
  for (int e = 0; e < P::SE; ++e) {
    const int c = (e ^ (e >> 1) ^ (e >> 2) ^ (e >> 3)) & 1;
    const i64 lx = mad_wu((unsigned)v[e].x, w[e], (i64)(unsigned long long)f[c].rnd);
    const i64 ly = mad_wu((unsigned)v[e].y, w[e], (i64)(unsigned long long)f[1 - c].rnd);
    const i64 hx = mad_w((int)(v[e].x >> 32), (int)w[e], (i64)((unsigned long long)lx >> 32));
    const i64 hy = mad_w((int)(v[e].y >> 32), (int)w[e], (i64)((unsigned long long)ly >> 32));
    // (h 2^32 + low word) >> s, s < 32
    v[e].x = (i64)(((unsigned long long)__funnelshift_r((unsigned)hx, (unsigned)(hx >> 32), s) << 32) |
                   __funnelshift_r((unsigned)lx, (unsigned)hx, s));
    v[e].y = (i64)(((unsigned long long)__funnelshift_r((unsigned)hy, (unsigned)(hy >> 32), s) << 32) |
                   __funnelshift_r((unsigned)ly, (unsigned)hy, s));
    if (e % P::SR >= P::SR / 2) {
      v[e].x = (v[e].x ^ flip) - flip;
      v[e].y = (v[e].y ^ flip) - flip;
    }
  }
}
// wavenumber of element e of a thread's spectral side, N for none
template <class P> __device__ __forceinline__ int col_k(int e, int q) {
  const int job = q + P::TT * (e / P::SR);
  return job < P::SJ ? job + P::SJ * (e % P::SR) : P::N;
}
// weights of ky: |k| or N - |k|, none for the Nyquist row
template <class P> __device__ __forceinline__ void ky_weights(unsigned (&w)[P::SE], int q, bool zero) {
#pragma unroll
  for (int e = 0; e < P::SE; ++e) {
    const int k = col_k<P>(e, q);
    w[e] = zero || k == P::N / 2 || k >= P::N ? 0u : (unsigned)(k < P::N / 2 ? k : P::N - k);
  }
}
// row of element e of a thread's physical side, negative for none
template <class P> __device__ __forceinline__ int col_row(int e, int q) {
  const int job = q + P::TT * (e / P::R1);
  return job < P::N1 ? job + P::N1 * (e % P::R1) : -1;
}
// outputs while the integers stay in use: converted four at a time
template <int CNT, class V, class St>
__device__ __forceinline__ void fix_groups(V&& val, St&& store, int ex, double factor) {
#pragma unroll
  for (int g = 0; g < CNT; g += 4) {
    cfix t[4];
    double2 r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = val(g + i < CNT ? g + i : CNT - 1);
    fix_out(t, r, ex, factor);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (g + i < CNT) store(g + i, r[i]);
  }
}
__device__ __forceinline__ bool col_direct(const ColJob& J, int o) {  // needs no y transform
  const int code = J.coef[o][0];
  return J.dir == DIR_BOTH && ((J.inv_mask >> o) & 1u) && (code == CC_ONE || code == CC_KILL || code == CC_IKX);
}

// One input, same length.  DIR: the job's direction; ngen: inverse outputs
// that need a transform (MULTI: several, the spectrum waits in shared memory).
template <class P, int MB, int DIR, bool MULTI>
__global__ void __launch_bounds__(ICOL_TX * P::TT, MB)
    k_icol(ColJob J, const int4* __restrict__ tw, int total, int ndirect, int nspec, int ngen) {
  pdl_wait();
  constexpr int TX = ICOL_TX, N = P::N, NT = TX * P::TT;
  static_assert(NT % 32 == 0, "whole warps");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  cfix* K = S + N * TX;  // the spectrum, kept for later outputs (MULTI)
  __shared__ unsigned slots[ICOL_SLOTS * TX];
  __shared__ i64 sums[2 * TX];
  for (int t = threadIdx.x; t < ICOL_SLOTS * TX; t += NT) slots[t] = 0;
  if (threadIdx.x < 2 * TX) sums[threadIdx.x] = 0;
  const int b = threadIdx.x % TX, q = threadIdx.x / TX;
  const int col = blockIdx.x * TX + b;
  const bool ok = col < total;
  const int lev = ok ? col / J.ncols : 0, jx = ok ? col - lev * J.ncols : 0;
  const size_t in0 = (size_t)lev * J.ps_in + (size_t)blockIdx.y * J.fs_in + jx;
  const size_t out0 = (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
  const double2* src = reinterpret_cast<const double2*>(J.in[0]) + in0;
  constexpr bool fwd = (DIR & DIR_FWD) != 0;
  const bool last = jx == J.lh - 1;  // kx = nx/2: removed by KILL and by the derivatives
  const bool coin = fix_coin((unsigned)(jx * P::TT + q));
  cfix v[P::E];
  int ex;
  bool bad = false;
  {
    double2 x[P::E];
    constexpr int cnt = fwd ? P::PE : P::SE;
#pragma unroll
    for (int e = 0; e < cnt; ++e) {
      const int row = fwd ? col_row<P>(e, q) : col_k<P>(e, q);
      x[e] = make_double2(0.0, 0.0);
      if (ok && row >= 0 && row < N) x[e] = src[(size_t)row * J.wc_in];
    }
    if (DIR == DIR_INV && !MULTI && q == 0) {  // row 0 has no part in i ky: it must not set the scale
      const int code = J.coef[0][0];
      if ((code == CC_IKY || code == CC_MIKY) && max(fix_mag(x[0].x), fix_mag(x[0].y)) < 0x7ff00000u)
        x[0] = make_double2(0.0, 0.0);
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, cnt>(x, v, slots, b, fwd ? fix_in(P::R1) : 60, bad);
  }
  double ax = 0.0, ay = 0.0;  // (-1)^row times the alternating sum
  if (DIR == DIR_BOTH && ndirect) {
    constexpr int SH = P::ALT;
    constexpr i64 SR = 1ll << (SH - 1);
    i64 sx = 0, sy = 0;
#pragma unroll
    for (int e = 0; e < P::PE; ++e) { sx += (v[e].x + SR) >> SH; sy += (v[e].y + SR) >> SH; }
    if (q & 1) { sx = -sx; sy = -sy; }
    col_sum<TX>(sx, sy, sums, b);
    if (q & 1) { sx = -sx; sy = -sy; }
    const cfix t[1] = {{sx, sy}};
    double2 r[1];
    fix_out(t, r, ex + SH, 1.0);
    ax = nan_if(bad, r[0].x);
    ay = nan_if(bad, r[0].y);
  }
  auto direct = [&]() {
    if (DIR != DIR_BOTH || ndirect == 0 || !ok) return;
    for (int o = 0; o < J.nout; ++o) {
      if (!col_direct(J, o)) continue;
      const int code = J.coef[o][0];
      const bool one = code == CC_ONE, ikx = code == CC_IKX;
      const double f = !one && last ? 0.0 : (ikx ? J.kx[jx] : 1.0);
      const double fn = f * (double)N, bx = one ? 0.0 : f * ax, by = one ? 0.0 : f * ay;
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
#pragma unroll
      for (int e = 0; e < P::PE; ++e) {  // N f - (-1)^row sum, from the input again
        const int row = col_row<P>(e, q);
        if (row >= 0) {
          const double2 a = src[(size_t)row * J.wc_in];
          const double rx = fma(fn, a.x, -bx), ry = fma(fn, a.y, -by);
          dst[(size_t)row * J.wc_out] = ikx ? make_double2(-ry, rx) : make_double2(rx, ry);
        }
      }
    }
  };
  if (nspec + ngen == 0) {
    direct();
    return;
  }
  if constexpr (fwd) col_fwd<P, TX>(v, S, slots + 2 * TX, tw, q, b, coin, ex);
  if (DIR != DIR_INV && nspec && ok) {
    for (int o = 0; o < J.nout; ++o) {
      if ((J.inv_mask >> o) & 1u) continue;
      const bool kill = J.coef[o][0] == CC_KILL;
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
      fix_groups<P::SE>([&](int e) { return v[e]; }, [&](int e, double2 r) {
        const int k = col_k<P>(e, q);
        if (k < N) dst[(size_t)k * J.wc_out] = kill && k == N / 2 ? make_double2(0.0, 0.0) : r;
      }, ex, kill && last ? 0.0 : nan_if(bad, 1.0));
    }
  }
  if (DIR == DIR_FWD || ngen == 0) {
    direct();
    return;
  }
  const int ex0 = ex;
  auto output = [&](int o) {
    const int code = J.coef[o][0];
    unsigned* so = slots + (4 + 2 * o) * TX;
    double f = 1.0;
    const bool iky = code == CC_IKY || code == CC_MIKY, rot = iky || code == CC_IKX;
    unsigned w[P::SE];
    if (iky) {
      f = code == CC_IKY ? J.ky[J.lh] : -J.ky[J.lh];  // row 1: the unit of ky
      ky_weights<P>(w, q, last);
    } else if (code == CC_ONE || code == CC_KILL || code == CC_IKX) {
      if (code == CC_IKX) f = J.kx[jx];
#pragma unroll
      for (int e = 0; e < P::SE; ++e) {
        const int k = col_k<P>(e, q);
        w[e] = k >= N || (code != CC_ONE && (last || k == N / 2)) ? 0u : 1u;
      }
    } else {  // cutoff filters: pass or drop, one common factor
      const bool wide = code == CC_G || code == CC_MASK;
      const float* T = wide ? J.Gf : J.GGf;
      if (code == CC_G || code == CC_GG) f = (wide ? J.G : J.GG)[0];
#pragma unroll
      for (int e = 0; e < P::SE; ++e) {
        const int k = col_k<P>(e, q);
        w[e] = k >= N || __ldg(&T[(size_t)J.lh * k + jx]) == 0.f ? 0u : 1u;
      }
    }
    col_weigh<P, TX>(v, w, iky, so, b, coin, ex);
    col_inv<P, TX>(v, S, so + TX, tw, q, b, coin, ex);
    if (ok) {
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
      double2 r[P::PE];
      fix_out(v, r, ex, nan_if(bad, f));
#pragma unroll
      for (int e = 0; e < P::PE; ++e) {
        const int row = col_row<P>(e, q);
        if (row >= 0) dst[(size_t)row * J.wc_out] = make_double2(rot ? -r[e].y : r[e].x, rot ? r[e].x : r[e].y);
      }
    }
  };
  auto general = [&](int o) { return ((J.inv_mask >> o) & 1u) && !col_direct(J, o); };
  if constexpr (MULTI) {
#pragma unroll
    for (int e = 0; e < P::SE; ++e) K[(e * P::TT + q) * TX + b] = v[e];
    for (int o = 0; o < J.nout; ++o) {
      if (!general(o)) continue;
#pragma unroll
      for (int e = 0; e < P::SE; ++e) v[e] = K[(e * P::TT + q) * TX + b];
      ex = ex0;
      output(o);
    }
  } else {
    int o = 0;
    while (o + 1 < J.nout && !general(o)) ++o;
    output(o);
  }
  direct();
}

// i kx in0 + i ky in1 (the horizontal divergences): in1 makes the round trip;
// in0 needs none, only its Nyquist row removed, and is added on the way out.
template <class P, int MB>
__global__ void __launch_bounds__(ICOL_TX * P::TT, MB) k_icol_div(ColJob J, const int4* __restrict__ tw, int total) {
  pdl_wait();
  constexpr int TX = ICOL_TX, N = P::N, NT = TX * P::TT, NW = NT / 32;
  static_assert(NT % 32 == 0, "whole warps");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  __shared__ unsigned slots[6 * TX];
  __shared__ double2 part[NW * TX];
  for (int t = threadIdx.x; t < 6 * TX; t += NT) slots[t] = 0;
  const int b = threadIdx.x % TX, q = threadIdx.x / TX;
  const int col = blockIdx.x * TX + b;
  const bool ok = col < total;
  const int lev = ok ? col / J.ncols : 0, jx = ok ? col - lev * J.ncols : 0;
  const size_t in0 = (size_t)lev * J.ps_in + (size_t)blockIdx.y * J.fs_in + jx;
  const double2* sx = reinterpret_cast<const double2*>(J.in[0]) + in0;
  const double2* sy = reinterpret_cast<const double2*>(J.in[1]) + in0;
  cfix v[P::E];
  int ex;
  bool bad = false;
  {
    double2 x[P::E];
    double ax = 0.0, ay = 0.0;  // alternating sum of in0
#pragma unroll
    for (int e = 0; e < P::PE; ++e) {
      const int row = col_row<P>(e, q);
      x[e] = ok && row >= 0 ? sx[(size_t)row * J.wc_in] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int e = 0; e < P::PE; ++e) { ax += x[e].x; ay += x[e].y; }
    if (q & 1) { ax = -ax; ay = -ay; }
#pragma unroll
    for (int o = TX; o < 32; o <<= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    if ((threadIdx.x & 31) < TX) part[(threadIdx.x >> 5) * TX + b] = make_double2(ax, ay);
#pragma unroll
    for (int e = 0; e < P::PE; ++e) {
      const int row = col_row<P>(e, q);
      x[e] = ok && row >= 0 ? sy[(size_t)row * J.wc_in] : make_double2(0.0, 0.0);
    }
    __syncthreads();  // slots are zero, partial sums are written
    ex = col_fix<TX, P::PE>(x, v, slots, b, fix_in(P::R1), bad);
  }
  const bool coin = fix_coin((unsigned)(jx * P::TT + q));
  col_fwd<P, TX>(v, S, slots + 2 * TX, tw, q, b, coin, ex);
  const bool last = jx == J.lh - 1;
  {
    unsigned w[P::SE];
    ky_weights<P>(w, q, last);
    col_weigh<P, TX>(v, w, true, slots + 4 * TX, b, coin, ex);
  }
  col_inv<P, TX>(v, S, slots + 5 * TX, tw, q, b, coin, ex);
  if (!ok) return;
  double cx = 0.0, cy = 0.0;
#pragma unroll
  for (int w = 0; w < NW; ++w) { cx += part[w * TX + b].x; cy += part[w * TX + b].y; }
  const double kx = last ? 0.0 : J.kx[jx], kn = kx * (double)N;
  cx *= q & 1 ? -kx : kx;
  cy *= q & 1 ? -kx : kx;
  double2* dst = reinterpret_cast<double2*>(J.out[0]) + (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
  double2 r[P::PE];
  fix_out(v, r, ex, nan_if(bad, J.ky[J.lh]));
#pragma unroll
  for (int e = 0; e < P::PE; ++e) {
    const int row = col_row<P>(e, q);
    if (row >= 0) {
      const double2 a = sx[(size_t)row * J.wc_in];
      // i kx N (a - (-1)^y c / N)
      dst[(size_t)row * J.wc_out] = make_double2(fma(-kn, a.y, cy - r[e].y), fma(kn, a.x, r[e].x - cx));
    }
  }
}

// 3/2 padding (padd.f90:123-133) and truncation (unpadd.f90:143-155): PA::N
// rows in, PB::N rows out, unit coefficient.  From a spectrum each thread
// loads the rows it needs; otherwise the two layouts meet in shared memory.
template <class PA, class PB, int MB>
__global__ void __launch_bounds__(ICOL_TX * cmax(PA::TT, PB::TT), MB)
    k_icol_pad(ColJob J, const int4* __restrict__ twa, const int4* __restrict__ twb, int total) {
  pdl_wait();
  constexpr int TX = ICOL_TX, NA = PA::N, NB = PB::N, NT = TX * cmax(PA::TT, PB::TT), E = cmax(PA::E, PB::E);
  constexpr bool PAD = NB > NA;
  constexpr int NS = PAD ? NA : NB, NL = PAD ? NB : NA;
  static_assert(NT % 32 == 0, "whole warps");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  __shared__ unsigned slots[6 * TX];
  for (int t = threadIdx.x; t < 6 * TX; t += NT) slots[t] = 0;
  const int b = threadIdx.x % TX, q0 = threadIdx.x / TX;
  const int qa = q0 < PA::TT ? q0 : 1 << 20, qb = q0 < PB::TT ? q0 : 1 << 20;  // beyond a side's threads: no jobs
  const int col = blockIdx.x * TX + b;
  const bool ok = col < total;
  const int lev = ok ? col / J.ncols : 0, jx = ok ? col - lev * J.ncols : 0;
  const double2* src = reinterpret_cast<const double2*>(J.in[0]) + (size_t)lev * J.ps_in + (size_t)blockIdx.y * J.fs_in + jx;
  double2* dst = reinterpret_cast<double2*>(J.out[0]) + (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
  auto from = [](int k) {  // input wavenumber row of output row k (negative: none)
    if (k >= NB) return -1;
    if (PAD) return k < NS / 2 ? k : (k > NL - NS / 2 ? k - (NL - NS) : -1);
    return k < NS / 2 ? k : (k == NS / 2 ? -1 : k + (NL - NS));
  };
  const bool coin = fix_coin((unsigned)(jx * cmax(PA::TT, PB::TT) + q0));
  cfix v[E];
  int ex;
  bool bad = false;
  double2 x[E];
#pragma unroll
  for (int e = 0; e < E; ++e) x[e] = make_double2(0.0, 0.0);
  if (J.dir & DIR_FWD) {
#pragma unroll
    for (int e = 0; e < PA::PE; ++e) {
      const int row = col_row<PA>(e, qa);
      if (ok && row >= 0) x[e] = src[(size_t)row * J.wc_in];
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, PA::PE>(x, v, slots, b, fix_in(PA::R1), bad);
    col_fwd<PA, TX>(v, S, slots + 2 * TX, twa, qa, b, coin, ex);
    __syncthreads();  // the exchange buffer is read
#pragma unroll
    for (int e = 0; e < PA::SE; ++e) {
      const int k = col_k<PA>(e, qa);
      if (k < NA) S[k * TX + b] = v[e];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < PB::SE; ++e) {
      const int k = from(col_k<PB>(e, qb));
      v[e].x = v[e].y = 0;
      if (k >= 0) v[e] = S[k * TX + b];
    }
  } else {
#pragma unroll
    for (int e = 0; e < PB::SE; ++e) {
      const int k = from(col_k<PB>(e, qb));
      if (ok && k >= 0) x[e] = src[(size_t)k * J.wc_in];
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, PB::SE>(x, v, slots, b, 60, bad);
  }
  {
    unsigned w[PB::SE];
#pragma unroll
    for (int e = 0; e < PB::SE; ++e) w[e] = 1u;
    col_weigh<PB, TX>(v, w, false, slots + 4 * TX, b, coin, ex);
  }
  col_inv<PB, TX>(v, S, slots + 5 * TX, twb, qb, b, coin, ex);
  if (ok) {
    double2 r[PB::PE];
    fix_out(v, r, ex, nan_if(bad, 1.0));
#pragma unroll
    for (int e = 0; e < PB::PE; ++e) {
      const int row = col_row<PB>(e, qb);
      if (row >= 0) dst[(size_t)row * J.wc_out] = r[e];
    }
  }
}

template <typename K> void smem_of(K kernel, size_t sm, size_t& set) {
  if (sm > set) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    set = sm;
  }
}

// resident blocks for about 1024 threads (three steps, 64 registers) or 512
template <class P> constexpr int icol_mb(int tt) {
  return cmax(1, (P::E <= 8 ? 1024 : (P::E <= 12 ? 640 : 512)) / (ICOL_TX * tt));
}
template <class P> bool run_same(const ColJob& J, const FftPlanDev& F, cudaStream_t s) {
  constexpr int TX = ICOL_TX, NT = TX * P::TT, MB = icol_mb<P>(P::TT);
  const int total = J.ncols * J.nlev;
  const dim3 grid((total + TX - 1) / TX, J.nf > 0 ? J.nf : 1);
  if (J.nin == 1) {
    int nd = 0, ns = 0, ng = 0;
    for (int o = 0; o < J.nout; ++o) {
      const int code = J.coef[o][0];
      const bool inv = (J.inv_mask >> o) & 1u;
      if (code == CC_NONE) return false;
      if (!inv) {
        if (code != CC_ONE && code != CC_KILL) return false;
        ++ns;
      } else if (J.dir == DIR_BOTH && (code == CC_ONE || code == CC_KILL || code == CC_IKX)) {
        ++nd;
      } else {
        ++ng;
      }
    }
    const size_t sm = (size_t)(P::N + (ng > 1 ? P::SE * P::TT : 0)) * TX * sizeof(cfix);
    auto run = [&](auto kernel, size_t& set) {
      smem_of(kernel, sm, set);
      pdl(kernel, grid, NT, sm, s)(J, F.uniti, total, nd, ns, ng);
    };
    static size_t set[5] = {40 * 1024, 40 * 1024, 40 * 1024, 40 * 1024, 40 * 1024};  // the static arrays count too
    if (J.dir == DIR_FWD && ng == 0) run(k_icol<P, MB, DIR_FWD, false>, set[0]);
    else if (J.dir == DIR_INV && ns == 0 && ng == 1) run(k_icol<P, MB, DIR_INV, false>, set[1]);
    else if (J.dir == DIR_INV && ns == 0) run(k_icol<P, MB, DIR_INV, true>, set[2]);
    else if (J.dir == DIR_BOTH && ng <= 1) run(k_icol<P, MB, DIR_BOTH, false>, set[3]);
    else if (J.dir == DIR_BOTH) run(k_icol<P, MB, DIR_BOTH, true>, set[4]);
    else return false;
    return true;
  }
  // sums: every output i kx of one input plus i ky of another
  if (J.dir != DIR_BOTH) return false;
  int a[COL_MAXO], c[COL_MAXO];
  for (int o = 0; o < J.nout; ++o) {
    a[o] = c[o] = -1;
    if (!((J.inv_mask >> o) & 1u)) return false;
    for (int i = 0; i < J.nin; ++i) {
      if (J.coef[o][i] == CC_IKX && a[o] < 0) a[o] = i;
      else if (J.coef[o][i] == CC_IKY && c[o] < 0) c[o] = i;
      else if (J.coef[o][i] != CC_NONE) return false;
    }
    if (a[o] < 0 || c[o] < 0) return false;
  }
  const size_t sm = (size_t)P::N * TX * sizeof(cfix);
  static size_t set = 40 * 1024;  // the static arrays count too
  smem_of(k_icol_div<P, MB>, sm, set);
  for (int o = 0; o < J.nout; ++o) {
    ColJob K = J;
    K.in[0] = J.in[a[o]];
    K.in[1] = J.in[c[o]];
    K.out[0] = J.out[o];
    pdl(k_icol_div<P, MB>, grid, NT, sm, s)(K, F.uniti, total);
    if (o > 0) LES_COUNT_LAUNCH();  // the caller counts one
  }
  return true;
}
template <class PA, class PB> bool run_pad(const ColJob& J, const FftPlanDev& Fa, const FftPlanDev& Fb, cudaStream_t s) {
  constexpr int TX = ICOL_TX, TT = cmax(PA::TT, PB::TT);
  constexpr int MB = cmax(PA::E, PB::E) == PA::E ? icol_mb<PA>(TT) : icol_mb<PB>(TT);
  constexpr bool pad = PB::N > PA::N;
  if (J.nin != 1 || J.nout != 1 || J.coef[0][0] != CC_ONE || !(J.inv_mask & 1u) ||
      J.map != (pad ? MAP_PAD : MAP_UNPAD) || J.ny_small != (pad ? PA::N : PB::N) || (!pad && !(J.dir & DIR_FWD)))
    return false;
  const int total = J.ncols * J.nlev;
  const size_t sm = (size_t)std::max(PA::N, PB::N) * TX * sizeof(cfix);
  static size_t set = 40 * 1024;  // the static arrays count too
  smem_of(k_icol_pad<PA, PB, MB>, sm, set);
  pdl(k_icol_pad<PA, PB, MB>, dim3((total + TX - 1) / TX, J.nf > 0 ? J.nf : 1), TX * TT, sm, s)(J, Fa.uniti, Fb.uniti,
                                                                                               total);
  return true;
}

// shapes (R1, R2, R3, threads per column)
template <int N> struct ColOf;
#define LES_ICOLS(X)                                                                                        \
  X(16, 4, 4, 1, 4) X(24, 6, 4, 1, 8) X(32, 4, 8, 1, 8) X(36, 6, 6, 1, 8) X(48, 6, 8, 1, 8) X(64, 8, 8, 1, 8) \
  X(72, 6, 6, 2, 12) X(96, 6, 4, 4, 16) X(108, 9, 12, 1, 12) X(128, 8, 4, 4, 16) X(144, 6, 6, 4, 24)        \
  X(192, 6, 8, 4, 32) X(216, 6, 6, 6, 36) X(256, 8, 8, 4, 32) X(288, 6, 8, 6, 48) X(384, 6, 8, 8, 64)
#define LES_DEF(n, a, b, c, t) \
  template <> struct ColOf<n> { typedef ColShape<a, b, c, t> type; };
LES_ICOLS(LES_DEF)
#undef LES_DEF
}  // namespace

#define LES_IPADS(X)                                                                                  \
  X(16, 24) X(24, 36) X(32, 48) X(48, 72) X(64, 96) X(72, 108) X(96, 144) X(128, 192) X(144, 216) X(192, 288) \
  X(256, 384)

bool int_cols_length(int ny) {  // ny and its 3/2 padding
  switch (ny) {
#define LES_CASE(n, m) case n:
    LES_IPADS(LES_CASE)
#undef LES_CASE
    return true;
    default: return false;
  }
}
bool launch_cols_int(const ColJob& J, const FftPlanDev& Pin, const FftPlanDev& Pout, cudaStream_t s) {
  if (!Pin.uniti || !Pout.uniti) return false;
  if (J.map == MAP_SAME) {
    if (J.ny_in != J.ny_out || J.ny_small != J.ny_in) return false;
    switch (J.ny_in) {
#define LES_CASE(n, a, b, c, t) \
  case n: return run_same<ColOf<n>::type>(J, Pin, s);
      LES_ICOLS(LES_CASE)
#undef LES_CASE
      default: return false;
    }
  }
  switch (J.ny_in * 10000 + J.ny_out) {
#define LES_CASE(n, m)                                                                      \
  case n * 10000 + m: return run_pad<ColOf<n>::type, ColOf<m>::type>(J, Pin, Pout, s);      \
  case m * 10000 + n: return run_pad<ColOf<m>::type, ColOf<n>::type>(J, Pin, Pout, s);
    LES_IPADS(LES_CASE)
#undef LES_CASE
    default: return false;
  }
}

}  // namespace les
