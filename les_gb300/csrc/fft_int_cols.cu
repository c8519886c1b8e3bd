// FP64 y pass (cols) on the integer pipe; see fft_int.cuh.
//
// TX columns per block; a column of N = N1 N2 rows is served by
// max(N1, N2) threads.  Thread q holds the rows q + N1 n2 (n2 < N2) of the
// physical side or the wavenumbers q + N2 k1 (k1 < N1) of the spectral side;
// one exchange through shared memory turns one into the other, so a column
// goes through the registers once per transform.  Columns are numbered
// through all levels, so that only the last block of a launch has idle ones.
//
// Outputs that only drop the Nyquist row (filt_da's field) or multiply by
// the column's kx need no transform at all in y: the field less its
// alternating sum, sum_y (-1)^y f / ny, is what the round trip gives.
#include <algorithm>
#include "fft_int.cuh"
#include "les_internal.h"

namespace les {
namespace {

constexpr int ICOL_TX = 8;
constexpr int ICOL_SLOTS = 3 + 2 * COL_MAXO;

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
  const int s = fix_shift(m, bits), s20 = s * (1 << 20);
  bad = bad || m >= 0x7ff00000u;
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    v[i].x = fix_of(x[i].x, s20);
    v[i].y = fix_of(x[i].y, s20);
  }
  return -s - pre;
}

// forward: v[n2] = x[q + N1 n2], components below 2^fix_in(N2), to
// v[k1] = X[q + N2 k1]
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_fwd(cfix (&v)[NV], cfix* S, unsigned* slot, const int4* __restrict__ tw, int q, int b,
                                        int& ex) {
  unsigned top = 0;
  if (q < N1) {
    fdft<N2, -1>(v);
#pragma unroll
    for (int i = 0; i < N2; ++i) {
      if (i > 0) v[i] = ftw(v[i], __ldg(&tw[q * i]));
      top = max(top, max(fix_top(v[i].x), fix_top(v[i].y)));
      S[(i * N1 + q) * TX + b] = v[i];
    }
  }
  const int s = fix_down(col_max<TX>(top, slot, b), fix_in(N1));
  const i64 rnd = fix_rnd(s);
  ex += s;
  if (q < N2) {
#pragma unroll
    for (int i = 0; i < N1; ++i) {
      const cfix a = S[(q * N1 + i) * TX + b];
      v[i].x = fix_shr(a.x, s, rnd);
      v[i].y = fix_shr(a.y, s, rnd);
    }
    fdft<N1, -1>(v);
  }
}
// inverse: v[k1] = X[q + N2 k1], sums of N1 moduli below 2^60, to
// v[n2] = x[q + N1 n2]
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_inv(cfix (&v)[NV], cfix* S, unsigned* slot, const int4* __restrict__ tw, int q, int b,
                                        int& ex) {
  unsigned top = 0;
  if (q < N2) {
    fdft<N1, 1>(v);
#pragma unroll
    for (int i = 0; i < N1; ++i) {
      if (i > 0) v[i] = ftwc(v[i], __ldg(&tw[q * i]));
      top = max(top, max(fix_top(v[i].x), fix_top(v[i].y)));
      S[(q * N1 + i) * TX + b] = v[i];
    }
  }
  const int s = fix_down(col_max<TX>(top, slot, b), fix_in(N2));
  const i64 rnd = fix_rnd(s);
  ex += s;
  if (q < N1) {
#pragma unroll
    for (int i = 0; i < N2; ++i) {
      const cfix a = S[(i * N1 + q) * TX + b];
      v[i].x = fix_shr(a.x, s, rnd);
      v[i].y = fix_shr(a.y, s, rnd);
    }
    fdft<N2, 1>(v);
  }
}
// the sums of moduli below 2^60 that col_inv needs
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_room(cfix (&v)[NV], unsigned* slot, int q, int b, int& ex) {
  unsigned sum = 0;
  if (q < N2) {
#pragma unroll
    for (int i = 0; i < N1; ++i) sum += fix_l1(v[i]);
  }
  const int s = fix_down_sum(col_max<TX>(sum, slot, b));
  const i64 rnd = fix_rnd(s);
  ex += s;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    v[i].x = fix_shr(v[i].x, s, rnd);
    v[i].y = fix_shr(v[i].y, s, rnd);
  }
}
// i ky X with ky = k - (k >= N/2) N as an integer (its unit is a factor of
// the output), with the same bound; `neg`: -i ky.  The products are exact
// 96-bit integers before the shift.
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_iky(cfix (&v)[NV], unsigned* slot, int q, int b, bool zero, bool neg, int& ex) {
  constexpr int N = N1 * N2;
  unsigned sum = 0;
  if (q < N2 && !zero) {
#pragma unroll
    for (int i = 0; i < N1; ++i) {
      const int k = q + N2 * i;
      const unsigned m = i < N1 / 2 ? k : N - k;
      if (k != N / 2) sum += fix_l1(v[i]) * m;
    }
  }
  const int s = fix_down_sum(col_max<TX>(sum, slot, b));
  const i64 rnd = fix_rnd(s);
  ex += s;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    const int k = q + N2 * i;
    unsigned m = i < N1 / 2 ? k : N - k;
    if (k == N / 2 || zero || q >= N2) m = 0;
    const i64 lx = mad_wu((unsigned)v[i].x, m, rnd), ly = mad_wu((unsigned)v[i].y, m, rnd);
    const i64 hx = mad_w((int)(v[i].x >> 32), (int)m, (i64)((unsigned long long)lx >> 32));
    const i64 hy = mad_w((int)(v[i].y >> 32), (int)m, (i64)((unsigned long long)ly >> 32));
    // (h 2^32 + low word) >> s, s < 32
    const i64 px = (i64)(((unsigned long long)__funnelshift_r((unsigned)hx, (unsigned)(hx >> 32), s) << 32) |
                         __funnelshift_r((unsigned)lx, (unsigned)hx, s));
    const i64 py = (i64)(((unsigned long long)__funnelshift_r((unsigned)hy, (unsigned)(hy >> 32), s) << 32) |
                         __funnelshift_r((unsigned)ly, (unsigned)hy, s));
    if ((i < N1 / 2) != neg) {  // +i
      v[i].x = -py;
      v[i].y = px;
    } else {
      v[i].x = py;
      v[i].y = -px;
    }
  }
}

__device__ __forceinline__ double nan_if(bool bad, double f) {
  return bad ? __longlong_as_double(0x7ff8000000000000ll) : f;
}
__device__ __forceinline__ bool col_direct(const ColJob& J, int o) {  // needs no y transform
  const int code = J.coef[o][0];
  return J.dir == DIR_BOTH && ((J.inv_mask >> o) & 1u) && (code == CC_ONE || code == CC_KILL || code == CC_IKX);
}

// One input, same length.  ngen: inverse outputs that need a transform.
template <int N1, int N2, int MB>
__global__ void __launch_bounds__(ICOL_TX * (N1 > N2 ? N1 : N2), MB)
    k_icol(ColJob J, const int4* __restrict__ tw, int total, int ndirect, int nspec, int ngen) {
  constexpr int TX = ICOL_TX, N = N1 * N2, NV = N1 > N2 ? N1 : N2, NT = TX * NV;
  static_assert(NT % 32 == 0 && N1 % 2 == 0, "whole warps; row parity by thread");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  cfix* K = S + N * TX;  // the spectrum, kept for later outputs (ngen > 1)
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
  const bool fwd = (J.dir & DIR_FWD) != 0;
  const bool last = jx == J.lh - 1;  // kx = nx/2: removed by KILL and by the derivatives
  cfix v[NV];
  int ex;
  bool bad = false;
  {
    double2 x[NV];
    const int r0 = q, step = fwd ? N1 : N2, cnt = fwd ? N2 : N1;
    const bool act = ok && q < step;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      x[i] = make_double2(0.0, 0.0);
      if (act && i < cnt) x[i] = src[(size_t)(r0 + step * i) * J.wc_in];
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, NV>(x, v, slots, b, fwd ? fix_in(N2) : 60, bad);
  }
  if (ndirect) {
    double cx = 0.0, cy = 0.0;
    {
      i64 sx = 0, sy = 0;
#pragma unroll
      for (int i = 0; i < N2; ++i) { sx += (v[i].x + 2) >> 2; sy += (v[i].y + 2) >> 2; }
      if (q & 1) { sx = -sx; sy = -sy; }
      col_sum<TX>(sx, sy, sums, b);
      cx = (double)sx * (4.0 / N);
      cy = (double)sy * (4.0 / N);
    }
    const i64 ax = __double2ll_rn(q & 1 ? -cx : cx), ay = __double2ll_rn(q & 1 ? -cy : cy);
    if (ok && q < N1) {
      for (int o = 0; o < J.nout; ++o) {
        if (!col_direct(J, o)) continue;
        const int code = J.coef[o][0];
        const bool one = code == CC_ONE, ikx = code == CC_IKX;
        double f = nan_if(bad, ikx ? J.kx[jx] * (double)N : (double)N);
        if (!one && last) f = 0.0;
        const FixOut out(ex, f);
        const i64 bx = one ? 0 : ax, by = one ? 0 : ay;
        double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
#pragma unroll
        for (int i = 0; i < N2; ++i) {
          const double rx = out(v[i].x - bx), ry = out(v[i].y - by);
          dst[(size_t)(q + N1 * i) * J.wc_out] = ikx ? make_double2(-ry, rx) : make_double2(rx, ry);
        }
      }
    }
  }
  if (nspec + ngen == 0) return;
  if (fwd) col_fwd<N1, N2, TX>(v, S, slots + 2 * TX, tw, q, b, ex);
  if (nspec && ok && q < N2) {
    for (int o = 0; o < J.nout; ++o) {
      if ((J.inv_mask >> o) & 1u) continue;
      const bool kill = J.coef[o][0] == CC_KILL;
      const FixOut out(ex, kill && last ? 0.0 : nan_if(bad, 1.0));
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        const int k = q + N2 * i;
        double2 r = make_double2(out(v[i].x), out(v[i].y));
        if (kill && k == N / 2) r = make_double2(0.0, 0.0);
        dst[(size_t)k * J.wc_out] = r;
      }
    }
  }
  if (ngen == 0) return;
  if (ngen > 1) {
#pragma unroll
    for (int i = 0; i < NV; ++i) K[(i * NV + q) * TX + b] = v[i];
  }
  const int ex0 = ex;
  int done = 0;
  for (int o = 0; o < J.nout; ++o) {
    if (!((J.inv_mask >> o) & 1u) || col_direct(J, o)) continue;
    if (done++ > 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) v[i] = K[(i * NV + q) * TX + b];
    }
    ex = ex0;
    const int code = J.coef[o][0];
    unsigned* so = slots + (3 + 2 * o) * TX;
    double f = 1.0;
    bool rot = false;
    if (code == CC_IKY || code == CC_MIKY) {
      f = J.ky[J.lh];  // row 1: the unit of ky
      col_iky<N1, N2, TX>(v, so, q, b, last, code == CC_MIKY, ex);
    } else {
      if (code == CC_KILL || code == CC_IKX) {
        if (code == CC_IKX) { f = J.kx[jx]; rot = true; }
#pragma unroll
        for (int i = 0; i < N1; ++i)
          if (last || q + N2 * i == N / 2) v[i].x = v[i].y = 0;
      } else if (code != CC_ONE) {  // cutoff filters: pass or drop, one common factor
        const bool wide = code == CC_G || code == CC_MASK;
        const float* T = wide ? J.Gf : J.GGf;
        if (code == CC_G || code == CC_GG) f = (wide ? J.G : J.GG)[0];
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          const int k = q + N2 * i;
          if (q < N2 && __ldg(&T[(size_t)J.lh * k + jx]) == 0.f) v[i].x = v[i].y = 0;
        }
      }
      col_room<N1, N2, TX>(v, so, q, b, ex);
    }
    col_inv<N1, N2, TX>(v, S, so + TX, tw, q, b, ex);
    if (ok && q < N1) {
      const FixOut out(ex, nan_if(bad, f));
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        const double rx = out(v[i].x), ry = out(v[i].y);
        dst[(size_t)(q + N1 * i) * J.wc_out] = rot ? make_double2(-ry, rx) : make_double2(rx, ry);
      }
    }
  }
}

// i kx in0 + i ky in1 (the horizontal divergences): in1 makes the round trip;
// in0 needs none, only its Nyquist row removed, and is added on the way out.
template <int N1, int N2, int MB>
__global__ void __launch_bounds__(ICOL_TX * (N1 > N2 ? N1 : N2), MB)
    k_icol_div(ColJob J, const int4* __restrict__ tw, int total) {
  constexpr int TX = ICOL_TX, N = N1 * N2, NV = N1 > N2 ? N1 : N2, NT = TX * NV, NW = NT / 32;
  static_assert(NT % 32 == 0 && N1 % 2 == 0, "whole warps; row parity by thread");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  __shared__ unsigned slots[5 * TX];
  __shared__ double2 part[NW * TX];
  for (int t = threadIdx.x; t < 5 * TX; t += NT) slots[t] = 0;
  const int b = threadIdx.x % TX, q = threadIdx.x / TX;
  const int col = blockIdx.x * TX + b;
  const bool ok = col < total;
  const int lev = ok ? col / J.ncols : 0, jx = ok ? col - lev * J.ncols : 0;
  const size_t in0 = (size_t)lev * J.ps_in + (size_t)blockIdx.y * J.fs_in + jx;
  const double2* sx = reinterpret_cast<const double2*>(J.in[0]) + in0;
  const double2* sy = reinterpret_cast<const double2*>(J.in[1]) + in0;
  const bool act = ok && q < N1;
  cfix v[NV];
  int ex;
  bool bad = false;
  {
    double2 x[NV];
    double ax = 0.0, ay = 0.0;  // alternating sum of in0
#pragma unroll
    for (int i = 0; i < N2; ++i) x[i] = act ? sx[(size_t)(q + N1 * i) * J.wc_in] : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < N2; ++i) { ax += x[i].x; ay += x[i].y; }
    if (q & 1) { ax = -ax; ay = -ay; }
#pragma unroll
    for (int o = TX; o < 32; o <<= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    if ((threadIdx.x & 31) < TX) part[(threadIdx.x >> 5) * TX + b] = make_double2(ax, ay);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      x[i] = make_double2(0.0, 0.0);
      if (act && i < N2) x[i] = sy[(size_t)(q + N1 * i) * J.wc_in];
    }
    __syncthreads();  // slots are zero, partial sums are written
    ex = col_fix<TX, NV>(x, v, slots, b, fix_in(N2), bad);
  }
  col_fwd<N1, N2, TX>(v, S, slots + 2 * TX, tw, q, b, ex);
  const bool last = jx == J.lh - 1;
  col_iky<N1, N2, TX>(v, slots + 3 * TX, q, b, last, false, ex);
  col_inv<N1, N2, TX>(v, S, slots + 4 * TX, tw, q, b, ex);
  if (!act) return;
  double cx = 0.0, cy = 0.0;
#pragma unroll
  for (int w = 0; w < NW; ++w) { cx += part[w * TX + b].x; cy += part[w * TX + b].y; }
  const double kx = last ? 0.0 : J.kx[jx], kn = kx * (double)N;
  cx *= q & 1 ? -kx : kx;
  cy *= q & 1 ? -kx : kx;
  const FixOut out(ex, nan_if(bad, J.ky[J.lh]));
  double2* dst = reinterpret_cast<double2*>(J.out[0]) + (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
#pragma unroll
  for (int i = 0; i < N2; ++i) {
    const size_t row = (size_t)(q + N1 * i);
    const double2 a = sx[row * J.wc_in];
    // i kx N (a - (-1)^y c / N)
    dst[row * J.wc_out] = make_double2(fma(-kn, a.y, out(v[i].x) + cy), fma(kn, a.x, out(v[i].y) - cx));
  }
}

// 3/2 padding (padd.f90:123-133) and truncation (unpadd.f90:143-155): A1 A2
// rows in, B1 B2 rows out, unit coefficient.  From a spectrum each thread
// loads the rows it needs; otherwise the two layouts meet in shared memory.
template <int A1, int A2, int B1, int B2, int MB> struct PadT {
  static constexpr int NA = A1 * A2, NB = B1 * B2;
  static constexpr int ta = A1 > A2 ? A1 : A2, tb = B1 > B2 ? B1 : B2, nv = ta > tb ? ta : tb;
};
template <int A1, int A2, int B1, int B2, int MB>
__global__ void __launch_bounds__(ICOL_TX * (PadT<A1, A2, B1, B2, MB>::nv), MB)
    k_icol_pad(ColJob J, const int4* __restrict__ twa, const int4* __restrict__ twb, int total) {
  typedef PadT<A1, A2, B1, B2, MB> PT;
  constexpr int TX = ICOL_TX, NA = PT::NA, NB = PT::NB, NV = PT::nv, NT = TX * NV;
  constexpr bool PAD = NB > NA;
  constexpr int NS = PAD ? NA : NB, NL = PAD ? NB : NA;
  static_assert(NT % 32 == 0, "whole warps");
  extern __shared__ __align__(16) unsigned char smraw[];
  cfix* S = reinterpret_cast<cfix*>(smraw);
  __shared__ unsigned slots[5 * TX];
  for (int t = threadIdx.x; t < 5 * TX; t += NT) slots[t] = 0;
  const int b = threadIdx.x % TX, q = threadIdx.x / TX;
  const int col = blockIdx.x * TX + b;
  const bool ok = col < total;
  const int lev = ok ? col / J.ncols : 0, jx = ok ? col - lev * J.ncols : 0;
  const double2* src = reinterpret_cast<const double2*>(J.in[0]) + (size_t)lev * J.ps_in + (size_t)blockIdx.y * J.fs_in + jx;
  double2* dst = reinterpret_cast<double2*>(J.out[0]) + (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
  auto from = [](int k) {  // input wavenumber row of output row k (negative: none)
    if (PAD) return k < NS / 2 ? k : (k > NL - NS / 2 ? k - (NL - NS) : -1);
    return k < NS / 2 ? k : (k == NS / 2 ? -1 : k + (NL - NS));
  };
  cfix v[NV];
  int ex;
  bool bad = false;
  double2 x[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) x[i] = make_double2(0.0, 0.0);
  if (J.dir & DIR_FWD) {
    if (ok && q < A1) {
#pragma unroll
      for (int i = 0; i < A2; ++i) x[i] = src[(size_t)(q + A1 * i) * J.wc_in];
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, A2>(x, v, slots, b, fix_in(A2), bad);
    col_fwd<A1, A2, TX>(v, S, slots + 2 * TX, twa, q, b, ex);
    __syncthreads();  // the exchange buffer is read
    if (q < A2) {
#pragma unroll
      for (int i = 0; i < A1; ++i) S[(q + A2 * i) * TX + b] = v[i];
    }
    __syncthreads();
    if (q < B2) {
#pragma unroll
      for (int i = 0; i < B1; ++i) {
        const int k = from(q + B2 * i);
        v[i].x = v[i].y = 0;
        if (k >= 0) v[i] = S[k * TX + b];
      }
    }
  } else {
    if (ok && q < B2) {
#pragma unroll
      for (int i = 0; i < B1; ++i) {
        const int k = from(q + B2 * i);
        if (k >= 0) x[i] = src[(size_t)k * J.wc_in];
      }
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, B1>(x, v, slots, b, 60, bad);
  }
  col_room<B1, B2, TX>(v, slots + 3 * TX, q, b, ex);
  col_inv<B1, B2, TX>(v, S, slots + 4 * TX, twb, q, b, ex);
  if (ok && q < B1) {
    const FixOut out(ex, nan_if(bad, 1.0));
#pragma unroll
    for (int i = 0; i < B2; ++i) dst[(size_t)(q + B1 * i) * J.wc_out] = make_double2(out(v[i].x), out(v[i].y));
  }
}

template <typename K> void smem_of(K kernel, size_t sm, size_t& set) {
  if (sm > set) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    set = sm;
  }
}

template <int N1, int N2, int MB> bool run_same(const ColJob& J, const FftPlanDev& P, cudaStream_t s) {
  constexpr int TX = ICOL_TX, NV = N1 > N2 ? N1 : N2, NT = TX * NV;
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
    const size_t sm = (size_t)(N1 * N2 + (ng > 1 ? NV * NV : 0)) * TX * sizeof(cfix);
    static size_t set = 40 * 1024;  // the static arrays count too
    smem_of(k_icol<N1, N2, MB>, sm, set);
    k_icol<N1, N2, MB><<<grid, NT, sm, s>>>(J, P.uniti, total, nd, ns, ng);
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
  const size_t sm = (size_t)N1 * N2 * TX * sizeof(cfix);
  static size_t set = 40 * 1024;  // the static arrays count too
  smem_of(k_icol_div<N1, N2, MB>, sm, set);
  for (int o = 0; o < J.nout; ++o) {
    ColJob K = J;
    K.in[0] = J.in[a[o]];
    K.in[1] = J.in[c[o]];
    K.out[0] = J.out[o];
    k_icol_div<N1, N2, MB><<<grid, NT, sm, s>>>(K, P.uniti, total);
    if (o > 0) LES_COUNT_LAUNCH();  // the caller counts one
  }
  return true;
}
template <int A1, int A2, int B1, int B2, int MB>
bool run_pad(const ColJob& J, const FftPlanDev& Pa, const FftPlanDev& Pb, cudaStream_t s) {
  constexpr int TX = ICOL_TX;
  typedef PadT<A1, A2, B1, B2, MB> PT;
  constexpr bool pad = PT::NB > PT::NA;
  if (J.nin != 1 || J.nout != 1 || J.coef[0][0] != CC_ONE || !(J.inv_mask & 1u) ||
      J.map != (pad ? MAP_PAD : MAP_UNPAD) || J.ny_small != (pad ? PT::NA : PT::NB) || (!pad && !(J.dir & DIR_FWD)))
    return false;
  const int total = J.ncols * J.nlev;
  const size_t sm = (size_t)std::max(PT::NA, PT::NB) * TX * sizeof(cfix);
  static size_t set = 40 * 1024;  // the static arrays count too
  smem_of(k_icol_pad<A1, A2, B1, B2, MB>, sm, set);
  k_icol_pad<A1, A2, B1, B2, MB><<<dim3((total + TX - 1) / TX, J.nf > 0 ? J.nf : 1), TX * PT::nv, sm, s>>>(
      J, Pa.uniti, Pb.uniti, total);
  return true;
}

}  // namespace

// length: (N1, N2, resident blocks per SM)
#define LES_ICOLS(X)                                                                                        \
  X(16, 4, 4, 8) X(24, 8, 3, 6) X(32, 8, 4, 6) X(36, 12, 3, 5) X(48, 12, 4, 5) X(64, 8, 8, 8) X(72, 12, 6, 5)  \
  X(96, 12, 8, 5) X(108, 12, 9, 5) X(128, 16, 8, 4) X(144, 12, 12, 5) X(192, 16, 12, 4) X(216, 24, 9, 2)     \
  X(256, 16, 16, 4) X(288, 24, 12, 2) X(384, 24, 16, 2)
#define LES_IPADS(X)                                                                                       \
  X(16, 4, 4, 24, 8, 3, 6) X(24, 8, 3, 36, 12, 3, 5) X(32, 8, 4, 48, 12, 4, 5) X(48, 12, 4, 72, 12, 6, 5)  \
  X(64, 8, 8, 96, 12, 8, 5) X(72, 12, 6, 108, 12, 9, 5) X(96, 12, 8, 144, 12, 12, 5)                       \
  X(128, 16, 8, 192, 16, 12, 4) X(144, 12, 12, 216, 24, 9, 2) X(192, 16, 12, 288, 24, 12, 2)               \
  X(256, 16, 16, 384, 24, 16, 2)

bool launch_cols_int(const ColJob& J, const FftPlanDev& Pin, const FftPlanDev& Pout, cudaStream_t s) {
  if (!Pin.uniti || !Pout.uniti) return false;
  if (J.map == MAP_SAME) {
    if (J.ny_in != J.ny_out || J.ny_small != J.ny_in) return false;
    switch (J.ny_in) {
#define LES_CASE(n, a, b, mb) \
  case n: return run_same<a, b, mb>(J, Pin, s);
      LES_ICOLS(LES_CASE)
#undef LES_CASE
      default: return false;
    }
  }
  switch (J.ny_in * 10000 + J.ny_out) {
#define LES_CASE(n, a, b, m, c, d, mb)                                                \
  case n * 10000 + m: return run_pad<a, b, c, d, mb>(J, Pin, Pout, s);                \
  case m * 10000 + n: return run_pad<c, d, a, b, mb>(J, Pin, Pout, s);
    LES_IPADS(LES_CASE)
#undef LES_CASE
    default: return false;
  }
}

}  // namespace les
