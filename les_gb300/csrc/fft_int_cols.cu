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
// alternating sum, sum_y (-1)^y f / ny, is what the round trip gives.  They are
// written last, from the input again (cached), so that no register holds it.
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
  const int s = fix_shift(m, bits), c = 1082 - s;
  bad = bad || m >= 0x7ff00000u;
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    v[i].x = fix_of(x[i].x, c);
    v[i].y = fix_of(x[i].y, c);
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
// v[n2] = x[q + N1 n2].  (One bound from the whole column's sum would save
// the second shift, 2 % of a step, but leaves 256 to 384 values of noise four
// bits fewer: 3/2 round trip at 256^2 4.2e-16 against 1.6e-16.)
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
// the sums of moduli below 2^60 that col_inv needs: a thread's values, up to
// 24 with weights up to 192, stay below 2^31 units of 2^44
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_room(cfix (&v)[NV], unsigned* slot, int q, int b, int& ex) {
  unsigned sum = 0;
  if (q < N2) {
#pragma unroll
    for (int i = 0; i < N1; ++i) sum += fix_l1<12>(v[i]);
  }
  const int s = fix_down_sum(col_max<TX>(sum, slot, b), 44);
  const i64 rnd = fix_rnd(s);
  ex += s;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    v[i].x = fix_shr(v[i].x, s, rnd);
    v[i].y = fix_shr(v[i].y, s, rnd);
  }
}
// the same for w(k) v with integer weights: 0 or 1, or (sgn) |ky| as an
// integer, negative wavenumbers (i >= N1/2) changing sign.  The products are
// exact 96-bit integers before the shift.
template <int N1, int N2, int TX, int NV>
__device__ __forceinline__ void col_weigh(cfix (&v)[NV], const unsigned (&w)[N1], bool sgn, unsigned* slot, int q, int b,
                                          int& ex) {
  unsigned sum = 0;
#pragma unroll
  for (int i = 0; i < N1; ++i)
    if (w[i]) sum += fix_l1<12>(v[i]) * w[i];
  const int s = fix_down_sum(col_max<TX>(sum, slot, b), 44);
  const i64 rnd = fix_rnd(s);
  const i64 flip = sgn ? -1 : 0;
  ex += s;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    const i64 lx = mad_wu((unsigned)v[i].x, w[i], rnd), ly = mad_wu((unsigned)v[i].y, w[i], rnd);
    const i64 hx = mad_w((int)(v[i].x >> 32), (int)w[i], (i64)((unsigned long long)lx >> 32));
    const i64 hy = mad_w((int)(v[i].y >> 32), (int)w[i], (i64)((unsigned long long)ly >> 32));
    // (h 2^32 + low word) >> s, s < 32
    v[i].x = (i64)(((unsigned long long)__funnelshift_r((unsigned)hx, (unsigned)(hx >> 32), s) << 32) |
                   __funnelshift_r((unsigned)lx, (unsigned)hx, s));
    v[i].y = (i64)(((unsigned long long)__funnelshift_r((unsigned)hy, (unsigned)(hy >> 32), s) << 32) |
                   __funnelshift_r((unsigned)ly, (unsigned)hy, s));
    if (i >= N1 / 2) {
      v[i].x = (v[i].x ^ flip) - flip;
      v[i].y = (v[i].y ^ flip) - flip;
    }
  }
}
// weights of ky: |k| or N - |k|, none for the Nyquist row
template <int N1, int N2> __device__ __forceinline__ void ky_weights(unsigned (&w)[N1], int q, bool zero) {
  constexpr int N = N1 * N2;
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    const int k = q + N2 * i;
    w[i] = zero || q >= N2 || k == N / 2 ? 0u : (unsigned)(i < N1 / 2 ? k : N - k);
  }
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
template <int N1, int N2, int MB, int DIR, bool MULTI>
__global__ void __launch_bounds__(ICOL_TX * (N1 > N2 ? N1 : N2), MB)
    k_icol(ColJob J, const int4* __restrict__ tw, int total, int ndirect, int nspec, int ngen) {
  pdl_wait();
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
  constexpr bool fwd = (DIR & DIR_FWD) != 0;
  const bool last = jx == J.lh - 1;  // kx = nx/2: removed by KILL and by the derivatives
  cfix v[NV];
  int ex;
  bool bad = false;
  {
    double2 x[NV];
    constexpr int step = fwd ? N1 : N2, cnt = fwd ? N2 : N1;
    const bool act = ok && q < step;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      x[i] = make_double2(0.0, 0.0);
      if (act && i < cnt) x[i] = src[(size_t)(q + step * i) * J.wc_in];
    }
    __syncthreads();  // slots are zero
    ex = col_fix<TX, cnt>(x, v, slots, b, fwd ? fix_in(N2) : 60, bad);
  }
  double ax = 0.0, ay = 0.0;  // (-1)^row times the alternating sum
  if (DIR == DIR_BOTH && ndirect) {
    i64 sx = 0, sy = 0;
#pragma unroll
    for (int i = 0; i < N2; ++i) { sx += (v[i].x + 2) >> 2; sy += (v[i].y + 2) >> 2; }
    if (q & 1) { sx = -sx; sy = -sy; }
    col_sum<TX>(sx, sy, sums, b);
    if (q & 1) { sx = -sx; sy = -sy; }
    const cfix t[1] = {{sx, sy}};
    double2 r[1];
    fix_out(t, r, ex + 2, 1.0);
    ax = nan_if(bad, r[0].x);
    ay = nan_if(bad, r[0].y);
  }
  auto direct = [&]() {
    if (DIR != DIR_BOTH || ndirect == 0 || !ok || q >= N1) return;
    for (int o = 0; o < J.nout; ++o) {
      if (!col_direct(J, o)) continue;
      const int code = J.coef[o][0];
      const bool one = code == CC_ONE, ikx = code == CC_IKX;
      const double f = !one && last ? 0.0 : (ikx ? J.kx[jx] : 1.0);
      const double fn = f * (double)N, bx = one ? 0.0 : f * ax, by = one ? 0.0 : f * ay;
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
#pragma unroll
      for (int i = 0; i < N2; ++i) {  // N f - (-1)^row sum, from the input again
        const size_t row = (size_t)(q + N1 * i);
        const double2 a = src[row * J.wc_in];
        const double rx = fma(fn, a.x, -bx), ry = fma(fn, a.y, -by);
        dst[row * J.wc_out] = ikx ? make_double2(-ry, rx) : make_double2(rx, ry);
      }
    }
  };
  if (nspec + ngen == 0) {
    direct();
    return;
  }
  if constexpr (fwd) col_fwd<N1, N2, TX>(v, S, slots + 2 * TX, tw, q, b, ex);
  if (DIR != DIR_INV && nspec && ok && q < N2) {
    for (int o = 0; o < J.nout; ++o) {
      if ((J.inv_mask >> o) & 1u) continue;
      const bool kill = J.coef[o][0] == CC_KILL;
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
      fix_groups<N1>([&](int i) { return v[i]; }, [&](int i, double2 r) {
        const int k = q + N2 * i;
        dst[(size_t)k * J.wc_out] = kill && k == N / 2 ? make_double2(0.0, 0.0) : r;
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
    unsigned* so = slots + (3 + 2 * o) * TX;
    double f = 1.0;
    const bool iky = code == CC_IKY || code == CC_MIKY, rot = iky || code == CC_IKX;
    unsigned w[N1];
    if (iky) {
      f = code == CC_IKY ? J.ky[J.lh] : -J.ky[J.lh];  // row 1: the unit of ky
      ky_weights<N1, N2>(w, q, last);
    } else if (code == CC_ONE || code == CC_KILL || code == CC_IKX) {
      if (code == CC_IKX) f = J.kx[jx];
#pragma unroll
      for (int i = 0; i < N1; ++i) w[i] = q >= N2 || (code != CC_ONE && (last || q + N2 * i == N / 2)) ? 0u : 1u;
    } else {  // cutoff filters: pass or drop, one common factor
      const bool wide = code == CC_G || code == CC_MASK;
      const float* T = wide ? J.Gf : J.GGf;
      if (code == CC_G || code == CC_GG) f = (wide ? J.G : J.GG)[0];
#pragma unroll
      for (int i = 0; i < N1; ++i)
        w[i] = q >= N2 || __ldg(&T[(size_t)J.lh * (q + N2 * i) + jx]) == 0.f ? 0u : 1u;
    }
    col_weigh<N1, N2, TX>(v, w, iky, so, q, b, ex);
    col_inv<N1, N2, TX>(v, S, so + TX, tw, q, b, ex);
    if (ok && q < N1) {
      double2* dst = reinterpret_cast<double2*>(J.out[o]) + out0;
      double2 r[N2];
      fix_out(v, r, ex, nan_if(bad, f));
#pragma unroll
      for (int i = 0; i < N2; ++i)
        dst[(size_t)(q + N1 * i) * J.wc_out] = make_double2(rot ? -r[i].y : r[i].x, rot ? r[i].x : r[i].y);
    }
  };
  auto general = [&](int o) { return ((J.inv_mask >> o) & 1u) && !col_direct(J, o); };
  if constexpr (MULTI) {
#pragma unroll
    for (int i = 0; i < NV; ++i) K[(i * NV + q) * TX + b] = v[i];
    for (int o = 0; o < J.nout; ++o) {
      if (!general(o)) continue;
#pragma unroll
      for (int i = 0; i < NV; ++i) v[i] = K[(i * NV + q) * TX + b];
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
template <int N1, int N2, int MB>
__global__ void __launch_bounds__(ICOL_TX * (N1 > N2 ? N1 : N2), MB)
    k_icol_div(ColJob J, const int4* __restrict__ tw, int total) {
  pdl_wait();
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
  {
    unsigned w[N1];
    ky_weights<N1, N2>(w, q, last);
    col_weigh<N1, N2, TX>(v, w, true, slots + 3 * TX, q, b, ex);
  }
  col_inv<N1, N2, TX>(v, S, slots + 4 * TX, tw, q, b, ex);
  if (!act) return;
  double cx = 0.0, cy = 0.0;
#pragma unroll
  for (int w = 0; w < NW; ++w) { cx += part[w * TX + b].x; cy += part[w * TX + b].y; }
  const double kx = last ? 0.0 : J.kx[jx], kn = kx * (double)N;
  cx *= q & 1 ? -kx : kx;
  cy *= q & 1 ? -kx : kx;
  double2* dst = reinterpret_cast<double2*>(J.out[0]) + (size_t)lev * J.ps_out + (size_t)blockIdx.y * J.fs_out + jx;
  double2 r[N2];
  fix_out(v, r, ex, nan_if(bad, J.ky[J.lh]));
#pragma unroll
  for (int i = 0; i < N2; ++i) {
    const size_t row = (size_t)(q + N1 * i);
    const double2 a = sx[row * J.wc_in];
    // i kx N (a - (-1)^y c / N)
    dst[row * J.wc_out] = make_double2(fma(-kn, a.y, cy - r[i].y), fma(kn, a.x, r[i].x - cx));
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
  pdl_wait();
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
    double2 r[B2];
    fix_out(v, r, ex, nan_if(bad, 1.0));
#pragma unroll
    for (int i = 0; i < B2; ++i) dst[(size_t)(q + B1 * i) * J.wc_out] = r[i];
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
    auto run = [&](auto kernel, size_t& set) {
      smem_of(kernel, sm, set);
      pdl(kernel, grid, NT, sm, s)(J, P.uniti, total, nd, ns, ng);
    };
    static size_t set[5] = {40 * 1024, 40 * 1024, 40 * 1024, 40 * 1024, 40 * 1024};  // the static arrays count too
    if (J.dir == DIR_FWD && ng == 0) run(k_icol<N1, N2, MB, DIR_FWD, false>, set[0]);
    else if (J.dir == DIR_INV && ns == 0 && ng == 1) run(k_icol<N1, N2, MB, DIR_INV, false>, set[1]);
    else if (J.dir == DIR_INV && ns == 0) run(k_icol<N1, N2, MB, DIR_INV, true>, set[2]);
    else if (J.dir == DIR_BOTH && ng <= 1) run(k_icol<N1, N2, MB, DIR_BOTH, false>, set[3]);
    else if (J.dir == DIR_BOTH) run(k_icol<N1, N2, MB, DIR_BOTH, true>, set[4]);
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
  const size_t sm = (size_t)N1 * N2 * TX * sizeof(cfix);
  static size_t set = 40 * 1024;  // the static arrays count too
  smem_of(k_icol_div<N1, N2, MB>, sm, set);
  for (int o = 0; o < J.nout; ++o) {
    ColJob K = J;
    K.in[0] = J.in[a[o]];
    K.in[1] = J.in[c[o]];
    K.out[0] = J.out[o];
    pdl(k_icol_div<N1, N2, MB>, grid, NT, sm, s)(K, P.uniti, total);
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
  pdl(k_icol_pad<A1, A2, B1, B2, MB>, dim3((total + TX - 1) / TX, J.nf > 0 ? J.nf : 1), TX * PT::nv, sm, s)(
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

bool int_cols_length(int ny) {  // ny and its 3/2 padding
  switch (ny) {
#define LES_CASE(n, a, b, m, c, d, mb) case n:
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
