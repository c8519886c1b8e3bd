// FP64 x pass (rows_r2c, rows_c2r) on the integer pipe; see fft_int.cuh.
//
// Half length M = N1 N2.  A row is served by TT lanes of one warp (no block
// barrier anywhere): n = n1 + N1 n2, k = k2 + N2 k1, the N1 first-step and
// the N2 second-step transforms dealt out to the lanes, one exchange through
// shared memory between them.  The Hermitian post- and pre-processing works
// on the pairs (k, M - k): one twiddle product serves both members and every
// element is read and written once.  The blocks of one group of rows in all
// fields of a job are neighbours, so that a field and its x derivative, which
// the inverse pass makes from the same spectrum, read it from memory once.
#include <algorithm>
#include "fft_int.cuh"
#include "les_internal.h"

namespace les {
namespace {

template <int TT> __device__ __forceinline__ unsigned row_max(unsigned m) {
#pragma unroll
  for (int o = 1; o < TT; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}
template <int TT> __device__ __forceinline__ unsigned row_sum(unsigned m) {
#pragma unroll
  for (int o = 1; o < TT; o <<= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
  return m;
}
// the row's scale: x to integers below 2^bits; returns the exponent of one unit
template <int TT, int CNT>
__device__ __forceinline__ int row_fix(double2 (&x)[CNT], cfix (&v)[CNT], int bits, bool& bad) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < CNT; ++i) m = max(m, max(fix_mag(x[i].x), fix_mag(x[i].y)));
  const unsigned lm = m;
  m = row_max<TT>(m);
  int pre = 0;
  if (__any_sync(0xffffffffu, lm != 0u && lm < (unsigned)FIX_TINY)) {  // near the smallest FP64 exponents
    if (m != 0u && m < (unsigned)FIX_TINY) {
      pre = FIX_PRE;
      const double f = fix_pow2(FIX_PRE);
#pragma unroll
      for (int i = 0; i < CNT; ++i) { x[i].x *= f; x[i].y *= f; }
    }
    m = 0;
#pragma unroll
    for (int i = 0; i < CNT; ++i) m = max(m, max(fix_mag(x[i].x), fix_mag(x[i].y)));
    m = row_max<TT>(m);
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

// the same for i k x with the integers k(i) of the row's elements, below 2^57
template <int TT, int CNT, class KF>
__device__ __forceinline__ int row_fix_ik(double2 (&x)[CNT], cfix (&v)[CNT], bool& bad, KF&& kof) {
  auto top = [&](int i) {  // exponent field bound of k x (x = 0: 0)
    const unsigned m = max(fix_mag(x[i].x), fix_mag(x[i].y));
    return m >= 0x7ff00000u ? 0x7fffffffu : (m ? (m >> 20) + 32u - __clz((int)kof(i)) : 0u);
  };
  unsigned m = 0;
  bool low = false;
#pragma unroll
  for (int i = 0; i < CNT; ++i) m = max(m, top(i));
  low = m != 0u && m < 72u;
  m = row_max<TT>(m);
  int pre = 0;
  if (__any_sync(0xffffffffu, low)) {  // near the smallest FP64 exponents
    if (m != 0u && m < 72u) {
      pre = FIX_PRE;
      const double f = fix_pow2(FIX_PRE);
#pragma unroll
      for (int i = 0; i < CNT; ++i) { x[i].x *= f; x[i].y *= f; }
    }
    m = 0;
#pragma unroll
    for (int i = 0; i < CNT; ++i) m = max(m, top(i));
    m = row_max<TT>(m);
  }
  bad = bad || m == 0x7fffffffu;
  const int e1 = m ? (int)min(m, 4000u) - 1 : 4000;
#pragma unroll
  for (int i = 0; i < CNT; ++i) {
    const unsigned k = kof(i);
    v[i].x = -fix_times(x[i].y, k, e1);
    v[i].y = fix_times(x[i].x, k, e1);
  }
  return e1 - 1078 - pre;
}

template <int N1, int N2, int TT> struct RowShape {
  static constexpr int M = N1 * N2, J1 = (N1 + TT - 1) / TT, J2 = (N2 + TT - 1) / TT;
  static constexpr int LD1 = N1 | 1;              // odd stride: the transposed read is free of bank conflicts
  static constexpr int MS = N2 * LD1 > M + 1 ? N2 * LD1 : M + 1;
  static constexpr int NT = 128, RPB = NT / TT, KP = (M / 2 + TT - 1) / TT;
  static_assert(32 % TT == 0 && M % 2 == 0, "a row within one warp");
  // Inverse pass, scaled by the largest sum of moduli of the first step's transforms
  // (FINE) instead of the whole row's.  Rows of 384: the row's leaves a flat spectrum (a
  // single point's) 52 bits, 2.2 x 2^-53 of error (the FP64 kernels 1.7); with the
  // steps' 0.4 to 0.8.  Shorter rows stay below the FP64 kernels with the row's (288
  // points 1.2 against 1.9), which takes one reduction less.
  static constexpr bool FINE = M > 144;
  static_assert(!FINE || (TT == N1 && N1 == 16), "a lane's elements at k, and those at M - k, belong to one k1 each");
  static constexpr size_t smem = (size_t)RPB * MS * sizeof(cfix);
};

template <int N1, int N2, int TT, int MB>
__global__ void __launch_bounds__(128, MB) k_ir2c(RowJob J, const int4* __restrict__ tw, const int4* __restrict__ wr,
                                                  int nrows) {
  pdl_wait();
  typedef RowShape<N1, N2, TT> R;
  constexpr int M = R::M, J1 = R::J1, J2 = R::J2, LD1 = R::LD1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int q = threadIdx.x % TT, r = threadIdx.x / TT;
  cfix* S = reinterpret_cast<cfix*>(smraw) + r * R::MS;
  const int f = blockIdx.x % J.nfield, row = (blockIdx.x / J.nfield) * R::RPB + r;
  const bool ok = row < nrows;
  const int lev = ok ? row / J.ny : 0, y = ok ? row - lev * J.ny : 0;
  const double2* src = reinterpret_cast<const double2*>(reinterpret_cast<const double*>(J.phys[f]) +
                                                        (size_t)lev * J.pstride_phys + (size_t)y * J.ld);
  double2 x[J1 * N2];
#pragma unroll
  for (int j = 0; j < J1; ++j)
#pragma unroll
    for (int i = 0; i < N2; ++i) {
      const int n1 = q + TT * j;
      x[j * N2 + i] = make_double2(0.0, 0.0);
      if (ok && (N1 % TT == 0 || n1 < N1)) x[j * N2 + i] = src[n1 + N1 * i];
    }
  if (J.off[f]) {
    const double off = J.off[f][lev];
#pragma unroll
    for (int i = 0; i < J1 * N2; ++i) { x[i].x -= off; x[i].y -= off; }
  }
  bool bad = false;
  cfix v[J1 * N2];
  int ex = row_fix<TT, J1 * N2>(x, v, fix_in(N2), bad);
  unsigned top = 0;
#pragma unroll
  for (int j = 0; j < J1; ++j) {
    const int n1 = q + TT * j;
    if (N1 % TT == 0 || n1 < N1) {
      fdft<N2, -1>(v + j * N2);  // over n2
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        if (i > 0) v[j * N2 + i] = ftw(v[j * N2 + i], __ldg(&tw[n1 * i]));
        top = max(top, max(fix_top(v[j * N2 + i].x), fix_top(v[j * N2 + i].y)));
        S[i * LD1 + n1] = v[j * N2 + i];
      }
    }
  }
  // one bit spare for the sums of the post-processing
  const FixShift s(fix_down(row_max<TT>(top), fix_in(N1) - 1), fix_coin((unsigned)y));
  ex += s.s;
  __syncwarp();
  cfix w[J2 * N1];
#pragma unroll
  for (int j = 0; j < J2; ++j) {
    const int k2 = q + TT * j;
    if (N2 % TT == 0 || k2 < N2) {
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        const cfix a = S[k2 * LD1 + i];
        w[j * N1 + i].x = s(a.x);
        w[j * N1 + i].y = s(a.y);
      }
      fdft<N1, -1>(w + j * N1);  // over n1: Z[k2 + N2 i]
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < J2; ++j) {
    const int k2 = q + TT * j;
    if (N2 % TT == 0 || k2 < N2) {
#pragma unroll
      for (int i = 0; i < N1; ++i) S[k2 + N2 * i] = w[j * N1 + i];
    }
  }
  __syncwarp();
  if (!ok) return;
  // X[k] = (E + O) / 2, X[M - k] = conj(E - O) / 2; lane 0: X[0], X[M], X[M / 2]
  double2* dst = reinterpret_cast<double2*>(J.work[f]) + (size_t)lev * J.pstride_work + (size_t)y * J.wc;
  const int nc = J.ncols;
  cfix g[2 * R::KP + 1];
#pragma unroll
  for (int i = 0; i < R::KP; ++i) {
    const int k = q + TT * i;
    g[2 * i].x = g[2 * i].y = g[2 * i + 1].x = g[2 * i + 1].y = 0;
    if (k < nc && ((M / 2) % TT == 0 || k < M / 2)) {
      const cfix a = S[k];
      if (i == 0 && k == 0) {
        g[0].x = (a.x + a.y) << 1;
        g[1].x = (a.x - a.y) << 1;
      } else {
        const cfix c = S[M - k];
        const int4 t = __ldg(&wr[k]);
        cfix e, d;  // Z[k] +- conj(Z[M - k])
        e.x = a.x + c.x; e.y = a.y - c.y;
        d.x = a.x - c.x; d.y = a.y + c.y;
        const cfix o = fcmul(d, t.z, t.w, -t.x, -t.y);  // -i w d
        g[2 * i].x = e.x + o.x; g[2 * i].y = e.y + o.y;
        g[2 * i + 1].x = e.x - o.x; g[2 * i + 1].y = o.y - e.y;
      }
    }
  }
  g[2 * R::KP].x = S[M / 2].x << 1;
  g[2 * R::KP].y = -(S[M / 2].y << 1);
  double2 o[2 * R::KP + 1];
  fix_out(g, o, ex - 1, nan_if(bad, J.div[f] != 0.0 ? J.scale[f] / J.div[f] : J.scale[f]));
#pragma unroll
  for (int i = 0; i < R::KP; ++i) {
    const int k = q + TT * i;
    if ((M / 2) % TT == 0 || k < M / 2) {
      if (k < nc) dst[k] = o[2 * i];
      if (M - k < nc) dst[M - k] = o[2 * i + 1];
    }
  }
  if (q == 0 && M / 2 < nc) dst[M / 2] = o[2 * R::KP];
}

template <int N1, int N2, int TT, int MB>
__global__ void __launch_bounds__(128, MB) k_ic2r(RowJob J, const int4* __restrict__ tw, const int4* __restrict__ wr,
                                                  int nrows) {
  pdl_wait();
  typedef RowShape<N1, N2, TT> R;
  constexpr int M = R::M, J1 = R::J1, J2 = R::J2, LD1 = R::LD1, KP = R::KP;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int q = threadIdx.x % TT, r = threadIdx.x / TT;
  cfix* S = reinterpret_cast<cfix*>(smraw) + r * R::MS;
  const int f = blockIdx.x % J.nfield, row = (blockIdx.x / J.nfield) * R::RPB + r;
  const bool ok = row < nrows;
  const int lev = ok ? row / J.ny : 0, y = ok ? row - lev * J.ny : 0;
  const double2* src = reinterpret_cast<const double2*>(J.work[f]) + (size_t)lev * J.pstride_work + (size_t)y * J.wc;
  const int nc = ok ? J.ncols : 0;
  int ex;
  bool bad = false;
  unsigned sum = 0, sum2 = 0;  // moduli of the elements at k and at M - k
  {
    double2 x[2 * KP + 1];  // X[k], X[M - k], and lane 0's X[M / 2]
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const int k = q + TT * i;
      x[2 * i] = x[2 * i + 1] = make_double2(0.0, 0.0);
      if ((M / 2) % TT == 0 || k < M / 2) {
        if (k < nc) x[2 * i] = src[k];
        if (M - k < nc) x[2 * i + 1] = src[M - k];
      }
    }
    x[2 * KP] = make_double2(0.0, 0.0);
    if (q == 0) {
      if (M / 2 < nc) x[2 * KP] = src[M / 2];
      x[0].y = 0.0;  // the halfcomplex pass ignores Im of X[0], X[M]
      x[1].y = 0.0;
    }
    cfix g[2 * KP + 1];
    if (J.deriv[f]) {  // i kx X, kx = 0 at k = 0 and k = M; the unit of kx is a factor of the output
      if (q == 0) {
        x[1] = make_double2(0.0, 0.0);
        // a mean adds nothing, so it must not set the scale either (p at 10^6 times
        // its fluctuations: 20 bits); not-a-number and infinity stay
        if (fix_mag(x[0].x) < 0x7ff00000u) x[0].x = 0.0;
      }
      ex = row_fix_ik<TT, 2 * KP + 1>(x, g, bad, [&](int i) {
        const int k = q + TT * (i / 2);
        return (unsigned)(i == 2 * KP ? M / 2 : (i & 1 ? M - k : k));
      });
    } else {
      ex = row_fix<TT, 2 * KP + 1>(x, g, 58, bad);
    }
    auto put = [&](int k, cfix u, unsigned& total) {  // element k = k1 + N1 k2 at k2 LD1 + k1
      S[(k / N1) * LD1 + k % N1] = u;
      total += fix_l1<4>(u);
    };
#pragma unroll
    for (int i = 0; i < KP; ++i) {
      const int k = q + TT * i;
      if ((M / 2) % TT == 0 || k < M / 2) {
        const cfix a = g[2 * i], c = g[2 * i + 1];
        cfix e, d, o;
        e.x = a.x + c.x; e.y = a.y - c.y;
        d.x = a.x - c.x; d.y = a.y + c.y;
        if (i == 0 && k == 0) {
          o = d;  // w = 1
        } else {
          o = ftwc(d, __ldg(&wr[k]));
        }
        cfix u;  // A[k] = E + i D, A[M - k] = conj(E - i D)
        u.x = e.x - o.y; u.y = e.y + o.x;
        put(k, u, sum);
        if (!(i == 0 && k == 0)) {
          u.x = e.x + o.y; u.y = o.x - e.y;
          put(M - k, u, sum2);
        }
      }
    }
    if (q == 0) {
      cfix u;
      u.x = g[2 * KP].x << 1;
      u.y = -(g[2 * KP].y << 1);
      put(M / 2, u, sum);
    }
  }
  // at most 25 values a lane: below 2^31 units of 2^36; the row's in units of 2^40.
  // FINE: lane q holds all of the first step's transform k1 = q, so the two largest
  // parts bound each of them.  Below 2^58, the second step's inner four-point
  // transforms stay below 2^60 before its rotations and its results below 2^62.
  const int s1 = R::FINE ? fix_down_sum(row_max<TT>(sum) + row_max<TT>(sum2), 36 + 2)
                         : fix_down_sum(row_sum<TT>(((sum + sum2) >> 4) + 1u), 40);
  const FixShift s(s1, fix_coin((unsigned)y));
  ex += s.s;
  __syncwarp();
  // first step in place: a lane's transforms read and write their own slots,
  // so the loop needs no registers for the others (and half the code)
#pragma unroll 1
  for (int j = 0; j < J1; ++j) {
    const int k1 = q + TT * j;
    if (N1 % TT == 0 || k1 < N1) {
      cfix v[N2];
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        const cfix a = S[i * LD1 + k1];
        v[i].x = s(a.x);
        v[i].y = s(a.y);
      }
      fdft<N2, 1>(v);  // over k2
#pragma unroll
      for (int i = 0; i < N2; ++i) {
        if (i > 0) v[i] = ftwc(v[i], __ldg(&tw[k1 * i]));
        S[i * LD1 + k1] = v[i];
      }
    }
  }
  __syncwarp();
  if (!ok) return;
  const double factor = nan_if(bad, J.deriv[f] ? J.scale[f] * J.kunit : J.scale[f]);
  double2* dst = reinterpret_cast<double2*>(reinterpret_cast<double*>(const_cast<void*>(J.phys[f])) +
                                            (size_t)lev * J.pstride_phys + (size_t)y * J.ld);
  const double* offs = J.off[f];
#pragma unroll
  for (int j = 0; j < J2; ++j) {
    const int n2 = q + TT * j;
    if (N2 % TT == 0 || n2 < N2) {
      cfix w[N1];
#pragma unroll
      for (int i = 0; i < N1; ++i) w[i] = S[n2 * LD1 + i];
      fdft<N1, 1>(w);  // over k1: z[n2 + N2 i]
      double2 o[N1];
      fix_out(w, o, ex, factor);
      if (offs) {
        const double off = offs[lev];
#pragma unroll
        for (int i = 0; i < N1; ++i) { o[i].x += off; o[i].y += off; }
      }
#pragma unroll
      for (int i = 0; i < N1; ++i) dst[n2 + N2 * i] = o[i];
    }
  }
  if (q == 0) dst[M] = make_double2(0.0, 0.0);  // padding columns ld-1:ld
}

template <int N1, int N2, int TT, int MB>
void run_r2c(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  typedef RowShape<N1, N2, TT> R;
  static bool set = false;
  if (!set) {
    if (R::smem > 40 * 1024)
      cudaFuncSetAttribute(k_ir2c<N1, N2, TT, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::smem);
    set = true;
  }
  const int nrows = J.ny * J.nlev;
  pdl(k_ir2c<N1, N2, TT, MB>, (nrows + R::RPB - 1) / R::RPB * J.nfield, R::NT, R::smem, s)(J, P.c.uniti, P.wi, nrows);
}
template <int N1, int N2, int TT, int MB>
void run_c2r(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  typedef RowShape<N1, N2, TT> R;
  static bool set = false;
  if (!set) {
    if (R::smem > 40 * 1024)
      cudaFuncSetAttribute(k_ic2r<N1, N2, TT, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::smem);
    set = true;
  }
  const int nrows = J.ny * J.nlev;
  pdl(k_ic2r<N1, N2, TT, MB>, (nrows + R::RPB - 1) / R::RPB * J.nfield, R::NT, R::smem, s)(J, P.c.uniti, P.wi, nrows);
}

}  // namespace

// half length: (N1, N2, lanes per row, resident blocks per SM)
#define LES_IROWS(X)                                                                                    \
  X(16, 4, 4, 4, 6) X(24, 8, 3, 4, 6) X(32, 8, 4, 4, 5) X(36, 12, 3, 4, 5) X(48, 12, 4, 4, 5)           \
  X(54, 6, 9, 4, 3) X(64, 8, 8, 8, 6) X(72, 12, 6, 4, 3) X(96, 12, 8, 8, 4) X(108, 12, 9, 16, 5)       \
  X(128, 16, 8, 8, 4) X(144, 12, 12, 16, 5) X(192, 16, 12, 16, 4)

bool int_rows_length(int m) {
  switch (m) {
#define LES_CASE(m, a, b, t, mb) case m:
    LES_IROWS(LES_CASE)
#undef LES_CASE
    return true;
    default: return false;
  }
}
bool launch_rows_r2c_int(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  if (!P.c.uniti) return false;
  switch (P.nx / 2) {
#define LES_CASE(m, a, b, t, mb) \
  case m: run_r2c<a, b, t, mb>(J, P, s); return true;
    LES_IROWS(LES_CASE)
#undef LES_CASE
    default: return false;
  }
}
bool launch_rows_c2r_int(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  if (!P.c.uniti) return false;
  switch (P.nx / 2) {
#define LES_CASE(m, a, b, t, mb) \
  case m: run_c2r<a, b, t, mb>(J, P, s); return true;
    LES_IROWS(LES_CASE)
#undef LES_CASE
    default: return false;
  }
}

}  // namespace les
