// Shared device/host helpers for the GB300 LES core.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <type_traits>

#define LES_PI 3.1415926535897932384626433   /* param.f90:51 */
#define LES_BOGUS (-1234567890.0)              /* param.f90:50 */

namespace les {

// Complex type traits for the two arithmetic precisions.
template <typename T> struct CT;
template <> struct CT<double> { typedef double2 type; };
template <> struct CT<float> { typedef float2 type; };

template <typename T> __host__ __device__ __forceinline__ typename CT<T>::type mk(T a, T b) {
  typename CT<T>::type r; r.x = a; r.y = b; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
template <typename C, typename T> __device__ __forceinline__ C cscale(C a, T s) { a.x *= s; a.y *= s; return a; }
// i * a
template <typename C> __device__ __forceinline__ C cmuli(C a) { C r; r.x = -a.y; r.y = a.x; return r; }
// -i * a
template <typename C> __device__ __forceinline__ C cmulmi(C a) { C r; r.x = a.y; r.y = -a.x; return r; }
template <typename C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }

// eye * k * f = (-k f.im, k f.re), the reference's spectral derivative
// (ddx.f90:152, filt_da.f90:117-118).
template <typename C, typename T> __device__ __forceinline__ C ik(C f, T k) {
  C r; r.x = -(k * f.y); r.y = k * f.x; return r;
}

// IEEE-754 binary32 <-> binary64 conversions done with integer operations.
// On this part a hardware float<->double conversion issues on the FP64 pipe,
// which is as scarce as FP64 arithmetic; these run on the integer pipe for
// the normal range and zeros, and fall back to the hardware conversion for
// the rest (subnormals, overflow, infinities, NaN).  Results are identical
// to the hardware's: exact widening; narrowing rounds to nearest, ties to
// even, from the definition of the two formats.
// The integer pipe bounds the float-float row passes, so the operations count:
// 8 and 11 each, where a form with separate exponent and mantissa fields took 11
// and 17 (8 mixed members of 32^3 to 128^3: 3.86 -> 3.58 ms a step).
__device__ __forceinline__ double cvt_f2d(float f) {
  const unsigned u = __float_as_uint(f);
  if ((u & 0x7fffffffu) - 0x00800000u >= 0x7f000000u) {  // biased exponent 0 or 255
    if ((u << 1) == 0u) return __hiloint2double((int)u, 0);  // +-0
    return (double)f;
  }
  // sign, exponent + 896 and the mantissa's upper 20 bits; its lower three
  return __hiloint2double((int)(((unsigned)((int)u >> 3) & 0x8fffffffu) + (896u << 20)), (int)(u << 29));
}
__device__ __forceinline__ float cvt_d2f(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  if ((hi & 0x7fffffffu) - (897u << 20) >= (254u << 20)) {  // outside the normal range of binary32
    if (((hi << 1) | lo) == 0u) return __uint_as_float(hi);  // +-0
    return (float)x;
  }
  // 29 mantissa bits go: add half of the last kept unit, less one where that
  // unit is even; a carry rounds into the exponent
  const unsigned long long b = ((unsigned long long)hi << 32 | lo) + (0x0fffffffu + ((lo >> 29) & 1u));
  const unsigned m = (unsigned)(b >> 29) - (896u << 23);  // exponent and mantissa: the 9 exponent bits kept suffice
  return __uint_as_float((m & 0x7fffffffu) | (hi & 0x80000000u));
}
// FP32 truncation max(real(a), real(b)) of the reference's default-real MAX.
__device__ __forceinline__ double fmax32(double a, double b) {
  const float fa = cvt_d2f(a), fb = cvt_d2f(b);
  return cvt_f2d(fa > fb ? fa : fb);
}
// x / 2 and -2 x through the exponent field: exact products with powers of
// two need no operation of the FP64 pipe (about 1.7 per clock per SM, which
// bounds the pointwise FP64 kernels).  Infinities and NaN pass; subnormals
// are shifted, x / 2 to the nearest with halves to the even one: the bits of the
// products in every case.
__device__ __forceinline__ double half_of(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(b >> 32), e = (hi >> 20) & 0x7ffu;
  if (e > 1u) return e == 0x7ffu ? x : __hiloint2double((int)(hi - (1u << 20)), (int)(unsigned)b);
  const unsigned long long m = b & 0x7fffffffffffffffull;
  return __longlong_as_double((long long)((b & 0x8000000000000000ull) | ((m >> 1) + (m & (m >> 1) & 1ull))));
}
__device__ __forceinline__ double minus_twice(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) ^ 0x8000000000000000ull;
  const unsigned hi = (unsigned)(b >> 32), e = (hi >> 20) & 0x7ffu;
  if (e - 1u < 0x7fdu) return __hiloint2double((int)(hi + (1u << 20)), (int)(unsigned)b);
  if (e == 0u) return __longlong_as_double((long long)((b & 0x8000000000000000ull) | (b << 1)));
  return __longlong_as_double((long long)(e == 0x7ffu ? b : (b & 0x8000000000000000ull) | 0x7ff0000000000000ull));
}
// Float-float number ("double-single"): value hi + lo with |lo| <= ulp(hi)/2,
// about 48 significant bits, computed on the FP32 pipe with error-free
// transformations (Knuth's two-sum for additions, products through fused
// multiply-add, Dekker).  The mixed form runs its projection-path transforms
// in it: FP64-like accuracy at FP32-pipe throughput.
struct __align__(8) dfloat {
  float hi, lo;
  __host__ __device__ dfloat() {}
  __host__ __device__ constexpr dfloat(float h, float l) : hi(h), lo(l) {}
  __host__ __device__ constexpr dfloat(double d) : hi((float)d), lo((float)(d - (double)(float)d)) {}
  __host__ __device__ constexpr dfloat(int i) : hi((float)i), lo(0.f) {}
};
struct __align__(16) dcomplex {
  dfloat x, y;
};
template <> struct CT<dfloat> { typedef dcomplex type; };
__device__ __forceinline__ dfloat split_slow(double x) {
  const float h = cvt_d2f(x);
  return dfloat(h, cvt_d2f(x - cvt_f2d(h)));
}
// x as hi + lo, both rounded to nearest: the remainder is what the rounding of
// hi left of the mantissa, a signed 30-bit integer, so that no FP64 subtraction
// and no second narrowing are needed (mixed 256^3: k_dpdz_project32 466 -> 374 us,
// the float-float rows of p 467 -> 410 us).  The same for the sum of a pair did not
// pay: the conversion to an integer sits in the way of the small launches.
__device__ __forceinline__ dfloat split_d(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned a = hi & 0x7fffffffu;
  // hi normal and below the largest binade, lo's unit 2^(e - 52) a normal float
  if (a - ((896u + 53u) << 20) >= (201u << 20)) return split_slow(x);
  const unsigned long long b = ((unsigned long long)hi << 32 | lo) + (0x0fffffffu + ((lo >> 29) & 1u));
  const unsigned m = (unsigned)(b >> 29) - (896u << 23);
  const int r = (int)(lo - ((unsigned)b & 0xe0000000u)), s = (int)hi >> 31;
  const float unit = __uint_as_float(((a >> 20) - (896u + 52u)) << 23);
  return dfloat(__uint_as_float((m & 0x7fffffffu) | (hi & 0x80000000u)), __int2float_rn((r ^ s) - s) * unit);
}
__device__ __forceinline__ dfloat df_quick(float a, float b) {  // |a| >= |b|
  const float s = a + b;
  return dfloat(s, b - (s - a));
}
// Sums and products are left unnormalised (hi = the rounded leading term,
// lo = its exact error plus the low parts, |lo| a few ulp(hi) at most): the
// next operation's two-sum / FMA product absorbs it, and a conversion to
// FP64 adds the two.  Saves the quick-two-sum on the FP32 pipe.
__device__ __forceinline__ dfloat operator+(dfloat a, dfloat b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b.hi - bb) + (a.lo + b.lo);
  return dfloat(s, e);
}
__device__ __forceinline__ dfloat operator-(dfloat a) { return dfloat(-a.hi, -a.lo); }
__device__ __forceinline__ dfloat operator-(dfloat a, dfloat b) { return a + (-b); }
__device__ __forceinline__ dfloat operator*(dfloat a, dfloat b) {
  const float p = a.hi * b.hi;
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  e = fmaf(a.lo, b.hi, e);
  return dfloat(p, e);
}
__device__ __forceinline__ dfloat operator/(dfloat a, dfloat b) {
  const float q1 = a.hi / b.hi;
  const dfloat r = a - b * dfloat(q1, 0.f);
  const float q2 = r.hi / b.hi;
  return df_quick(q1, q2);
}
__device__ __forceinline__ dfloat& operator+=(dfloat& a, dfloat b) { return a = a + b; }
__device__ __forceinline__ dfloat& operator-=(dfloat& a, dfloat b) { return a = a - b; }
__device__ __forceinline__ dfloat& operator*=(dfloat& a, dfloat b) { return a = a * b; }
__device__ __forceinline__ bool operator!=(dfloat a, dfloat b) { return a.hi != b.hi || a.lo != b.lo; }

// element conversions between a transform's precision and the storage type
template <typename To, typename From> __device__ __forceinline__ To cvt(From v) { return (To)v; }
template <> __device__ __forceinline__ double cvt<double, float>(float v) { return cvt_f2d(v); }
template <> __device__ __forceinline__ float cvt<float, double>(double v) { return cvt_d2f(v); }
template <> __device__ __forceinline__ dfloat cvt<dfloat, double>(double v) {
  return split_d(v);
}
template <> __device__ __forceinline__ double cvt<double, dfloat>(dfloat v) { return cvt_f2d(v.hi) + cvt_f2d(v.lo); }
template <> __device__ __forceinline__ dfloat cvt<dfloat, dfloat>(dfloat v) { return v; }
__device__ __forceinline__ double2 to_d2(double2 v) { return v; }
__device__ __forceinline__ double2 to_d2(dcomplex v) { return make_double2(cvt<double>(v.x), cvt<double>(v.y)); }
template <typename CO> __device__ __forceinline__ CO from_d2(double2 v);
template <> __device__ __forceinline__ double2 from_d2<double2>(double2 v) { return v; }
template <> __device__ __forceinline__ dcomplex from_d2<dcomplex>(double2 v) {
  dcomplex r;
  r.x = cvt<dfloat>(v.x);
  r.y = cvt<dfloat>(v.y);
  return r;
}

}  // namespace les

#define LES_CUDA_CHECK(expr)                                                           \
  do {                                                                                 \
    cudaError_t _e = (expr);                                                           \
    if (_e != cudaSuccess) {                                                           \
      les_set_error("%s:%d %s: %s", __FILE__, __LINE__, #expr, cudaGetErrorString(_e)); \
      return LES_ERR_CUDA;                                                             \
    }                                                                                  \
  } while (0)

void les_set_error(const char* fmt, ...);

// Number of kernels this library has launched (diagnostic counter).
extern unsigned long long g_les_launches;
#define LES_COUNT_LAUNCH() (++g_les_launches)

namespace les {
// Launches with programmatic stream serialization: a kernel may be scheduled
// while the one before it in its stream drains, and its first statement,
// pdl_wait(), holds it until that kernel has finished and its writes are
// visible.  Kernel to kernel in a graph 1.0 to 1.15 -> 0.76 to 0.9 us (8 to 304
// blocks), in a stream 3.1 to 4.1 -> 1.6 us.  Every kernel launched this way
// begins with pdl_wait(), also one that needs nothing from its predecessor:
// the order of all earlier work rests on it.
template <class... P> struct PdlCall {
  void (*kernel)(P...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  // the kernel's own parameter types: arguments convert as in a call, never by a cast
  void operator()(P... args) const {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, args...);  // a failure stays for cudaGetLastError, as with <<<>>>
  }
};
static_assert(std::is_invocable<PdlCall<const double*, int>, double*, int>::value &&
                  !std::is_invocable<PdlCall<double*, int>, float*, int>::value &&
                  !std::is_invocable<PdlCall<double*, int>, const double*, int>::value,
              "a launch takes its kernel's argument types");
template <class... P>
PdlCall<P...> pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem = 0, cudaStream_t stream = 0) {
  return PdlCall<P...>{kernel, grid, block, smem, stream};
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Measurement hook (les_profile_begin/end): while a session is open, every
// launch of one kernel family on the session's stream is bracketed by CUDA
// events and its algorithmic bytes (inputs read once + outputs written once)
// are summed.  Families: 1 FP64 y-pass, 2 FP32 y-pass, 3 FP64 x-pass,
// 4 FP32 x-pass (forward and inverse).
enum ProfFamily { PROF_COLS64 = 1, PROF_COLS32 = 2, PROF_ROWS64 = 3, PROF_ROWS32 = 4 };
struct ProfSession {
  int family = 0;
  cudaStream_t stream = nullptr;
  int n = 0, cap = 0;
  cudaEvent_t* ev = nullptr;
  double bytes = 0.0;
};
extern ProfSession* g_prof;
bool prof_mark(int family, cudaStream_t s);         // true: the launch that follows is measured
void prof_done(cudaStream_t s, double bytes);       // after that launch
}  // namespace les
