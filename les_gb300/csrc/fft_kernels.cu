// Batched plane FFT kernels (rows_r2c, cols, rows_c2r); see fft.cuh.
#include "fft_kernels.cuh"
#include "les_internal.h"

namespace les {

// ---------------------------------------------------------------------------
// host launchers

// rows per CTA of a job.  An FP64 job of one or two planes takes single rows,
// so that it reaches every SM (two planes of 96 x 64: 8 CTAs of 16 rows, 10 us;
// 128 of one row, 8 us), in CTAs of two warps.
template <typename T> inline int rows_of(const RowJob& J, int nx) {
  int r = J.rpc > 0 ? J.rpc : rows_pc<T>(nx);
  if (std::is_same<T, double>::value)
    while (r > 1 && (long)((J.ny + r - 1) / r) * J.nlev * J.nfield < 2 * 152) r = (r + 1) / 2;
  return r;
}
template <typename T> inline int threads_of(int work) {  // of the runtime-length kernels
  return std::is_same<T, double>::value && work <= 256 ? 64 : 256;
}

template <typename T, typename TIn>
int launch_rows_r2c(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  typedef typename CT<T>::type C;
  const int rpc = rows_of<T>(J, P.nx);
  const size_t sm = (size_t)2 * rpc * (P.nx / 2) * sizeof(C);
  RowJob JJ = J;
  JJ.dnc = FastDiv((unsigned)J.ncols);
  dim3 grid((J.ny + rpc - 1) / rpc, J.nlev, J.nfield);
  const bool pr = g_prof && prof_mark(sizeof(T) == 8 ? PROF_ROWS64 : PROF_ROWS32, s);
  bool done = false;
  if constexpr (std::is_same<T, double>::value) done = launch_rows_r2c_int(JJ, P, s);
  else done = launch_rows_r2c_fixed<T, TIn>(JJ, P, rpc, sm, s);
  if (!done) {
    static size_t sm_set = 48 * 1024;  // opt-in raised once per instantiation (not during capture)
    if (sm > sm_set) {
      cudaFuncSetAttribute(k_rows_r2c<T, TIn, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      sm_set = sm;
    }
    pdl(k_rows_r2c<T, TIn, 0>, grid, threads_of<T>(rpc * P.nx / 2), sm, s)(JJ, P, rpc);
  }
  LES_COUNT_LAUNCH();
  if (pr)
    prof_done(s, (double)J.nfield * J.nlev * J.ny * ((double)P.nx * sizeof(TIn) + (double)J.ncols * sizeof(C)));
  return 0;
}

template <typename T, typename TOut>
int launch_rows_c2r(const RowJob& J, const RealPlanDev& P, cudaStream_t s) {
  typedef typename CT<T>::type C;
  const int rpc = rows_of<T>(J, P.nx);
  const int m = P.nx / 2;
  const size_t sm = (size_t)rpc * ((m + 1) + 2 * m) * sizeof(C);
  dim3 grid((J.ny + rpc - 1) / rpc, J.nlev, J.nfield);
  const bool pr = g_prof && prof_mark(sizeof(T) == 8 ? PROF_ROWS64 : PROF_ROWS32, s);
  bool done = false;
  if constexpr (std::is_same<T, double>::value) done = launch_rows_c2r_int(J, P, s);
  else done = launch_rows_c2r_fixed<T, TOut>(J, P, rpc, sm, s);
  if (!done) {
    static size_t sm_set = 48 * 1024;  // opt-in raised once per instantiation (not during capture)
    if (sm > sm_set) {
      cudaFuncSetAttribute(k_rows_c2r<T, TOut, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      sm_set = sm;
    }
    pdl(k_rows_c2r<T, TOut, 0>, grid, threads_of<T>(rpc * m), sm, s)(J, P, rpc);
  }
  LES_COUNT_LAUNCH();
  if (pr)
    prof_done(s, (double)J.nfield * J.nlev * J.ny * ((double)J.ncols * sizeof(C) + (double)J.ld * sizeof(TOut)));
  return 0;
}

template <typename T, int TX, typename CIn>
static int launch_cols_tx(const ColJob& J, const FftPlanDev& Pin, const FftPlanDev& Pout, cudaStream_t s) {
  typedef typename CT<T>::type C;
  const int nymax = J.ny_in > J.ny_out ? J.ny_in : J.ny_out;
  const size_t sm = (size_t)(J.nin * J.ny_in + 2 * nymax) * TX * sizeof(C);
  dim3 grid((J.ncols + TX - 1) / TX, J.nlev, J.nf > 0 ? J.nf : 1);
  const bool pr = g_prof && prof_mark(sizeof(T) == 8 ? PROF_COLS64 : PROF_COLS32, s);
  bool done = false;
  if constexpr (std::is_same<T, double>::value) done = launch_cols_int(J, Pin, Pout, s);
  else done = launch_cols_fixed<T, TX, CIn>(J, Pin, Pout, sm, grid, s);
  if (!done) {
    static size_t sm_set = 48 * 1024;  // opt-in raised once per instantiation (not during capture)
    if (sm > sm_set) {
      cudaFuncSetAttribute(k_cols<T, TX, CIn>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      sm_set = sm;
    }
    pdl(k_cols<T, TX, CIn>, grid, threads_of<T>(nymax * TX), sm, s)(J, Pin, Pout);
  }
  LES_COUNT_LAUNCH();
  if (pr) {
    const double nf = J.nf > 0 ? J.nf : 1;
    prof_done(s, nf * J.nlev * J.ncols *
                     ((double)J.nin * J.ny_in * sizeof(CIn) + (double)J.nout * J.ny_out * sizeof(C)));
  }
  return 0;
}

// kx tile width: 8-byte reals (FP64, float-float) {2, 4, 8} (default 4),
// FP32 {4, 8, 16} (default 8); the autotuner picks one per grid size
template <typename T, typename CIn>
int launch_cols(const ColJob& J, const FftPlanDev& Pin, const FftPlanDev& Pout, cudaStream_t s) {
  if (sizeof(T) == 8) {
    if constexpr (std::is_same<T, double>::value) {
      // one or two planes: single columns reach every SM
      const long tiles = (long)((J.ncols + 3) / 4) * J.nlev * (J.nf > 0 ? J.nf : 1);
      if (tiles < 152) return launch_cols_tx<T, 1, CIn>(J, Pin, Pout, s);
    }
    switch (J.tx) {
      case 2: return launch_cols_tx<T, 2, CIn>(J, Pin, Pout, s);
      case 8: return launch_cols_tx<T, 8, CIn>(J, Pin, Pout, s);
      default: return launch_cols_tx<T, 4, CIn>(J, Pin, Pout, s);
    }
  } else {
    switch (J.tx) {
      case 4: return launch_cols_tx<T, 4, CIn>(J, Pin, Pout, s);
      case 16: return launch_cols_tx<T, 16, CIn>(J, Pin, Pout, s);
      default: return launch_cols_tx<T, 8, CIn>(J, Pin, Pout, s);
    }
  }
}

template int launch_rows_r2c<double, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_c2r<double, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_cols<double, double2>(const ColJob&, const FftPlanDev&, const FftPlanDev&, cudaStream_t);
template int launch_rows_r2c<float, float>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_r2c<float, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_c2r<float, float>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_c2r<float, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_cols<float, float2>(const ColJob&, const FftPlanDev&, const FftPlanDev&, cudaStream_t);
template int launch_cols<float, double2>(const ColJob&, const FftPlanDev&, const FftPlanDev&, cudaStream_t);
template int launch_rows_r2c<dfloat, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_r2c<dfloat, dfloat>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_c2r<dfloat, double>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_rows_c2r<dfloat, dfloat>(const RowJob&, const RealPlanDev&, cudaStream_t);
template int launch_cols<dfloat, dcomplex>(const ColJob&, const FftPlanDev&, const FftPlanDev&, cudaStream_t);
template int launch_cols<dfloat, double2>(const ColJob&, const FftPlanDev&, const FftPlanDev&, cudaStream_t);

}  // namespace les
