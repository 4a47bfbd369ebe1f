// The pair-solve kernels of one shape group and field type: a translation unit defines GATO_FAST_T
// (float or double), GATO_FAST_G (group number) and GATO_FAST_SHAPES (its table) and includes this.
#include "fast_shapes.cuh"
#include "poisson_fast.cuh"

namespace gato {
namespace fast {

using T = GATO_FAST_T;
using T2 = typename Cplx<T>::type;
constexpr bool kF32 = sizeof(T) == 4;
constexpr int kG = GATO_FAST_G;

// the launcher of a table row
template <int A, int B, int L32, int L64>
using Row = Launch<T, A, B, kF32 ? L32 : L64>;

#define GATO_FAST_CALL(CALL)                  \
  switch (M) { GATO_FAST_SHAPES(CALL) }       \
  return kNotHandled

template <>
int rows_L_g<T, kG>(int M) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return kF32 ? L32 : L64;
  switch (M) { GATO_FAST_SHAPES(X) }
#undef X
  return 0;
}

template <>
int cols_g<T, kG>(int M, int mode, const T2* in, T2* out, const ColGeom& g, int outer, int nf, const T2* tw,
                  const T* ghat, int H, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::cols(mode, in, out, g, outer, nf, tw, ghat, H, s);
  GATO_FAST_CALL(X);
#undef X
}

template <>
int rows_fwd_g<T, kG>(int M, const PassArgs& a, int f0, int nfg, T2* S1, const T2* tw, int multi, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::rows_fwd(a, f0, nfg, S1, tw, multi, s);
  GATO_FAST_CALL(X);
#undef X
}

template <>
int rows_inv_g<T, kG>(int M, const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, int accumulate,
                      bool energy, double* partials, int64_t slot_stride, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::rows_inv(a, f0, nfg, S1, tw, accumulate, energy, partials, slot_stride, s);
  GATO_FAST_CALL(X);
#undef X
}

template <>
int rows_inv_j_g<T, kG>(int M, const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::rows_inv_j(a, f0, nfg, S1, tw, s);
  GATO_FAST_CALL(X);
#undef X
}

template <>
int rows_fwd_real_g<T, kG>(int M, const PassArgs& a, int f0, int nfg, T2* S1, const T2* tw, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::rows_fwd_real(a, f0, nfg, S1, tw, s);
  GATO_FAST_CALL(X);
#undef X
}

template <>
int rows_inv_real_g<T, kG>(int M, const PassArgs& a, int f0, int nfg, const T2* S1, const T2* tw, int accumulate,
                           bool j, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::rows_inv_real(a, f0, nfg, S1, tw, accumulate, j, s);
  GATO_FAST_CALL(X);
#undef X
}

#ifdef GATO_FAST_FE   // the spectral energy pass (FP64 only)
template <>
int cols_fe_g<T, kG>(int M, const T2* in, const ColGeom& g, int outer, int nf, const T2* tw, const T* ghat, int H,
                     const FeArgs& fa, cudaStream_t s) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return Row<A, B, L32, L64>::cols_fe(in, g, outer, nf, tw, ghat, H, fa, s);
  GATO_FAST_CALL(X);
#undef X
}
#endif

}  // namespace fast
}  // namespace gato
