// Instantiations of the packed two-line FP32 column passes, and the register engine's shape lookup.
#include "fast_shapes.cuh"
#include "poisson_packed.cuh"

namespace gato {
namespace fast {

int shape_r2(int M) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return B;
  switch (M) { GATO_FAST_SHAPES_ALL(X) }
#undef X
  return 0;
}

int strand_fields(int M, bool j) {
#define X(MM, A, B, L32, L64, A32, J32) \
  case MM: return j ? J32 : A32;
  switch (M) { GATO_FAST_SHAPES_ALL(X) }
#undef X
  return 0;
}

// Packed two-line column passes: M -> (R1, R2), 8 line pairs per CTA.
#define GATO_PACKED_SHAPES(X) X(128, 8, 16) X(160, 10, 16) X(192, 12, 16) X(256, 16, 16) X(320, 20, 16)

int packed_r2(int M) {
#define X(MM, A, B) \
  case MM: return B;
  switch (M) { GATO_PACKED_SHAPES(X) }
#undef X
  return 0;
}

int packed_cols(int M, int mode, const float2* in, float2* out, const ColGeom& g, int outer, int nf,
                const float4* tw4, const float* ghat2, int H, cudaStream_t s) {
#define X(MM, A, B) \
  case MM: return packed::LaunchP<A, B, 8>::cols(mode, in, out, g, outer, nf, tw4, ghat2, s);
  switch (M) { GATO_PACKED_SHAPES(X) }
#undef X
  return kNotHandled;
}

}  // namespace fast
}  // namespace gato
