// Internal entry of the stencil kernels (used by the operator and the C ABI).
#pragma once
#include "common.cuh"

namespace gato {
// How the TMA kernel chains (ptx.cuh). Late: the kernel ahead of it in the stream calls gdc_launch only once
// its own predecessor has ended, and touches neither psi, V nor out, so the stencil runs beside it and waits
// for it at its end. Open: the next chained kernel may begin beside the stencil; psi is complete then, out is
// after its gdc_wait.
constexpr int kChainLate = 1, kChainOpen = 2;
// out[b] = coef * L(psi[b]) + V * psi[b]; dot_dev[b] = dv * <psi[b], out[b]>. beside: other kernels run
// on the GPU at the same time (a choice of tiles, not of results).
int stencil_apply(int dtype, const void* psi, const void* V, void* out, int nb, int nx, int ny,
                  int nz, int64_t bstride, double coef, int boundary, int order, double* dot_dev,
                  double dv, cudaStream_t s, bool beside = false, int chain = 0);
}  // namespace gato
