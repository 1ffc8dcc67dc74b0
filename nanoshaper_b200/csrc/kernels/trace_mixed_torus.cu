// Mixed-precision torus intersection kernels, compiled without fused multiply-adds like the
// double-precision path: their clipping-sphere entry and quartic solve repeat the FP64 path's
// operations (only the feasibility tests run in FP32), so that the reference's solver, which is
// ill-conditioned for some rays, returns the same roots in both precisions.
#include "isect.cuh"

namespace nsg {

void launch_isect_mixed_torus(const TraceSets& T, dim3 grid, int threads, cudaStream_t s) {
  k_isect_mixed<true><<<grid, threads, 0, s>>>(T);
}

}  // namespace nsg
