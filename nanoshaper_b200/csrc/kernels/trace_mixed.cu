// Mixed-precision ray-patch intersection kernels of spheres and skin cells, compiled with fused
// multiply-adds (the build gives this file --fmad=true; every other device file, the mixed torus
// kernels of trace_mixed_torus.cu included, is compiled with --fmad=false).
#include "isect.cuh"

namespace nsg {

void launch_isect_mixed_sphere(const TraceSets& T, dim3 grid, int threads, cudaStream_t s) {
  k_isect_mixed<false><<<grid, threads, 0, s>>>(T);
}

void launch_isect_quad_mixed(const TraceSets& T, dim3 grid, int threads, cudaStream_t s) {
  k_isect_quad_mixed<<<grid, threads, 0, s>>>(T);
}

}  // namespace nsg
