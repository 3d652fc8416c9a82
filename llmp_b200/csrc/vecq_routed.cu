// The routed Q4_K vecq kernel's instantiations.
#include "vecq_routed.cuh"

namespace llmp_b200 {
namespace vecq {
namespace {
template <bool kGlu>
cudaError_t LaunchRoutedOne(const Desc& d, const RoutedPlan& plan, cudaStream_t stream) {
  auto* kernel = VecQRoutedKernel<kGlu>;
  static thread_local int configured_device = -1;
  int device = -1;
  cudaGetDevice(&device);
  if (configured_device != device) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               225 * 1024);
    if (e != cudaSuccess) return e;
    configured_device = device;
  }
  return LaunchPdl(kernel, dim3(static_cast<unsigned>(plan.grid)),
                   dim3(static_cast<unsigned>(plan.groups * plan.col_groups * 32)),
                   static_cast<std::size_t>(plan.smem_bytes), stream, d, plan);
}
}  // namespace

cudaError_t LaunchRouted(const Desc& d, const RoutedPlan& plan, cudaStream_t stream) {
  return d.glu != LLMP_B200_GLU_NONE ? LaunchRoutedOne<true>(d, plan, stream)
                                     : LaunchRoutedOne<false>(d, plan, stream);
}
}  // namespace vecq
}  // namespace llmp_b200
