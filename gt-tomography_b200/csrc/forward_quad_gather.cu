// forward_quad_gather.cu -- row-quad forward projector in the gather kernel's form
// (LerpForm): instantiations of forward_quad.cuh for launches whose rows TMA cannot
// read in place.
#include "forward_quad.cuh"

namespace cbct {

template <class V>
QuadKernel<V> quad_kernel_gather(const cbct_plan* p) {
  QuadKernel<V> k = nullptr;
  with_quad<V>(p, [&](auto BX, auto SHAPE) { k = quad_kernel_of<V, decltype(BX)::value, decltype(SHAPE)::value, true>(); });
  return k;
}

template QuadKernel<float> quad_kernel_gather<float>(const cbct_plan*);
template QuadKernel<__half> quad_kernel_gather<__half>(const cbct_plan*);
template QuadKernel<__nv_bfloat16> quad_kernel_gather<__nv_bfloat16>(const cbct_plan*);

}  // namespace cbct
