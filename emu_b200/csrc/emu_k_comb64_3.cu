// emu_k_comb64_3.cu -- FP64 stage and deposit kernels on combined meshes for
// 3 flavors.
#include "emu_fp64_impl.cuh"

namespace emu {
template void launch_stage64_t<3>(const DevParams&, const DevState&, int, const double*, double*, double*, double*,
                                  StepCtl*, int, cudaStream_t, const DevState*, const unsigned*, unsigned*,
                                  unsigned*);
template void launch_deposit_comb64_t<3>(const DevParams&, const DevState&, double*, const StepCtl*, cudaStream_t);
template void launch_deposit_full64_t<3>(const DevParams&, const DevState&, const double*, double*, StepCtl*,
                                         cudaStream_t);
}  // namespace emu
