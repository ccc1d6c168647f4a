// Local-potential kernels of one sphere, FP32.
#include "local_kernels.cuh"

namespace qgb {

template int launch_ifft_yz<float>(const qgb_sphere&, const LocalParams&, const void*, void*, cudaStream_t);
template int launch_chunk<float>(const qgb_sphere&, const LocalParams&, const void*, void*, void*, cudaStream_t,
                            cudaEvent_t);
#ifdef QGB_DEBUG_CHECKS
int violation_local_f32(unsigned long long* out4) { return unit_violation(out4); }
#endif

}  // namespace qgb
