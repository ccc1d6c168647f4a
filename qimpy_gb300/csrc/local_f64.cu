// Local-potential kernels of one sphere, FP64.
#include "local_kernels.cuh"

namespace qgb {

template int launch_ifft_yz<double>(const qgb_sphere&, const LocalParams&, const void*, void*, cudaStream_t);
template int launch_chunk<double>(const qgb_sphere&, const LocalParams&, const void*, void*, void*, cudaStream_t,
                            cudaEvent_t);
#ifdef QGB_DEBUG_CHECKS
int violation_local_f64(unsigned long long* out4) { return unit_violation(out4); }
#endif

}  // namespace qgb
