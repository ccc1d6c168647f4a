// Density kernel, FP32.
#include "density_kernels.cuh"

namespace qgb {

template int launch_density_chunk<float>(const qgb_sphere&, const LocalParams&, const void*, void*, const double*,
                                    double*, cudaStream_t);
#ifdef QGB_DEBUG_CHECKS
int violation_density_f32(unsigned long long* out4) { return unit_violation(out4); }
#endif

}  // namespace qgb
