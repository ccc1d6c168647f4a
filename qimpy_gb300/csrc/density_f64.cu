// Density kernel, FP64.
#include "density_kernels.cuh"

namespace qgb {

template int launch_density_chunk<double>(const qgb_sphere&, const LocalParams&, const void*, void*, const double*,
                                    double*, cudaStream_t);
#ifdef QGB_DEBUG_CHECKS
int violation_density_f64(unsigned long long* out4) { return unit_violation(out4); }
#endif

}  // namespace qgb
