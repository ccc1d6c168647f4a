// Density kernel, FP32.
#include "density_kernels.cuh"

namespace qgb {

template int launch_density_chunk<float>(const qgb_sphere&, const LocalParams&, const void*, void*, const double*,
                                    double*, cudaStream_t);

}  // namespace qgb
