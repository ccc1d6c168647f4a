// Batched local-potential kernels, FP32.
#include "batched_kernels.cuh"

namespace qgb {

template int launch_batched<float>(const qgb_batch_item*, const int*, const long long*, const int*, const long long*,
                              long long, long long, size_t, size_t, cudaStream_t);
#ifdef QGB_DEBUG_CHECKS
int violation_batched_f32(unsigned long long* out4) { return unit_violation(out4); }
#endif

}  // namespace qgb
