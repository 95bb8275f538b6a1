// The decode GEMV (decode_gemv.cu) over block-scaled float planes and the re-laid 32-value block types.
#include "gemv_kernel.cuh"

namespace bl {
template cudaError_t gemv_family<true, 2>(const GemvArgs&, const GemvPlan&, cudaStream_t);
template cudaError_t gemv_family<false, 2>(const GemvArgs&, const GemvPlan&, cudaStream_t);
}  // namespace bl
