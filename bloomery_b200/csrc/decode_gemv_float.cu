// The decode GEMV (decode_gemv.cu) of calls with F32 / F16 / BF16 rows among their weights.
#include "gemv_kernel.cuh"

namespace bl {
template cudaError_t gemv_family<true, 1>(const GemvArgs&, const GemvPlan&, cudaStream_t);
}  // namespace bl
