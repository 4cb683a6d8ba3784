// FP32 instantiation of the resident LLG steps.
#include "llg_resident.cuh"

namespace vgpu {
template cudaError_t resident_capacity<float>(const LLGArgs<float>&, int, int, const ResidentPlan&, int, int*);
template cudaError_t launch_resident_check<float>(const LLGArgs<float>&, int*, cudaStream_t);
template cudaError_t launch_llg_resident<float>(const LLGArgs<float>&, int, int, int, const ResidentPlan&, int, cudaStream_t);
template cudaError_t path_fits<float>(const LLGArgs<float>&, int, const ResidentPlan&, int, bool*);
template cudaError_t launch_llg_path<float>(const LLGArgs<float>&, int, int, const ResidentPlan&, int, float*, float*, int, float*, double*, cudaStream_t);
}  // namespace vgpu
