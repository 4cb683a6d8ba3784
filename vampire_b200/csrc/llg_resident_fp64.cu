// FP64 instantiation of the resident LLG steps (built without FMA contraction, as
// the FP64 passes are).
#include "llg_resident.cuh"

namespace vgpu {
template cudaError_t resident_capacity<double>(const LLGArgs<double>&, int, int, const ResidentPlan&, int, int*);
template cudaError_t launch_resident_check<double>(const LLGArgs<double>&, int*, cudaStream_t);
template cudaError_t launch_llg_resident<double>(const LLGArgs<double>&, int, int, int, const ResidentPlan&, int, cudaStream_t);
template cudaError_t path_fits<double>(const LLGArgs<double>&, int, const ResidentPlan&, int, bool*);
template cudaError_t launch_llg_path<double>(const LLGArgs<double>&, int, int, const ResidentPlan&, int, double*, double*, int, double*, double*, cudaStream_t);
}  // namespace vgpu
