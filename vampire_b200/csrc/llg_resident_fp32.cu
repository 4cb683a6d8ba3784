// FP32 instantiation of the resident LLG steps.
#include "llg_resident.cuh"

namespace vgpu {
template cudaError_t resident_capacity<float>(const LLGArgs<float>&, int, int, const ResidentPlan&, int, int*);
template cudaError_t launch_resident_check<float>(const LLGArgs<float>&, int*, cudaStream_t);
template cudaError_t launch_llg_resident<float>(const LLGArgs<float>&, int, int, int, const ResidentPlan&, int, cudaStream_t);
template cudaError_t cluster_capacity<float>(const LLGArgs<float>&, int, int, const ClusterShape&, int*);
template cudaError_t launch_llg_cluster<float>(const LLGArgs<float>&, int, int, int, const ClusterShape&, cudaStream_t);
}  // namespace vgpu
