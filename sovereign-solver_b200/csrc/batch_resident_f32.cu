// batch_resident_f32.cu -- batch_resident.cuh in FP32.
#include "batch_resident.cuh"

namespace pdhg {

template void init_resident_kernels<float>();
template bool plan_resident<float>(const std::vector<ResParts>&, int, int, bool, ResPlan&);
template cudaError_t launch_batch_resident<float>(const std::vector<ResClass>&, const ResBuffers&, int, int,
                                                const BatchView&, const Iterates<float>&, const BatchParams&, long long,
                                                long long, long long, cudaStream_t, const ResStreams&);

}  // namespace pdhg
