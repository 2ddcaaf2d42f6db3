// batch_resident_f64.cu -- batch_resident.cuh in FP64.
#include "batch_resident.cuh"

namespace pdhg {

template void init_resident_kernels<double>();
template bool plan_resident<double>(const std::vector<ResParts>&, int, int, bool, ResPlan&);
template cudaError_t launch_batch_resident<double>(const std::vector<ResClass>&, const ResBuffers&, int, int,
                                                const BatchView&, const Iterates<double>&, const BatchParams&, long long,
                                                long long, long long, cudaStream_t, const ResStreams&);

}  // namespace pdhg
