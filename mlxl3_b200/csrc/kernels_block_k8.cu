// Instantiates the cluster-per-column-block linear-layer kernels for K = 8 bits per weight.
#include "kernels_block_impl.cuh"

namespace b200exl3 {
cudaError_t block_dispatch_k8(const QmvArgs& p, int cb, bool exact, const BlockPlan& plan, cudaStream_t stream) {
    return block_launch_k<8>(p, cb, exact, plan, stream);
}
}  // namespace b200exl3
