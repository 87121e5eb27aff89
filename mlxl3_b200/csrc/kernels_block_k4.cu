// Instantiates the cluster-per-column-block linear-layer kernels for K = 4 bits per weight.
#include "kernels_block_impl.cuh"

namespace b200exl3 {
cudaError_t block_dispatch_k4(const QmvArgs& p, int cb, bool exact, const BlockPlan& plan, cudaStream_t stream) {
    return block_launch_k<4>(p, cb, exact, plan, stream);
}
// the count depends on the board and the shared memory, not on the bits: asked of one instantiation
cudaError_t block_resident_clusters(int cluster, int* clusters) { return block_resident<4, 0, 0, 0>(cluster, clusters); }
}  // namespace b200exl3
