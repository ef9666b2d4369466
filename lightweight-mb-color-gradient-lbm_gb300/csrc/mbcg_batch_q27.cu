// Batch kernels for D3Q27 and their table of step parameters.
#include "mbcg_batch_kernel.cuh"

namespace mbcg {

cudaError_t upload_batch_params_q27(const StepParams* params, int n, cudaStream_t s) {
    return cudaMemcpyToSymbolAsync(c_batch_params, params, sizeof(StepParams) * 2 * n, 0, cudaMemcpyHostToDevice, s);
}

cudaError_t launch_batch_q27(int kind, const BatchCase* cases, const BatchTile* tiles, int ntiles, const ChunkState* chunk,
                             int* counter, int j, int grid, cudaStream_t s) {
    return launch_batch_kind<27>(kind, cases, tiles, ntiles, chunk, counter, j, grid, s);
}

} // namespace mbcg
