// mbcg_batch.cu -- the batch step's dispatch (kernels in mbcg_batch_q{19,27}.cu) and the state hash.
#include <algorithm>

#include "mbcg_batch.h"

namespace mbcg {

namespace {

// order-independent: sum over nodes of mix64(field, index, bits), wrapping
template <typename S>
__global__ void state_hash_kernel(const StepParams P, unsigned long long* out) {
    const long long nxf = P.nx - 2, nyf = P.ny - 2, nzf = P.nz - 2;
    const long long total = nxf * nyf * nzf;
    unsigned long long acc = 0;
    for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long x = 1 + e % nxf, y = 1 + (e / nxf) % nyf, z = 1 + e / (nxf * nyf);
        const long long o = z * P.plane + y * P.pitch + x;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            unsigned long long bits;
            if constexpr (sizeof(S) == 4) bits = __float_as_uint(static_cast<const float*>(P.a[f])[o]);
            else bits = *reinterpret_cast<const unsigned short*>(static_cast<const S*>(P.a[f]) + o);
            acc += mix64((static_cast<unsigned long long>(e) * 16ULL + f) * 0x9E3779B97F4A7C15ULL ^ (bits << 1));
        }
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

} // namespace

cudaError_t upload_batch_params(const StepParams* params, int n, cudaStream_t s) {
    if (n < 0 || n > kBatchParamSlots) return cudaErrorInvalidValue;
    if (cudaError_t e = upload_batch_params_q19(params, n, s)) return e;
    return upload_batch_params_q27(params, n, s);
}

cudaError_t launch_batch(int kind, const BatchCase* cases, const BatchTile* tiles, int ntiles, const ChunkState* chunk,
                         int* counter, int j, int grid, cudaStream_t s) {
    if (kind < 0 || kind >= BK_COUNT) return cudaErrorInvalidValue;
    return batch_q(kind) == 27 ? launch_batch_q27(kind, cases, tiles, ntiles, chunk, counter, j, grid, s)
                               : launch_batch_q19(kind, cases, tiles, ntiles, chunk, counter, j, grid, s);
}

cudaError_t launch_state_hash(int precision, const StepParams& P, unsigned long long* out, cudaStream_t s) {
    const long long n = static_cast<long long>(P.nx - 2) * (P.ny - 2) * (P.nz - 2);
    const int grid = static_cast<int>(std::min<long long>((n + 255) / 256, 1184));
    switch (precision) {
    case MBCG_FP16: state_hash_kernel<__half><<<grid, 256, 0, s>>>(P, out); break;
    case MBCG_BF16: state_hash_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>(P, out); break;
    default: state_hash_kernel<float><<<grid, 256, 0, s>>>(P, out); break;
    }
    return cudaGetLastError();
}

} // namespace mbcg
