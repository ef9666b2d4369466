// mbcg_batch_kernel.cuh -- persistent batch step: one launch per kind of body advances every live lattice
// of that kind by one time step.
//
// The work is a flat queue of tiles (BatchTile) over the live lattices of one kind (Q, storage, feature
// set), sorted by the host, largest tiles first.  Each CTA of a grid of at most one CTA per SM takes the
// next tile with an atomic counter and runs the same step_tile(), or pop::tile(), as the plain kernel on that
// lattice's step parameters in a constant-memory table indexed by slot.  The mbarriers are initialised once
// per CTA; their parities carry from tile to tile.  The kinds' launches of one step are branches of the
// server's graph and overlap: a kind's next step waits for its own tiles only.
//
// One kernel per kind, not one with every body: side by side in one kernel the bodies spilled 280 bytes
// each (values hoisted across them), as functions 170 to 770; alone they spill nothing, or 4 to 240 bytes
// in the parts for walls and inlets.
#pragma once

#include "mbcg_batch.h"
#include "mbcg_step.cuh"
#include "mbcg_step_pop.cuh"

namespace mbcg {

namespace {

__constant__ StepParams c_batch_params[kBatchParamSlots * 2]; // [slot][parity]

// kPop: the step by populations, W warps of one row each; otherwise W / 2 of two.
template <int Q, typename S, int W, int kFeat, bool kPop>
__global__ void __launch_bounds__(kPop ? 32 * W : 16 * W, 1)
    batch_kernel(const BatchCase* __restrict__ cases, const BatchTile* __restrict__ tiles, int ntiles,
                 const ChunkState* __restrict__ chunk, int* __restrict__ counter, int j) {
    __shared__ int s_tile;
    init_barriers<kPop ? 0 : W / 2>(aligned_smem_base());
    uint32_t phase = 0;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    for (;;) {
        __syncthreads(); // everyone is done with the previous tile's s_tile
        if (tid == 0) s_tile = atomicAdd(counter, 1);
        __syncthreads();
        const int t = s_tile;
        if (t >= ntiles) return;
        const BatchTile bt = tiles[t];
        const ChunkState cs = chunk[bt.slot];
        if (j >= cs.nsteps) continue;
        const int par = cs.parity0 ^ (j & 1);
        const StepParams& P = c_batch_params[bt.slot * 2 + par]; // this lattice, this parity
        const CUtensorMap* maps = cases[bt.slot].maps[par];
        const long long step = cs.step0 + j + 1;
        bool ok;
        if constexpr (kPop) {
            ok = pop::tile<Q, S, W, true, kFeat>(P, maps, bt.bx, bt.by, bt.bz, step, aligned_smem_base(), phase);
        } else if constexpr ((kFeat & (F_WALL | F_INOUT)) != 0) {
            constexpr int kInner = kFeat & ~(F_WALL | F_INOUT);
            ok = tile_is_interior<W>(P, bt.bx, bt.by, bt.bz)
                     ? step_tile<Q, S, W, true, kInner, true>(P, maps, bt.bx, bt.by, bt.bz, step, aligned_smem_base(), phase)
                     : step_tile<Q, S, W, true, kFeat, true>(P, maps, bt.bx, bt.by, bt.bz, step, aligned_smem_base(), phase);
        } else {
            ok = step_tile<Q, S, W, true, kFeat, true>(P, maps, bt.bx, bt.by, bt.bz, step, aligned_smem_base(), phase);
        }
        if (!ok) return; // the tile has set the lattice's status word
    }
}

template <int Q, typename S, int kFeat, bool kPop = false>
cudaError_t launch_batch_one(const BatchCase* cases, const BatchTile* tiles, int ntiles, const ChunkState* chunk,
                             int* counter, int j, int grid, cudaStream_t s) {
    constexpr int W = kPop ? kBatchW : step_rows(kBatchW);
    constexpr int smem = kPop ? pop::Geo<S, W>::smem : Geo<S, W>::smem;
    auto kern = batch_kernel<Q, S, W, kFeat, kPop>;
    static std::atomic<unsigned long long> configured{0};
    if (cudaError_t e = configure_once(kern, smem, configured)) return e;
    if (grid < 1 || ntiles < 1) return cudaSuccess;
    kern<<<grid, dim3(32, kPop ? W : W / 2, 1), smem, s>>>(cases, tiles, ntiles, chunk, counter, j);
    return cudaGetLastError();
}

template <int Q>
cudaError_t launch_batch_kind(int kind, const BatchCase* cases, const BatchTile* tiles, int ntiles,
                              const ChunkState* chunk, int* counter, int j, int grid, cudaStream_t s) {
    switch (kind) {
    case BK_Q19_F32:
    case BK_Q27_F32: return launch_batch_one<Q, float, F_ALL>(cases, tiles, ntiles, chunk, counter, j, grid, s);
    case BK_Q19_F16:
    case BK_Q27_F16: return launch_batch_one<Q, __half, F_ALL>(cases, tiles, ntiles, chunk, counter, j, grid, s);
    case BK_Q19_BF16:
    case BK_Q27_BF16: return launch_batch_one<Q, __nv_bfloat16, F_ALL>(cases, tiles, ntiles, chunk, counter, j, grid, s);
    case BK_Q19_F32_P:
    case BK_Q27_F32_P: return launch_batch_one<Q, float, 0>(cases, tiles, ntiles, chunk, counter, j, grid, s);
    case BK_Q19_F16_P:
    case BK_Q27_F16_P: return launch_batch_one<Q, __half, 0, true>(cases, tiles, ntiles, chunk, counter, j, grid, s);
    case BK_Q19_BF16_N:
    case BK_Q27_BF16_N:
        return launch_batch_one<Q, __nv_bfloat16, pop::pop_features<__nv_bfloat16>(), true>(cases, tiles, ntiles, chunk,
                                                                                             counter, j, grid, s);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace

} // namespace mbcg
