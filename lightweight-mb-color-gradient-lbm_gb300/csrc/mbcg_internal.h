// mbcg_internal.h -- declarations shared by the translation units of libmbcg.so.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "mbcg.h"
#include "mbcg_lattice.cuh"

namespace mbcg {

// Step CTA shapes.  A warp is 32 lanes (30 destination columns plus halo) and two source rows, one in
// each half of packed registers; a CTA of R source rows (R / 2 warps) owns R - 2 destination rows.
// The plain step is built for two shapes, named by the block_rows of the C ABI:
//   16 (default): 24 source rows, 12 warps, one CTA per SM (168 registers a thread)
//    8:            8 source rows,  4 warps, two CTAs per SM
constexpr int kStepW = 16;
constexpr int kStepWSmall = 8;
constexpr int step_rows(int w) { return w == kStepWSmall ? 8 : 24; }
// Lattices in BF16 storage without an inlet, and in FP16 storage fully periodic and unforced ones, step by
// populations, one node a thread, w source rows, on every path: cases, the server, plain loads (the reason
// stands in mbcg_step_pop.cuh).
constexpr bool uses_pop(int precision, int features) {
    return precision == MBCG_BF16 ? (features & F_INOUT) == 0 : precision == MBCG_FP16 && features == 0;
}
constexpr int kStepTileX = 30; // destination columns per tile
constexpr int kStepRBX = 48;   // staged width of the rhor / rhob boxes
constexpr int kStepMX = 40;    // staged width of the other nine boxes

struct TensorMaps {
    CUtensorMap m[NF];
};

// fused step (mbcg_step.cu; instantiations in mbcg_step_q{19,27}_{f32,f16,bf16}.cu)
cudaError_t launch_step(int q, int precision, bool tma, int w, const StepParams& P, const TensorMaps& T,
                        cudaStream_t s);
cudaError_t launch_step_q19_f32(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
cudaError_t launch_step_q19_f16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
cudaError_t launch_step_q19_bf16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
cudaError_t launch_step_q27_f32(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
cudaError_t launch_step_q27_f16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
cudaError_t launch_step_q27_bf16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s);
int step_smem_bytes(int precision, int w);
inline int step_tile_rows(int w) { return step_rows(w) - 2; } // destination rows
// The step addresses the planes of a tile by 32-bit byte offsets: the deepest tile it may be given.
inline int max_zchunk(long long plane, int elem_bytes) {
    const long long bytes = plane * elem_bytes;
    return static_cast<int>(std::min<long long>(1 << 20, std::max<long long>(1, ((1LL << 32) - 1) / bytes - 1)));
}

// boundary functors, initial conditions, diagnostics, layout conversion (mbcg_aux.cu)
cudaError_t launch_bc(int precision, const StepParams& P, cudaStream_t s);
cudaError_t launch_fill_ghosts(int precision, const StepParams& P, cudaStream_t s); // on P.b
cudaError_t launch_init(int precision, const StepParams& P, const mbcg_params& p, cudaStream_t s);
cudaError_t launch_diag(int precision, const StepParams& P, const mbcg_params& p, double* partials, int nparts,
                        double* result, cudaStream_t s);
int diag_partials_needed(const StepParams& P);
// one field between the state and the reference's dense FP32 layout (P.a -> dst; src -> P.b,
// where the 16-bit forms take rhor and rhob together as field 0 and skip field 1)
cudaError_t launch_to_dense(int precision, const StepParams& P, int field, float* dst, cudaStream_t s);
// all fields between the state (P.a for the read, P.b for the write) and dense FP32 fields in
// host memory the device accesses directly (device pointers of pinned host memory)
cudaError_t launch_state_to_host(int precision, const StepParams& P, float* const host[NF], cudaStream_t s);
cudaError_t launch_host_to_state(int precision, const StepParams& P, const float* const host[NF], cudaStream_t s);
cudaError_t launch_from_dense(int precision, const StepParams& P, int field, const float* src, const float* src_b,
                              cudaStream_t s);

// sets the message mbcg_last_error() returns on the calling thread (mbcg_capi.cu)
void set_last_error(const std::string& msg);
// one field of a case's current state as dense FP32 (reference layout) into dst, on stream s;
// the step counter of a case (restart from a checkpoint) (mbcg_capi.cu)
int case_field_to_dense(mbcg_case* c, int field, float* dst, cudaStream_t s);
int case_state_params(mbcg_case* c, StepParams* out); // parameter block with P.a = current state
int mirror_state(mbcg_case* c, cudaStream_t s); // current state -> the other (never-written layers agree)
void case_set_steps(mbcg_case* c, long long steps);
// parameter checks, the step's constant chain and TMA descriptors, shared by the case API and
// the server (mbcg_capi.cu); validate_params sets the last-error message on failure
int validate_params(const mbcg_params* p);
void fill_step_physics(const mbcg_params& p, StepParams& P);
bool state_tma_capable(const mbcg_params& p, const void* const* f, long long pitch);
int encode_state_maps(const mbcg_params& p, const void* const* f, long long pitch, int rows, TensorMaps& T);

constexpr int kDiagSlots = 12; // mass_r, mass_b, mom x/y/z, p_in sum, n_in, p_out sum, n_out, nonfinite, nodes, spare

} // namespace mbcg
