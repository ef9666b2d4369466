// Plain step kernels for D3Q27 with __nv_bfloat16 storage: block shapes 8 and 16, feature sets
// {inlet/outlet, all} on the TMA path and all features on the plain-load path; the step by populations.
#include "mbcg_step_pop.cuh"

namespace mbcg {

cudaError_t launch_step_q27_bf16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    if (uses_pop(MBCG_BF16, features_of(P))) return pop::launch<27, __nv_bfloat16>(tma, w, P, T, s);
    return launch_qs<27, __nv_bfloat16>(tma, w, P, T, s);
}

} // namespace mbcg
