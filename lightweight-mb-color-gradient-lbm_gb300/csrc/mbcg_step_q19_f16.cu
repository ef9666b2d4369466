// Plain step kernels for D3Q19 with __half storage: block shapes 8 and 16, feature sets
// {inlet/outlet, walls + force, all} on the TMA path and all features on the plain-load path; the step by
// populations.
#include "mbcg_step_pop.cuh"

namespace mbcg {

cudaError_t launch_step_q19_f16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    if (uses_pop(MBCG_FP16, features_of(P))) return pop::launch<19, __half>(tma, w, P, T, s);
    return launch_qs<19, __half>(tma, w, P, T, s);
}

} // namespace mbcg
