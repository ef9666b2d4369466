// Plain step kernels for D3Q19 with __half storage: block shapes W = 8 and 16, feature sets
// {none, inlet/outlet, all} on the TMA path and all features on the plain-load path.
#include "mbcg_step_pop.cuh"

namespace mbcg {

cudaError_t launch_step_q19_f16(bool tma, int w, const StepParams& P, const TensorMaps& T, cudaStream_t s) {
    if (tma && uses_pop(sizeof(__half) == 2, features_of(P)))
        return w == kStepWSmall ? pop::launch<19, __half, kStepWSmall>(P, T, s) : pop::launch<19, __half, kStepW>(P, T, s);
    return launch_qs<19, __half>(tma, w, P, T, s);
}

} // namespace mbcg
