// step_single64.cu -- FP64 instantiations of the single-component steps
// (fused_single.cuh), compiled with -fmad=false (bit-exact with the reference).
#include "fused_single.cuh"

namespace sclbm {

cudaError_t launch_single_fp64(const Fused1Args<double, double> &a, int K, int steps, cudaStream_t s)
{
    return launch_single_any(a, K, steps, s);
}

} // namespace sclbm
