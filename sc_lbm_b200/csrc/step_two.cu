// step_two.cu -- the two-steps-per-launch kernels (fused_two.cuh) of the FP32-
// and FP16-shifted forms.
#include "fused_two.cuh"

namespace sclbm {

cudaError_t launch_two2_f32(const Fused2Args<float, float> &a, int rows, cudaStream_t s)
{
    return launch_two2_any(a, rows, s);
}
cudaError_t launch_two2_f16(const Fused2Args<__half, float> &a, int rows, cudaStream_t s)
{
    return launch_two2_any(a, rows, s);
}
cudaError_t launch_batch_two_f32(const Fused2Args<float, float> *doms, const TwoUnit *units, int nunits,
                                 int parity, int flags, cudaStream_t s)
{
    return launch_batch_two_any(doms, units, nunits, parity, flags, s);
}
cudaError_t launch_batch_two_f16(const Fused2Args<__half, float> *doms, const TwoUnit *units, int nunits,
                                 int parity, int flags, cudaStream_t s)
{
    return launch_batch_two_any(doms, units, nunits, parity, flags, s);
}

} // namespace sclbm
