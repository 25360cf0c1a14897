// step_single.cu -- FP32-arithmetic instantiations of the single-component
// steps (fused_single.cuh).
#include "fused_single.cuh"

namespace sclbm {

// 32-bit element offsets and the grid's y limit (tiles of at least six rows)
bool single_fits(size_t nx, size_t ny)
{
    return nx >= 1 && ny >= 1 && nx < ((size_t)1 << 30) && !needs_wide_offsets(nx * ny) && ny / 6 < 65535;
}

cudaError_t launch_single_f32(const Fused1Args<float, float> &a, int K, int steps, cudaStream_t s)
{
    return launch_single_any(a, K, steps, s);
}
cudaError_t launch_single_f16(const Fused1Args<__half, float> &a, int K, int steps, cudaStream_t s)
{
    return launch_single_any(a, K, steps, s);
}

} // namespace sclbm
