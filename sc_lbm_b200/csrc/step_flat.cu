// step_flat.cu -- FP32-arithmetic instantiations of the one-node-per-thread
// step (fused_flat.cuh).
#include "fused_flat.cuh"

namespace sclbm {

// 32-bit element offsets and the grid's y limit
bool flat_fits(size_t nx, size_t ny)
{
    return nx >= 1 && ny >= 1 && !needs_wide_offsets(nx * ny) && (ny + FLAT_ROWS - 1) / FLAT_ROWS <= 65535;
}

cudaError_t launch_flat2_f32(const Fused2Args<float, float> &a, cudaStream_t s)
{
    return launch_flat2_any<float, float, KF_UNIFORM>(a, s);
}
cudaError_t launch_flat2_f16(const Fused2Args<__half, float> &a, cudaStream_t s)
{
    return launch_flat2_any<__half, float, KF_UNIFORM>(a, s);
}

} // namespace sclbm
