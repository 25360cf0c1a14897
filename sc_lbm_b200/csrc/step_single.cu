// step_single.cu -- FP32-arithmetic instantiations of the single-component
// steps (fused_single.cuh).
#include "fused_single.cuh"

namespace sclbm {

// 32-bit element offsets and the grid's y limit (tiles of at least six rows)
bool single_fits(size_t nx, size_t ny)
{
    return nx >= 1 && ny >= 1 && nx < ((size_t)1 << 30) && !needs_wide_offsets(nx * ny) && ny / 6 < 65535;
}

// Steps per launch.  While the tiles of six steps (22 x 6 nodes) fit the GPU at
// once a launch's latency is worth the halo's work; then five steps for the
// shifted forms up to one and a half waves of their tiles (24 x 8), and as many
// as pay for the repeated halo: three for the shifted forms, three for FP64 up
// to one wave (28 x 12), then two.  us per step for K = 2 / 3 / 5 / 6: FP64 200 x
// 50 2.16 / 1.74 / 1.36 / 1.23, 400 x 200 3.07 / 2.66 / 2.81 / 3.85, 1500 x 600
// 18.5 / 19.0 / 24.7 / 32.6; FP32 200 x 50 1.64 / 1.31 / 0.96 / 0.85, 400 x 200
// 2.29 / 2.33 / 1.77 / 2.38, 1500 x 600 12.9 / 11.2 / 14.5 / 18.9.
int single_depth(size_t nx, size_t ny, bool fp64)
{
    const size_t wave = 2 * (size_t)sm_count();
    auto tiles = [&](size_t w, size_t h) { return ((nx + w - 1) / w) * ((ny + h - 1) / h); };
    if (tiles(22, 6) <= wave) return 6;
    if (fp64) return tiles(28, 12) <= wave ? 3 : 2;
    return tiles(24, 8) <= wave + wave / 2 ? 5 : 3;
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
