// step_flat64.cu -- FP64 instantiations of the one-node-per-thread step
// (fused_flat.cuh), compiled with -fmad=false (bit-exact with the reference).
#include "fused_flat.cuh"

namespace sclbm {

cudaError_t launch_flat2_fp64(const Fused2Args<double, double> &a, cudaStream_t s)
{
    return launch_flat2_any<double, double, 0>(a, s);
}
cudaError_t launch_batch_flat_fp64(const Fused2Args<double, double> *doms, const FlatTile *tiles, int ntiles,
                                   int parity, int flags, cudaStream_t s)
{
    return launch_batch_flat_any<double, double, 0>(doms, tiles, ntiles, parity, flags, s);
}

} // namespace sclbm
