// fused_single.cuh -- several single-component time steps in one launch
// (collide, volume force, stream: src/lbm.cpp:275-288, 315-325, 343-384).
//
// Why.  One step of a small lattice is launch latency, one round of loads and
// the mask bytes behind them: the 200 x 50 channel took 4.6 us a step with 40
// of its CTAs on 148 SMs.  A single component couples nodes only through the
// streaming, one node per step, so a tile with a halo of K - 1 nodes can be
// advanced K steps in shared memory before it is written back.
//
// Measured on one B200, us per step, one step per launch before and K steps now
// (K by single_depth): FP64 200 x 50 4.7 -> 1.2, 700 x 333 8.2 -> 5.3, 4096^2 439
// -> 306; FP32 200 x 50 4.15 -> 0.85, 1024^2 18.6 -> 13.0, 4096^2 273 -> 196.
// Lattices a few nodes wide, and large ones stepped one step a call, do not fill
// the tiles or pay for the halo in vain: they take one node per thread (routes.h).
// Small lattices are bound by the chain of a step (loads from shared memory, a
// collision, a barrier) and a launch every K steps, large ones by instructions:
// the halo's repeated work against the DRAM traffic it saves.
//
// A CTA owns 32 - 2(K-1) columns and 16 - 2(K-1) rows; each of its 512 threads
// stands for one node of the tile with its halo.  Step s of k collides the
// nodes within k - s of the tile; all but the last step push into one of two
// shared buffers (the state between the steps, in the storage type), the last
// one pushes the tile's nodes into the output arrays.  A halo node is advanced
// by several CTAs from the same inputs, so the values are the same and equal
// to k single steps byte for byte.
#pragma once
#include "fused_step.cuh"
#include "launch.cuh"

namespace sclbm {

constexpr int SINGLE_W = 32, SINGLE_H = 16; // nodes of a tile with its halo

// two CTAs per SM: 64 registers for FP64, without spills (one CTA, 4096^2: 321
// us a step at K = 3; three, 40 registers: 426)
constexpr int SINGLE_CTAS = 2;

template <typename S, typename T, int K>
__global__ void __launch_bounds__(SINGLE_W * SINGLE_H, SINGLE_CTAS)
    k_single(const __grid_constant__ Fused1Args<S, T> a, int steps)
{
    constexpr int H = K - 1, TW = SINGLE_W - 2 * H, TH = SINGLE_H - 2 * H;
    constexpr int P = SINGLE_W + 2, NP = P * (SINGLE_H + 2); // one more node around: pushes off the halo
    constexpr int BUFS = K > 2 ? 2 : 1;
    static_assert(TW > 0 && TH > 0, "halo");
    extern __shared__ __align__(16) unsigned char single_raw[];
    S *const buf = reinterpret_cast<S *>(single_raw);                 // [BUFS][9][NP]
    uint8_t *const msk = single_raw + sizeof(S) * BUFS * 9 * NP;       // [NP]
    const int t = threadIdx.x, lx = t % SINGLE_W, ly = t / SINGLE_W;
    const int nx = a.nx, ny = a.ny;
    const int bx = blockIdx.x * TW, by = blockIdx.y * TH;
    const int ncol = min(TW, nx - bx), nrow = min(TH, ny - by);
    // distance of this node from the tile
    const int dx = lx < H ? H - lx : max(lx - (H + ncol - 1), 0);
    const int dy = ly < H ? H - ly : max(ly - (H + nrow - 1), 0);
    const int d = max(dx, dy);
    // a halo may wrap around a small lattice more than once
    int x = (bx - H + lx) % nx, y = (by - H + ly) % ny;
    x += x < 0 ? nx : 0;
    y += y < 0 ? ny : 0;
    const uint32_t node = (uint32_t)y * (uint32_t)nx + (uint32_t)x;
    const int p = (ly + 1) * P + lx + 1;
    dependent_wait();
    dependent_launch();
    T f[9];
    if (d < steps) {
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = Load<S>::value(a.fin + elem<false>(i, a.N, node));
    }
    const bool fluid = a.mask[node] == 1;
    msk[p] = fluid ? 1 : 0;
    // off the halo: a push goes to a slot that is never read, as would its
    // bounce-back
    if (t < 2 * P) msk[t < P ? t : (SINGLE_H + 1) * P + t - P] = 1;
    else if (t < 2 * P + 2 * SINGLE_H) msk[((t - 2 * P) / 2 + 1) * P + ((t & 1) ? P - 1 : 0)] = 1;
    __syncthreads();
    // bit i: the neighbour along c_i is fluid
    uint32_t nf = 1;
    if (d < steps) {
#pragma unroll
        for (int i = 1; i < 9; ++i) nf |= (uint32_t)msk[p + cy(i) * P + cx(i)] << i;
    }
    for (int s = 1; s < steps; ++s) {
        if (s > 1 && d <= steps - s) {
            const S *in = buf + ((s - 1) & (BUFS - 1)) * 9 * NP + p;
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i] = T(in[i * NP]);
        }
        if (fluid && d <= steps - s) {
            T out[9];
            collide_single<S, T>(a.c, f, out);
            S *to = buf + (s & (BUFS - 1)) * 9 * NP + p;
            to[0] = S(out[0]);
#pragma unroll
            for (int i = 1; i < 9; ++i)
                to[(nf >> i) & 1 ? i * NP + cy(i) * P + cx(i) : opp(i) * NP] = S(out[i]);
        }
        __syncthreads();
    }
    if (d != 0) return;
    if (!fluid) {
#pragma unroll
        for (int i = 0; i < 9; ++i) Store<S>::st(a.fout + elem<false>(i, a.N, node), T(0));
        return;
    }
    if (steps > 1) {
        const S *in = buf + ((steps - 1) & (BUFS - 1)) * 9 * NP + p;
#pragma unroll
        for (int i = 0; i < 9; ++i) f[i] = T(in[i * NP]);
    }
    T out[9];
    collide_single<S, T>(a.c, f, out);
    const Nbr n = make_nbr(nx, x, wrap1(x - 1, nx), wrap1(x + 1, nx), y, wrap1(y - 1, ny), wrap1(y + 1, ny));
    Store<S>::st(a.fout + elem<false>(0, a.N, node), out[0]);
#pragma unroll
    for (int i = 1; i < 9; ++i)
        Store<S>::st(a.fout + ((nf >> i) & 1 ? elem<false>(i, a.N, n.nb[i]) : elem<false>(opp(i), a.N, node)),
                     out[i]);
}

template <typename S, typename T, int K>
inline cudaError_t launch_single_k(const Fused1Args<S, T> &a, int steps, cudaStream_t s)
{
    constexpr int H = K - 1, TW = SINGLE_W - 2 * H, TH = SINGLE_H - 2 * H;
    constexpr size_t bytes = ((K > 2 ? 2 : 1) * 9 * sizeof(S) + 1) * (SINGLE_W + 2) * (SINGLE_H + 2);
    auto kern = k_single<S, T, K>;
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    const dim3 grid((a.nx + TW - 1) / TW, (a.ny + TH - 1) / TH);
    return launch_dependent(kern, grid, dim3(SINGLE_W * SINGLE_H), bytes, s, a, steps);
}

template <typename S, typename T>
inline cudaError_t launch_single_any(const Fused1Args<S, T> &a, int K, int steps, cudaStream_t s)
{
    if (steps < 1 || steps > K || !single_fits(a.nx, a.ny)) return cudaErrorInvalidValue;
    switch (K) {
    case 2: return launch_single_k<S, T, 2>(a, steps, s);
    case 3: return launch_single_k<S, T, 3>(a, steps, s);
    case 5: return launch_single_k<S, T, 5>(a, steps, s);
    case 6: return launch_single_k<S, T, 6>(a, steps, s);
    }
    return cudaErrorInvalidValue;
}

} // namespace sclbm
