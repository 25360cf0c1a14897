// fused_flat.cuh -- the fused two-component step with one node per thread.
//
// Why.  The register tile marches a CTA along the rows: an iteration waits for
// a row's loads and a collision, about 1.8 us for FP64, and small lattices pay
// it six times or more with a few warps per SM at work (256^2 FP64: 12 us a
// step, 8 % of the warps busy).  Here every node has a thread, so one load
// round, one barrier and one collision are all there is; what bounds it is that
// chain's latency on small lattices, then L2 (512^2 FP64: 374 B per node
// counting the halo, 8 TB/s), and DRAM once both buffers outgrow L2; FP64 runs into
// the board's power limit within a third of a second (1.49 of 1.965 GHz at 995 W:
// 1024^2 54 -> 61 us).
//
// A CTA owns a tile of 32 columns and four rows, a warp per row (eight rows
// have fewer halo nodes but ran 5-15 % slower above 256^2).  Each thread loads
// its node's populations, and the first 76 also those of one halo node each
// (the ring around the tile, densities only); all loads are in flight at once.
// The arithmetic per node is collide_push's, so the results equal the other
// kernels' byte for byte.
//
// The kernel is launched as a programmatic dependent (launch.cuh).
//
// Measured on one B200, us per step (before: register tile or pipelined
// kernel): FP64 64^2 4.0 (10.3), 256^2 5.4 (12.3), 512^2 12.3 (18.5), 1024^2
// 53.5 (63.8), 2048 x 1024 106 (121), the last two with 40 % solid nodes 68
// (87), 130 (150); FP32 256^2 3.5 (8.2), 512^2 7.5 (12.3); FP16 1024^2 24 (32).
#pragma once
#include "fused_step.cuh"
#include "launch.cuh"

namespace sclbm {

constexpr int FLAT_ROWS = 4;

// a tile of a batch's list: columns from x0, rows from y0 of domain dom
struct FlatTile {
    int dom, x0, y0;
};

// Resident CTAs per SM the register cap aims at: six for float arithmetic (80
// registers; five ran 2-5 % slower with solid nodes), four for FP64 (its
// solid forms take 108 registers; capped at 96 for five they ran 8-25 % slower)
template <typename T> constexpr int flat_ctas() { return sizeof(T) == 8 ? 4 : 6; }

// One step of the tile [x0, x0 + 32) x [y0, y0 + TY) of a's lattice.
template <typename S, typename T, int TY, int FLAGS>
__device__ __forceinline__ void flat_tile(const Fused2Args<S, T> &a, const int x0, const int y0)
{
    constexpr bool SOLID = (FLAGS & KF_SOLID) != 0;
    constexpr int C = 34, HALO = 2 * C + 2 * TY;
    static_assert(HALO <= 32 * TY, "one halo node per thread");
    __shared__ V2<T> rho[TY + 2][C];
    __shared__ uint8_t msk[TY + 2][C];
    const int t = threadIdx.x, nx = a.nx, ny = a.ny;
    const int ncol = min(32, nx - x0), nrow = min(TY, ny - y0);
    // this thread's node: column c, row r of the tile with its halo
    const int c = (t & 31) + 1, r = t / 32 + 1;
    const bool own = c <= ncol && r <= nrow;
    const int x = x0 + (own ? c - 1 : 0), y = y0 + (own ? r - 1 : 0);
    // halo node: the rows below and above, then the columns left and right
    int hc, hr;
    bool halo;
    if (t < 2 * C) {
        hc = t < C ? t : t - C;
        hr = t < C ? 0 : nrow + 1;
        halo = hc <= ncol + 1;
    } else {
        const int u = t - 2 * C;
        hc = u < TY ? 0 : ncol + 1;
        hr = (u < TY ? u : u - TY) + 1;
        halo = u < 2 * TY && hr <= nrow;
    }
    dependent_wait();
    dependent_launch();
    T f[2][9], h[2][9];
    // FP16: node codes (1024^2 26.4 us a step against 28.6 for mask bytes); else
    // mask bytes, shared like the densities (FP32 with codes gained 3 % on
    // 512^2 and lost 6 % on 1024^2, where another byte per node comes from DRAM)
    constexpr bool CODES = SOLID && sizeof(S) == 2;
    uint32_t m = CODES ? 0x1ff : 1, mh = 1;
    const uint32_t node = (uint32_t)y * (uint32_t)nx + (uint32_t)x;
    if (SOLID) m = CODES ? (uint32_t)a.codes[node] : (uint32_t)a.mask[node];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 9; ++i) f[k][i] = Load<S>::value(a.fin[k] + elem<false>(i, a.N, node));
    if (halo) {
        const uint32_t hn = (uint32_t)wrap1(y0 - 1 + hr, ny) * (uint32_t)nx + (uint32_t)wrap1(x0 - 1 + hc, nx);
        if (SOLID) mh = CODES ? (uint32_t)a.codes[hn] & 1u : (uint32_t)a.mask[hn];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 9; ++i) h[k][i] = Load<S>::value(a.fin[k] + elem<false>(i, a.N, hn));
        T r0, r1;
        node_density(h, r0, r1);
        if (SOLID && !mh) r0 = r1 = T(0);
        rho[hr][hc] = Vec2<T>::make(r0, r1);
        if (!CODES) msk[hr][hc] = (uint8_t)mh;
    }
    if (own) {
        T r0, r1;
        node_density(f, r0, r1);
        if (SOLID && !(m & 1u)) r0 = r1 = T(0);
        rho[r][c] = Vec2<T>::make(r0, r1);
        if (!CODES) msk[r][c] = (uint8_t)m;
    }
    __syncthreads();
    if (!own) return;
    const Stencil<T> st{{rho[r - 1], rho[r], rho[r + 1]}, {msk[r - 1], msk[r], msk[r + 1]}, c};
    const Nbr n = make_nbr(nx, x, wrap1(x - 1, nx), wrap1(x + 1, nx), y, wrap1(y - 1, ny), wrap1(y + 1, ny));
    if constexpr (CODES)
        collide_node<S, T, FLAGS>(a, f, st, GlobalSink<S, T, true, false>{a, n}, CodeMask{m, a.sums});
    else
        collide_push<S, T, FLAGS>(a, f, st, n);
}

template <typename S, typename T, int TY, int FLAGS>
__global__ void __launch_bounds__(32 * TY, (flat_ctas<T>()))
    k_flat2(const __grid_constant__ Fused2Args<S, T> a)
{
    flat_tile<S, T, TY, FLAGS>(a, blockIdx.x * 32, blockIdx.y * TY);
}

// A batch: CTA b takes tile b of the list.  doms holds two entries per domain
// (buffer parity 0 and 1); the tile's argument block, which no step writes, is
// copied into shared memory while the step before ends.
template <typename S, typename T, int TY, int FLAGS>
__global__ void __launch_bounds__(32 * TY, (flat_ctas<T>()))
    k_batch_flat(const Fused2Args<S, T> *__restrict__ doms, const FlatTile *__restrict__ tiles, int parity)
{
    __shared__ __align__(16) Fused2Args<S, T> sa;
    static_assert(sizeof(sa) % 4 == 0, "argument block copied as words");
    const FlatTile u = tiles[blockIdx.x];
    const uint32_t *src = reinterpret_cast<const uint32_t *>(doms + 2 * u.dom + parity);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(sa) / 4); w += 32 * TY) dst[w] = src[w];
    __syncthreads();
    flat_tile<S, T, TY, FLAGS>(sa, u.x0, u.y0);
}

// UNI: lattices with solid nodes run the uniform solid form (FP32/FP16; FP64
// ran 15 % slower in it on 520 x 260 and 1.5 % faster from 1024^2)
template <typename S, typename T, int UNI>
inline cudaError_t launch_flat2_any(const Fused2Args<S, T> &a, cudaStream_t s)
{
    constexpr int TY = FLAT_ROWS;
    if (!flat_fits(a.nx, a.ny)) return cudaErrorInvalidValue;
    const dim3 grid((a.nx + 31) / 32, (a.ny + TY - 1) / TY), block(32 * TY);
    switch (kernel_flags(a)) {
    case 0: return launch_dependent(k_flat2<S, T, TY, 0>, grid, block, 0, s, a);
    case KF_FORCE: return launch_dependent(k_flat2<S, T, TY, KF_FORCE>, grid, block, 0, s, a);
    case KF_SOLID: return launch_dependent(k_flat2<S, T, TY, KF_SOLID | UNI>, grid, block, 0, s, a);
    default: return launch_dependent(k_flat2<S, T, TY, KF_FORCE | KF_SOLID | UNI>, grid, block, 0, s, a);
    }
}

// flags: KF_FORCE / KF_SOLID when any domain of the batch has a volume force /
// a solid node
template <typename S, typename T, int UNI>
inline cudaError_t launch_batch_flat_any(const Fused2Args<S, T> *doms, const FlatTile *tiles, int ntiles,
                                         int parity, int flags, cudaStream_t s)
{
    constexpr int TY = FLAT_ROWS;
    const dim3 grid(ntiles), block(32 * TY);
    if (flags & KF_SOLID)
        return launch_dependent(k_batch_flat<S, T, TY, KF_FORCE | KF_SOLID | UNI>, grid, block, 0, s, doms, tiles,
                                parity);
    if (flags & KF_FORCE)
        return launch_dependent(k_batch_flat<S, T, TY, KF_FORCE>, grid, block, 0, s, doms, tiles, parity);
    return launch_dependent(k_batch_flat<S, T, TY, 0>, grid, block, 0, s, doms, tiles, parity);
}

} // namespace sclbm
