// fused_two.cuh -- two time steps of a two-component FP32- or FP16-shifted
// lattice in one launch.
//
// Why.  A step on its own reads and writes every population once, and the
// one-step kernels run at the memory's copy rate on large lattices.  Two steps
// per pass read and write the populations once for both: the state between the
// steps lives in shared memory, a few rows at a time.  Nothing is saturated then:
// issue slots 55-64 % taken, the FP32 pipe about 56 % busy (a packed pair takes two
// cycles), DRAM 24-45 %.  Three warps per scheduler share 316-410 instructions per
// node and step, and the largest stall is their fixed latency.  FP32 also runs into
// the board's power limit within half a second (1.65 of 1.965 GHz at 995 W: 267 ->
// 291 us on 4096^2); FP16 does not.  Measured on one B200, us per step
// (the one-step kernels before): FP32 4096^2 267 (407), its 60 % fluid form 322
// (459), FP16 4096^2 277 (334) and 324 (442), FP32 2048 x 1024 with 40 % solid
// nodes 46 (78), 1024^2 22.6 (35.5).  With solid nodes a node step took 469
// instructions against 309; node codes in place of mask bytes and sums (and no
// zeros between the steps) gave 4 to 12 % there.  FP64 stays with the one-step kernels: its rows between the steps
// leave two CTAs per SM, and 12 % busy warps ran no faster (398 against 388
// on 4096 x 2048, 546 against 485 with solid nodes).
//
// Work decomposition.  A CTA of TX threads owns a strip of up to TX - 6
// columns and a band of rows; thread t stands for column xb - 3 + t and
// marches along the band.  One step reads densities one node around a node and
// pushes one node further, so the second step's nodes need the first step's
// results two nodes around them and the first densities three: the outer
// three columns and rows are recomputed by neighbouring CTAs (same inputs,
// same arithmetic, so the same values).  Iteration q of the march:
//
//   A  row q-3's densities after the first step, from the shared rows; row
//      q's densities from its populations (registers, loaded during the
//      previous iteration);                                       -- barrier
//   B  collide row q-1 (first step), pushing into the shared rows q-2..q;
//      request the populations of row q+1; collide row q-4 (second step),
//      pushing into the output arrays;                            -- barrier
//
// Plain loads of one row ahead are enough here (half the bytes per step, and
// a whole collision between request and use), so rows may start anywhere:
// unlike the ring kernel this one has no alignment rule.
//
// The arithmetic per node is collide_node's, and the values between the steps
// are held in the storage type, so the result equals two one-step launches
// byte for byte.
#pragma once
#include "fused_step.cuh"
#include "launch.cuh"

namespace sclbm {

// 128 threads: 256 ran 2-8 % slower (barrier over eight warps), 64 3-4 %
// (halo columns)
constexpr int TWO_TX = 128;

// one direction of both components' populations between the steps
template <typename S> struct TwoCell;
template <> struct TwoCell<float> {
    using type = float2;
};
template <> struct TwoCell<__half> {
    using type = __half2;
};

// The rows between the steps, kept per direction only as long as they are
// needed.  With the march pointing "ahead", the populations of row r that came
// from behind (their direction points ahead) are pushed when row r-1 is
// collided, the level ones with row r, and those that come back with row r+1,
// half-way bounce-backs with row r; all are read two rows later.  Rings of
// three, two and two rows of three directions each hold them.  Every slot has
// one writer; slots of columns and rows that only feed the halo are never
// read, and a solid node's slots never matter: densities and stencils are
// masked.  31 KB for FP32: 100 KB of an SM stay with its L1 beside four CTAs.
template <typename S, int TX> struct __align__(16) TwoShared {
    static constexpr int ROW = 3 * TX; // three directions of a row
    static constexpr int LEVEL = 3 * ROW, BEHIND = 5 * ROW;
    typename TwoCell<S>::type m[7 * ROW];
    float2 rho1[3][TX], rho2[3][TX]; // densities before the first and second step
    uint16_t code[8][TX];            // node codes of the rows q-7 .. q, each read by its own thread
    float2 sums[256];                // Fused2Args::sums (read from L1 it cost 5 %: the rows stream through)
};

// place of direction i among the three of its class (opposite ones alike)
__host__ __device__ constexpr int two_place(int i)
{
    return i == 0 || i == 2 || i == 4 ? 0 : (i == 1 || i == 5 || i == 7 ? 1 : 2);
}

// Offsets (elements of the row storage, this thread's column) of one row's
// three classes of directions: c_y = -1, 0, +1.
struct TwoRow {
    int dn, level, up;
    __device__ __forceinline__ int at(int i) const { return cy(i) == 0 ? level : (cy(i) > 0 ? up : dn); }
};

// pushes a first-step node's populations into the rows between the steps;
// to: the destination rows of the three classes, own: the node's own row
template <typename S, int TX, bool SOLID> struct SharedSink {
    static constexpr bool SOLID_ZEROS = false; // solid nodes' slots are never used
    typename TwoCell<S>::type *m;
    TwoRow to, own;
    __device__ __forceinline__ int slot(int i, uint32_t nf) const
    {
        const int fwd = to.at(i) + two_place(i) * TX + cx(i);
        if (i == 0 || !SOLID) return fwd;
        const int back = own.at(opp(i)) + two_place(opp(i)) * TX;
        return back ^ ((fwd ^ back) & (0 - (int)nf)); // nf is 0 or 1
    }
    __device__ __forceinline__ void pair(int i, float v0, float v1, uint32_t nf) const
    {
        m[slot(i, nf)] = make_float2(v0, v1);
    }
    __device__ __forceinline__ void pair_half(int i, __half h0, __half h1, uint32_t nf) const
    {
        m[slot(i, nf)] = __halves2half2(h0, h1);
    }
    __device__ __forceinline__ void solid() const {}
};

// populations of one row between the steps
template <typename S, int TX>
__device__ __forceinline__ void two_read(const TwoShared<S, TX> &sh, const TwoRow &r, float (&f)[2][9])
{
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        float2 v;
        if constexpr (sizeof(S) == 4) v = sh.m[r.at(i) + two_place(i) * TX];
        else v = __half22float2(sh.m[r.at(i) + two_place(i) * TX]);
        f[0][i] = v.x;
        f[1][i] = v.y;
    }
}

// wrap for offsets in [-3, n + 2] (n >= 3)
__device__ __forceinline__ int wrap3(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// Two steps of the columns [xb, xb + ncol) and rows [y0, y0 + nrow) of a's
// lattice (nx, ny >= 4), rows marched upward or (down) downward.
template <typename S, int TX, int FLAGS>
__device__ __forceinline__ void two_unit(const Fused2Args<S, float> &a, const int xb, const int ncol,
                                         const int y0, const int nrow, const bool down,
                                         TwoShared<S, TX> &sh)
{
    using L = TwoShared<S, TX>;
    constexpr bool SOLID = (FLAGS & KF_SOLID) != 0;
    const int t = threadIdx.x;
    const int nx = a.nx, ny = a.ny;
    // columns of this thread that each stage computes
    const bool load = t < ncol + 6;            // populations and densities before step 1
    const bool step1 = t >= 1 && t < ncol + 5; // collisions of step 1
    const bool dens2 = t >= 2 && t < ncol + 4; // densities before step 2
    const bool step2 = t >= 3 && t < ncol + 3; // collisions of step 2
    const int x = load ? wrap3(xb - 3 + t, nx) : 0;
    const int xl = wrap1(x - 1, nx), xr = wrap1(x + 1, nx);
    auto gy = [&](int q) { return wrap3(y0 + (down ? nrow - 1 - q : q), ny); };

    uint16_t code_ahead = 0x1ff;
    // loads on every thread (idle ones column 0), without a branch around them:
    // the loads of a row sit earlier.  us per step with / without: FP16 4096^2
    // 289 / 309, with solid nodes 324 / 328; FP32 280 / 286, but with solid nodes
    // 343 / 320, the form in which the compiler keeps the branch
    constexpr bool EVERY = !SOLID || sizeof(S) == 2;
    auto load_row = [&](int q, float(&f)[2][9]) {
        if (!EVERY && !load) return;
        const uint32_t node = (uint32_t)gy(q) * (uint32_t)nx + (uint32_t)x;
        if (SOLID) code_ahead = a.codes[node];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                // FP16 without solid nodes: the array's base first (280 -> 273 us
                // on 4096^2: fewer wide multiplies on the FP32 pipe; no gain elsewhere)
                const S *p = sizeof(S) == 2 && !SOLID ? a.fin[k] + (size_t)i * a.N + node
                                                      : a.fin[k] + elem<false>(i, a.N, node);
                f[k][i] = Load<S>::value(p);
            }
    };
    // L2 is asked for the row after the one being loaded, one 128-byte line per
    // thread (FP16 289 -> 277 us a step, with solid nodes 343 -> 328; FP32 1-2 %; a
    // batch of 64 mixed domains 73 -> 69)
    constexpr int LINES = (TX * (int)sizeof(S) + 127) / 128 + 1; // lines a row segment touches
    const S *pf = nullptr;
    if (t < 18 * LINES) {
        const int arr = t / LINES, l = t % LINES;
        const int col = min(max(xb - 3, 0) + l * (128 / (int)sizeof(S)), nx - 1);
        pf = a.fin[arr >= 9 ? 1 : 0] + (size_t)(arr % 9) * a.N + col;
    }

    // slots of the rows q (s0), q - 1 (s1), q - 2 (s2) of the rings of three;
    // rows three apart share one
    int s0 = 0, s1 = 2, s2 = 1;
    // the classes of row r (any value of its parity) whose slot in the rings of
    // three is s
    auto row_at = [&](int s, int r) {
        const int ahead = s * L::ROW + t, two = (r & 1) * L::ROW + t;
        return TwoRow{down ? ahead : L::BEHIND + two, L::LEVEL + two, down ? L::BEHIND + two : ahead};
    };
    // mask of this thread's node in row r (without solid nodes not used)
    auto code_of = [&](int r) { return SOLID ? (uint32_t)sh.code[(r + 8) & 7][t] : 0x1ffu; };

    // cur: row q, prev: row q - 1, both before step 1; mcur: row q - 3, mprev:
    // row q - 4, both after it
    auto row = [&](const int q, float(&cur)[2][9], float(&prev)[2][9], float(&mcur)[2][9],
                   const float(&mprev)[2][9]) {
        if (dens2 && q >= 2 && q <= nrow + 3) {
            float r0, r1;
            two_read<S, TX>(sh, row_at(s0, q - 3), mcur);
            node_density(mcur, r0, r1);
            if (SOLID && !(code_of(q - 3) & 1u)) r0 = r1 = 0.f;
            sh.rho2[s0][t] = make_float2(r0, r1);
        }
        if (load && q <= nrow + 2) {
            float r0, r1;
            node_density(cur, r0, r1);
            if (SOLID) {
                if (!(code_ahead & 1u)) r0 = r1 = 0.f;
                sh.code[(q + 8) & 7][t] = code_ahead;
            }
            sh.rho1[s0][t] = make_float2(r0, r1);
        }
        __syncthreads();
        const int lo = down ? s0 : s2, hi = down ? s2 : s0; // rows below and above the node
        if (step1 && q >= -1 && q <= nrow + 2) {
            const Stencil<float> st{{sh.rho1[lo], sh.rho1[s1], sh.rho1[hi]}, {}, t};
            // ahead: row q; level: row q - 1; behind: row q - 2
            const TwoRow own = row_at(s1, q - 1);
            const int ahead = s0 * L::ROW + t, behind = L::BEHIND + (q & 1) * L::ROW + t;
            const TwoRow to{down ? ahead : behind, own.level, down ? behind : ahead};
            collide_node<S, float, FLAGS>(a, prev, st, SharedSink<S, TX, SOLID>{sh.m, to, own},
                                          CodeMask{code_of(q - 1), sh.sums});
        }
        if (EVERY) load_row(min(q + 1, nrow + 2), prev);
        else if (q < nrow + 2) load_row(q + 1, prev);
        if (pf != nullptr && q + 2 <= nrow + 2)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(pf + (size_t)gy(q + 2) * (size_t)nx));
        if (step2 && q >= 4 && q <= nrow + 3) {
            const Stencil<float> st{{sh.rho2[lo], sh.rho2[s1], sh.rho2[hi]}, {}, t};
            const int yc = gy(q - 4);
            const Nbr n = make_nbr(nx, x, xl, xr, yc, wrap1(yc - 1, ny), wrap1(yc + 1, ny));
            collide_node<S, float, FLAGS>(a, mprev, st, GlobalSink<S, float, SOLID, false>{a, n},
                                          CodeMask{code_of(q - 4), sh.sums});
        }
        __syncthreads();
        const int s = s2;
        s2 = s1;
        s1 = s0;
        s0 = s;
    };

    if (SOLID) // read after the first barrier
        for (int i = t; i < 256; i += TX) sh.sums[i] = a.sums[i];
    float A[2][9], B[2][9], C[2][9], D[2][9];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 9; ++i) A[k][i] = B[k][i] = C[k][i] = D[k][i] = 0.f;
    load_row(-3, A);
    // two rows per trip so the register buffers swap roles instead of being copied
    for (int q = -3; q <= nrow + 3; q += 2) {
        row(q, A, B, C, D);
        row(q + 1, B, A, D, C);
    }
}

// Four CTAs per SM (128 registers, no spills).  A fifth needs 96 registers:
// the spills and the smaller L1 beside five CTAs' shared memory cost a quarter
// (362 against 288 us on 4096^2).
constexpr int TWO_CTAS = 4;

// Launched as a programmatic dependent (launch.cuh): 1024^2 22.6 -> 21.5 us a
// step, 700^2 15.4 -> 14.3.  Strip s covers the columns [s*w, min(nx, (s+1)*w)), band b the rows
// [b*ny/bands, (b+1)*ny/bands); neighbouring bands march in opposite
// directions, so the rows they share are read by both near the same time
template <typename S, int TX, int FLAGS>
__global__ void __launch_bounds__(TX, TWO_CTAS)
    k_two2(const __grid_constant__ Fused2Args<S, float> a, int w, int bands)
{
    __shared__ TwoShared<S, TX> sh;
    const int band = blockIdx.y, xb = blockIdx.x * w;
    const int y0 = (int)((long long)band * a.ny / bands);
    const int nrow = (int)((long long)(band + 1) * a.ny / bands) - y0;
    dependent_wait();
    dependent_launch();
    two_unit<S, TX, FLAGS>(a, xb, min(w, a.nx - xb), y0, nrow, (band & 1) != 0, sh);
}

// Width of a lattice's strips (the last one may be narrower): as few strips as
// hold the columns, and of the widths that give as few, the one with the
// fewest warps at work -- a strip of n columns keeps the warps of n + 6 threads
// busy, the rest of its CTA waits at the barriers.  128 columns: 90 + 38 run
// on five warps, 64 + 64 on six.
inline int two_width(int nx)
{
    constexpr int W = TWO_COLUMNS;
    static_assert(W == TWO_TX - 6, "a strip's columns and three more on each side");
    const int strips = (nx + W - 1) / W, even = (nx + strips - 1) / strips;
    int best = even, least = 0;
    for (int w = even; w <= W; ++w) {
        const int warps = (nx / w) * ((w + 6 + 31) / 32) + (nx % w ? (nx % w + 6 + 31) / 32 : 0);
        if (least == 0 || warps < least) {
            least = warps;
            best = w;
        }
    }
    return best;
}

// Rows per band: the relative time of `units` bands of r rows each.  A band
// computes r + 4 rows of the first step, r of the second and takes r + 8
// iterations, about r + 4 full ones; four CTAs are resident per SM and a full
// wave of them takes four shares of an SM's throughput per iteration.  In the
// last, partial wave an iteration with n CTAs on an SM takes longer than n
// shares, down to the latency of one (measured with solid nodes, where a share
// is 0.66 us: 1.6, 1.9, 2.45 and 2.9 us for one to four).  Measured by this
// choice / other heights, us per step: 1021 x 763 12 rows 20.5 / 16 rows 21.4;
// 1024^2 16 rows 22.6 / 12 rows 26.0, 24 rows 24.7; 2048 x 1024 32 rows 47.3 / 40
// rows 48.2; a batch of eight 400 x 306 20 rows 32.9 / 24 rows 34.1; 4096^2
// within 2 % from 48 to 96 rows.
constexpr int TWO_ROWS[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64};
inline double two_cost(long units, int r, int sms)
{
    const double last[TWO_CTAS + 1] = {0.0, 2.4, 2.9, 3.7, 4.2};
    const long wave = (long)TWO_CTAS * sms, rest = units % wave;
    return (r + 4) * ((double)(units / wave) * TWO_CTAS + last[(rest + sms - 1) / sms]);
}
inline int two_rows(int nx, int ny, int sms)
{
    const int w = two_width(nx), strips = (nx + w - 1) / w;
    int best = 1;
    double least = 0.0;
    for (int r : TWO_ROWS) {
        const double cost = two_cost((long)strips * ((ny + r - 1) / r), r, sms);
        if (least == 0.0 || cost < least) {
            least = cost;
            best = r;
        }
    }
    return best;
}

template <typename S, int TX, int FLAGS>
inline cudaError_t launch_two2_f(const Fused2Args<S, float> &a, int rows, cudaStream_t s)
{
    const int w = two_width(a.nx), strips = (a.nx + w - 1) / w;
    const int bands = std::min((a.ny + rows - 1) / rows, 65535);
    return launch_dependent(k_two2<S, TX, FLAGS>, dim3(strips, bands), dim3(TX), 0, s, a, w, bands);
}

// rows: rows per band (0: two_rows); lattices with solid nodes run the uniform
// solid form.  Refuses lattices that need 64-bit offsets and those that a halo
// of three wraps around more than once.
template <typename S>
inline cudaError_t launch_two2_any(const Fused2Args<S, float> &a, int rows, cudaStream_t s)
{
    if (needs_wide_offsets(a.N) || a.nx < 4 || a.ny < 4) return cudaErrorInvalidValue;
    if (rows < 1) rows = two_rows(a.nx, a.ny, sm_count());
    switch (kernel_flags(a)) {
    case 0: return launch_two2_f<S, TWO_TX, 0>(a, rows, s);
    case KF_FORCE: return launch_two2_f<S, TWO_TX, KF_FORCE>(a, rows, s);
    case KF_SOLID: return launch_two2_f<S, TWO_TX, KF_SOLID | KF_UNIFORM>(a, rows, s);
    default: return launch_two2_f<S, TWO_TX, KF_FORCE | KF_SOLID | KF_UNIFORM>(a, rows, s);
    }
}

// ---------------------------------------------------------------- batches
// A unit of the batched kernel: the columns [xb, xb + ncol) and rows
// [y0, y0 + nrow) of domain dom; down: the march direction (alternating
// between a domain's bands).
struct TwoUnit {
    int dom, xb, ncol, y0, nrow, down;
};

// One CTA per unit, in the list's order (largest first): the block scheduler
// balances them, no counter to take turns at.  An ordinary launch: as a
// programmatic dependent the next step's uneven units fill the free places
// first, which put four on some SMs (eight mixed domains 9.2 -> 10.6 us a step,
// others 1-3 % faster).  doms holds two entries per
// domain (buffer parity 0 and 1); the unit's argument block is copied into
// shared memory.
template <typename S, int FLAGS>
__global__ void __launch_bounds__(TWO_TX, TWO_CTAS)
    k_batch_two(const Fused2Args<S, float> *__restrict__ doms, const TwoUnit *__restrict__ units, int parity)
{
    __shared__ TwoShared<S, TWO_TX> sh;
    __shared__ __align__(16) Fused2Args<S, float> sa;
    static_assert(sizeof(sa) % 4 == 0, "argument block copied as words");
    const TwoUnit u = units[blockIdx.x];
    const uint32_t *src = reinterpret_cast<const uint32_t *>(doms + 2 * u.dom + parity);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&sa);
    for (int w = threadIdx.x; w < (int)(sizeof(sa) / 4); w += TWO_TX) dst[w] = src[w];
    __syncthreads();
    two_unit<S, TWO_TX, FLAGS>(sa, u.xb, u.ncol, u.y0, u.nrow, u.down != 0, sh);
}

// flags: KF_FORCE / KF_SOLID when any domain of the batch has a volume force /
// a solid node
template <typename S>
inline cudaError_t launch_batch_two_any(const Fused2Args<S, float> *doms, const TwoUnit *units, int nunits,
                                        int parity, int flags, cudaStream_t s)
{
    if (flags & KF_SOLID)
        k_batch_two<S, KF_FORCE | KF_SOLID | KF_UNIFORM><<<nunits, TWO_TX, 0, s>>>(doms, units, parity);
    else if (flags & KF_FORCE)
        k_batch_two<S, KF_FORCE><<<nunits, TWO_TX, 0, s>>>(doms, units, parity);
    else
        k_batch_two<S, 0><<<nunits, TWO_TX, 0, s>>>(doms, units, parity);
    return cudaGetLastError();
}

} // namespace sclbm
