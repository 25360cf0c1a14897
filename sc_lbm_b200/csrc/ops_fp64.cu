// ops_fp64.cu -- per-operator FP64 kernels (one per reference method) and the
// FP64 instantiations of the fused step.  Compiled with -fmad=false: every
// product and sum is rounded separately, in the reference's order, so results
// are bit-identical to the serial reference (g++ on x86-64 has no FMA).
#include "fused_step.cuh"
#include "launch.cuh"
#include "ops_fp64.h"

namespace sclbm {

#define GRID_STRIDE(n, N)                                                                      \
    for (size_t n = blockIdx.x * (size_t)blockDim.x + threadIdx.x; n < (N);                    \
         n += (size_t)gridDim.x * blockDim.x)

// The operators of a driver's step (density, velocities, forces, collisions,
// stream).  A lattice of a driver's size leaves a few warps on an SM, so a
// kernel costs its launch and its rounds of dependent loads: each reads all it
// needs before its first store (arrays may alias, so the compiler keeps a load
// behind an earlier store: the collision's nine read-modify-writes took 9.3 us
// on 256^2, one after the other), both fluids of a pair share a launch, and
// launches are programmatic dependents (launch.cuh) in CTAs of 128.  Six
// operators of a 256^2 step: 39 us before, 18 now; of 800 x 500: 108, 71-75; of
// 2048^2, beyond L2: 941, 842.
//
// I: index type, 32 bits while the nine arrays of a fluid hold fewer elements.

// Fluid::compute_density, src/fluid.cpp:175-183 (all nodes)
template <typename I> __global__ void __launch_bounds__(128) k_density(I N, const double *f, double *rho)
{
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        double r = 0.0;
#pragma unroll
        for (int j = 0; j < 9; ++j) r += f[j * N + n];
        rho[n] = r;
    }
}

// Fluid::compute_velocities, src/fluid.cpp:186-200
__device__ __forceinline__ void velocity_node(bool fluid, const double (&f)[9], double rho, double &ux,
                                              double &uy)
{
    double x = 0.0, y = 0.0;
    if (fluid) {
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            x += f[j] * double(cx(j));
            y += f[j] * double(cy(j));
        }
        x /= rho;
        y /= rho;
    }
    ux = x;
    uy = y;
}

template <typename I> __device__ __forceinline__ void load_pops(I N, I n, const double *f, double (&v)[9])
{
#pragma unroll
    for (int j = 0; j < 9; ++j) v[j] = f[j * N + n];
}

template <typename I>
__global__ void __launch_bounds__(128)
    k_velocities(I N, const uint8_t *__restrict__ g, const double *f, const double *rho, double *ux, double *uy)
{
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        double v[9], a, b;
        load_pops(N, n, f, v);
        velocity_node(g[n] == 1, v, rho[n], a, b);
        ux[n] = a;
        uy[n] = b;
    }
}

// Fluid::compute_f_equilibrium(geom), src/fluid.cpp:210-243; with COLLIDE also
// LBM::collide(geom, fluid), src/lbm.cpp:275-288
template <typename I, bool COLLIDE>
__global__ void __launch_bounds__(128)
    k_feq_single(I N, const uint8_t *__restrict__ g, double *f, double *rho, double *ux, double *uy,
                 double *feq, double omega)
{
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        double v[9], r = 0.0, a, b;
        load_pops(N, n, f, v);
#pragma unroll
        for (int j = 0; j < 9; ++j) r += v[j];
        velocity_node(g[n] == 1, v, r, a, b);
        rho[n] = r;
        ux[n] = a;
        uy[n] = b;
        double fe[9];
        feq_exact(r, a, b, fe);
#pragma unroll
        for (int i = 0; i < 9; ++i) feq[i * N + n] = fe[i];
        if (COLLIDE) {
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i * N + n] = (1.0 - omega) * v[i] + omega * fe[i];
        }
    }
}

// Fluid::compute_f_equilibrium(), src/fluid.cpp:246-278; with COLLIDE also the
// collision loop of LBM::collide(f1, f2), src/lbm.cpp:305-311; fluid blockIdx.y
template <typename I, bool COLLIDE>
__global__ void __launch_bounds__(128) k_feq_multi(I N, FeqArgs a0, FeqArgs a1)
{
    const FeqArgs &a = blockIdx.y ? a1 : a0;
    double *const f = a.f, *const feq = a.feq;
    const double omega = a.omega;
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        double v[9], fe[9];
        if (COLLIDE) load_pops(N, n, f, v);
        feq_exact(a.rho[n], a.uex[n], a.uey[n], fe);
#pragma unroll
        for (int i = 0; i < 9; ++i) feq[i * N + n] = fe[i];
        if (COLLIDE) {
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i * N + n] = (1.0 - omega) * v[i] + omega * fe[i];
        }
    }
}

// LBM::compute_solid_surface_force common sums, src/lbm.cpp:110-136
__global__ void k_solid_sums(int nx, int ny, const uint8_t *__restrict__ g, double *__restrict__ sx,
                             double *__restrict__ sy)
{
    const size_t N = (size_t)nx * ny;
    GRID_STRIDE(n, N)
    {
        double a = 0.0, b = 0.0;
        const int x = int(n % nx), y = int(n / nx);
        if (g[n] != 0) {
#pragma unroll
            for (int i = 1; i < 9; ++i) {
                const int xn = wrap1(x + cx(i), nx), yn = wrap1(y + cy(i), ny);
                if (g[(size_t)yn * nx + xn] == 0) {
                    a += w_sc(i) * cx(i);
                    b += w_sc(i) * cy(i);
                }
            }
        }
        sx[n] = a;
        sy[n] = b;
    }
}

// LBM::compute_fluid_repulsive_interactions, src/lbm.cpp:144-206 (masked
// terms are selected away: the loads do not wait for the mask)
template <typename I>
__global__ void __launch_bounds__(128)
    k_repulsive(int nx, int ny, const uint8_t *__restrict__ g, const double *psi1, const double *psi2,
                double gf1, double gf2, double *f1x, double *f1y, double *f2x, double *f2y)
{
    const I N = (I)nx * (I)ny;
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        const int y = int(n / (I)nx), x = int(n - (I)y * (I)nx);
        const int xl = wrap1(x - 1, nx), xr = wrap1(x + 1, nx), yd = wrap1(y - 1, ny), yu = wrap1(y + 1, ny);
        double p1[9], p2[9];
        bool fl[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const I ij = (I)(cy(i) == 0 ? y : (cy(i) > 0 ? yu : yd)) * (I)nx +
                         (I)(cx(i) == 0 ? x : (cx(i) > 0 ? xr : xl));
            p1[i] = psi1[ij];
            p2[i] = psi2[ij];
            fl[i] = g[ij] != 0;
        }
        double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
        if (fl[0]) {
#pragma unroll
            for (int i = 1; i < 9; ++i) {
                const double wcx = w_sc(i) * cx(i), wcy = w_sc(i) * cy(i);
                ax = fl[i] ? ax + wcx * p2[i] : ax;
                ay = fl[i] ? ay + wcy * p2[i] : ay;
                bx = fl[i] ? bx + wcx * p1[i] : bx;
                by = fl[i] ? by + wcy * p1[i] : by;
            }
            ax *= gf1 * p1[0];
            ay *= gf1 * p1[0];
            bx *= gf2 * p2[0];
            by *= gf2 * p2[0];
        }
        f1x[n] = ax;
        f1y[n] = ay;
        f2x[n] = bx;
        f2y[n] = by;
    }
}

struct EqvelFluid {
    const double *f, *rho, *frx, *fry, *fsx, *fsy;
    double *ux, *uy, *uex, *uey;
    double omega, inv_omega;
};

// LBM::compute_equilibrium_velocities, src/lbm.cpp:209-272
template <typename I>
__global__ void __launch_bounds__(128)
    k_eqvel(I N, const uint8_t *__restrict__ g, EqvelFluid a, EqvelFluid b)
{
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        double fa[9], fb[9];
        load_pops(N, n, a.f, fa);
        load_pops(N, n, b.f, fb);
        const double ra = a.rho[n], rb = b.rho[n];
        const double farx = a.frx[n], fary = a.fry[n], fasx = a.fsx[n], fasy = a.fsy[n];
        const double fbrx = b.frx[n], fbry = b.fry[n], fbsx = b.fsx[n], fbsy = b.fsy[n];
        if (g[n] != 1) {
            a.ux[n] = a.uy[n] = b.ux[n] = b.uy[n] = 0.0;
            continue;
        }
        double p = 0.0, q = 0.0, r = 0.0, s = 0.0;
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            p += fa[j] * double(cx(j));
            q += fa[j] * double(cy(j));
            r += fb[j] * double(cx(j));
            s += fb[j] * double(cy(j));
        }
        a.ux[n] = p;
        a.uy[n] = q;
        b.ux[n] = r;
        b.uy[n] = s;
        const double ucx = (p * a.omega + r * b.omega) / (ra * a.omega + rb * b.omega);
        const double ucy = (q * a.omega + s * b.omega) / (ra * a.omega + rb * b.omega);
        if (!rho_is_zero(ra)) {
            a.uex[n] = ucx + farx * a.inv_omega / ra + fasx * a.inv_omega;
            a.uey[n] = ucy + fary * a.inv_omega / ra + fasy * a.inv_omega;
        }
        if (!rho_is_zero(rb)) {
            b.uex[n] = ucx + fbrx * b.inv_omega / rb + fbsx * b.inv_omega;
            b.uey[n] = ucy + fbry * b.inv_omega / rb + fbsy * b.inv_omega;
        }
    }
}

struct ForceVec {
    double v[9];
};

// LBM::add_volume_force, src/lbm.cpp:315-340; fluid blockIdx.y
template <typename I>
__global__ void __launch_bounds__(128)
    k_volume_force(I N, const uint8_t *__restrict__ g, double *f0, double *f1, ForceVec F)
{
    double *const f = blockIdx.y ? f1 : f0;
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        if (g[n] == 1) {
            double v[9];
            load_pops(N, n, f, v);
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i * N + n] = v[i] + F.v[i];
        }
    }
}

// LBM::stream, src/lbm.cpp:343-384, written in gather form: every destination
// slot is assigned exactly the value the reference pushes into it (zero at
// solid nodes, bounce-back where the upstream node is solid); fluid blockIdx.y
template <typename I, bool SOLID>
__global__ void __launch_bounds__(128)
    k_stream(int nx, int ny, const uint8_t *__restrict__ g, const double *in0, double *out0, const double *in1,
             double *out1)
{
    const double *const f = blockIdx.y ? in1 : in0;
    double *const out = blockIdx.y ? out1 : out0;
    const I N = (I)nx * (I)ny;
    dependent_wait();
    dependent_launch();
    for (I n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        const int y = int(n / (I)nx), x = int(n - (I)y * (I)nx);
        const int xl = wrap1(x - 1, nx), xr = wrap1(x + 1, nx), yd = wrap1(y - 1, ny), yu = wrap1(y + 1, ny);
        double v[9], own[9];
        bool fl[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const I src = (I)(cy(i) == 0 ? y : (cy(i) > 0 ? yd : yu)) * (I)nx +
                          (I)(cx(i) == 0 ? x : (cx(i) > 0 ? xl : xr));
            v[i] = f[i * N + src];
            if (SOLID) {
                own[i] = f[i * N + n];
                fl[i] = g[src] == 1;
            }
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            if (SOLID) out[i * N + n] = !fl[0] ? 0.0 : (fl[i] ? v[i] : own[opp(i)]);
            else out[i * N + n] = v[i];
        }
    }
}

// f = value on fluid nodes (Fluid::simple_ini, src/fluid.cpp:86-101)
__global__ void k_fill_fluid(size_t N, const uint8_t *__restrict__ g, double *__restrict__ f,
                             double v)
{
    GRID_STRIDE(n, N)
    {
        if (g[n] == 1) {
#pragma unroll
            for (int i = 0; i < 9; ++i) f[i * N + n] = v;
        }
    }
}

// LBM::initialize_droplet, src/lbm.cpp:11-48
__global__ void k_init_droplet(int nx, int ny, const uint8_t *__restrict__ g, double *fb,
                               double *fd, double rb, double rd, double rbd, double rdb, double xc,
                               double yc, double radius)
{
    const size_t N = (size_t)nx * ny;
    GRID_STRIDE(n, N)
    {
        const int xi = int(n % nx), yj = int(n / nx);
        if (g[n] == 0) continue;
        const bool in = (((double)xi - xc) * ((double)xi - xc) +
                         ((double)yj - yc) * ((double)yj - yc)) <= radius * radius;
        const double vb = (in ? rbd : rb) / 9.0, vd = (in ? rd : rdb) / 9.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            fb[i * N + n] = vb;
            fd[i * N + n] = vd;
        }
    }
}

// LBM::initialize_fluid_rectangle, src/lbm.cpp:51-99 (both passes; the caller
// has already checked that the rectangle indexes stay inside the lattice)
__global__ void k_init_rect(int nx, int ny, const uint8_t *__restrict__ g, double *fb, double *fd,
                            double rb, double rd, double rbd, double rdb, long long x0,
                            long long xf, long long y0, long long yf)
{
    const size_t N = (size_t)nx * ny;
    GRID_STRIDE(n, N)
    {
        if (g[n] == 0) continue;
        const long long xi = (long long)(n % nx), yj = (long long)(n / nx);
        // a rectangle node (xi', yj') touches linear index yj'*nx + xi'; xi' may
        // exceed nx and wrap into the next row exactly like the reference's
        // geom(xi, yj) = geom.at(yj*Nx + xi)
        bool in = false;
        for (long long yy = y0; yy <= yf && !in; ++yy) {
            const long long rem = (long long)n - yy * nx;
            if (rem >= x0 && rem <= xf) in = true;
        }
        (void)xi;
        (void)yj;
        const double vb = (in ? rbd : rb) / 9.0, vd = (in ? rd : rdb) / 9.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            fb[i * N + n] = vb;
            fd[i * N + n] = vd;
        }
    }
}

// ----------------------------------------------------------------- launchers
#define LAUNCH(kern, N, ...)                                                                   \
    do {                                                                                       \
        kern<<<grid_for((N), 256), 256, 0, s>>>(__VA_ARGS__);                                  \
        return cudaGetLastError();                                                             \
    } while (0)

// one thread per node in CTAs of 128 (grid-stride beyond the cap), `fluids`
// rows of CTAs; i32: 9N elements fit 32-bit indices
static dim3 op_grid(size_t N, int fluids = 1) { return dim3(grid_for(N, 128), fluids); }
#define LAUNCH_OP(N, fluids, kern32, kern64, ...)                                              \
    (needs_wide_offsets(N) ? launch_dependent(kern64, op_grid(N, fluids), dim3(128), 0, s, __VA_ARGS__)       \
                           : launch_dependent(kern32, op_grid(N, fluids), dim3(128), 0, s, __VA_ARGS__))

cudaError_t op_density(size_t N, const double *f, double *rho, cudaStream_t s)
{
    return LAUNCH_OP(N, 1, k_density<uint32_t>, k_density<size_t>, N, f, rho);
}
cudaError_t op_velocities(size_t N, const uint8_t *g, const double *f, const double *rho,
                          double *ux, double *uy, cudaStream_t s)
{
    return LAUNCH_OP(N, 1, k_velocities<uint32_t>, k_velocities<size_t>, N, g, f, rho, ux, uy);
}
cudaError_t op_feq_single(size_t N, const uint8_t *g, double *f, double *rho, double *ux,
                          double *uy, double *feq, double omega, int collide, cudaStream_t s)
{
    if (collide)
        return LAUNCH_OP(N, 1, (k_feq_single<uint32_t, true>), (k_feq_single<size_t, true>), N, g, f, rho, ux,
                         uy, feq, omega);
    return LAUNCH_OP(N, 1, (k_feq_single<uint32_t, false>), (k_feq_single<size_t, false>), N, g, f, rho, ux, uy,
                     feq, omega);
}
cudaError_t op_feq(size_t N, const FeqArgs &a, cudaStream_t s)
{
    return LAUNCH_OP(N, 1, (k_feq_multi<uint32_t, false>), (k_feq_multi<size_t, false>), N, a, a);
}
cudaError_t op_collide(size_t N, const FeqArgs &a, const FeqArgs &b, cudaStream_t s)
{
    if (a.f != b.f)
        return LAUNCH_OP(N, 2, (k_feq_multi<uint32_t, true>), (k_feq_multi<size_t, true>), N, a, b);
    // the same fluid twice: one collision after the other
    const cudaError_t e = LAUNCH_OP(N, 1, (k_feq_multi<uint32_t, true>), (k_feq_multi<size_t, true>), N, a, a);
    if (e != cudaSuccess) return e;
    return LAUNCH_OP(N, 1, (k_feq_multi<uint32_t, true>), (k_feq_multi<size_t, true>), N, b, b);
}
cudaError_t op_solid_sums(int nx, int ny, const uint8_t *g, double *sx, double *sy, cudaStream_t s)
{
    LAUNCH(k_solid_sums, (size_t)nx * ny, nx, ny, g, sx, sy);
}
cudaError_t op_repulsive(int nx, int ny, const uint8_t *g, const double *psi1, const double *psi2,
                         double gf1, double gf2, double *f1x, double *f1y, double *f2x,
                         double *f2y, cudaStream_t s)
{
    return LAUNCH_OP((size_t)nx * ny, 1, k_repulsive<uint32_t>, k_repulsive<size_t>, nx, ny, g, psi1, psi2, gf1,
                     gf2, f1x, f1y, f2x, f2y);
}
cudaError_t op_eqvel(size_t N, const uint8_t *g, const EqvelArgs &a, const EqvelArgs &b,
                     cudaStream_t s)
{
    const EqvelFluid A{a.f, a.rho, a.frx, a.fry, a.fsx, a.fsy, a.ux, a.uy, a.uex, a.uey, a.omega,
                       1.0 / a.omega};
    const EqvelFluid B{b.f, b.rho, b.frx, b.fry, b.fsx, b.fsy, b.ux, b.uy, b.uex, b.uey, b.omega,
                       1.0 / b.omega};
    return LAUNCH_OP(N, 1, k_eqvel<uint32_t>, k_eqvel<size_t>, N, g, A, B);
}
cudaError_t op_volume_force(size_t N, const uint8_t *g, double *f0, double *f1, const double *force9,
                            cudaStream_t s)
{
    ForceVec F;
    for (int i = 0; i < 9; ++i) F.v[i] = force9[i];
    if (f1 && f1 != f0) return LAUNCH_OP(N, 2, k_volume_force<uint32_t>, k_volume_force<size_t>, N, g, f0, f1, F);
    const cudaError_t e = LAUNCH_OP(N, 1, k_volume_force<uint32_t>, k_volume_force<size_t>, N, g, f0, f0, F);
    if (e != cudaSuccess || !f1) return e;
    // the same fluid twice: one addition after the other
    return LAUNCH_OP(N, 1, k_volume_force<uint32_t>, k_volume_force<size_t>, N, g, f0, f0, F);
}
cudaError_t op_stream(int nx, int ny, const uint8_t *g, bool has_solid, const double *in0, double *out0,
                      const double *in1, double *out1, cudaStream_t s)
{
    const size_t N = (size_t)nx * ny;
    const int fluids = in1 ? 2 : 1;
    if (has_solid)
        return LAUNCH_OP(N, fluids, (k_stream<uint32_t, true>), (k_stream<size_t, true>), nx, ny, g, in0, out0,
                         in1, out1);
    return LAUNCH_OP(N, fluids, (k_stream<uint32_t, false>), (k_stream<size_t, false>), nx, ny, g, in0, out0, in1,
                     out1);
}
cudaError_t op_fill_fluid(size_t N, const uint8_t *g, double *f, double v, cudaStream_t s)
{
    LAUNCH(k_fill_fluid, N, N, g, f, v);
}
cudaError_t op_init_droplet(int nx, int ny, const uint8_t *g, double *fb, double *fd, double rb,
                            double rd, double rbd, double rdb, double xc, double yc, double radius,
                            cudaStream_t s)
{
    LAUNCH(k_init_droplet, (size_t)nx * ny, nx, ny, g, fb, fd, rb, rd, rbd, rdb, xc, yc, radius);
}
cudaError_t op_init_rect(int nx, int ny, const uint8_t *g, double *fb, double *fd, double rb,
                         double rd, double rbd, double rdb, long long x0, long long xf,
                         long long y0, long long yf, cudaStream_t s)
{
    LAUNCH(k_init_rect, (size_t)nx * ny, nx, ny, g, fb, fd, rb, rd, rbd, rdb, x0, xf, y0, yf);
}

cudaError_t launch_fused2_fp64(const Fused2Args<double, double> &a, int variant, int tx,
                               cudaStream_t s)
{
    return launch_fused2_any<double, double>(a, variant, tx, s);
}
cudaError_t launch_fused1_fp64(const Fused1Args<double, double> &a, cudaStream_t s)
{
    k_fused1<double, double><<<grid_for(a.N, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}
cudaError_t launch_density_fp64(const uint8_t *mask, const double *f0, const double *f1,
                                double *r0, double *r1, size_t N, cudaStream_t s)
{
    k_density2<double, double><<<grid_for(N, 256), 256, 0, s>>>(mask, f0, f1, r0, r1, N);
    return cudaGetLastError();
}

} // namespace sclbm

// the FP64 batched kernel lives in this -fmad=false translation unit
#include "batch_kernel.cuh"
namespace sclbm {
cudaError_t launch_batch_fp64(const Fused2Args<double, double> *doms, const TileRef *tiles,
                              int ntiles, int parity, int grid, int flags, cudaStream_t s)
{
    return launch_batch_t<double, double>(doms, tiles, ntiles, parity, grid, flags, s);
}
int batch_blocks_per_sm_fp64() { return batch_blocks_per_sm_t<double, double>(); }
} // namespace sclbm

// pipelined persistent FP64 kernels (-fmad=false keeps them bit-exact)
#include "fused_async.cuh"
namespace sclbm {
cudaError_t launch_fused2_async_fp64(const Fused2Args<double, double> &a, cudaStream_t s,
                                     bool uniform)
{
    if (uniform) return launch_fused2_async_t<double, double, 128, 3, KF_UNIFORM>(a, s);
    return launch_fused2_async_t<double, double, 128, 3>(a, s);
}
cudaError_t launch_batch2_async_fp64(const Fused2Args<double, double> *doms, const BandTile *tiles,
                                     int ntiles, int grid, int parity, cudaStream_t s)
{
    return launch_batch2_async_t<double, double, 128, 3>(doms, tiles, ntiles, grid, parity, s);
}
int async_resident_fp64() { return async_resident_ctas<double, double, 128, 3>(); }
} // namespace sclbm

// ring kernel, FP64 storage (-fmad=false keeps it bit-exact): 19 KB per stage,
// three stages beside the three CTAs per SM that the registers allow; solid
// lanes branch around the collision as in the FP64 register tile
#include "fused_ring.cuh"
namespace sclbm {
cudaError_t launch_ring2_fp64(const Fused2Args<double, double> &a, int stages, int rows, cudaStream_t s,
                              bool edge)
{
    // FP64 keeps its halo boxes: its registers, not its stages, set its residency
    if (edge) return launch_ring2_any<double, double, 2, 0>(a, rows, s);
    if (stages < 0) return launch_ring2_any<double, double, 2, 0>(a, rows, s);
    if (stages > 0) return launch_ring2_any<double, double, 4, 0>(a, rows, s);
    return launch_ring2_any<double, double, 3, 0>(a, rows, s);
}
constexpr int RING_BATCH_R64 = 3;
cudaError_t launch_batch_ring_fp64(const Fused2Args<double, double> *doms, const RingMaps *maps,
                                   const RingUnit *units, int nunits, int parity, int grid, int flags,
                                   unsigned *counters, int width, cudaStream_t s)
{
    if (width == 64)
        return launch_batch_ring<double, double, RING_BATCH_R64, 0, 64>(doms, maps, units, nunits, parity,
                                                                         grid, flags, counters, s);
    return launch_batch_ring<double, double, RING_BATCH_R64, 0, 128>(doms, maps, units, nunits, parity,
                                                                      grid, flags, counters, s);
}
int batch_ring_prepare_shifted(sclbm_precision p, int width, int *per_sm);
int batch_ring_prepare(sclbm_precision p, int width, int *per_sm)
{
    if (p != SCLBM_FP64) return batch_ring_prepare_shifted(p, width, per_sm);
    const cudaError_t e = width == 64 ? batch_ring_prepare<double, double, RING_BATCH_R64, 0, 64>(per_sm)
                                      : batch_ring_prepare<double, double, RING_BATCH_R64, 0, 128>(per_sm);
    return e == cudaSuccess ? 0 : cuda_fail(e, "ring batch set-up");
}
int ring_maps_of(const Fused2Args<double, double> &a, int width, RingMaps *m)
{
    const cudaError_t e = width == 64 ? ring_maps<double, double, RING_BATCH_R64, 64>(a, *m)
                                      : ring_maps<double, double, RING_BATCH_R64, 128>(a, *m);
    return e == cudaSuccess ? 0 : 1;
}
} // namespace sclbm
