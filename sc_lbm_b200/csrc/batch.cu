// batch.cu -- many independent two-component domains advanced together, one
// launch per step or per two steps, the launches of a run captured once into a
// CUDA graph and replayed.  All domains of a batch share the storage precision
// and the buffer parity.  The bodies that variant 0 takes:
//
//  * pairs (FP32/FP16, k_batch_two in fused_two.cuh): every domain is cut into
//    strips of up to 122 columns and bands of rows, a CTA per strip and band, two
//    steps per launch;
//  * one node per thread (FP64, k_batch_flat in fused_flat.cuh): a CTA per tile of
//    32 x 4 nodes, on all-fluid batches below 4 M nodes and, with solid nodes, where
//    it beats the ring (routes.h);
//  * for what these leave (steps left over from pairs, lattices or heights that
//    pairs do not take, larger FP64 batches) and by set_kernel the persistent
//    one-step bodies:
//    - ring (fused_ring.cuh): CTAs take units of a strip and a band from a
//      counter; the automatic choice with solid nodes on rows that start on
//      16-byte boundaries;
//    - bands (FP64/FP32): every domain is cut into 128-column strips and row
//      bands of one common height, chosen as the smallest for which all
//      (domain, strip, band) tiles are resident at once; neighbouring strips of
//      a band are adjacent in the list so they walk the same rows together; the
//      pipelined single-pass body (fused_async.cuh) runs each tile;
//    - tile list: every tile (126 columns x tile_y rows) of every domain,
//      largest first; CTA b takes tiles b, b+grid, ... and runs the
//      register-tile body (batch_kernel.cuh).
// Among the persistent bodies the automatic choice and the rows per tile come
// from the autotuned size-class table (tuning.h), weighted by the nodes of each
// class in the batch.
#include <algorithm>
#include <memory>
#include <numeric>
#include <utility>

#include "domain.h"
#include "batch_kernel.cuh"
#include "fused_async.cuh"
#include "fused_flat.cuh"
#include "fused_ring.cuh"
#include "fused_two.cuh"
#include "routes.h"
#include "tuning.h"


using namespace sclbm;

static constexpr int GRAPH_STEPS = 20; // steps per captured graph (a multiple of 4: the parity returns)

struct sclbm_batch {
    std::vector<sclbm_domain *> doms;
    sclbm_precision prec = SCLBM_FP32_SHIFTED;
    void *d_lists = nullptr; // the allocation that holds all device lists
    void *d_args = nullptr;  // Fused2Args<S,T>[2*ndom] (parity 0, parity 1)
    TileRef *d_tiles = nullptr;
    TileRef *d_tiles_half = nullptr; // 64-column tiles of the two-tiles-per-CTA body
    int ntiles_half = 0;
    TileRef *d_tiles_warp = nullptr; // 32-column tiles of the one-tile-per-warp body
    int ntiles_warp = 0;
    BandTile *d_bands = nullptr; // (domain, strip, band) tiles of the pipelined kernel
    int nbands = 0, band_grid = 0, band_rows = 0;
    int ntiles = 0, grid = 0, parity = 0;
    int use_units = 1;
    int auto_units = 1; // tuned choice for variant 0
    int body = BODY_TILE; // tile-list body: 2 register tile, 5 load ahead, 6 compacted, 8 uniform
    int auto_body = BODY_TILE; // tile-list body of variant 0
    int grid_body[BODY_COUNT] = {};  // resident grid of each body
    int flags = 0;                 // KF_FORCE / KF_SOLID if any domain needs them
    cudaGraphExec_t graph[2] = {nullptr, nullptr}; // by starting parity
    cudaStream_t graph_stream = nullptr;
    // ring bodies (variant 11: 128-column strips, 12: 64-column strips): units
    // of (domain, strip, band), tensor maps per domain and parity, the work
    // counters; absent when a domain's rows do not start on 16-byte boundaries
    bool ring = false;
    int use_ring = 0;  // 0, or the strip width of the ring body in use
    int auto_ring = 0; // the ring body of variant 0
    RingUnit *d_units[2] = {nullptr, nullptr}; // [0] 128 wide, [1] 64 wide
    RingMaps *d_maps[2] = {nullptr, nullptr};
    unsigned *d_counters = nullptr;
    int nunits[2] = {0, 0}, ring_grid[2] = {0, 0};
    // steps in pairs (variant 0 of FP32/FP16 batches): units of the two-step
    // kernel; absent (0) when a domain is too small for it
    TwoUnit *d_two = nullptr;
    int ntwo = 0;
    bool use_two = false;
    // one node per thread (variant 0 of FP64 batches): tiles of all domains;
    // absent (0) where another body is the faster one
    FlatTile *d_flat = nullptr;
    int nflat = 0;
    bool use_flat = false;
};

// Device lists of a batch: one allocation, filled by copies in the stream that
// the batch's kernels run in, all of them done when send returns (a cudaMemcpy
// of pageable memory may return before its data has arrived, and does not order
// other streams).  The lists stay on the host until then.
struct DeviceLists {
    struct Part {
        void **list;
        std::shared_ptr<void> keep;
        const void *data;
        size_t bytes, at;
    };
    std::vector<Part> parts;
    size_t bytes = 0;

    template <typename P, typename T> void add(P **list, std::vector<T> v)
    {
        auto keep = std::make_shared<std::vector<T>>(std::move(v));
        const size_t n = keep->size() * sizeof(T), at = (bytes + 255) / 256 * 256;
        parts.push_back(Part{(void **)list, keep, keep->data(), n, at});
        bytes = at + n;
    }
    int send(void **base)
    {
        cudaStream_t s = stream();
        SCLBM_CUDA(cudaMalloc(base, std::max<size_t>(bytes, 16)));
        for (auto &p : parts) {
            *p.list = (char *)*base + p.at;
            if (p.bytes) SCLBM_CUDA(cudaMemcpyAsync(*p.list, p.data, p.bytes, cudaMemcpyHostToDevice, s));
        }
        SCLBM_CUDA(cudaStreamSynchronize(s));
        return SCLBM_OK;
    }
};

// the tile list of the current body
static const TileRef *batch_tiles(const sclbm_batch *b)
{
    return b->body == BODY_HALF ? b->d_tiles_half : b->body == BODY_WARP ? b->d_tiles_warp : b->d_tiles;
}
static int batch_ntiles(const sclbm_batch *b)
{
    return b->body == BODY_HALF ? b->ntiles_half : b->body == BODY_WARP ? b->ntiles_warp : b->ntiles;
}

static cudaError_t batch_launch_any(sclbm_batch *b, int parity, cudaStream_t s)
{
    if (b->use_flat)
        return launch_batch_flat_fp64((const Fused2Args<double, double> *)b->d_args, b->d_flat, b->nflat, parity,
                                      b->flags, s);
    if (b->use_ring) {
        const int w = b->use_ring, r = w == 64 ? 1 : 0;
        switch (b->prec) {
        case SCLBM_FP64:
            return launch_batch_ring_fp64((const Fused2Args<double, double> *)b->d_args, b->d_maps[r],
                                          b->d_units[r], b->nunits[r], parity, b->ring_grid[r], b->flags,
                                          b->d_counters, w, s);
        case SCLBM_FP32_SHIFTED:
            return launch_batch_ring_f32((const Fused2Args<float, float> *)b->d_args, b->d_maps[r],
                                         b->d_units[r], b->nunits[r], parity, b->ring_grid[r], b->flags,
                                         b->d_counters, w, s);
        default:
            return launch_batch_ring_f16((const Fused2Args<__half, float> *)b->d_args, b->d_maps[r],
                                         b->d_units[r], b->nunits[r], parity, b->ring_grid[r], b->flags,
                                         b->d_counters, w, s);
        }
    }
    if (b->use_units && b->prec == SCLBM_FP64)
        return launch_batch2_async_fp64((const Fused2Args<double, double> *)b->d_args, b->d_bands,
                                        b->nbands, b->band_grid, parity, s);
    if (b->use_units && b->prec == SCLBM_FP32_SHIFTED)
        return launch_batch2_async_f32((const Fused2Args<float, float> *)b->d_args, b->d_bands,
                                       b->nbands, b->band_grid, parity, s);
    switch (b->prec) {
    case SCLBM_FP64:
        return launch_batch_fp64((const Fused2Args<double, double> *)b->d_args, b->d_tiles,
                                 b->ntiles, parity, b->grid, b->flags, s);
    case SCLBM_FP32_SHIFTED:
        return launch_batch_f32((const Fused2Args<float, float> *)b->d_args, batch_tiles(b),
                                batch_ntiles(b), parity, b->grid_body[b->body], b->flags, b->body, s);
    default:
        return launch_batch_f16((const Fused2Args<__half, float> *)b->d_args, batch_tiles(b),
                                batch_ntiles(b), parity, b->grid_body[b->body], b->flags, b->body, s);
    }
}

// Ring bodies: every domain cut into strips `width` columns wide and bands of
// about `rows` rows (a domain's bands alternate their march direction),
// largest units first; tensor maps of both parities of every domain.
template <typename S, typename T>
static int build_ring(sclbm_batch *b, const std::vector<Fused2Args<S, T>> &h, const std::vector<int> &rows,
                      int width, DeviceLists &lists)
{
    const int r = width == 64 ? 1 : 0;
    std::vector<RingUnit> units;
    std::vector<long> cost;
    for (int k = 0; k < (int)b->doms.size(); ++k) {
        const sclbm_domain *d = b->doms[k];
        const int nb = std::max(1, (int)((d->ny + rows[k] / 2) / rows[k]));
        for (int j = 0; j < nb; ++j) {
            const int y0 = (int)((long long)d->ny * j / nb), y1 = (int)((long long)d->ny * (j + 1) / nb);
            for (int xb = 0; xb < (int)d->nx; xb += width) {
                units.push_back(RingUnit{k, xb, y0, y1, j & 1, {0, 0, 0}});
                cost.push_back((long)std::min(width, (int)d->nx - xb) * (y1 - y0 + 2));
            }
        }
    }
    // Largest first at domain granularity: a domain's units stay together in
    // band-major order, so vertically neighbouring bands (opposite march
    // directions) start within a few claims of each other and the halo rows
    // they share are read from L2 the second time; domains are ordered by
    // their largest unit.
    std::vector<long> dom_cost(b->doms.size(), 0);
    for (size_t i = 0; i < units.size(); ++i)
        dom_cost[units[i].dom] = std::max(dom_cost[units[i].dom], cost[i]);
    std::vector<int> order(units.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int c) { return dom_cost[units[a].dom] > dom_cost[units[c].dom]; });
    std::vector<RingUnit> sorted(units.size());
    for (size_t i = 0; i < order.size(); ++i) sorted[i] = units[order[i]];
    std::vector<RingMaps> maps(h.size());
    for (size_t i = 0; i < h.size(); ++i)
        if (ring_maps_of(h[i], width, &maps[i])) return set_error(SCLBM_E_CUDA, "tensor map encoding");
    int per_sm = 0;
    int rc = batch_ring_prepare(b->prec, width, &per_sm);
    if (rc) return rc;
    b->nunits[r] = (int)sorted.size();
    b->ring_grid[r] = std::max(1, std::min(b->nunits[r], std::max(1, per_sm) * sm_count()));
    lists.add(&b->d_units[r], std::move(sorted));
    lists.add(&b->d_maps[r], std::move(maps));
    return SCLBM_OK;
}

template <typename S, typename T>
static int build_rings(sclbm_batch *b, const std::vector<Fused2Args<S, T>> &h, const std::vector<int> &rows,
                       DeviceLists &lists)
{
    const int A = 16 / (int)sizeof(S);
    for (auto *d : b->doms)
        if (d->nx % A != 0) return SCLBM_OK; // no ring body for this batch
    int rc = build_ring<S, T>(b, h, rows, 128, lists);
    if (!rc) rc = build_ring<S, T>(b, h, rows, 64, lists);
    if (rc) return rc;
    lists.add(&b->d_counters, std::vector<unsigned>(2, 0u));
    b->ring = true;
    return SCLBM_OK;
}

// rows per unit of the ring body (a unit reads two halo rows), unless the
// caller gives tile_y per domain or the tuned batch default sets them
constexpr int RING_BATCH_ROWS = 32;

template <typename S, typename T>
static int build_args(sclbm_batch *b, const std::vector<int> &ty, const std::vector<int> &ring_rows,
                      DeviceLists &lists)
{
    std::vector<Fused2Args<S, T>> h(2 * b->doms.size());
    for (size_t k = 0; k < b->doms.size(); ++k) {
        sclbm_domain *d = b->doms[k];
        const int par = d->parity, saved_ty = d->tile_y;
        d->tile_y = ty[k];
        for (int p = 0; p < 2; ++p) {
            d->parity = p;
            Fused2Args<double, double> a64;
            Fused2Args<float, float> a32;
            Fused2Args<__half, float> a16;
            domain_fused2_args(d, &a64, &a32, &a16);
            if constexpr (sizeof(S) == 8) h[2 * k + p] = a64;
            else if constexpr (sizeof(S) == 4) h[2 * k + p] = a32;
            else h[2 * k + p] = a16;
        }
        d->parity = par;
        d->tile_y = saved_ty;
    }
    const int rc = build_rings<S, T>(b, h, ring_rows, lists);
    lists.add(&b->d_args, std::move(h));
    return rc;
}

// Units of the two-step kernel: per domain its strips and bands, all of about
// the rows that two_cost finds best for the batch's units (the caller's height
// where given; none when one of those is too low for pairs).  64 mixed domains, before the node codes: 24 rows 80 us per
// step, 16 rows 85, 32 rows 98, 64 rows 92 (ring body 104).
static void build_two(sclbm_batch *b, const int *tile_y, DeviceLists &lists)
{
    if (b->prec == SCLBM_FP64) return;
    for (auto *d : b->doms)
        if (d->nx < 4 || d->ny < 4) return;
    auto bands_of = [&](const sclbm_domain *d, int k, int rows) {
        const int r = tile_y && tile_y[k] > 0 ? tile_y[k] : rows;
        return std::max(1, (int)((d->ny + r - 1) / r));
    };
    std::vector<int> width(b->doms.size()), strips(b->doms.size());
    for (size_t k = 0; k < b->doms.size(); ++k) {
        width[k] = two_width((int)b->doms[k]->nx);
        strips[k] = ((int)b->doms[k]->nx + width[k] - 1) / width[k];
    }
    int rows = 1;
    double least = 0.0;
    for (int r : TWO_ROWS) {
        long n = 0;
        for (size_t k = 0; k < b->doms.size(); ++k) n += (long)strips[k] * bands_of(b->doms[k], (int)k, r);
        const double cost = two_cost(n, r, sm_count());
        if (least == 0.0 || cost < least) {
            least = cost;
            rows = r;
        }
    }
    if (tile_y) {
        long n = 0;
        for (size_t k = 0; k < b->doms.size(); ++k) n += (long)strips[k] * bands_of(b->doms[k], (int)k, rows);
        for (size_t k = 0; k < b->doms.size(); ++k)
            if (!two_rows_pay(b->prec, std::max(0, tile_y[k]), n, b->flags & KF_SOLID, sm_count())) return;
    }
    std::vector<TwoUnit> units;
    std::vector<long> cost;
    double nodes = 0.0, strip_rows = 0.0;
    for (size_t k = 0; k < b->doms.size(); ++k) {
        const sclbm_domain *d = b->doms[k];
        constexpr size_t W = TWO_COLUMNS;
        nodes += (double)d->N;
        strip_rows += (double)((d->nx + W - 1) / W) * (double)d->ny;
        const int w = width[k], bands = bands_of(d, (int)k, rows);
        for (int j = 0; j < bands; ++j) {
            const int y0 = (int)((long long)d->ny * j / bands), y1 = (int)((long long)d->ny * (j + 1) / bands);
            for (int xb = 0; xb < (int)d->nx; xb += w) {
                units.push_back(TwoUnit{(int)k, xb, std::min(w, (int)d->nx - xb), y0, y1 - y0, j & 1});
                cost.push_back(y1 - y0);
            }
        }
    }
    if (b->body == BODY_WARP && !b->use_ring &&
        !batch_two_beats_warp(strip_rows, nodes / (strip_rows * TWO_COLUMNS), sm_count()))
        return;
    // largest first at domain granularity, as the ring's units
    std::vector<long> dom_cost(b->doms.size(), 0);
    for (size_t i = 0; i < units.size(); ++i)
        dom_cost[units[i].dom] = std::max(dom_cost[units[i].dom], cost[i]);
    std::vector<int> order(units.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return dom_cost[units[x].dom] > dom_cost[units[y].dom]; });
    std::vector<TwoUnit> sorted(units.size());
    for (size_t i = 0; i < order.size(); ++i) sorted[i] = units[order[i]];
    b->ntwo = (int)sorted.size();
    lists.add(&b->d_two, std::move(sorted));
    b->use_two = true;
}

// Turns from fluid to solid or back along the rows of some masks; CTA rows
// (blockIdx.y) take one each.
struct MaskGroup {
    static constexpr int MOST = 128;
    const uint8_t *mask[MOST];
    uint32_t N[MOST]; // a batch's domains have fewer than 2^32 / 9 nodes
};
__global__ void __launch_bounds__(256)
    k_mask_changes(const __grid_constant__ MaskGroup g, unsigned long long *__restrict__ sum)
{
    const uint8_t *mask = g.mask[blockIdx.y];
    const uint32_t N = g.N[blockIdx.y];
    unsigned n = 0;
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i + 1 < N; i += gridDim.x * 256) n += mask[i] != mask[i + 1];
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(sum, n);
}

static int mask_changes(const sclbm_batch *b, double *out)
{
    cudaStream_t s = stream();
    auto *sum = (unsigned long long *)b->doms[0]->partials; // scratch of the monitor
    unsigned long long n = 0;
    SCLBM_CUDA(cudaMemsetAsync(sum, 0, sizeof n, s));
    for (size_t k = 0; k < b->doms.size(); k += MaskGroup::MOST) {
        MaskGroup g;
        const int n_g = (int)std::min<size_t>(MaskGroup::MOST, b->doms.size() - k);
        for (int j = 0; j < n_g; ++j) {
            g.mask[j] = b->doms[k + j]->d_mask;
            g.N[j] = (uint32_t)b->doms[k + j]->N;
        }
        k_mask_changes<<<dim3(16, n_g), 256, 0, s>>>(g, sum);
        SCLBM_LAUNCHED("mask changes");
    }
    SCLBM_CUDA(cudaMemcpyAsync(&n, sum, sizeof n, cudaMemcpyDeviceToHost, s));
    SCLBM_CUDA(cudaStreamSynchronize(s));
    *out = (double)n;
    return SCLBM_OK;
}

// Tiles of the one-node-per-thread kernel for FP64 batches: with solid nodes
// where it is faster than the ring body (routes.h; eight mixed domains 12.9 / 27.8
// us per step), without, as for a single lattice, up to 4 M nodes.  Heights of
// the caller's choice ask for marching tiles.
static int build_flat(sclbm_batch *b, const int *tile_y, DeviceLists &lists)
{
    if (b->prec != SCLBM_FP64 || tile_y) return SCLBM_OK;
    size_t nodes = 0, count = 0, strips = 0;
    for (auto *d : b->doms) {
        nodes += d->N;
        if (const size_t w = (size_t)b->auto_ring) strips += (d->nx + w - 1) / w * w * d->ny;
        count += ((d->nx + 31) / 32) * ((d->ny + FLAT_ROWS - 1) / FLAT_ROWS);
    }
    if ((!(b->flags & KF_SOLID) && nodes >= ((size_t)1 << 22)) || count > ((size_t)1 << 30)) return SCLBM_OK;
    if ((b->flags & KF_SOLID) && b->auto_ring) {
        const double full = (double)nodes / (double)strips;
        double changes = 0.0; // counted where they decide
        if (batch_flat_beats_ring((double)nodes, full, 0.0) != batch_flat_beats_ring((double)nodes, full, 1.0)) {
            const int rc = mask_changes(b, &changes);
            if (rc) return rc;
        }
        if (!batch_flat_beats_ring((double)nodes, full, changes / (double)nodes)) return SCLBM_OK;
    }
    std::vector<FlatTile> tiles;
    tiles.reserve(count);
    for (size_t k = 0; k < b->doms.size(); ++k)
        for (size_t y = 0; y < b->doms[k]->ny; y += FLAT_ROWS)
            for (size_t x = 0; x < b->doms[k]->nx; x += 32) tiles.push_back(FlatTile{(int)k, (int)x, (int)y});
    b->nflat = (int)tiles.size();
    lists.add(&b->d_flat, std::move(tiles));
    b->use_flat = true;
    return SCLBM_OK;
}

static cudaError_t batch_launch_two(sclbm_batch *b, int parity, cudaStream_t s)
{
    if (b->prec == SCLBM_FP32_SHIFTED)
        return launch_batch_two_f32((const Fused2Args<float, float> *)b->d_args, b->d_two, b->ntwo, parity,
                                    b->flags, s);
    return launch_batch_two_f16((const Fused2Args<__half, float> *)b->d_args, b->d_two, b->ntwo, parity,
                                b->flags, s);
}

extern "C" {

void sclbm_batch_destroy(sclbm_batch *b)
{
    if (!b) return;
    for (auto &g : b->graph)
        if (g) cudaGraphExecDestroy(g);
    if (b->d_lists) cudaFree(b->d_lists);
    delete b;
}

int sclbm_batch_create(sclbm_domain *const *domains, int ndomains, const int *tile_y_per_domain,
                       sclbm_batch **out)
{
    if (!domains || ndomains < 1 || !out) return set_error(SCLBM_E_INVALID_ARGUMENT, "bad batch");
    int rc = ensure_device();
    if (rc) return rc;
    auto *b = new (std::nothrow) sclbm_batch();
    if (!b) return set_error(SCLBM_E_ALLOC, "host allocation failed");
    b->doms.assign(domains, domains + ndomains);
    if (!b->doms[0]) {
        delete b;
        return set_error(SCLBM_E_INVALID_ARGUMENT, "null domain in batch");
    }
    b->prec = b->doms[0]->prec;
    b->parity = b->doms[0]->parity;
    std::vector<int> ty(ndomains);
    double nodes_units = 0.0, nodes_tiles = 0.0;
    const SclbmTunedShape bd = tuned_batch_default(b->prec);
    const bool bd_list = bd.variant == 2 || bd.variant == 8 || bd.variant == 9 || bd.variant == 10;
    for (int k = 0; k < ndomains; ++k) {
        sclbm_domain *d = b->doms[k];
        if (!d || d->ncomp != 2 || d->prec != b->prec || d->parity != b->parity) {
            sclbm_batch_destroy(b);
            return set_error(SCLBM_E_INVALID_ARGUMENT,
                             "batch domains must be two-component, of one precision and in step");
        }
        if (needs_wide_offsets(d->N)) {
            sclbm_batch_destroy(b);
            return set_error(SCLBM_E_INVALID_ARGUMENT,
                             "batch domains must have fewer than 2^32/9 nodes (step larger ones alone)");
        }
        d->held = true;
        if (d->has_solid) b->flags |= KF_SOLID;
        if (d->p.force_on[0] || d->p.force_on[1]) b->flags |= KF_FORCE;
        const SclbmTunedShape ts = tuned_shape(d->nx, d->ny, b->prec);
        ty[k] = tile_y_per_domain && tile_y_per_domain[k] > 0 ? tile_y_per_domain[k]
                : (bd_list && bd.tile_y > 0 && d->has_solid ? bd.tile_y : ts.tile_y);
        (ts.variant == 3 ? nodes_units : nodes_tiles) += (double)d->nx * (double)d->ny;
    }
    // Small batches: tiles as tall as the table's (tuned on batches of ~4M
    // nodes) would leave most CTAs idle -- a batch of five 256^2 domains got 60
    // tiles of 64 rows for 740 resident CTAs.  Heights the caller did not set
    // are halved (down to 4 rows) until there are four tiles per resident CTA.
    {
        const long resident = (long)std::max(1, batch_blocks_per_sm(b->prec)) * sm_count();
        auto count = [&]() {
            long n = 0;
            for (int k = 0; k < ndomains; ++k)
                n += (long)((b->doms[k]->nx + BATCH_TX - 3) / (BATCH_TX - 2)) *
                     (long)((b->doms[k]->ny + ty[k] - 1) / ty[k]);
            return n;
        };
        const bool given = tile_y_per_domain != nullptr;
        while (!given && count() < 4 * resident) {
            bool changed = false;
            for (int k = 0; k < ndomains; ++k)
                if (ty[k] > 4) {
                    ty[k] = std::max(4, ty[k] / 2);
                    changed = true;
                }
            if (!changed) break;
        }
    }
    // tile lists of tiles `width` columns wide, largest tiles first
    auto tile_list = [&](int width) {
        const int w = width - 2;
        std::vector<TileRef> list;
        std::vector<long> cost;
        for (int k = 0; k < ndomains; ++k) {
            const sclbm_domain *d = b->doms[k];
            for (int yb = 0; yb < (int)d->ny; yb += ty[k])
                for (int xb = 0; xb < (int)d->nx; xb += w) {
                    list.push_back(TileRef{k, xb, yb, 0});
                    cost.push_back((long)std::min(w, (int)d->nx - xb) *
                                   (std::min(ty[k], (int)d->ny - yb) + 2));
                }
        }
        std::vector<int> order(list.size());
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return cost[a] > cost[c]; });
        std::vector<TileRef> sorted(list.size());
        for (size_t i = 0; i < order.size(); ++i) sorted[i] = list[order[i]];
        return sorted;
    };
    std::vector<TileRef> sorted = tile_list(BATCH_TX);
    std::vector<TileRef> halves = tile_list(HALF_TX);
    std::vector<TileRef> warps = tile_list(WARP_TX);
    b->ntiles = (int)sorted.size();
    b->ntiles_half = (int)halves.size();
    b->ntiles_warp = (int)warps.size();
    int per_sm = batch_blocks_per_sm(b->prec);
    if (per_sm < 1) per_sm = 1;
    b->grid = std::max(1, std::min(b->ntiles, per_sm * sm_count()));
    for (int body = 0; body < BODY_COUNT; ++body) {
        const int pb = b->prec == SCLBM_FP64 ? per_sm : std::max(1, batch_blocks_per_sm(b->prec, body));
        const int units = body == BODY_HALF   ? (b->ntiles_half + 1) / 2
                          : body == BODY_WARP ? (b->ntiles_warp + BATCH_TX / WARP_TX - 1) / (BATCH_TX / WARP_TX)
                                              : b->ntiles;
        b->grid_body[body] = std::max(1, std::min(units, pb * sm_count()));
    }
    // rows per unit of the ring bodies: the caller's tile_y, else the tuned
    // batch default's, else RING_BATCH_ROWS
    std::vector<int> ring_rows(ndomains);
    for (int k = 0; k < ndomains; ++k)
        ring_rows[k] = tile_y_per_domain && tile_y_per_domain[k] > 0
                           ? tile_y_per_domain[k]
                           : ((bd.variant == 11 || bd.variant == 12) && bd.tile_y > 0 ? bd.tile_y : RING_BATCH_ROWS);
    if (!tile_y_per_domain) {
        // as for the tile lists: four units per resident CTA, units of at least 8 rows
        const long resident = (long)std::max(1, per_sm) * sm_count();
        auto units = [&]() {
            long n = 0;
            for (int k = 0; k < ndomains; ++k)
                n += (long)((b->doms[k]->nx + 127) / 128) *
                     std::max(1L, (long)((b->doms[k]->ny + ring_rows[k] / 2) / ring_rows[k]));
            return n;
        };
        while (units() < 4 * resident) {
            bool changed = false;
            for (int k = 0; k < ndomains; ++k)
                if (ring_rows[k] > 8) {
                    ring_rows[k] = std::max(8, ring_rows[k] / 2);
                    changed = true;
                }
            if (!changed) break;
        }
    }
    DeviceLists lists;
    switch (b->prec) {
    case SCLBM_FP64: rc = build_args<double, double>(b, ty, ring_rows, lists); break;
    case SCLBM_FP32_SHIFTED: rc = build_args<float, float>(b, ty, ring_rows, lists); break;
    default: rc = build_args<__half, float>(b, ty, ring_rows, lists); break;
    }
    // pipelined kernel: the smallest band height whose (domain, strip, band)
    // tiles all fit resident at once, bands of one domain split its rows evenly.
    // Default: the tuned variant of the size classes holding most nodes (the
    // FP16 form has no band kernel)
    b->auto_units = b->prec != SCLBM_FP16_SHIFTED && nodes_units > nodes_tiles;
    // FP32/FP16 tile lists with solid nodes: the uniform solid body (512-domain
    // ensemble, FP32: 21.7 vs 19.6 GLUPS), on one-warp tiles for FP16 storage
    // (25.3 vs 23.5 GLUPS)
    b->auto_body = !(b->flags & KF_SOLID) || b->prec == SCLBM_FP64 ? BODY_TILE
                   : b->prec == SCLBM_FP16_SHIFTED                 ? BODY_WARP
                                                                   : BODY_UNIFORM;
    b->body = b->auto_body;
    b->use_units = b->auto_units;
    // Batches with solid nodes run the body that the autotuner's sweep of the
    // whole mixed 512-domain ensemble found fastest for the precision (the
    // tuned batch default); without one recorded, FP32/FP64 take the ring body
    // on 128-column strips (ensemble: FP32 24.5 vs 21.3 GLUPS for the uniform
    // tile list, FP64 12.0 vs 10.3) and FP16 its one-warp tile list.
    if (b->flags & KF_SOLID) {
        if ((bd.variant == 11 || bd.variant == 12) && b->ring) {
            b->auto_ring = bd.variant == 11 ? 128 : 64;
        } else if (bd.variant == 2 || bd.variant == 8 || bd.variant == 10 || bd.variant == 9) {
            if (b->prec != SCLBM_FP64)
                b->auto_body = bd.variant == 8 ? BODY_UNIFORM : bd.variant == 10 ? BODY_WARP
                               : bd.variant == 9 ? BODY_HALF : BODY_TILE;
            b->auto_units = 0;
        } else if (bd.variant == 3 && b->prec != SCLBM_FP16_SHIFTED) {
            b->auto_units = 1;
        } else if (bd.variant == 0) {
            b->auto_ring = b->ring && b->prec != SCLBM_FP16_SHIFTED ? 128 : 0;
        }
        b->body = b->auto_body;
        b->use_units = b->auto_units;
    }
    b->use_ring = b->auto_ring;
    std::vector<BandTile> bands;
    if (b->prec != SCLBM_FP16_SHIFTED) {
        const int res = std::max(1, b->prec == SCLBM_FP64 ? async_resident_fp64() : async_resident_f32());
        int H = 4;
        auto count = [&](int h) {
            long long n = 0;
            for (auto *d : b->doms)
                n += (long long)((d->nx + ASYNC_STRIP - 1) / ASYNC_STRIP) * ((d->ny + h - 1) / h);
            return n;
        };
        int max_ny = 1;
        for (auto *d : b->doms) max_ny = std::max(max_ny, (int)d->ny);
        while (count(H) > res && H < max_ny) ++H;
        b->band_rows = H;
        for (int k = 0; k < ndomains; ++k) {
            const sclbm_domain *d = b->doms[k];
            const int nb = (int)((d->ny + H - 1) / H), ns = (int)((d->nx + ASYNC_STRIP - 1) / ASYNC_STRIP);
            for (int j = 0; j < nb; ++j) {
                const int y0 = (int)((long long)d->ny * j / nb), y1 = (int)((long long)d->ny * (j + 1) / nb);
                for (int s = 0; s < ns; ++s) bands.push_back(BandTile{k, s * ASYNC_STRIP, y0, y1});
            }
        }
        b->nbands = (int)bands.size();
        b->band_grid = std::max(1, std::min(b->nbands, res));
        lists.add(&b->d_bands, std::move(bands));
    }
    lists.add(&b->d_tiles, std::move(sorted));
    lists.add(&b->d_tiles_warp, std::move(warps));
    lists.add(&b->d_tiles_half, std::move(halves));
    if (!rc) build_two(b, tile_y_per_domain, lists);
    if (!rc) rc = build_flat(b, tile_y_per_domain, lists);
    if (!rc) rc = lists.send(&b->d_lists);
    if (rc) {
        sclbm_batch_destroy(b);
        return rc;
    }
    *out = b;
    return SCLBM_OK;
}

int sclbm_batch_set_kernel(sclbm_batch *b, int variant)
{
    if (!b) return set_error(SCLBM_E_INVALID_ARGUMENT, "null batch");
    if (variant != 0 && variant != 2 && variant != 3 && variant != 5 && variant != 6 && variant != 8 &&
        variant != 9 && variant != 10 && variant != 11 && variant != 12)
        return set_error(SCLBM_E_INVALID_ARGUMENT, "variant is 0, 2, 3, 5, 6, 8, 9, 10, 11 or 12");
    if ((variant == 11 || variant == 12) && !b->ring)
        return set_error(SCLBM_E_INVALID_ARGUMENT,
                         "the ring body needs every domain's width to be a multiple of "
                         "16 bytes of storage (nx a multiple of 2, 4 or 8 for FP64, FP32, FP16)");
    if (variant == 3 && b->prec == SCLBM_FP16_SHIFTED)
        return set_error(SCLBM_E_INVALID_ARGUMENT, "the FP16 form uses the tile list (variant 2)");
    if ((variant == 5 || variant == 6 || (variant >= 8 && variant <= 10)) && b->prec == SCLBM_FP64)
        return set_error(SCLBM_E_INVALID_ARGUMENT,
                         "the load-ahead, compacted and uniform tile lists are for FP32/FP16 storage");
    b->use_ring = variant == 11 ? 128 : (variant == 12 ? 64 : (variant == 0 ? b->auto_ring : 0));
    b->use_units = variant == 3 || (variant == 0 && b->auto_units);
    b->body = variant == 5   ? BODY_AHEAD
              : variant == 6 ? BODY_COMPACT
              : variant == 8 ? BODY_UNIFORM
              : variant == 9 ? BODY_HALF
              : variant == 10 ? BODY_WARP
              : variant == 0 ? b->auto_body
                             : BODY_TILE;
    b->use_two = variant == 0 && b->ntwo > 0;
    b->use_flat = variant == 0 && b->nflat > 0;
    for (auto &g : b->graph)
        if (g) {
            cudaGraphExecDestroy(g);
            g = nullptr;
        }
    return SCLBM_OK;
}

int sclbm_batch_info(const sclbm_batch *b, int *ntiles, int *grid_ctas)
{
    if (!b) return set_error(SCLBM_E_INVALID_ARGUMENT, "null batch");
    if (b->use_two || b->use_flat) { // one CTA per unit or tile
        const int n = b->use_two ? b->ntwo : b->nflat;
        if (ntiles) *ntiles = n;
        if (grid_ctas) *grid_ctas = n;
        return SCLBM_OK;
    }
    const int r = b->use_ring == 64 ? 1 : 0;
    if (ntiles) *ntiles = b->use_ring ? b->nunits[r] : (b->use_units ? b->ntiles : batch_ntiles(b));
    if (grid_ctas)
        *grid_ctas = b->use_ring    ? b->ring_grid[r]
                     : b->use_units ? b->band_grid
                                    : (b->prec == SCLBM_FP64 ? b->grid : b->grid_body[b->body]);
    return SCLBM_OK;
}

int sclbm_batch_step(sclbm_batch *b, int nsteps, int use_graph)
{
    if (!b) return set_error(SCLBM_E_INVALID_ARGUMENT, "null batch");
    if (nsteps < 0) return set_error(SCLBM_E_INVALID_ARGUMENT, "negative step count");
    for (auto *d : b->doms)
        if (d->parity != b->parity)
            return set_error(SCLBM_E_RUNTIME, "a batch domain was stepped outside the batch");
    cudaStream_t s = stream();
    if (use_graph && b->graph_stream != s) {
        for (auto &g : b->graph)
            if (g) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
        b->graph_stream = s;
    }
    int done = 0;
    while (use_graph && nsteps - done >= GRAPH_STEPS) {
        cudaGraphExec_t &ge = b->graph[b->parity];
        if (!ge) {
            cudaGraph_t g;
            SCLBM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            cudaError_t e = cudaSuccess;
            const int launches = b->use_two ? GRAPH_STEPS / 2 : GRAPH_STEPS; // even: the parity returns
            for (int k = 0; k < launches && e == cudaSuccess; ++k)
                e = b->use_two ? batch_launch_two(b, b->parity ^ (k & 1), s)
                               : batch_launch_any(b, b->parity ^ (k & 1), s);
            cudaError_t e2 = cudaStreamEndCapture(s, &g);
            if (e != cudaSuccess) return cuda_fail(e, "batch capture");
            if (e2 != cudaSuccess) return cuda_fail(e2, "batch capture end");
            e = cudaGraphInstantiate(&ge, g, 0);
            cudaGraphDestroy(g);
            if (e != cudaSuccess) return cuda_fail(e, "graph instantiate");
        }
        SCLBM_CUDA(cudaGraphLaunch(ge, s));
        done += GRAPH_STEPS; // even: parity unchanged
    }
    // pairs in twos, so that the buffers' parity follows the steps'
    for (; b->use_two && nsteps - done >= 4; done += 4)
        for (int k = 0; k < 2; ++k) {
            cudaError_t e = batch_launch_two(b, b->parity ^ k, s);
            if (e != cudaSuccess) return cuda_fail(e, "batch step");
        }
    for (; done < nsteps; ++done) {
        cudaError_t e = batch_launch_any(b, b->parity, s);
        if (e != cudaSuccess) return cuda_fail(e, "batch step");
        b->parity ^= 1;
    }
    for (auto *d : b->doms) d->parity = b->parity;
    return SCLBM_OK;
}

} // extern "C"
