// routes.h -- which kernel a call's steps run, by sizes and precision alone
// (host rules without CUDA calls).
#pragma once
#include <algorithm>
#include <cstddef>

#include "sclbm.h"

namespace sclbm {

// --------------------------------------------------- two-component lattices
// Single steps on lattices that the ring kernel does not take: one node per
// thread, or the register tile.  The tile keeps its rate on large lattices
// where the halo loads of one node per thread come from DRAM; it loses the
// columns that its last strip of 126 does not have.  us per step, one node per
// thread / register tile: FP32 1200 x 1100 40.4 / 44.7, 1800 x 1500 78.8 / 84.9, 1500 x
// 1100 52.4 / 50.1 (99 % of its strips full), 2047^2 123 / 118, 4095^2 484 / 450,
// with disks 2801 x 2401 226 / 233, 3501 x 3001 355 / 351; FP16 2801 x 2401 145 / 155,
// 3001 x 2701 184 / 176, with disks 4095^2 431 / 463; FP64 1501 x 1101 84 / 96, 4095^2
// 808 / 953.
inline bool flat_beats_tile(size_t nx, size_t ny, sclbm_precision p, bool solid)
{
    const size_t n = nx * ny, M = 1000000;
    if (p == SCLBM_FP64) return true;
    if (p == SCLBM_FP16_SHIFTED) return solid || n < 7 * M;
    if (solid) return n < 9 * M;
    const double full = (double)nx / (double)((nx + 125) / 126 * 126);
    return n < 3 * M / 2 || (n < 3 * M && full < 0.985);
}

// Whether bands of a height of the caller's choice (0: none) run in pairs
// (fused_two.cuh).  A band of r rows computes r + 4 rows of the first step, so low
// ones lose to single steps of that height, unless all units (four CTAs per SM)
// are under way at once and latency counts.  us per step, pairs / single steps:
// FP32 2048^2 2 rows 151 / 121, 512^2 3 rows 11.2 / 10.4, 1024^2 3 rows 33.7 / 37.1, 256^2
// 2 rows 5.6 / 6.3; FP16 2048^2 4 rows 115 / 103, 5 rows 104 / 100, 6 rows equal or
// faster, 300^2 5 rows 7.0 / 10.4, with solid nodes 1024^2 3 rows 42.3 / 39.1, 4 rows
// equal, 5 rows 35.7 / 41.0.
inline bool two_rows_pay(sclbm_precision p, int rows, long units, bool solid, int sms)
{
    return rows == 0 || units <= 4L * sms || rows >= (p == SCLBM_FP32_SHIFTED ? 3 : solid ? 4 : 6);
}

// Whether an FP16 batch with solid nodes, off the ring body, runs in pairs or in
// the one-warp tiles that are its single-step body: strips of few columns leave
// most of a pair kernel's CTA idle, which counts once the strips have more than
// some 25 rows per SM.  rows: of all strips together; full: nodes over the columns
// of whole strips.  us per step, pairs / one-warp tiles: 300 domains of 20 x 20 20.0
// / 12.2 (41 rows per SM, full 0.16), 60 x 60 50 / 46 (122, 0.49), 90 x 60 57 / 71 (122,
// 0.74), 12 x 8 9.4 / 9.7 (16, 0.10); 60 domains of 20 x 20 6.2 / 9.8 (8, 0.16), 44 x 60
// 12.6 / 14.0 (24, 0.36).
inline bool batch_two_beats_warp(double rows, double full, int sms) { return rows <= 25.0 * sms || full >= 0.6; }

// FP64 batches with solid nodes that the ring body takes: one node per thread, or
// the ring.  full: nodes over the columns of whole ring strips (which the ring
// computes in vain); changes: how often a row turns from fluid to solid or back,
// per node (the scattered stores of one node per thread).  us per step, one node
// per thread / ring: 2 x 1024^2 with disks of radius 10-30 (0.027) 139 / 155, 4-16
// (0.052) 155 / 163, 2-4 (0.079) 179 / 173, 10 % of all nodes solid (0.18) 198 / 183;
// 24 x (400 x 306), strips 78 % full, (0.027) 203 / 257, (0.18) 272 / 285; 16 x 512^2
// (0.056) 309 / 301; 200 x (320 x 160) 769 / 784; 4 x 256^2 (0.18) 20 / 28; every fourth
// node solid (0.375), 4 x 512^2 100 / 107, 256 x 64^2, strips half full, 97 / 143, 24 x
// (400 x 306) 280 / 288, 64 x (300 x 200) 401 / 371.
inline bool batch_flat_beats_ring(double nodes, double full, double changes)
{
    if (nodes < 1.2e6 || (nodes < 8e6 && full < 0.7)) return true;
    const bool loose = full < 0.9;
    if (nodes < 4e6) return changes < (!loose ? 0.06 : nodes < 3e6 ? 0.5 : 0.15);
    return nodes < 8e6 && loose && changes < 0.06;
}

// ------------------------------------------------- single-component lattices
// A launch of k_single (fused_single.cuh) takes as long as its tiles of 32 x 16
// nodes with halo, however few nodes of their own they hold: 0.7 us and, per
// tile, a + b n ns for n steps.  A tile of fewer rows costs less (8 + rows of
// 24), one of fewer columns does not.  A step of the kernel with one node per
// thread takes 4.2 us and c ns per node.  Measured us per step by tiles / by
// nodes: FP64 2048^2 78 / 116, 29 x 40000 23 / 35, 33 x 30000 32 / 31, 4 x 100000
// 49 / 10.4; FP32 2048^2 49 / 73, 29 x 40000 25.5 / 20.6, 4 x 100000 31 / 9.7; FP16
// 2048^2 55 / 76, 33 x 30000 21.8 / 18.6; one step a call: FP64 500^2 9.0 / 9.4,
// 1024^2 37.4 / 34.6, FP32 500^2 6.7 / 8.4, 1024^2 20.9 / 19.0.
struct SingleCost {
    int K;          // steps per launch on lattices of many tiles
    double a, b, c; // ns
};
inline SingleCost single_cost(sclbm_precision p)
{
    if (p == SCLBM_FP64) return {2, 10.6, 2.4, 0.025};
    if (p == SCLBM_FP32_SHIFTED) return {3, 5.0, 2.15, 0.0135};
    return {3, 5.3, 2.5, 0.0155};
}

// whether n steps of the lattice in one launch of depth K beat n launches of
// one node per thread; lattices whose tiles of a greater depth than K fit the
// GPU at once: always (3.5 us against 4.2 for a single step)
inline bool single_pays(size_t nx, size_t ny, sclbm_precision p, int K, int n)
{
    const SingleCost s = single_cost(p);
    if (K > s.K) return true;
    if (K < s.K) return false;
    const size_t H = K - 1, w = 32 - 2 * H, h = 16 - 2 * H, rest = ny % h;
    const double tiles = (double)((nx + w - 1) / w) * ((double)(ny / h) + (rest ? (8 + rest + 2 * H) / 24.0 : 0.0));
    return 700 + tiles * (s.a + s.b * n) < n * (4200 + s.c * (double)nx * (double)ny);
}

// Steps per launch.  While the tiles of six steps (22 x 6 nodes) fit the GPU at
// once (wave: two CTAs per SM) a launch's latency is worth the halo's work;
// then five steps for the shifted forms up to one and a half waves of their
// tiles (24 x 8), three for FP64 up to one wave (28 x 12), and as many as pay for
// the repeated halo: three for the shifted forms, two for FP64, or one (no
// tiles at all) on lattices a few nodes wide.  us per step for K = 2 / 3 / 5 / 6:
// FP64 200 x 50 2.16 / 1.74 / 1.36 / 1.23, 400 x 200 3.07 / 2.66 / 2.81 / 3.85, 1500 x
// 600 18.5 / 19.0 / 24.7 / 32.6; FP32 200 x 50 1.64 / 1.31 / 0.96 / 0.85, 400 x 200
// 2.29 / 2.33 / 1.77 / 2.38, 1500 x 600 12.9 / 11.2 / 14.5 / 18.9.
inline int single_depth(size_t nx, size_t ny, sclbm_precision p, int sms)
{
    const size_t wave = 2 * (size_t)sms;
    auto tiles = [&](size_t w, size_t h) { return ((nx + w - 1) / w) * ((ny + h - 1) / h); };
    if (tiles(22, 6) <= wave) return 6;
    if (p == SCLBM_FP64 && tiles(28, 12) <= wave) return 3;
    if (p != SCLBM_FP64 && tiles(24, 8) <= wave + wave / 2) return 5;
    const int K = single_cost(p).K;
    return single_pays(nx, ny, p, K, K) ? K : 1;
}

// launches for nsteps, at most K each; keep: an odd number of them exactly when
// nsteps is odd, so that two buffers in turn end as after single steps (one
// more launch at most)
inline int single_launches(int nsteps, int K, bool keep)
{
    const int n = nsteps / K + (nsteps % K != 0);
    return keep && ((n ^ nsteps) & 1) ? n + 1 : n;
}

} // namespace sclbm
