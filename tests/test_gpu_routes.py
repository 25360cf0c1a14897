"""Lattices at the edges of the dispatch rules: the same bytes on both sides."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def median_time(sclbm, call):
    t = []
    for _ in range(7):
        sclbm.synchronize()
        t0 = time.perf_counter()
        call()
        sclbm.synchronize()
        t.append(time.perf_counter() - t0)
    return np.median(t)


@pytest.mark.parametrize("prec_name", ["FP64", "FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("nx", [1, 3, 4])
def test_narrow_single_component_lattices(sclbm, prec_name, nx):
    """A few columns (one node per thread) against the same columns repeated
    (several steps per launch)."""
    from sc_lbm_b200 import workloads as W
    ny, wide = 12000, 28 // nx * nx
    mask = (W.uniform(2, nx * ny) < 0.8).astype(np.int32).reshape(ny, nx)
    rho = (1 + 0.1 * (2 * W.uniform(3, nx * ny) - 1)).reshape(ny, nx)
    p = sclbm.make_params(ncomp=1, tau=(0.9, 1.0), force=(W.force_vec(1e-5, "x"), None))
    out = []
    for cols in (nx, wide):
        m, r = (np.tile(a, (1, cols // nx)).ravel() for a in (mask, rho))
        d = sclbm.Domain(cols, ny, m, p, getattr(sclbm, prec_name))
        d.upload_f(0, W.populations(r, m))
        for k in (7, 1, 2):
            d.step(k)
        out.append(d.download_f(0).reshape(9, ny, cols)[:, :, :nx].tobytes())
    assert out[0] == out[1]


def test_narrow_single_component_lattices_cost_their_nodes(sclbm):
    """4 x 100000 in no more than three times the time of 400 x 1000 (seven times
    by tiles that hold four columns each)."""
    def per_call(nx, ny):
        d = sclbm.Domain(nx, ny, np.ones(nx * ny, np.int32), sclbm.make_params(ncomp=1), sclbm.FP64)
        d.init_noise(0, 1.0, 0.01, 1)
        return median_time(sclbm, lambda: d.step(200))
    assert per_call(4, 100000) < 3 * per_call(400, 1000)


def pair_domain(sclbm, nx, ny, prec, variant, rows, seed=1):
    from sc_lbm_b200 import workloads as W
    mask = (W.uniform(2, nx * ny) < 0.8).astype(np.int32)
    p = sclbm.make_params(ncomp=2, g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1))
    d = sclbm.Domain(nx, ny, mask, p, prec)
    d.set_kernel(variant, rows)
    for k in range(2):
        d.init_noise(k, 1.0, 0.1, seed + k)
    return d


@pytest.mark.parametrize("prec_name", ["FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("nx,ny,rows", [(4, 4, 6), (5, 7, 6), (64, 33, 6), (121, 13, 6), (122, 9, 8), (123, 6, 64),
                                        (64, 33, 5), (64, 33, 4), (64, 33, 3)])
def test_bands_on_both_sides_of_the_lowest_pair(sclbm, prec_name, nx, ny, rows):
    prec = getattr(sclbm, prec_name)
    a, b = (pair_domain(sclbm, nx, ny, prec, v, r) for v, r in ((0, rows), (2, 0)))
    a.step(7)
    b.step(7)
    assert [a.download_f(k).tobytes() for k in range(2)] == [b.download_f(k).tobytes() for k in range(2)]


def test_low_bands_cost_no_more_than_single_steps(sclbm):
    """Bands of one row asked for: within half as much again as the register tile
    (twice its time in pairs)."""
    t = [median_time(sclbm, lambda d=d: d.step(100))
         for d in (pair_domain(sclbm, 1024, 1024, sclbm.FP16_SHIFTED, v, r) for v, r in ((0, 1), (8, 0)))]
    assert t[0] < 1.5 * t[1], t


def small_batch(sclbm, nx, ny, count, body):
    doms = [pair_domain(sclbm, nx, ny, sclbm.FP16_SHIFTED, 2, 0, seed=k) for k in range(count)]
    batch = sclbm.Batch(doms)
    batch.set_kernel(body)
    return doms, batch


def test_many_narrow_domains_keep_their_one_warp_tiles(sclbm):
    """300 domains of 20 x 20 with solid nodes: no slower than the one-warp body
    asked for by name (1.6 times its time in pairs)."""
    (a, x), (b, y) = (small_batch(sclbm, 20, 20, 300, body) for body in (0, 10))
    t = [median_time(sclbm, lambda x=x: x.step(200)) for x in (x, y)]
    assert t[0] < 1.3 * t[1], t
    assert all(p.download_f(0).tobytes() == q.download_f(0).tobytes() for p, q in zip(a[::37], b[::37]))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("porous", [False, True])
def test_fp64_batch_of_ragged_lattices(sclbm, graph, porous):
    """One node per thread on heights off its tiles' four rows and widths off 32."""
    from sc_lbm_b200 import workloads as W
    sizes = [(1, 9), (7, 1), (33, 5), (129, 130), (31, 3), (1, 1), (64, 37)]
    doms, alone = [], []
    for out, variant in ((doms, 0), (alone, 2)):
        for k, (nx, ny) in enumerate(sizes):
            n = nx * ny
            mask = (W.uniform(k, n) < 0.75).astype(np.int32) if porous else np.ones(n, np.int32)
            F = (W.force_vec(1e-4, "x"), W.force_vec(2e-4, "y")) if k % 2 else (None, None)
            d = sclbm.Domain(nx, ny, mask, sclbm.make_params(g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1), force=F),
                             sclbm.FP64)
            d.set_kernel(variant)
            for c in range(2):
                d.upload_f(c, W.populations(1 + 0.1 * (2 * W.uniform(5 + c + k, n) - 1), mask))
            out.append(d)
    batch = sclbm.Batch(doms)
    batch.step(23, graph)
    for d, a, size in zip(doms, alone, sizes):
        a.step(23)
        for c in range(2):
            assert d.download_f(c).tobytes() == a.download_f(c).tobytes(), size


@pytest.mark.parametrize("radii,flat", [((10, 30), True), (None, False)])
def test_fp64_batch_of_scattered_solids(sclbm, radii, flat):
    """Large disks: one node per thread; every tenth node solid: the ring."""
    from sc_lbm_b200 import workloads as W
    nx, ny, n = 1024, 512, 1024 * 512
    mask = np.ones(n, np.int32) if radii else (W.uniform(1, n) < 0.9).astype(np.int32)
    p = sclbm.make_params(g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1))
    doms = [sclbm.Domain(nx, ny, mask, p, sclbm.FP64) for _ in range(3)]
    for d in doms:
        if radii:
            d.add_random_disks(0.7, *radii, 3)
        for c in range(2):
            d.init_noise(c, 1.0, 0.1, 3 + c)
    batch = sclbm.Batch(doms)
    tiles = 3 * (nx // 32) * (ny // 4)
    assert (batch.info()[0] == tiles) == flat
    batch.step(3)
    one = sclbm.Domain(nx, ny, doms[0].download_mask(), p, sclbm.FP64)
    one.set_kernel(2)
    for c in range(2):
        one.init_noise(c, 1.0, 0.1, 3 + c)
    one.step(3)
    assert all(d.download_f(0).tobytes() == one.download_f(0).tobytes() for d in doms)


@pytest.mark.parametrize("prec_name,rows", [("FP32_SHIFTED", 16), ("FP16_SHIFTED", 16), ("FP16_SHIFTED", 0)])
def test_disks_added_on_the_device_reach_the_node_codes(sclbm, prec_name, rows):
    """Pairs and the FP16 form of one node per thread read node codes, the register
    tile the mask: the same bytes after disks are added, and as on a domain made
    from the finished mask."""
    nx, ny = 150, 131
    p = sclbm.make_params(g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1))
    disks = dict(porosity=0.7, rmin=3, rmax=9, seed=11)
    out = []
    for variant, r in ((0, rows), (2, 0), (0, rows)):
        mask = np.ones(nx * ny, np.int32)
        if len(out) == 2:
            mask = packed
        d = sclbm.Domain(nx, ny, mask, p, getattr(sclbm, prec_name))
        if len(out) < 2:
            assert d.add_random_disks(**disks) > 0
            packed = d.download_mask()
        d.set_kernel(variant, r)
        for k in range(2):
            d.init_noise(k, 1.0, 0.1, 3 + k)
        d.step(5)
        out.append([d.download_f(k).tobytes() for k in range(2)])
    assert out[0] == out[1] == out[2]
