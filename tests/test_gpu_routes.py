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
