"""Lattices at the edges of the dispatch rules: the same bytes on both sides."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
        t = []
        for _ in range(7):
            sclbm.synchronize()
            t0 = time.perf_counter()
            d.step(200)
            sclbm.synchronize()
            t.append(time.perf_counter() - t0)
        return np.median(t)
    assert per_call(4, 100000) < 3 * per_call(400, 1000)
