"""The default step kernels -- one node per thread, and steps run in pairs (two
per launch) -- against the register tile.

Their nodes run the same arithmetic as the register tile's, and pairs
hold the state between the steps in the storage type, so the populations are
equal byte for byte: at widths around its strips (122 columns), with bands of
one row and of uneven heights, on lattices that its halo wraps around, for odd
and even step counts.  The parity a batch relies on, and a captured step call,
behave as with one step per launch.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(sclbm, nx, ny, prec, porous, force, seed=5):
    from sc_lbm_b200 import workloads as W
    n = nx * ny
    mask = (W.uniform(seed, n) < 0.75).astype(np.int32) if porous else np.ones(n, np.int32)
    F = (W.force_vec(1e-4, "x"), W.force_vec(2e-4, "y")) if force else (None, None)
    p = sclbm.make_params(ncomp=2, tau=(1.0, 0.9), g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1),
                          rho_ref=(1.0, 1.2), force=F)
    f = [W.populations((1 + 0.2 * k) * (1 + 0.1 * (2 * W.uniform(seed + k, n) - 1)), mask)
         for k in range(2)]

    def build(variant=0, rows=0):
        d = sclbm.Domain(nx, ny, mask, p, prec)
        d.set_kernel(variant, rows)  # a band height asks for pairs
        for k in range(2):
            d.upload_f(k, f[k])
        return d
    return build


def state(d):
    return [d.download_f(k).tobytes() for k in range(2)]


@pytest.mark.parametrize("prec_name", ["FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("nx,ny,rows", [(4, 4, 2), (5, 7, 1), (64, 33, 5), (121, 20, 20), (122, 9, 4),
                                        (123, 40, 32), (245, 31, 3), (1021, 77, 7), (1400, 1100, 0)])
def test_pairs_match_single_steps(sclbm, prec_name, nx, ny, rows):
    prec = getattr(sclbm, prec_name)
    for porous in (False, True):
        for force in (False, True):
            build = make(sclbm, nx, ny, prec, porous, force)
            for steps in (2, 5):
                a, b = build(0, rows), build(2, 0)
                a.step(steps)
                b.step(steps)
                assert state(a) == state(b), (porous, force, steps)


@pytest.mark.parametrize("prec_name", ["FP64", "FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 9), (7, 1), (31, 3), (32, 4), (33, 5), (64, 37), (129, 130)])
def test_one_node_per_thread_matches_tiles(sclbm, prec_name, nx, ny):
    """Tiles of 32 x 4 nodes: full, partial and wrapping around the lattice."""
    prec = getattr(sclbm, prec_name)
    for porous in (False, True):
        for force in (False, True):
            build = make(sclbm, nx, ny, prec, porous, force)
            a, b = build(), build(2)
            a.step(5)
            b.step(5)
            assert state(a) == state(b), (porous, force)


def test_pairs_keep_a_domain_in_step_with_its_batch(sclbm):
    """Two steps outside the batch leave it usable, one does not."""
    build = [make(sclbm, nx, 48, sclbm.FP32_SHIFTED, True, False) for nx in (96, 60)]
    doms, alone = [b() for b in build], [b(2) for b in build]
    for d in doms:
        d.set_kernel(0, 16)
    doms[0].step(2)  # before the batch takes the buffers' addresses
    batch = sclbm.Batch(doms)
    doms[1].step(6)
    batch.step(3)
    alone[0].step(5)
    alone[1].step(9)
    for d, a in zip(doms, alone):
        assert state(d) == state(a)
    doms[1].step(1)
    with pytest.raises(RuntimeError):
        batch.step(1)


@pytest.mark.parametrize("rows", [0, 16])
def test_captured_steps_replay(sclbm, rows):
    import torch
    build = make(sclbm, 130, 50, sclbm.FP32_SHIFTED, False, True)
    d, one = build(), build(2)
    st = torch.cuda.Stream()
    sclbm.synchronize()
    sclbm.set_stream(st.cuda_stream)
    try:
        d.set_kernel(0, rows)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            d.step(6)
        with torch.cuda.stream(st):
            for _ in range(3):
                g.replay()
        st.synchronize()
        one.step(18)
        assert state(d) == state(one)
    finally:
        sclbm.synchronize()
        sclbm.set_stream(None)


@pytest.mark.parametrize("prec_name", ["FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("porous", [False, True])
def test_batch_pairs_match_single_steps(sclbm, prec_name, porous):
    """Uneven domains, a caller's band height, runs of whole graphs and of a few steps."""
    prec = getattr(sclbm, prec_name)
    sizes = [(4, 4), (64, 33), (128, 70), (130, 17), (245, 31), (512, 9)]
    build = [make(sclbm, nx, ny, prec, porous, k % 2 == 1, seed=9 + k) for k, (nx, ny) in enumerate(sizes)]
    alone = [b(2) for b in build]
    for a in alone:
        a.step(27)
    for tile_y in (None, [7] * len(sizes)):
        doms = [b() for b in build]
        batch = sclbm.Batch(doms, tile_y)
        batch.step(1)
        batch.step(26)
        for d, a, size in zip(doms, alone, sizes):
            assert state(d) == state(a), (size, tile_y)


@pytest.mark.parametrize("prec_name", ["FP64", "FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 9), (7, 1), (22, 6), (23, 13), (64, 33), (400, 180), (420, 200),
                                   (700, 333)])
def test_single_component_steps_per_launch(sclbm, prec_name, nx, ny):
    """K steps in one launch (K = 6, 5, 3 or 2 by size) against K calls of one
    step, whose tiles hold the halo but use one node of it."""
    from sc_lbm_b200 import workloads as W
    n = nx * ny
    for porous in (False, True):
        mask = (W.uniform(3, n) < 0.75).astype(np.int32) if porous else np.ones(n, np.int32)
        p = sclbm.make_params(ncomp=1, tau=(0.9, 1.0), force=(W.force_vec(1e-5, "x") if porous else None, None))
        f = W.populations(1 + 0.1 * (2 * W.uniform(4, n) - 1), mask)
        out = []
        for calls in ([13], [1] * 13, [2, 5, 6]):
            d = sclbm.Domain(nx, ny, mask, p, getattr(sclbm, prec_name))
            d.upload_f(0, f)
            for k in calls:
                d.step(k)
            out.append(d.download_f(0).tobytes())
        assert out[0] == out[1] == out[2], porous


def test_single_component_matches_reference_steps(sclbm):
    """FP64, a wall, random solids and a force, at sizes around the tiles."""
    from sc_lbm_b200 import workloads as W
    for nx, ny in ((3, 2), (23, 7), (45, 30), (120, 50)):
        n = nx * ny
        mask = (W.uniform(nx, n) < 0.8).astype(np.int32)
        mask[:nx] = 0
        F = W.force_vec(1e-4, "x")
        g = sclbm.Geometry.from_mask(nx, ny, mask)
        fl, lbm = sclbm.Fluid(g, 0.8), sclbm.LBM(g)
        f = W.populations(1 + 0.1 * (2 * W.uniform(5, n) - 1), mask)
        fl.set("f", f)
        for _ in range(9):  # the reference's operators, one call each
            lbm.collide(g, fl)
            lbm.add_volume_force(g, fl, F)
            lbm.stream(g, fl)
        want = fl.get("f").tobytes()
        fl.set("f", f)
        lbm.step_single(g, fl, 9, F)
        assert fl.get("f").tobytes() == want
        d = sclbm.Domain(nx, ny, mask, sclbm.make_params(ncomp=1, tau=(0.8, 1.0), force=(F, None)), sclbm.FP64)
        d.upload_f(0, f)
        d.step(9)
        assert d.download_f(0).tobytes() == want
