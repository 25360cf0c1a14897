"""Captured calls replayed between eager ones.

A graph holds the addresses of the buffers it was captured with.  Steps taken
outside it, however many a launch advances, leave the state where single steps
would: in the same buffers after an even number of them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Captured:
    """Calls of the library captured into a graph on a stream of their own."""

    def __init__(self, sclbm):
        import torch
        self.torch, self.sclbm = torch, sclbm

    def __enter__(self):
        self.sclbm.synchronize()
        self.stream = self.torch.cuda.Stream()
        self.sclbm.set_stream(self.stream.cuda_stream)
        return self

    def capture(self, call):
        self.graph = self.torch.cuda.CUDAGraph()
        with self.torch.cuda.graph(self.graph, stream=self.stream):
            call()

    def replay(self):
        with self.torch.cuda.stream(self.stream):
            self.graph.replay()

    def __exit__(self, *exc):
        self.sclbm.synchronize()
        self.sclbm.set_stream(None)


def domain(sclbm, nx, ny, prec, ncomp, variant=0, rows=0):
    from sc_lbm_b200 import workloads as W
    n = nx * ny
    mask = (W.uniform(2, n) < 0.8).astype(np.int32)
    p = sclbm.make_params(ncomp=ncomp, tau=(0.9, 1.0), g_fluid=(0.9, 0.9), g_solid=(-0.1, 0.1),
                          rho_ref=(1.0, 1.0), force=(W.force_vec(1e-5, "x"), None))
    d = sclbm.Domain(nx, ny, mask, p, prec)
    d.set_kernel(variant, rows)
    for k in range(ncomp):
        d.upload_f(k, W.populations(1 + 0.1 * (2 * W.uniform(4 + k, n) - 1), mask))
    return d


def state(d):
    return [d.download_f(k).tobytes() for k in range(d.ncomp)]


@pytest.mark.parametrize("prec_name", ["FP64", "FP32_SHIFTED", "FP16_SHIFTED"])
@pytest.mark.parametrize("ncomp", [1, 2])
@pytest.mark.parametrize("captured", [1, 2, 6, 7])
def test_domain_steps_between_replays(sclbm, prec_name, ncomp, captured):
    """Eager counts that make odd numbers of launches of two, or of up to six, steps."""
    prec = getattr(sclbm, prec_name)
    rows = 16 if ncomp == 2 and prec_name != "FP64" else 0  # a band height asks for pairs
    d, one = domain(sclbm, 130, 50, prec, ncomp, 0, rows), domain(sclbm, 130, 50, prec, ncomp, 2 * (ncomp - 1))
    steps = 2
    d.step(2)  # before anybody holds an address
    with Captured(sclbm) as c:
        c.capture(lambda: d.step(captured))
        if captured % 2:  # the graph leaves the state in the other buffers
            c.replay()
            steps += captured
        else:
            for eager in (2, 6, 10, 0):
                c.replay()
                d.step(eager)
                steps += captured + eager
        for _ in range(steps):
            one.step(1)
        assert state(d) == state(one)


@pytest.mark.parametrize("how", ["step_single", "operators"])
@pytest.mark.parametrize("nx,ny", [(40, 30), (520, 300)])
def test_fluid_steps_between_replays(sclbm, how, nx, ny):
    from sc_lbm_b200 import workloads as W
    n = nx * ny
    mask = (W.uniform(6, n) < 0.8).astype(np.int32)
    g = sclbm.Geometry.from_mask(nx, ny, mask)
    fl, lbm, other = sclbm.Fluid(g, 0.8), sclbm.LBM(g), sclbm.Fluid(g, 0.8)
    f = W.populations(1 + 0.1 * (2 * W.uniform(5, n) - 1), mask)
    fl.set("f", f)
    lbm.step_single(g, fl, 0)  # the mask goes to the device

    def two_steps(x):
        if how == "step_single":
            lbm.step_single(g, x, 2)
        else:
            for _ in range(2):
                lbm.collide(g, x)
                lbm.stream(g, x)
    with Captured(sclbm) as c:
        c.capture(lambda: two_steps(fl))
        steps = 0
        for eager in (2, 6, 10, 0):
            c.replay()
            lbm.step_single(g, fl, eager)
            steps += 2 + eager
        # the LBM's scratch array is the graph's too: another fluid gives it back
        other.set("f", f)
        lbm.step_single(g, other, 2)
        c.replay()
        got, got2 = fl.get("f"), other.get("f")
    one = sclbm.Fluid(g, 0.8)
    one.set("f", f)
    for k in range(steps + 2):
        lbm.step_single(g, one, 1)
        if k == 1:
            assert got2.tobytes() == one.get("f").tobytes()
    assert got.tobytes() == one.get("f").tobytes()


def test_halo_rows_between_replays(sclbm):
    import torch
    d = domain(sclbm, 64, 48, sclbm.FP32_SHIFTED, 2, 0, 16)
    ghost = torch.zeros(2, d.halo_bytes(4), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with Captured(sclbm) as c:
        c.capture(lambda: d.halo_pack(4, 0, ghost[0].data_ptr()))
        d.step(2)
        c.replay()
        d.halo_pack(4, 0, ghost[1].data_ptr())
        sclbm.synchronize()
        assert torch.equal(ghost[0], ghost[1])
