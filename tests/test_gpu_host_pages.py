"""Fields read into fresh arrays: whole whatever their alignment, and no dearer
for a program that makes an object, reads one field and drops it."""
import mmap
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec_name", ["FP64", "FP32_SHIFTED"])
@pytest.mark.parametrize("n", [393216, 393217, 1100000, 2500001])
@pytest.mark.parametrize("off", [0, 8, 4088])
def test_fresh_arrays_are_filled(sclbm, prec_name, n, off):
    from sc_lbm_b200 import api, capi
    d = sclbm.Domain(n, 1, np.ones(n, np.int32), sclbm.make_params(ncomp=1), getattr(sclbm, prec_name))
    d.init_noise(0, 1.0, 0.1, 7)
    want = {}
    for call, size in (("f", 9 * n), ("rho", n)):
        got = []
        for fresh in (True, False):
            m = mmap.mmap(-1, 8 * size + 8192)
            a = np.frombuffer(m, np.float64, size, off)
            if not fresh:
                a[:] = -1.0
            capi.call("sclbm_domain_download_" + call, d.handle, 0, api._dp(a), size)
            got.append(a.tobytes())
            assert m[:off] == bytes(off) and m[off + 8 * size:] == bytes(8192 - off)
        assert got[0] == got[1]
        want[call] = np.frombuffer(got[0]).reshape(-1, n).sum(axis=0)
    np.testing.assert_allclose(want["f"], want["rho"], rtol=1e-6)


def test_one_field_of_a_short_lived_object(sclbm):
    """Reading one field costs no set-up beyond a slightly smaller one's: within
    a factor of two, where a buffer allocated for it costs five."""
    def median(n):
        mask, p, t = np.ones(n, np.int32), sclbm.make_params(ncomp=2), []
        for _ in range(9):
            t0 = time.perf_counter()
            d = sclbm.Domain(n, 1, mask, p, sclbm.FP32_SHIFTED)
            d.download_rho(0)
            del d
            t.append(time.perf_counter() - t0)
        return np.median(t)
    median(380000)
    small, large = median(380000), median(410000)  # 2.9 and 3.1 MiB
    assert large < 2 * small, (small, large)
