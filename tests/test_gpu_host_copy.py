"""Fields copied out through the pinned buffer: chunk edges, more chunks than
slots, several threads at once, arrays that start off a page."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [43690, 43691, 65536, 262144, 300001])
def test_large_fields_arrive_whole(sclbm, n):
    from sc_lbm_b200 import workloads as W
    g = sclbm.Geometry(n, 1)
    fl = sclbm.Fluid(g, 1.0)
    v = W.uniform(n, 9 * n)
    fl.set("f", v)
    assert fl.get("f").tobytes() == v.tobytes()
    assert fl.get("rho").tobytes() == np.zeros(n).tobytes()
    off = np.empty(9 * n + 1)[1:]
    from sc_lbm_b200 import api, capi
    capi.call("sclbm_fluid_read", fl.handle, capi.FIELDS["f"], api._dp(off), off.size)
    assert off.tobytes() == v.tobytes()


def test_copies_from_several_threads(sclbm):
    from sc_lbm_b200 import workloads as W
    n = 100000
    g = sclbm.Geometry(n, 1)
    fluids = [sclbm.Fluid(g, 1.0) for _ in range(4)]
    want = [W.uniform(k + 1, 9 * n) for k in range(4)]
    for f, v in zip(fluids, want):
        f.set("f", v)
    bad = []

    def read(k):
        for _ in range(6):
            if fluids[k].get("f").tobytes() != want[k].tobytes():
                bad.append(k)
    threads = [threading.Thread(target=read, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
