"""Records of more 1D lattices than a grid has rows."""
import numpy as np
import pytest

import swalbe_gb300 as sw

pytestmark = pytest.mark.gpu


def test_records_of_70000_lattices():
    count = 70000
    s = sw.SysConst_1D(5, sw.Taumucs())
    b = sw.Batch1D([s] * count, records=2)
    h = [1.0, 1.1, 0.9, 1.2, 0.8]
    one = sw.Sys(s, T=np.float64)
    for x in (0, 65535, 65536, count - 1):
        b.set_height(x, h)
    one.height = h
    b.step(7)
    one.step(7)
    b.sync()
    want = [(r.t, r.mass, r.hmax, r.hmin, r.wetted) for r in one.measures()[-2:]]
    for x in (0, 65535, 65536, count - 1):
        assert np.array_equal(b.height(x), one.height)
        assert [(r.t, r.mass, r.hmax, r.hmin, r.wetted) for r in b.measures(x)] == want
    flat = b.measures(123)
    assert [r.t for r in flat] == [6, 7] and flat[0].hmax == 1.0
