"""The mass record of FP32 states with heights of 2^24 and more, whose rounding
residues (half an ulp at most) reach 1: every cell's pulled height and residue, summed in
integers here, equal the record up to its conversion to Float64."""
import numpy as np
import pytest

import swalbe_gb300 as sw
from swalbe_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def pulled_mass(f):
    """Sum of h + residue over the cells, in units of 2^-32, from the streamed populations."""
    f = np.moveaxis(f, -1, 0).astype(np.float32)
    s = ((f[1] + f[3]) + (f[5] + f[7])) + ((f[2] + f[4]) + (f[6] + f[8]))
    h = f[0] + s
    lo = s - (h - f[0])
    unit = np.float32(2.0 ** 32)
    return sum(int(x) for x in np.concatenate([np.rint(h * unit).ravel(), np.rint(lo * unit).ravel()])), np.abs(lo).max()


@pytest.mark.parametrize("geo", [(64, 2), (128, 4), (-32, 2), (32, 16), (33, 0)], ids=str)
def test_record_of_large_heights(geo):
    Lx, Ly = 8, 4  # a sum of 64-bit integers holds 2^31 / 2^25 = 64 such heights
    s = sw.SysConst(Lx, Ly, sw.Taumucs(gamma=1e-12))
    st = sw.Sys(s, "GB300", T=np.float32)
    st.set_geometry(*geo)
    st.set_measures(L.MEAS_ALL)
    st.height = np.asfortranarray(2.0 ** 24 * np.random.default_rng(8).uniform(1.0, 1.9, (Lx, Ly)))
    st.velx = np.full((Lx, Ly), 0.02)
    largest = 0.0
    for t in range(1, 6):
        st.step(1)
        if t > 1:
            r = st.measures()[-1]
            assert r.t == t and abs(r.mass - total * 2.0 ** -32) <= 2 * np.spacing(r.mass)
        total, lo = pulled_mass(st.get("fout"))
        largest = max(largest, lo)
    assert largest > 0.5  # the case this test is for
