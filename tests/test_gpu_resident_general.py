"""Resident tiles with θ fields (at rest and moving), the θ wave, an
inclination and thermal noise against the general strips: full and partial
tiles, a lattice narrower than a tile, and runs of more than one launch."""
import numpy as np
import pytest

import swalbe_gb300 as sw
from swalbe_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def run(Lx, Ly, steps, T, geo, what):
    kbt = 1e-7 if "thermal" in what else 0.0
    s = sw.SysConst(Lx, Ly, sw.Taumucs(delta=2.0, kbt=kbt))
    st = sw.Sys(s, "GB300", T=T, kind="thermal" if kbt else "simple")
    rng = np.random.default_rng(Lx + Ly)
    if "field" in what:
        st.set_theta(np.asfortranarray(rng.uniform(0.05, 0.2, (Lx, Ly))))
        if "moving" in what:
            st.move_substrate(7, "diagonal")
    elif "wave" in what:
        st.set_theta_wave(1 / 9, 1 / 36, 1 / 98)
    if "incl" in what:
        st.set_inclination((2e-4, -1e-4), loop_time=True, tstart=20, tsmooth=10)
    st.set_geometry(*geo)
    st.set_measures(L.MEAS_ALL)
    st.height = np.asfortranarray(1.0 + 0.1 * rng.uniform(-1, 1, (Lx, Ly)))
    for n in (1, steps // 3, steps - 1 - steps // 3):
        st.step(n)
    st.sync()
    return st, st.height, st.measures_array(cap=steps)


@pytest.mark.parametrize("T", [np.float32, np.float16])
@pytest.mark.parametrize("what", [("incl",), ("field",), ("field", "moving", "incl"), ("wave",),
                                  ("thermal",), ("wave", "thermal", "incl")], ids="+".join)
def test_general_resident_equals_strips(what, T):
    for Lx, Ly, steps in [(130, 34, 90), (48, 40, 1300), (256, 131, 60)]:
        _, h_ref, r_ref = run(Lx, Ly, steps, T, (64, 8), what)
        for geo in (33, 34):
            st, h, r = run(Lx, Ly, steps, T, (geo, 0), what)
            assert st.geometry()[0] == geo and st.step_mode() == "multi"
            assert np.array_equal(h, h_ref), (Lx, Ly, geo)
            for f in ("t", "mass", "wetted", "hmax", "hmin", "area", "energy"):
                assert np.array_equal(r[f], r_ref[f]), (Lx, Ly, geo, f)
