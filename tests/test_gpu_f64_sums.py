"""Masses of Float64 records over the whole exponent range: the correctly
rounded sum of the heights, whatever their size, sign and order."""
import ctypes as C
import math

import numpy as np
import pytest

import swalbe_gb300 as sw
from swalbe_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def film(shape, exponents, seed, signs=False):
    rng = np.random.default_rng(seed)
    h = np.ldexp(rng.uniform(1, 2, shape), rng.integers(*exponents, shape))
    return np.asfortranarray(h * rng.choice([-1.0, 1.0], shape) if signs else h)


def masses(h0):
    """Masses recorded of h0, once from either parity."""
    Lx, Ly = h0.shape
    out = []
    for before in (0, 1):
        st = sw.Sys(sw.SysConst(Lx, Ly, sw.Taumucs()), "GB300")
        st.set_measures(L.MEAS_ALL)
        st.height = np.ones((Lx, Ly))
        st.step(before)
        st.sync()
        st.height = h0
        st.step(1)
        st.height = np.ones((Lx, Ly))  # so that no height is left that is not finite
        out.append(st)
    return out


def record(st):
    """The newest record, also of a state whose heights are not finite any more."""
    m = (L.Measure * 4)()
    n = C.c_int64()
    L.lib().swb_get_measures(st.handle, m, 4, C.byref(n))
    return m[n.value - 1]


@pytest.mark.parametrize("signs", [False, True], ids=["positive", "signed"])
@pytest.mark.parametrize("exponents", [(-3, 3), (-46, -40), (-60, -44), (-80, 40), (29, 34), (-1074, -1000),
                                       (-1074, 1000), (1000, 1010)], ids=str)
def test_mass_is_the_rounded_sum(exponents, signs):
    for shape in ((61, 11), (1, 1), (300, 7)):
        h0 = film(shape, exponents, shape[0], signs)
        for st in masses(h0):
            assert record(st).mass == math.fsum(h0.ravel()), shape


@pytest.mark.parametrize("odd,want", [((math.inf,), math.inf), ((-math.inf,), -math.inf), ((math.nan,), math.nan),
                                      ((math.inf, -math.inf), math.nan), ((1.7e308,) * 3, math.inf)], ids=str)
def test_mass_that_is_not_finite(odd, want):
    h0 = film((61, 11), (-60, 40), 5)
    h0[3:3 + len(odd), 4] = odd
    for st in masses(h0):
        got = record(st).mass
        assert got == want or (math.isnan(got) and math.isnan(want))


@pytest.mark.parametrize("exponents", [(-60, -58), (-80, -44), (-200, -190), (31, 40)], ids=str)
def test_1d_mass(exponents):
    n = 1000
    h0 = film((n,), exponents, 2)
    st = sw.Sys(sw.SysConst_1D(n, sw.Taumucs()), T=np.float64)
    st.height = h0
    st.step(1)
    m = st.measures()[0].mass
    # at worst a plain Float64 sum of what the integers do not hold
    assert abs(m - math.fsum(h0)) <= n * 2.0 ** -53 * math.fsum(h0)
