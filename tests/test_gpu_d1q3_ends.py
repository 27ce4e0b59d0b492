"""1D Float64 at the ends of its range against the oracle: heights that are not
finite (and a state set again after them), heights over the whole exponent
range, velocities and forces down to the smallest numbers.  L = 1000 runs CTAs
of 64 cells, the batch of 200 lattices CTAs of 128."""
import numpy as np
import pytest

import oracle
import swalbe_gb300 as sw

pytestmark = pytest.mark.gpu


class Run:
    """A lattice of L cells on the GPU, alone or as one of 200, beside its oracle."""

    def __init__(self, L, kw):
        s = sw.SysConst_1D(L, sw.Taumucs(**kw))
        p = s.param
        self.ref = oracle.State1D(oracle.params(L, 1, tau=p.tau, delta=p.delta, gamma=p.gamma, n=p.n, m=p.m,
                                                hmin=p.hmin, hcrit=p.hcrit, theta=p.theta, g=p.g))
        self.b = sw.Batch1D([s] * (1 if L > 128 else 200))
        self.i = len(self.b.systems) - 1

    def set(self, h, u):
        self.b.set_height(self.i, h)
        self.b.set_vel(self.i, u)
        self.ref.h[...], self.ref.u[...] = h, u

    def step(self, n):
        self.b.step(n)
        with np.errstate(all="ignore"):
            self.ref.run(n)
        try:
            self.b.sync()
        except sw.SwbError:
            pass
        for got, want in ((self.b.height(self.i), self.ref.h), (self.b.vel(self.i), self.ref.u),
                          (self.b.fout(self.i), self.ref.fout)):
            assert np.array_equal(got, want, equal_nan=True)


LENGTHS = pytest.mark.parametrize("L", [100, 1000])
KINDS = pytest.mark.parametrize("kw", [{}, {"g": 0.002}, {"tau": 0.8}, {"tau": 0.8, "g": 0.002}], ids=str)


@LENGTHS
@KINDS
@pytest.mark.parametrize("odd", [np.inf, -np.inf, np.nan])
def test_heights_that_are_not_finite(L, kw, odd):
    r = Run(L, kw)
    rng = np.random.default_rng(1)
    h, u = rng.uniform(0.5, 2, L), rng.uniform(-0.1, 0.1, L)
    u[20:23] = 0.0
    h[[7, 21, L - 1]] = odd
    r.set(h, u)
    r.step(1)
    r.step(2)
    h[[7, 21, L - 1]] = 1.0
    r.set(h, u)  # the populations are still what the first steps left
    r.step(1)
    r.step(1)


@LENGTHS
@KINDS
@pytest.mark.parametrize("exponents", [(-9, 9), (-60, 40), (-300, 300), (-1074, -1000), (-1074, 1023), (990, 1023)], ids=str)
def test_the_whole_exponent_range(L, kw, exponents):
    for gamma in (0.01, 1e-300):
        r = Run(L, dict(kw, gamma=gamma))
        rng = np.random.default_rng(L)
        h = np.ldexp(rng.uniform(1, 2, L), rng.integers(*exponents, L))
        u = np.ldexp(rng.uniform(-1, 1, L), rng.integers(-1074, 0, L))
        r.set(h, u)
        for _ in range(3):
            r.step(1)


@LENGTHS
@KINDS
def test_the_smallest_velocities(L, kw):
    """Films that come to rest: velocities and forces of a few units of 2^-1074."""
    for g in (kw.get("g", 0.0), 3e-308, 2e-323):
        r = Run(L, dict(kw, g=g, gamma=1e-320))
        rng = np.random.default_rng(L)
        r.set(rng.uniform(0.5, 2, L), rng.integers(-9, 10, L) * 2.0 ** -1074)
        for n in (1, 1, 1, 5, 40):
            r.step(n)
