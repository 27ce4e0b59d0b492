"""2D Float64 at the ends of its range against the oracle, by the cell kernels
and op by op: heights that are not finite (and a state set again after them),
heights over the whole exponent range, the smallest velocities."""
import numpy as np
import pytest

import oracle
import swalbe_gb300 as sw

pytestmark = pytest.mark.gpu
SHAPE = (37, 9)


class Run:
    def __init__(self, kw):
        s = sw.SysConst(*SHAPE, sw.Taumucs(**kw))
        p = s.param
        self.ref = oracle.LiteralState(oracle.params(*SHAPE, tau=p.tau, delta=p.delta, gamma=p.gamma, n=p.n, m=p.m,
                                                     hmin=p.hmin, hcrit=p.hcrit, theta=p.theta, g=p.g, mu=p.mu))
        self.states = [sw.Sys(s, d) for d in ("GB300", "GB300-plain")]

    def set(self, h, ux, uy):
        for f, v in (("height", h), ("velx", ux), ("vely", uy)):
            self.ref.field(f)[...] = v
            for st in self.states:
                setattr(st, f, np.asfortranarray(v))

    def step(self, n):
        self.ref.run(n)
        for st in self.states:
            st.step(n)
            try:
                st.sync()
            except sw.SwbError:
                pass
            for f in ("height", "velx", "vely", "fout"):
                assert np.array_equal(st.get(f), self.ref.field(f), equal_nan=True), (st.precision, f)


KINDS = pytest.mark.parametrize("kw", [{}, {"g": 0.002}, {"tau": 0.8}, {"tau": 0.8, "g": 0.002}, {"delta": 1e150}], ids=str)


@KINDS
@pytest.mark.parametrize("odd", [np.inf, -np.inf, np.nan])
def test_heights_that_are_not_finite(kw, odd):
    r = Run(kw)
    rng = np.random.default_rng(1)
    h, ux, uy = rng.uniform(0.5, 2, SHAPE), rng.uniform(-0.1, 0.1, SHAPE), rng.uniform(-0.1, 0.1, SHAPE)
    ux[:, 3] = uy[:, 3] = 0.0
    h[[3, 20, 36], [0, 3, 8]] = odd
    r.set(h, ux, uy)
    r.step(1)
    r.step(2)
    h[[3, 20, 36], [0, 3, 8]] = 1.0
    r.set(h, ux, uy)
    r.step(1)
    r.step(1)


@KINDS
@pytest.mark.parametrize("exponents", [(-9, 9), (-60, 40), (-300, 300), (500, 520), (-1074, -1000), (-1074, 1023), (990, 1023)], ids=str)
def test_the_whole_exponent_range(kw, exponents):
    for gamma in (0.01, 1e-300):
        r = Run(dict(kw, gamma=gamma))
        rng = np.random.default_rng(5)
        h = np.ldexp(rng.uniform(1, 2, SHAPE), rng.integers(*exponents, SHAPE))
        ux, uy = np.ldexp(rng.uniform(-1, 1, (2,) + SHAPE), rng.integers(-1074, 0, (2,) + SHAPE))
        r.set(h, ux, uy)
        for _ in range(3):
            r.step(1)


@KINDS
def test_the_smallest_velocities(kw):
    for g in (kw.get("g", 0.0), 3e-308, 2e-323):
        r = Run(dict(kw, g=g, gamma=1e-320))
        rng = np.random.default_rng(6)
        ux, uy = rng.integers(-9, 10, (2,) + SHAPE) * 2.0 ** -1074
        r.set(rng.uniform(0.5, 2, SHAPE), ux, uy)
        for n in (1, 1, 1, 5, 40):
            r.step(n)
