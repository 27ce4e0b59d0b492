"""The Float64 cell kernels where they can go wrong: block remainders, one-row
and one-column lattices, heights over many binades (the corrected quotients
and their general division), and measures the integer sums split or refuse."""
import math

import numpy as np
import pytest

import oracle
import swalbe_gb300 as sw
from swalbe_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def pair(Lx, Ly, h0, steps, theta=None, **kw):
    s = sw.SysConst(Lx, Ly, sw.Taumucs(Tmax=steps, **kw))
    p = s.param
    P = oracle.params(Lx, Ly, Tmax=steps, tau=p.tau, mu=p.mu, delta=p.delta, gamma=p.gamma, n=p.n, m=p.m,
                      hmin=p.hmin, hcrit=p.hcrit, theta=p.theta, g=p.g)
    st = sw.Sys(s, "GB300")
    if theta is not None:
        st.set_theta(theta)
    st.height = h0
    st.set_measures(L.MEAS_ALL)
    return st, oracle.time_loop_literal(P, h0, steps, theta_field=theta)


@pytest.mark.parametrize("kw", [{}, {"tau": 0.8, "g": 0.001}, {"n": 4, "m": 1}], ids=["plain", "tau_g", "n4m1"])
@pytest.mark.parametrize("Lx,Ly", [(1, 1), (127, 1), (1, 128), (43, 3), (32, 8), (67, 5), (129, 130)])
def test_sizes_equal_oracle(Lx, Ly, kw):
    rng = np.random.default_rng(Lx * 1000 + Ly)
    # three binades, and cells whose film pressure divides exactly
    h0 = np.asfortranarray(np.exp2(rng.uniform(-1, 2, (Lx, Ly))))
    h0[rng.uniform(size=(Lx, Ly)) < 0.2] = 0.15
    theta = np.asfortranarray(rng.uniform(0.05, 0.2, (Lx, Ly))) if kw else None
    st, ref = pair(Lx, Ly, h0, 5, theta, **kw)
    st.step(5)
    st.sync()
    assert np.array_equal(st.height, ref.height)
    assert np.array_equal(st.velx, ref.velx)
    assert np.array_equal(st.vely, ref.vely)
    r = st.measures()[0]
    assert r.wetted == np.count_nonzero(h0 > 0.055)
    assert (r.hmax, r.hmin) == (h0.max(), h0.min())
    # the sum is exact before one rounding of its upper and lower word each
    assert abs(r.mass - math.fsum(h0.ravel())) <= 2 * np.spacing(r.mass)
    assert len(st.measures()) == 0


@pytest.mark.parametrize("exponents", [(-9, 9), (-60, 40), (-300, 300), (-1000, 900)],
                         ids=["narrow", "units", "wide", "ends"])
def test_heights_over_many_binades(exponents):
    """One iteration from heights spread over the exponent range: the quotients
    near the ends of it, and masses beyond the integers' window."""
    Lx, Ly = 61, 11
    rng = np.random.default_rng(7)
    h0 = np.asfortranarray(np.ldexp(rng.uniform(1, 2, (Lx, Ly)), rng.integers(*exponents, (Lx, Ly))))
    with np.errstate(all="ignore"):
        st, ref = pair(Lx, Ly, h0, 1, gamma=1e-300 if exponents[1] > 100 else 0.01)
    st.step(1)
    try:
        st.sync()
    except sw.SwbError:
        pass
    for got, want in ((st.height, ref.height), (st.velx, ref.velx), (st.vely, ref.vely)):
        assert np.array_equal(got, want, equal_nan=True)
    if exponents[1] <= 40:
        r = st.measures()[0]
        # one rounding per height of 2^30 and more, which is summed in Float64
        ulps = 2 + np.count_nonzero(h0 >= 2.0 ** 30)
        assert abs(r.mass - math.fsum(h0.ravel())) <= ulps * np.spacing(r.mass)
        assert (r.hmax, r.hmin) == (h0.max(), h0.min())


def test_velocities_and_zeros():
    """Velocities of either sign, zero and tiny, on flat and stepped films."""
    Lx, Ly = 40, 9
    rng = np.random.default_rng(3)
    u = np.asfortranarray(rng.choice([0.0, -0.0, 1e-3, -2e-3, 1e-200, -1e-310], (Lx, Ly)))
    h0 = np.asfortranarray(np.where(np.arange(Lx)[:, None] < 20, 1.0, 0.5) * np.ones((Lx, Ly)))
    s = sw.SysConst(Lx, Ly, sw.Taumucs())
    lit = oracle.LiteralState(oracle.params(Lx, Ly))
    plain = sw.Sys(s, "GB300-plain")
    st = sw.Sys(s, "GB300")
    for x in (st, plain):
        x.height = h0
        x.velx = u
        x.vely = -u
    lit.field("height")[...] = h0
    lit.field("velx")[...] = u
    lit.field("vely")[...] = -u
    lit.run(4)
    for x in (st, plain):
        x.step(4)
        x.sync()
        assert np.array_equal(x.height, lit.field("height"))
        assert np.array_equal(x.velx, lit.field("velx"))
        assert np.array_equal(x.vely, lit.field("vely"))


@pytest.mark.parametrize("T,device", [(np.float64, "GB300"), (np.float64, "GB300-plain"), (np.float32, "GB300")])
def test_theta_field_equals_scalar_theta(T, device):
    """κ and cos θ of a field's cells are those of the same scalar θ: special
    values, both sides of every reduction, and angles a hair from a right one."""
    rng = np.random.default_rng(5)
    th = [0.0, 0.25, 0.5, 0.75, 1.0, 1.5, 2.0, -0.3, 7.1, 1 / 9, 1e-200, 0.5 - 2.0 ** -54, 0.5 + 2.0 ** -50]
    th += list(rng.uniform(0, 0.5, 60)) + list(rng.uniform(-3, 3, 20)) + list(0.25 + rng.uniform(-1e-9, 1e-9, 7))
    for group in (th[:-12], th[:10] + th[14:]):
        s = sw.SysConst(3, 1, sw.Taumucs())
        one = sw.Sys(s, device, T=T)
        want = []
        for t in group:
            one.set_theta(float(t))
            want.append((probe(one, 3), one.measure_now().energy / 3))
        s = sw.SysConst(len(group), 1, sw.Taumucs())
        st = sw.Sys(s, device, T=T)
        st.set_theta(np.array(group)[:, None])
        got = probe(st, len(group))
        assert np.array_equal(got, [w[0][0] for w in want])


def probe(st, n):
    """The film pressure of a flat film, which is κ times the same factor in every cell."""
    st.height = np.full((n, 1), 0.07)
    if st.precision == L.SWB_PLAIN64:
        sw.api.check(sw.api.lib().swb_op_filmpressure(st.handle))
    return st.pressure[:, 0]


@pytest.mark.parametrize("shape", [(8, 8), (33, 17)])
def test_captured_ops_replay(shape):
    """A graph of one streaming op, replayed three times, equals three calls: the
    ops that follow each other outside a graph may change buffers, a captured one not."""
    torch = pytest.importorskip("torch")
    lx, ly = shape
    c = sw.SysConst(lx, ly, sw.Taumucs(delta=1.0))
    h = 1 + 0.1 * np.random.default_rng(3).uniform(-1, 1, shape)

    def ops(s):
        sw.equilibrium_(s, c)
        sw.BGKandStream_(s, c)
        sw.moments_(s)

    a, b = (sw.Sys(c, "GB300-plain") for _ in range(2))
    for s in (a, b):
        s.height = h
        ops(s)
    st = torch.cuda.Stream()
    b.sync()
    b.set_stream(st.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        ops(b)
    for _ in range(3):
        ops(a)
        with torch.cuda.stream(st):
            g.replay()
    st.synchronize()
    a.sync()
    for f in ("height", "velx", "vely", "fout"):
        assert np.array_equal(a.get(f), b.get(f)), f
    b.set_stream(None)
