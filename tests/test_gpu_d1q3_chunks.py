"""1D lattices cut into chunks with halos: one CTA with no halo, the first
lengths that need several, and step counts that are no multiple of a launch."""
import math

import numpy as np
import pytest

import oracle
import swalbe_gb300 as sw

pytestmark = pytest.mark.gpu


def ref_of(s, h0):
    p = s.param
    return oracle.State1D(oracle.params(s.L, 1, tau=p.tau, delta=p.delta, gamma=p.gamma, n=p.n, m=p.m,
                                        hmin=p.hmin, hcrit=p.hcrit, theta=p.theta, g=p.g), h0)


def film(L):
    return 1.0 + np.random.default_rng(L).uniform(-0.2, 0.2, L)


@pytest.mark.parametrize("kw", [{}, {"tau": 0.8, "g": 0.002}], ids=["plain", "tau_g"])
@pytest.mark.parametrize("L", [3, 31, 127, 128, 129, 143, 1000, 2401])
def test_lengths_equal_oracle(L, kw):
    s = sw.SysConst_1D(L, sw.Taumucs(**kw))
    th = np.repeat(np.linspace(0.1, 0.2, 7), L)[:L] if kw else None
    gm = 0.01 + 0.001 * np.cos(2 * np.pi * np.arange(L) / L) if kw else None
    st = sw.Sys(s, T=np.float64)
    st.height = film(L)
    st.set_theta(th)
    st.set_gamma(gm)
    ref = ref_of(s, film(L))
    heights = []
    for n in (1, 7, 45):
        heights.append(st.height)
        st.step(n)
        ref.run(n, theta_field=th, gamma_field=gm)
    st.sync()
    assert np.array_equal(st.height, ref.h)
    assert np.array_equal(st.vel, ref.u)
    assert np.array_equal(st.fout, ref.fout)
    r = st.measures()
    assert [x.t for x in r] == list(range(1, 54))
    for k, h in zip((0, 1, 8), heights):  # the records of the heights each call started from
        assert (r[k].hmax, r[k].hmin, r[k].wetted) == (h.max(), h.min(), np.count_nonzero(h > 0.055))
        assert abs(r[k].mass - math.fsum(h)) <= 2 * np.spacing(r[k].mass)


@pytest.mark.parametrize("count", [3, 200])
def test_mixed_batch_equals_single(count):
    """Short and long lattices in one batch (and enough of them for short launches)."""
    Ls = [(40, 128, 700)[i % 3] for i in range(count)]
    systems = [sw.SysConst_1D(L, sw.Taumucs(tau=1.0 if i % 2 else 0.9)) for i, L in enumerate(Ls)]
    for T in (np.float64, np.float32):
        b = sw.Batch1D(systems, T=T, records=16)
        for i, L in enumerate(Ls):
            b.set_height(i, film(L))
        b.step(33)
        b.sync()
        for i in (0, 1, 2, count - 1):
            one = sw.Sys(systems[i], T=T)
            one.height = film(Ls[i])
            one.step(33)
            one.sync()
            assert np.array_equal(b.height(i), one.height)
            assert np.array_equal(b.fout(i), one.fout)
            assert [(x.t, x.mass, x.hmax) for x in b.measures(i)] == \
                   [(x.t, x.mass, x.hmax) for x in one.measures()[-16:]]
