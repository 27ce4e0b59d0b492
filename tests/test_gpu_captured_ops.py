"""Graphs of per-op calls mixed with calls outside them: a replay always uses
the populations that the last call or replay left."""
import numpy as np
import pytest

import swalbe_gb300 as sw

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def pair(tau, shape=(33, 17)):
    c = sw.SysConst(*shape, sw.Taumucs(delta=1.0, tau=tau))
    rng = np.random.default_rng(3)
    h = 1 + 0.1 * rng.uniform(-1, 1, shape)
    ux, uy = rng.uniform(-0.05, 0.05, (2,) + shape)
    out = []
    for _ in range(2):
        s = sw.Sys(c, "GB300-plain")
        s.height, s.velx, s.vely = h, ux, uy
        out.append(s)
    return c, *out


def stream_of(s):
    st = torch.cuda.Stream()
    s.sync()
    s.set_stream(st.cuda_stream)
    return st


def capture(s, st, ops):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        ops(s)
    return g


def replay(g, st):
    with torch.cuda.stream(st):
        g.replay()


def check(a, b, st):
    st.synchronize()
    a.sync()
    for f in ("height", "velx", "vely", "fout"):
        assert np.array_equal(a.get(f), b.get(f)), f
    b.set_stream(None)


@pytest.mark.parametrize("tau", [0.8, 1.0])
@pytest.mark.parametrize("before", [0, 1, 2])
def test_calls_between_replays(tau, before):
    c, a, b = pair(tau)

    def ops(s):
        sw.equilibrium_(s, c)
        sw.BGKandStream_(s, c)
        sw.moments_(s)

    st = stream_of(b)
    for s in (a, b):
        for _ in range(before):
            ops(s)
    g = capture(b, st, ops)
    for plain in (1, 0, 2, 3):  # calls outside the graph between its replays
        ops(a)
        replay(g, st)
        for s in (a, b):
            for _ in range(plain):
                ops(s)
    check(a, b, st)


def test_a_captured_moments_alone():
    c, a, b = pair(0.8)
    st = stream_of(b)
    g = capture(b, st, sw.moments_)
    for k in range(3):
        for s in (a, b):
            sw.equilibrium_(s, c)
            sw.BGKandStream_(s, c)
        sw.moments_(a)
        replay(g, st)
    check(a, b, st)


def test_captured_steps_and_calls():
    c, a, b = pair(0.9)
    st = stream_of(b)
    for s in (a, b):
        s.step(1)
    g = capture(b, st, lambda s: s.step(1))
    for k in range(4):
        a.step(1)
        replay(g, st)
        for s in (a, b):
            s.step(k)
    check(a, b, st)
