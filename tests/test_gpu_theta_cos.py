"""cos θ of every cell of a θ field, as the energy of a film that wets only that
cell: it is that of a state with the cell's θ as a scalar."""
import numpy as np
import pytest

import swalbe_gb300 as sw

pytestmark = pytest.mark.gpu

THETAS = [0.0, 0.25, 0.5, 0.75, 1.0, 1.5, 2.0, -0.3, 7.1, 1 / 9, 1e-200, 0.5 - 2.0 ** -54, 0.5 + 2.0 ** -50, 0.1, 0.9]


@pytest.mark.parametrize("T,device", [(np.float64, "GB300"), (np.float64, "GB300-plain"), (np.float32, "GB300")])
@pytest.mark.parametrize("shape", [(5, 3), (16, 9)])
def test_the_energy_of_one_wetted_cell(T, device, shape):
    n = shape[0] * shape[1]
    th = np.array((THETAS + list(np.random.default_rng(5).uniform(-1, 1, n)))[:n]).reshape(shape, order="F")
    c = sw.SysConst(*shape, sw.Taumucs())
    field, scalar = (sw.Sys(c, device, T=T) for _ in range(2))
    field.set_theta(th)
    for i in np.ndindex(shape):
        h = np.full(shape, 0.01)
        h[i] = 1.0
        field.height = scalar.height = h
        scalar.set_theta(float(th[i]))
        got, want = field.measure_now(), scalar.measure_now()
        assert got.wetted == want.wetted == 1 and got.area == want.area
        # cos θ of an FP32 field is rounded to FP32, half a unit of at most 2^-24;
        # the two energies then have an area below 2 and are rounded once each
        assert abs(got.energy - want.energy) <= (0.0 if T == np.float64 else 2.0 ** -25 + 2.0 ** -51), i
