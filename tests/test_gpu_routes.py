"""Calls in orders and shapes that take another route through the host runtime
or the dispatch than the plain run of one case."""
import numpy as np
import pytest

import sddc_oracle as O
from helpers import case_channel, case_cylinder, case_periodic, rel_l2
from sddc_b200 import cases, ensemble, host, mesh
from sddc_b200.solver import NumericalFault, Solver

pytestmark = pytest.mark.gpu


def _records(ncell, n, ph, dt):
    edges = np.linspace(0, ncell, n + 1).astype(int)
    return [dict(first_cell=int(a), ncell=int(b - a), dt=dt, rinf=ph.rinf, pinf=ph.pinf, uinf=ph.uinf, vinf=ph.vinf,
                 bxinf=ph.bxinf, byinf=ph.byinf) for a, b in zip(edges[:-1], edges[1:])]


def test_sensor_of_a_batch_set_after_a_smaller_one():
    m, t, ph, Q = case_periodic(6, 3)
    dt = 0.1 * m.min_edge() / 3

    def sensor(s, n):
        s.set_cases(_records(t.ncell, n, ph, dt))
        s.set_state(Q)
        s.step_cases(2)
        return s.state(sm_ind=True)["sm_ind"]

    s = Solver(t, ph, precision="fp64")
    got = [sensor(s, n) for n in (2, 40, 3)]
    s.close()
    for n, g in zip((2, 40, 3), got):
        s = Solver(t, ph, precision="fp64")
        assert np.array_equal(sensor(s, n), g, equal_nan=True), n
        s.close()
