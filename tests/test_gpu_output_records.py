"""Models that store the point records of output steps alone (store_ip_data =
0): sequences without such a step take the kernels that store none, and change
neither the state nor the records."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import cube_problem, critical_time_step

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from nimblesm_gb300 import build as B
    B.build()


# one point per lane in FP64; two; several rounds of the grid
@pytest.mark.parametrize("n", [3, 14, 30])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("frequency", [0, 1, 4])
def test_records_are_those_of_the_last_output_step(n, precision, frequency):
    p = cube_problem(n, jitter=0.2, seed=n)
    dt = 0.5 * critical_time_step(p)
    steps = 11
    outputs = [s for s in range(steps) if frequency and (s % frequency == 0 or s == steps - 1)]
    for graph_steps in (3, 50):
        m = E.Model(p, precision=precision, store_ip_data=False, graph_steps=graph_steps)
        full = E.Model(p, precision=precision, graph_steps=graph_steps)
        for model in (m, full):
            model.begin(steps * dt, steps, frequency)
        want = m.GetIntegrationPointData()  # F = I, sigma = 0
        for s in range(0, steps, 2):  # two steps at a time, the records of each output step from the full model
            for k in range(s, min(s + 2, steps)):
                full.advance(1)
                if k in outputs:
                    want = full.GetIntegrationPointData()
            m.advance(min(2, steps - s))
            got = m.GetIntegrationPointData()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (graph_steps, s)
        a, b = m.state(with_ip=False), full.state(with_ip=False)
        for key in a:
            assert np.array_equal(a[key], b[key]), key
        m.close()
        full.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_no_outputs_no_storing_kernels(precision):
    """A schedule without output steps launches the kernels of one whose records
    are overwritten: the same element time, where the storing kernels take 10%
    more (more runs of either on one mesh differ by less than 2%)."""
    p = cube_problem(64, jitter=0.2, seed=1)
    dt = 0.5 * critical_time_step(p)
    times = {}
    for stored in (True, False):
        m = E.Model(p, precision=precision, store_ip_data=stored)
        m.begin(400 * dt, 400, 0)
        m.advance_timed(50)
        times[stored] = min(m.advance_timed(50) for _ in range(6))
        m.close()
    assert times[False] <= 1.03 * times[True], times
