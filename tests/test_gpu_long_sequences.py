"""Launch sequences of more steps than a grid has rows, with few driven nodes:
the values of their expressions are evaluated in several launches."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import BoundaryCondition, cube_problem, critical_time_step


@pytest.mark.gpu
def test_more_steps_in_a_sequence_than_rows_in_a_grid():
    """One driven node, a sequence of 66,000 steps, against sequences of 50:
    bitwise the same state."""
    from nimblesm_gb300 import build as B
    B.build()
    p = cube_problem(1)
    p.node_sets["driven"] = np.array([7], np.int32)
    p.bcs.append(BoundaryCondition.parse('prescribed_velocity driven x "0.01 * sin(2e4 * t)"'))
    steps, dt = 66_000, 0.1 * critical_time_step(p)
    states = []
    for graph_steps in (steps, 50):
        m = E.Model(p, graph_steps=graph_steps)
        m.begin(steps * dt, steps, 0)
        m.advance(steps)
        states.append(m.state())
        m.close()
    assert np.abs(states[0]["u"]).max() > 0.0
    for key in states[0]:
        assert np.array_equal(states[0][key], states[1][key]), key
