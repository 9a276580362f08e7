"""Elements that the fixed-point kernel of the FP64 form leaves to the FP64
code: displacements that are not numbers."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Material, Problem, cube_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from nimblesm_gb300 import build as B
    B.build()


def block_problem(kind, n=4, seed=7):
    """A jittered cube of one material, or of an elastic and a neo-Hookean block."""
    p = cube_problem(n, jitter=0.2, seed=seed)
    names = {"elastic": ["elastic"], "neohookean": ["neohookean"], "mixed": ["elastic", "neohookean"]}[kind]
    p.blocks = [Material(k, p.density, p.bulk_modulus, p.shear_modulus) for k in names]
    p.elem_block = (np.arange(p.num_elem) * len(names) // p.num_elem).astype(np.int32)
    return p


@pytest.mark.parametrize("kind", ["elastic", "neohookean", "mixed"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1.5e308])
@pytest.mark.parametrize("where", ["one node", "one component", "everything"])
def test_displacements_that_are_not_numbers_are_reported(kind, value, where):
    """Wherever they stand: the same value at all corners cancels in every
    difference (1.5e308: its sums overflow)."""
    p = block_problem(kind)
    u = np.random.default_rng(1).normal(0, 1e-4, p.coords.shape)
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    bad = u.copy()
    if where == "one node":
        bad[p.conn[3][0], 1] = value
    elif where == "one component":
        bad[:, 0] = value
    else:
        bad[:] = value
    with pytest.raises(E.EngineError):
        m.ComputeInternalForceHost(bad)
    assert np.array_equal(m.ComputeInternalForceHost(u), f)  # and the handle still works
    if np.isnan(value) and where == "everything":
        m.begin(1e-6, 4, 0, v_init=bad)
        with pytest.raises(E.EngineError):
            m.advance_timed(4)
    m.close()
