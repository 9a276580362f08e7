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


def strip(n, seed):
    """n jittered elements in a row along x, and the columns of nodes between them."""
    rng = np.random.default_rng(seed)
    h = 1.0 / n
    k, j, i = np.meshgrid([0, 1], [0, 1], np.arange(n + 1), indexing="ij")
    coords = np.stack([i.ravel(), j.ravel(), k.ravel()], 1) * h
    coords += rng.uniform(-0.1, 0.1, coords.shape) * h
    a = np.arange(n)
    conn = np.stack([a, a + 1, a + n + 2, a + n + 1], 1)
    return Problem(coords=coords, conn=np.concatenate([conn, conn + 2 * (n + 1)], 1).astype(np.int32)), h


@pytest.mark.parametrize("n", [1, 16, 33, 2432, 2433, 20_001])  # 19,424 elements: one round of the grid
@pytest.mark.parametrize("left", ["none", "the last", "one in 40", "a stretch", "all"])
def test_elements_outside_the_domain_beside_others(n, left):
    """The FP64 code evaluates those a block has left 32 at a time, whichever
    they are: the forces are the oracle's (2^-53 of |X| / h over the strain: 1e-9
    at the largest n), the same bits from every launch shape and range, and the
    states of two steps in one sequence those of two sequences, whose last
    steps store records.  One column of nodes moved up by 0.8 h shears the
    elements on both sides of it beyond the domain."""
    from oracle import oracle as O
    O.build(ref=False)
    p, h = strip(n, 3 + n)
    rng = np.random.default_rng(n)
    u = rng.normal(0, 1e-3 * h, p.coords.shape)
    columns = {"none": [], "the last": [n], "one in 40": np.arange(0, n + 1, 80), "a stretch": np.arange(n // 3, n // 2 + 1, 2),
               "all": np.arange(0, n + 1, 2)}[left]
    up = np.zeros(n + 1)
    up[columns] = 0.8 * h
    u[:, 1] += np.tile(up, 4)
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    want = np.zeros_like(u)
    for e in range(n):
        np.add.at(want, p.conn[e], np.asarray(O.element(p.coords[p.conn[e]], u[p.conn[e]], p.bulk_modulus, p.shear_modulus)[2]).reshape(8, 3))
    assert np.linalg.norm(f - want) <= 1e-9 * np.linalg.norm(want)
    F, s = m.GetIntegrationPointData()
    if n > 5:
        m.set_host_chunks(5)
        assert np.array_equal(m.ComputeInternalForceHost(u), f)
        F1, s1 = m.GetIntegrationPointData()
        assert np.array_equal(F, F1) and np.array_equal(s, s1)
        m.set_host_chunks(0)
    dt = 0.1 * h * np.sqrt(p.density / p.bulk_modulus)
    states = []
    for shape in (None, 0, 1, 2, 5):
        for parts in ((2,), (1, 1)):
            if shape is not None:
                m.set_launch_candidate(shape)
            m.begin(2 * dt, 2, 0, v_init=u / dt)
            for k in parts:
                m.advance(k)
            states.append(m.state())
    m.close()
    for key in states[0]:
        for state in states[1:]:
            assert np.array_equal(states[0][key], state[key]), key
