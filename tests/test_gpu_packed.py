"""The FP32 form's steps inside an advance evaluate two integration points per
operation where all materials are neo-Hookean; the last step of an advance, and
models with an elastic block, one.  The bits are the same: an advance of three
steps equals three of one."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Material, cube_problem, critical_time_step, uq_ensemble

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from nimblesm_gb300 import build as B
    B.build()


def problems(kind):
    if kind == "ensemble":  # moduli per sample, 5 samples of uneven size
        return uq_ensemble(num_samples=5, n_min=2, n_max=6, seed=3)
    n = {"one": 1, "partial warp": 3, "whole warps": 8, "several rounds": 41}[kind]
    return cube_problem(n, jitter=0.2 if n > 1 else 0.0, seed=n)


@pytest.mark.parametrize("kind", ["one", "partial warp", "whole warps", "several rounds", "ensemble"])
@pytest.mark.parametrize("elastic", [False, True])
def test_steps_inside_an_advance_equal_steps_alone(kind, elastic):
    p = problems(kind)
    if elastic:
        if kind in ("one", "ensemble"):
            pytest.skip("two blocks of one mesh")
        p.blocks = [Material("neohookean", p.density, p.bulk_modulus, p.shear_modulus), Material("elastic", 7800.0, 140e9, 60e9)]
        p.elem_block = (np.arange(p.num_elem) >= p.num_elem // 2).astype(np.int32)
    states = []
    for parts in ((3,), (1, 1, 1)):
        m = E.Model(p, precision="fp32")
        if kind == "ensemble":
            m.begin([3 * 0.4 * d for d in m.sample_time_steps()], 3, 0)
        else:
            m.begin(3 * 0.4 * critical_time_step(p), 3, 0)
        for k in parts:
            m.advance(k)
        states.append(m.state())
        m.close()
    assert np.abs(states[0]["f_int"]).max() > 0.0
    for key in states[0]:
        assert np.array_equal(states[0][key], states[1][key]), key
