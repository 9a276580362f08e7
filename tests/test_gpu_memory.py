"""An FP64 model where the device has no room for its fixed-point geometry: the
same mesh runs, its elements evaluated by the FP64 code."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Material, cube_problem, critical_time_step


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 2])
def test_a_model_without_room_for_the_fixed_geometry(blocks):
    """Errors of either form against the other: 2^-53 over the strain (1e-3) and
    a few hundred steps of rounding, 1e-11."""
    torch = pytest.importorskip("torch")
    from nimblesm_gb300 import build as B
    B.build()
    p = cube_problem(64, jitter=0.2, seed=4)
    if blocks == 2:
        p.blocks = [Material(k, p.density, p.bulk_modulus, p.shear_modulus) for k in ("elastic", "neohookean")]
        p.elem_block = (np.arange(p.num_elem) >= p.num_elem // 2).astype(np.int32)
    u = np.random.default_rng(1).normal(0, 1e-3 / 64, p.coords.shape)
    dt = 0.5 * critical_time_step(p)

    def run(m):
        out = {"f": m.ComputeInternalForceHost(u)}
        m.begin(8 * dt, 8, 0)
        m.advance(8)
        out.update(m.state())
        out["volume"], out["stress"], out["H"] = m.ComputeDerivedElementData()
        return out

    torch.zeros(1, device="cuda")
    warm = E.Model(p)
    warm.close()
    free0 = torch.cuda.mem_get_info()[0]
    m = E.Model(p)
    used = free0 - torch.cuda.mem_get_info()[0]
    want = run(m)
    m.close()
    fixed, later = 673 * p.num_elem, 576 * p.num_elem + 24 * p.num_nodes
    assert used > fixed
    free0 = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free0 - (used - fixed) - later - fixed // 2, dtype=torch.uint8, device="cuda")
    try:
        left = torch.cuda.mem_get_info()[0]
        m = E.Model(p)
        assert left - torch.cuda.mem_get_info()[0] < used - fixed // 2
        got = run(m)
        m.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    for key in want:
        a, b = np.asarray(got[key], float), np.asarray(want[key], float)
        assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b), key
