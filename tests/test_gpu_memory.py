"""FP64 models without fixed-point geometry: the device has no room for it, or
(nearly) no element is inside the domain.  The same mesh runs, its elements
evaluated by the FP64 code."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.0, 0.5, 0.95, 1.0])
def test_meshes_out_of_the_domain_keep_no_fixed_geometry(share):
    """A share of the elements is elastic of a low shear modulus (K = 20 G), which
    fixed point does not take: from nine tenths on, the model is as large as an
    FP64 one without it, and the forces are the ones that the FP64 code gives
    those elements beside others."""
    torch = pytest.importorskip("torch")
    from nimblesm_gb300 import build as B
    B.build()
    torch.zeros(1, device="cuda")
    p = cube_problem(40, jitter=0.2, seed=4)
    E.Model(p).close()

    def size():
        free0 = torch.cuda.mem_get_info()[0]
        m = E.Model(p)
        return m, free0 - torch.cuda.mem_get_info()[0]

    m, whole = size()  # neo-Hookean, all of it inside
    m.close()
    p.blocks = [Material("elastic", p.density, 20 * p.shear_modulus, p.shear_modulus),
                Material("neohookean", p.density, p.bulk_modulus, p.shear_modulus)]
    p.elem_block = (np.arange(p.num_elem) >= share * p.num_elem).astype(np.int32)
    if share == 0.0 or share == 1.0:
        p.blocks, p.elem_block = [p.blocks[int(share == 0.0)]], np.zeros(p.num_elem, np.int32)
    u = np.random.default_rng(1).normal(0, 1e-3 / 40, p.coords.shape)
    m, used = size()
    assert (used < whole - 673 * p.num_elem // 2) == (share >= 0.9), (used, whole)
    f = m.ComputeInternalForceHost(u)
    m.close()
    if share == 1.0:  # the same elements beside enough others that there is fixed geometry
        extra = cube_problem(40, jitter=0.2, seed=5)
        extra.v_init = None
        q = cube_problem(40, jitter=0.2, seed=4)
        q.coords = np.concatenate([q.coords, extra.coords + 2.0])
        q.conn = np.concatenate([q.conn, extra.conn + p.num_nodes])
        q.blocks = [p.blocks[0], Material("neohookean", p.density, p.bulk_modulus, p.shear_modulus)]
        q.elem_block = (np.arange(2 * p.num_elem) >= p.num_elem).astype(np.int32)
        q.bcs, q.v_init = [], None
        both = E.Model(q)
        assert np.array_equal(both.ComputeInternalForceHost(np.concatenate([u, u]))[: p.num_nodes], f)
        both.close()
