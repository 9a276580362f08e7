"""The FP32 forms' two layouts of element forces: planes over elements where
consecutive nodes lie in consecutive elements, records at the node's place in a
mesh without such an order.  A node's contributions are summed in element order
either way, so a renumbering of the nodes moves the forces and changes no bit."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Problem
from tests.gpu_util import rel

pytestmark = pytest.mark.gpu

K, G = 160e9, 79.3e9


@pytest.fixture(scope="module", autouse=True)
def _built():
    from nimblesm_gb300 import build as B
    B.build()


def fan(m, layers, shuffled):
    """Five m x m sectors of parallelograms around an axis, extruded: interior
    axis nodes have ten elements, two more than the slots of a node.  Elements
    in the same order either way, nodes in the order of their first element or
    shuffled."""
    edge = [np.array([np.cos(2 * np.pi * s / 5), np.sin(2 * np.pi * s / 5), 0.0]) for s in range(6)]
    corners = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    k, s, j, i = (q.ravel() for q in np.meshgrid(np.arange(layers), np.arange(5), np.arange(m), np.arange(m), indexing="ij"))
    e0, e1 = np.array(edge)[s], np.array(edge)[s + 1]
    pts = np.stack([((i + a)[:, None] * e0 + (j + b)[:, None] * e1 + (k + c)[:, None] * [0.0, 0.0, 1.0]) / m
                    for a, b, c in corners], axis=1)
    _, first, ids = np.unique(np.round(pts.reshape(-1, 3), 9), axis=0, return_index=True, return_inverse=True)
    to = np.empty(len(first), int)
    to[np.argsort(first)] = np.arange(len(first))  # in the order of first use
    coords = pts.reshape(-1, 3)[np.sort(first)]
    conn = to[ids.reshape(-1, 8)].astype(np.int32)
    perm = np.random.default_rng(m).permutation(len(coords)) if shuffled else np.arange(len(coords))
    moved = np.empty_like(coords)
    moved[perm] = coords
    problem = Problem(coords=moved, conn=perm[conn].astype(np.int32), node_sets={}, density=7800.0, bulk_modulus=K,
                      shear_modulus=G, bcs=[], v_init=np.zeros_like(coords))
    return problem, perm


# nodes on both sides of the node kernel's choice between a thread per node and
# component and a thread per node (51,882 nodes); a last warp and block in part
@pytest.mark.parametrize("m,layers", [(5, 7), (20, 31)])
@pytest.mark.parametrize("closure", [False, True])
def test_renumbering_the_nodes_moves_the_forces(m, layers, closure):
    net = E.MLPClosure(K, G, seed=3) if closure else None
    if net is not None:
        net.generate(1 << 14)
    f, u = {}, None
    for shuffled in (False, True):
        p, perm = fan(m, layers, shuffled)
        assert np.bincount(p.conn.ravel()).max() == 10
        if u is None:
            u = np.random.default_rng(8).normal(0, 2e-3 / m, size=p.coords.shape)
        up = np.empty_like(u)
        up[perm] = u
        for precision in ("fp32", "fp64") if not (shuffled or closure) else ("fp32",):
            model = E.Model(p, precision=precision)
            if net is not None:
                model.set_closure(net)
            model.SetVectorNodeData("displacement", up)
            model.ComputeInternalForce()
            f[precision, shuffled] = model.GetVectorNodeData("internal_force")[perm]
            model.close()
    assert np.abs(f["fp32", False]).max() > 0.0
    assert np.array_equal(f["fp32", True], f["fp32", False])
    if not closure:
        # single-precision rounding (6e-8 relative, a few dozen operations) of
        # F and of stresses that are differences of terms 1 / 2e-3 times larger
        assert rel(f["fp32", True], f["fp64", False]) < 1e-3
