"""The host-buffer force call on pinned arrays (read and written by the
kernels), pageable ones (through the staging array) and parts of one pinned
allocation: the same bits, whole and in chunks."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import cube_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from nimblesm_gb300 import build as B
    B.build()


@pytest.mark.parametrize("n", [1, 9, 38])  # 8 nodes; one component per thread; past it (59,319 nodes)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_every_kind_of_host_array_gives_the_same_bits(n, precision):
    p = cube_problem(n, jitter=0.2 if n > 1 else 0.0, seed=n)
    u = np.random.default_rng(n).normal(0, 1e-3 / n, size=p.coords.shape)
    m = E.Model(p, precision=precision)
    m.SetVectorNodeData("displacement", u)
    m.ComputeInternalForce()
    want = m.GetVectorNodeData("internal_force")
    assert np.abs(want).max() > 0.0
    pins = E.PinnedArray((2 * p.num_nodes + 1, 3))  # u and f in one allocation, f at an odd multiple of 8 bytes
    parts = {"pageable": (u, np.empty_like(u)),
             "pinned": (pins.array[: p.num_nodes], pins.array[p.num_nodes + 1 :])}
    parts["pinned"][0][:] = u
    for chunks in (1, min(3, p.num_elem)):
        m.set_host_chunks(chunks)
        for u_kind in parts:
            for f_kind in parts:
                f = parts[f_kind][1]
                f[:] = np.nan
                m.ComputeInternalForceHost(parts[u_kind][0], out=f)
                assert np.array_equal(f, want), (chunks, u_kind, f_kind)
                assert np.array_equal(m.GetVectorNodeData("internal_force"), want)
    m.close()
