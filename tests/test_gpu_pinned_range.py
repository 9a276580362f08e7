"""Host arrays that are pinned at both ends and not between: no kernel addresses
them, and the copy that the force call makes instead refuses them."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import cube_problem


@pytest.mark.gpu
def test_arrays_pinned_at_both_ends_only():
    torch = pytest.importorskip("torch")
    from nimblesm_gb300 import build as B
    B.build()
    rt = torch.cuda.cudart()
    p = cube_problem(30, jitter=0.2, seed=2)  # 29,791 nodes: 715 KB, past the largest page by far
    u = np.random.default_rng(1).normal(0, 1e-5, p.coords.shape)
    m = E.Model(p)
    want = m.ComputeInternalForceHost(u).copy()
    page, bytes_ = 65536, u.nbytes
    raw = np.zeros(2 * (bytes_ + 4 * page), np.uint8)
    first = -raw.ctypes.data % page
    half = (bytes_ // page + 2) * page
    arrays = []
    registered = []
    for k in range(2):
        a = raw[first + k * half : first + k * half + bytes_].view(np.float64).reshape(u.shape)
        arrays.append(a)
        for lo in (0, bytes_ // page * page):
            at = raw.ctypes.data + first + k * half + lo
            assert int(rt.cudaHostRegister(at, page, 0)) == 0
            registered.append(at)
    try:
        arrays[0][:] = u
        with pytest.raises(E.EngineError):
            m.ComputeInternalForceHost(arrays[0], out=arrays[1])
        with pytest.raises(E.EngineError):
            m.ComputeInternalForceHost(u, out=arrays[1])
        for chunks in (3, 1):  # refused part of the way; and the handle still works
            m.set_host_chunks(chunks)
            with pytest.raises(E.EngineError):
                m.ComputeInternalForceHost(arrays[0], out=arrays[1])
            assert np.array_equal(m.ComputeInternalForceHost(u), want)
        for at in registered:
            assert int(rt.cudaHostUnregister(at)) == 0
        registered = [raw.ctypes.data + first]  # both in one piece
        assert int(rt.cudaHostRegister(registered[0], 2 * half, 0)) == 0
        arrays[1][:] = np.nan
        assert np.array_equal(m.ComputeInternalForceHost(arrays[0], out=arrays[1]), want)
    finally:
        for at in registered:
            rt.cudaHostUnregister(at)
    m.close()
