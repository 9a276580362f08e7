"""The host-buffer force call into pageable memory, in chunks: its copies out
hold the host, and must not hold the chunks after them."""
import time

import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import cube_problem


@pytest.mark.gpu
def test_copies_to_pageable_memory_do_not_hold_the_chunks_that_follow():
    """64^3 elements, FP32, six chunks: into pinned memory 150 us, into pageable
    memory 180 (its copies are slower), 290 when a chunk waited for the copy of
    the one before.  The same bits, also into an array never touched before."""
    from nimblesm_gb300 import build as B
    B.build()
    p = cube_problem(64, jitter=0.2, seed=2)
    m = E.Model(p, precision="fp32")
    u, f = E.PinnedArray(p.coords.shape), E.PinnedArray(p.coords.shape)
    u.array[:] = np.random.default_rng(1).normal(0, 1e-5, p.coords.shape)
    out = np.zeros(p.coords.shape)
    best = {}
    for name, target in (("pinned", f.array), ("pageable", out)):
        times = []
        for _ in range(40):
            t = time.perf_counter()
            m.ComputeInternalForceHost(u.array, out=target)
            times.append(time.perf_counter() - t)
        best[name] = min(times)
    assert np.abs(out).max() > 0 and np.array_equal(out, f.array)
    assert np.array_equal(m.ComputeInternalForceHost(u.array), out)
    assert best["pageable"] <= 1.5 * best["pinned"], best
    m.close()
