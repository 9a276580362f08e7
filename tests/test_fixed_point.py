"""The FP64 form's element arithmetic in 64-bit fixed point (hex_fixed.cuh,
element_fixed.cu).

On the host, the arithmetic as the kernel's lanes carry it out against the
same formulas in extended precision: over strains of 1e-9 to 3e-2, with and
without a rigid displacement, forces and stresses are at least as close to the
exact values as an FP64 evaluation's.  On the GPU, element counts at the edges
of the kernel's groups of 8, elements outside the fixed-point domain beside
elements inside it, and ranges of elements that start inside a group."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Material, Problem, cube_mesh
from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
# Both forms end in numbers rounded to FP64 (2^-53 each) after sums of 8 points:
# below this the two are equally exact.
ROUNDING = 3e-16


def test_fixed_point_is_no_less_exact_than_fp64(tmp_path):
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc"))
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fixed_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", os.path.join(HERE, "fixed_check.cc"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe, "400", "17"], capture_output=True, text=True, check=True)
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 2 * 3 * 8
    for model, rigid, strain, f_fixed, f_fp64, s_fixed, s_fp64, outside in rows:
        if float(strain) == 1.0:
            assert int(outside) == 400  # every element is left to the FP64 code
            continue
        assert int(outside) <= 8, (model, rigid, strain)
        assert float(f_fixed) <= max(float(f_fp64), ROUNDING), (model, rigid, strain)
        assert float(s_fixed) <= max(float(s_fp64), ROUNDING), (model, rigid, strain)


def test_sums_of_eight_are_no_less_exact_than_fp64(tmp_path):
    """The node kernel's sum of up to eight element forces: over the largest of
    them, within the rounding of the sum (2^-53 of at most 8 times it) and eight
    numbers cut at 2^-59 of its power of two, and never further off than FP64
    additions; infinities, NaN and zeros exactly as those."""
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc"))
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "fixed_sum_check")
    subprocess.run([nvcc, "-O2", "-std=c++17", os.path.join(HERE, "fixed_sum_check.cc"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe, "20000", "5"], capture_output=True, text=True, check=True)
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 8
    for kind, fixed, fp64 in rows:
        assert float(fixed) <= float(fp64), kind
        if kind not in ("tiny", "huge"):  # those are FP64 additions
            assert float(fixed) <= 2.0 ** -53 * 8 + 8 * 2.0 ** -59, kind


def strip(n, seed):
    """n jittered elements in a row along x."""
    coords, conn = cube_mesh(1)
    x = np.concatenate([coords + [k, 0.0, 0.0] for k in range(n)])
    xy, ids = np.unique(x, axis=0, return_inverse=True)
    conn = ids.reshape(n, 8)[:, conn[0]].astype(np.int32)
    rng = np.random.default_rng(seed)
    return Problem(coords=(xy + rng.uniform(-0.1, 0.1, xy.shape)) / n, conn=conn), rng


def oracle_force(p, u):
    f = np.zeros_like(u)
    for e in p.conn:
        np.add.at(f, e, np.asarray(O.element(p.coords[e], u[e], p.bulk_modulus, p.shear_modulus)[2]).reshape(8, 3))
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 8, 9, 33])
@pytest.mark.parametrize("kind", ["inside", "some outside", "translated", "far away"])
def test_forces_at_the_edges(n, kind):
    """Forces against the oracle.  Its own rounding is 2^-53 of |X| / h = n
    over the strain, 4e-12 at the largest n: 1e-10 as elsewhere."""
    from nimblesm_gb300 import build as B
    B.build()
    O.build(ref=False)
    p, rng = strip(n, 5 + n)
    h = 1.0 / n
    u = rng.normal(0, 1e-3 * h, p.coords.shape)
    if kind == "some outside":  # strains of about 0.3 at every other element's nodes
        u[p.conn[::2].ravel()] += rng.normal(0, 0.05 * h, (p.conn[::2].size, 3))
    elif kind == "translated":  # several element sizes: the modes are shifted up
        u += [3.0 * h, -40.0 * h, 0.5 * h]
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    if kind == "far away":  # beyond the domain's range of displacements: the FP64 code, the same forces
        u2 = np.ldexp(np.round(np.ldexp(u, 34)), -34)
        f = m.ComputeInternalForceHost(u2)
        far = m.ComputeInternalForceHost(u2 + np.ldexp(1.0, 18))  # exact sums
        assert np.linalg.norm(far - f) <= 2.0 ** -53 * 2.0 ** 18 / (1e-3 * h) * 8 * np.linalg.norm(f)
        return
    ref = oracle_force(p, u)
    err = np.linalg.norm(f - ref) / np.linalg.norm(ref)
    assert err <= (1e-10 if kind != "translated" else 1e-8), err
    F0, s0 = m.GetIntegrationPointData()
    if n == 33:  # element ranges that begin and end inside a group of 8
        m.set_host_chunks(5)
        assert np.array_equal(m.ComputeInternalForceHost(u), f)
        F1, s1 = m.GetIntegrationPointData()
        assert np.array_equal(F0, F1) and np.array_equal(s0, s1)


@pytest.mark.gpu
def test_a_node_without_a_number_is_reported():
    p, rng = strip(9, 3)
    u = rng.normal(0, 1e-4, p.coords.shape)
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    bad = u.copy()
    bad[p.conn[4][0], 1] = np.nan
    with pytest.raises(E.EngineError):
        m.ComputeInternalForceHost(bad)
    assert np.array_equal(m.ComputeInternalForceHost(u), f)  # and the handle still works


@pytest.mark.gpu
# a lane's share of the element changes past one warp of 4 elements per
# scheduler of the chip (2,432 elements)
@pytest.mark.parametrize("n", [1, 3, 4, 5, 2432, 2433])
@pytest.mark.parametrize("elastic", [False, True])
def test_one_point_per_lane_gives_the_bits_of_two(n, elastic):
    """The first of two steps in one sequence stores no records and may take
    the kernel of one point per lane; a step by itself stores them, with two.
    Some elements strain beyond the fixed-point domain."""
    p, rng = strip(n, 11 + n)
    h = 1.0 / n
    dt = 0.3 * h * np.sqrt(p.density / p.bulk_modulus)
    p.v_init = rng.normal(0, 1e-3 * h / dt, p.coords.shape)
    p.v_init[p.conn[::3].ravel()] += rng.uniform(-0.08, 0.08, (p.conn[::3].size, 3)) * h / dt
    if elastic:
        kind = [Material(m, p.density, p.bulk_modulus, p.shear_modulus) for m in ("elastic", "neohookean")]
        p.blocks, p.elem_block = (kind, (np.arange(n) >= (n + 1) // 2).astype(np.int32)) if n > 1 else (kind[:1], np.zeros(1, np.int32))
    states = []
    for parts in ((2,), (1, 1)):
        m = E.Model(p)
        m.begin(2 * dt, 2, 0)
        for k in parts:
            m.advance(k)
        states.append(m.state())
        m.close()
    assert np.abs(states[0]["f_int"]).max() > 0.0
    for key in states[0]:
        assert np.array_equal(states[0][key], states[1][key]), key
