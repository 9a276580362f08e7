"""Which elements the FP64 form evaluates in fixed point, and that they are at
least as exact there as the FP64 code is: flat elements, moduli far apart, tiny
strains, turned and moved elements; on the GPU, elastic forces that scale with
the displacement down to the smallest numbers."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from nimblesm_gb300.mesh import Material, cube_problem

HERE = os.path.dirname(os.path.abspath(__file__))
# no element of these kinds (neo-Hookean, elastic) is inside the domain
OUTSIDE = ({"soft_in_volume", "turned_far", "not_numbers"},
           {"soft_in_shear", "turned_far", "not_numbers", "very_flat"})
# some may be: beyond a range of sizes, or at its edge
EDGE = ({"very_flat", "strain", "large_strain", "turned", "turned_and_strained"},
        {"flat", "needle", "below_the_scales", "large_strain"})


def test_inside_the_domain_fixed_point_is_no_less_exact_than_the_fp64_code(tmp_path):
    nvcc, cxx = shutil.which(os.environ.get("NVCC", "nvcc")), shutil.which("g++")
    if nvcc is None or cxx is None:
        pytest.skip("nvcc or g++ not found")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "fixed_domain_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=fast", "-w", "-I" + include,
                    os.path.join(HERE, "fixed_domain_check.cc"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe, "1000"], capture_output=True, text=True, check=True)
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) > 90
    for model, kind, outside, f_fixed, f_fp64, s_fixed, s_fp64 in rows:
        model, outside = int(model), int(outside)
        if kind in OUTSIDE[model]:
            assert outside == 1000, (model, kind)
            continue
        assert outside == 0 or kind in EDGE[model], (model, kind, outside)
        if kind == "below_the_scales":  # zero or nothing but FP64's own noise is left of a neo-Hookean element
            continue
        if outside == 1000:
            continue
        assert float(f_fixed) <= float(f_fp64), (model, kind)
        assert float(s_fixed) <= float(s_fp64), (model, kind)


def elastic(thin, ratio, seed=2):
    p = cube_problem(3, jitter=0.1, seed=seed)
    p.coords = p.coords * [1.0, 1.0, 1.0 / thin]
    p.blocks = [Material("elastic", p.density, ratio * p.shear_modulus, p.shear_modulus)]
    p.elem_block = np.zeros(p.num_elem, np.int32)
    return p


@pytest.mark.gpu
# inside the domain; flatter, and softer in shear, than it takes
@pytest.mark.parametrize("thin,ratio", [(1.0, 2.0), (3.0, 2.0), (50.0, 2.0), (1.0, 20.0)])
def test_elastic_forces_scale_with_the_displacement(thin, ratio):
    """Below strains of 2^-60 the elastic force is linear in the displacement
    to far below its rounding, and a power of two changes no rounding but those
    of the cofactors' unit (2^-60 of the force): 2^-50 for sums of eight points
    and eight elements."""
    from nimblesm_gb300 import build as B
    B.build()
    p = elastic(thin, ratio)
    rng = np.random.default_rng(4)
    u = np.ldexp(rng.normal(0, 1.0, p.coords.shape), -70)
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    assert np.abs(f).max() > 0.0
    for k in (30, 200, 700, 860):  # 860: beyond the scales, the FP64 code
        g = m.ComputeInternalForceHost(np.ldexp(u, -k))
        assert np.linalg.norm(np.ldexp(g, k) - f) <= 2.0 ** -50 * np.linalg.norm(f), k
    # at rest: zeros of either sign
    z = np.where(rng.random(u.shape) < 0.5, 0.0, -0.0)
    assert not m.ComputeInternalForceHost(z).any()
    m.close()


@pytest.mark.gpu
@pytest.mark.parametrize("model,thin,ratio", [("elastic", 1.0, 2.0), ("elastic", 3.5, 2.0), ("elastic", 50.0, 2.0),
                                              ("elastic", 1.0, 7.0), ("elastic", 1.0, 20.0), ("neohookean", 1.0, 0.55),
                                              ("neohookean", 1.0, 0.3), ("neohookean", 50.0, 2.0)])
def test_forces_at_the_edges_of_the_domain(model, thin, ratio):
    """Against the formulas in NumPy, FP64, whose own error is 2^-53 over the
    strain (1e-3) and the aspect ratio: 1e-11 at the largest."""
    from nimblesm_gb300 import build as B
    B.build()
    p = elastic(thin, ratio)
    G = p.shear_modulus
    K = ratio * G
    p.blocks = [Material(model, p.density, K, G)]
    u = np.random.default_rng(6).normal(0, 1e-3 / 3 / thin, p.coords.shape)
    m = E.Model(p)
    f = m.ComputeInternalForceHost(u)
    m.close()
    signs = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
    want = np.zeros_like(u)
    for x, ids in zip(p.coords[p.conn], p.conn):
        for g in signs * 0.577350269189626:
            t = 1 + signs * g
            dn = np.stack([signs[:, 0] * t[:, 1] * t[:, 2], signs[:, 1] * t[:, 0] * t[:, 2], signs[:, 2] * t[:, 0] * t[:, 1]], 1) / 8
            J = x.T @ dn
            dnx = dn @ np.linalg.inv(J)
            H = u[ids].T @ dnx
            F = np.eye(3) + H
            if model == "elastic":
                s = G * (H + H.T) + (K - 2 * G / 3) * np.trace(H) * np.eye(3)
            else:
                B_ = H + H.T + H @ H.T
                d = np.linalg.det(F)
                s = K / 2 * (d - 1 / d) * np.eye(3) + G * d ** (-5 / 3) * (B_ - np.trace(B_) / 3 * np.eye(3))
            np.add.at(want, ids, -dnx @ (np.linalg.inv(F) * np.linalg.det(F)) @ s * np.linalg.det(J))
    assert np.linalg.norm(f - want) <= 1e-11 * np.linalg.norm(want)
