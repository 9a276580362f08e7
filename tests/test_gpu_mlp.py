"""The learned constitutive closure: training data from the material, the
tensor-core forward pass and loss gradient against the CPU oracle
(oracle/mlp_oracle.py), and what training buys over the closure's linear
part alone."""
import numpy as np
import pytest

from nimblesm_gb300 import engine as E
from oracle import mlp_oracle as M
from oracle import oracle as O
from tests.gpu_util import rel

pytestmark = pytest.mark.gpu
K, G = 160e9, 79.3e9


@pytest.fixture(scope="module")
def mlp():
    from nimblesm_gb300 import build as B
    B.build()
    O.build(ref=False)
    m = E.MLPClosure(K, G, seed=3)
    m.generate(1 << 20, seed=11)
    yield m
    m.close()


def to_reference_F(H):
    slot = [0, 3, 8, 6, 1, 4, 5, 7, 2]  # row-major (i,J) -> reference full-tensor slot
    F = np.zeros((H.shape[0], 9))
    for q in range(9):
        F[:, slot[q]] = H[:, q] + (1.0 if q % 4 == 0 else 0.0)
    return F


def test_training_pairs_are_the_material(mlp):
    H, Y = mlp.training_sample(1000, 512)
    assert np.abs(H).max() < 0.5 and 0.045 < H.std() < 0.055
    sig = O.stress(to_reference_F(H.astype(np.float64)), K, G)  # the reference's arithmetic
    assert rel(Y, sig / G) < 1e-6  # FP32 storage of the targets


def test_forward_matches_oracle(mlp):
    P, S = mlp.params()
    rng = np.random.default_rng(0)
    P = P + rng.normal(0, 0.05, P.shape).astype(np.float32)  # non-trivial biases too
    mlp.set_params(P, S)
    H, _ = mlp.training_sample(0, 2048)
    sig, fb = mlp.predict(to_reference_F(H.astype(np.float64)))
    inside = np.abs(H).max(axis=1) <= S[3]
    ref = M.stress_over_g(P, S, H) * G
    assert rel(sig[inside], ref[inside]) < 2e-3
    assert fb == int((~inside).sum())


def test_gradient_matches_oracle(mlp):
    P, S = mlp.params()
    rng = np.random.default_rng(1)
    P = P + rng.normal(0, 0.05, P.shape).astype(np.float32)
    mlp.set_params(P, S)
    H, Y = mlp.training_sample(4096, 1024)
    g, loss = mlp.gradient(H, Y)
    l_e, g_e = M.loss_and_gradient(P, S, H, Y, emulate=True)
    l_x, g_x = M.loss_and_gradient(P, S, H, Y, emulate=False)
    assert abs(loss - l_e) < 1e-3 * l_e
    assert rel(g, g_e) < 2e-2          # same BF16 rounding points as the GPU
    assert rel(g, g_x) < 5e-2          # the exact mathematical gradient, to BF16 precision
    for lo, hi in ((M.oW1, M.ob1), (M.oW2, M.ob2), (M.oW3, M.ob3)):
        assert rel(g[lo:hi], g_e[lo:hi]) < 3e-2


def test_training_gains_over_the_analytic_base(mlp):
    """What the trained network adds: on the training distribution its stress
    is closer to the material's than the analytic base alone (the stress to
    second order in H, with the network's term left out), and far closer than
    the small-strain linear part."""
    mlp.set_params(E.MLPClosure(K, G, seed=3).params()[0])  # fresh weights, keep the data's scales
    loss = mlp.train(epochs=40, batch_tiles=16, lr=5e-3)
    P, S = mlp.params()
    rng = np.random.default_rng(99)
    H = rng.normal(0, 0.05, size=(4096, 9))
    F = to_reference_F(H)
    exact = O.stress(F, K, G) / G
    sig, fb = mlp.predict(F)
    inside = np.abs(H).max(axis=1) <= S[3]
    base = M.base_part(H, S[2])
    lin = M.linear_part(H, S[2])
    e_mlp = rel(sig[inside] / G, exact[inside])
    e_base = rel(base[inside], exact[inside])
    e_lin = rel(lin[inside], exact[inside])
    print(f"loss {loss:.3e}  stress error: linear part {e_lin:.3e}, second-order base {e_base:.3e}, "
          f"with the trained network {e_mlp:.3e}")
    assert loss < 0.05
    assert e_mlp < 0.25 * e_base, (e_mlp, e_base)
    assert e_mlp < 0.03 * e_lin, (e_mlp, e_lin)


def test_fused_element_kernel_matches_predict(mlp):
    """The closure inside the element kernel computes the same stress as the
    standalone inference of the same points."""
    from nimblesm_gb300.mesh import cube_problem
    p = cube_problem(6, jitter=0.2, seed=4)
    m = E.Model(p, precision="fp32")
    m.set_closure(mlp)
    rng = np.random.default_rng(5)
    m.SetVectorNodeData("displacement", rng.normal(0, 2e-3, size=(p.num_nodes, 3)))
    m.ComputeInternalForce()
    F, sig = m.GetIntegrationPointData()
    ref, fb = mlp.predict(F.reshape(-1, 9))
    # predict() sees H = F - I rebuilt from the FP32-stored F: at strains of
    # ~1e-2 that carries ~6e-8 / 1e-2 relative quantisation in H
    assert rel(sig.reshape(-1, 6), ref) < 5e-5
    assert m.closure_fallbacks() == fb


def test_fused_forces_match_the_material(mlp):
    """Nodal internal forces of the fused kernel (per-point B^T sigma reduced
    over each element's lanes, then the deterministic gather) against the
    plain FP32 element kernel on the same displacement: they differ only by
    the closure's stress error, on every node."""
    from nimblesm_gb300.mesh import cube_problem
    p = cube_problem(8, jitter=0.2, seed=6)
    rng = np.random.default_rng(8)
    u = rng.normal(0, 2e-4, size=(p.num_nodes, 3))
    f, F = {}, {}
    for form in ("plain", "mlp"):
        m = E.Model(p, precision="fp32")
        if form == "mlp":
            m.set_closure(mlp)
        m.SetVectorNodeData("displacement", u)
        m.ComputeInternalForce()
        f[form] = m.GetVectorNodeData("internal_force")
        F[form] = m.GetIntegrationPointData()[0]
        m.close()
    # each point's F record lands where the plain kernel puts it (FP32 rounding apart)
    assert rel(F["mlp"], F["plain"]) < 1e-6, rel(F["mlp"], F["plain"])
    assert rel(f["mlp"], f["plain"]) < 2e-3, rel(f["mlp"], f["plain"])
    scale = np.abs(f["plain"]).max()
    assert np.abs(f["mlp"] - f["plain"]).max() < 5e-3 * scale


def test_small_strain_limit(mlp):
    """The gated closure reduces to the material's response near F = I: at
    strains of 1e-4 and 1e-3 its stress error is the FP32 evaluation's and the
    third-order remainder's, far below the second-order terms (1e-4 and 1e-3
    of the stress) that a network error near H = 0 would disturb."""
    P, S = mlp.params()
    rng = np.random.default_rng(7)
    for scale in (1e-4, 1e-3):
        H = rng.normal(0, scale, size=(2048, 9))
        F = to_reference_F(H)
        exact = O.stress(F, K, G) / G
        sig, fb = mlp.predict(F)
        assert fb == 0
        assert rel(sig / G, exact) < 2e-5, (scale, rel(sig / G, exact))


def test_explicit_run_with_the_closure(mlp):
    """An explicit run whose material is the trained network, against the FP64
    plain run: displacement error, and no envelope fallbacks at these strains."""
    from nimblesm_gb300.mesh import cube_problem, critical_time_step
    p = cube_problem(16, jitter=0.2, seed=2)
    dt = 0.5 * critical_time_step(p)
    steps = 400
    ref = E.run(p, steps * dt, steps, precision="fp64")
    m = E.Model(p, precision="fp32")
    m.set_closure(mlp)
    m.begin(steps * dt, steps, 0)
    m.advance(steps)
    st = m.state(with_ip=False)
    e = rel(st["u"], ref["u"])
    print(f"closure run: relative displacement error {e:.3e} after {steps} steps, fallbacks {m.closure_fallbacks()}")
    assert e < 1e-3
    assert m.closure_fallbacks() == 0


def test_closure_over_the_full_schedule():
    """The workload's whole schedule (2000 steps at dt = 0.5 dt_crit) with the
    closure as the material, trained as the benchmark trains it (20M pairs of
    the material, 20 epochs of batches of 152 tiles), on a 32^3 jittered cube: displacement within
    1e-3 of the FP64 plain run after the last step; the energy drift of both
    runs is reported.  (At 32^3 the schedule covers 4x the physical time of
    the 128^3 one, dt being proportional to the element size.)"""
    from nimblesm_gb300.mesh import cube_problem, critical_time_step
    p = cube_problem(32, jitter=0.2, seed=0)
    mlp = E.MLPClosure(p.bulk_modulus, p.shear_modulus, seed=1)
    mlp.generate(20_000_000, seed=7, perturbation=0.05, min_det=0.5)
    loss = mlp.train(epochs=20, batch_tiles=152, lr=2e-2)
    dt = 0.5 * critical_time_step(p)
    steps = 2000
    out = {}
    for form in ("fp64", "mlp"):
        m = E.Model(p, precision="fp64" if form == "fp64" else "fp32", graph_steps=100)
        if form == "mlp":
            m.set_closure(mlp)
        m.begin(steps * dt, steps, 0)
        m.advance(1)
        e0 = sum(m.GetEnergies())
        m.advance(steps - 1)
        st = m.state(with_ip=False)
        out[form] = (st, (sum(m.GetEnergies()) - e0) / e0, m.closure_fallbacks() if form == "mlp" else 0)
        m.close()
    mlp.close()
    (ref, drift64, _), (st, drift, fallbacks) = out["fp64"], out["mlp"]
    e_u, e_v = rel(st["u"], ref["u"]), rel(st["v"], ref["v"])
    print(f"closure (loss {loss:.2e}), 32^3 x {steps} steps: displacement error {e_u:.3e}, velocity error {e_v:.3e}, "
          f"energy drift {drift:.3e} (FP64 plain {drift64:.3e}), fallbacks {fallbacks}")
    assert e_u < 1e-3
    assert abs(drift) < 1e-2


@pytest.mark.parametrize("pairs, tiles", [(100, 1), (128, 2), (20_001, 160), (51_163, 400)])
def test_one_training_step_is_adam_on_the_gradient(pairs, tiles):
    """A step over one partial tile, an empty second one, a last wave of tiles
    and more tiles than the GPU holds at once: from zero moments the step is
    lr g / (|g| + eps), g the gradient of the whole set (summed in another
    order: 2^-24 sqrt(tiles) relative to the largest terms, so entries within
    1e-3 of the largest are held to 1e-3 of a step)."""
    m = E.MLPClosure(K, G, seed=2)
    m.generate(pairs, seed=5)
    P0, _ = m.params()
    H, Y = m.training_sample(0, pairs)
    g, loss = m.gradient(H, Y)
    lr = 2e-3
    final = m.train(epochs=1, batch_tiles=tiles, lr=lr)
    P1, _ = m.params()
    assert abs(final * 6.0 - loss) <= 1e-5 * loss
    big = np.abs(g) > 1e-3 * np.abs(g).max()
    step = P0 - lr * np.sign(g) - P1  # one step of the schedule runs at the full rate
    assert np.abs(step[big]).max() <= 1e-3 * lr
    m.close()
