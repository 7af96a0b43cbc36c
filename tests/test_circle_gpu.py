"""FP64 self sums on the circle of tiles (csrc/vpm_circle.cuh), forced on at small sizes: two,
three and four tiles (an even count's last distance is met by half of them), a last tile of one
particle, and shares that end inside a list; against the one-sided FP64 sweeps, which are pinned
to the reference (1e-12), and bitwise repeatable."""
import numpy as np
import pytest
import torch

from conftest import normwise

pytestmark = pytest.mark.gpu

OPS = ("selfinduced_velocity", "strength_gradients", "strength_gradients_pse",
       "velocity_and_strength_gradients", "les_step_sums", "rhs_vjp", "rhs_vjp_pse")


def _inputs(n, seed, ring=False):
    from openonda_b200 import configs

    f = configs.vortex_ring(32, -(-n // 32), 1.0, 1.0, 0.1) if ring \
        else configs.random_cloud(n, seed=seed)
    rng = np.random.default_rng(n)
    arrays = [f.positions[:n], f.strengths[:n], f.radii[:n] * (1 if ring else 4),
              rng.uniform(0.5, 1.5, n) * 1e-3, rng.normal(size=(n, 3)), rng.normal(size=(n, 3))]
    return [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in arrays]


def _call(op, x, a, s, v, gu, gs, uniform):
    from openonda_b200 import autodiff, kernels

    if op == "rhs_vjp":
        return autodiff.rhs_vjp(x, a, s, None, gu, gs)[:3]
    if op == "rhs_vjp_pse":
        return autodiff.rhs_vjp(x, a, s, v, gu, gs)
    args = (x, a, s, v) if op == "strength_gradients_pse" else (x, a, s)
    got = getattr(kernels, op)(*args, uniform_core=uniform)
    return got if isinstance(got, tuple) else (got,)


@pytest.fixture
def threshold():
    from openonda_b200 import kernels

    prev = kernels.set_symmetric_min_n(2400)
    yield kernels.set_symmetric_min_n
    kernels.set_symmetric_min_n(prev)


def _one_sided(threshold, *call):
    threshold(1 << 40)
    try:
        return _call(*call)
    finally:
        threshold(2400)


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("n,ring", [(601, False), (1023, False), (1024, True), (1025, False),
                                    (1537, False), (2049, True), (2399, False)])
def test_circle_vs_one_sided(op, n, ring, threshold):
    from openonda_b200 import kernels

    args = _inputs(n, 3 + n, ring)
    assert kernels.sweep_launches(op, "fp64", n, n) == (3 if op == "les_step_sums" else 2)
    got = _call(op, *args, ring)
    again = _call(op, *args, ring)
    ref = _one_sided(threshold, op, *args, ring)
    assert not any(torch.equal(g, r) for g, r in zip(got[:1], ref[:1]))  # another schedule
    for k, (g, r, h) in enumerate(zip(got, ref, again)):
        e = abs(float(g) - float(r)) / abs(float(r)) if g.dim() == 0 \
            else normwise(g.cpu().numpy(), r.cpu().numpy())
        assert e <= 1e-12, (k, e)
        assert torch.equal(g, h)
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("op", ["strength_gradients", "rhs_vjp", "rhs_vjp_pse"])
def test_large_sums_vs_one_sided(op):
    """The stretching and the adjoint stay on the circle above the both-sides threshold."""
    from openonda_b200 import kernels

    n = 26001
    args = _inputs(n, 7)
    assert kernels.sweep_launches(op, "fp64", n, n) == 2
    got = _call(op, *args, False)
    prev = kernels.set_symmetric_min_n(1 << 40)
    try:
        ref = _call(op, *args, False)
    finally:
        kernels.set_symmetric_min_n(prev)
    for g, r in zip(got, ref):
        assert normwise(g.cpu().numpy(), r.cpu().numpy()) <= 1e-12


@pytest.mark.parametrize("op", ["strength_gradients", "rhs_vjp", "rhs_vjp_pse"])
def test_many_launch_form_where_the_sets_exceed_the_budget(op, threshold):
    """Past the budget of partial sums these operators fall back to the accumulating schedule
    (vpm_rot.cuh): its plan is taken at a size whose circle sets exceed 4 GB."""
    from openonda_b200 import kernels

    n = 700001
    assert kernels.sweep_launches(op, "fp64", n, n) > 2
    assert kernels.workspace_bytes(op, "fp64", n, n) < 6 << 30


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("what", ["position", "strength"])
def test_non_finite_particles(bad, what, threshold):
    """A NaN or infinite particle reaches the same outputs as in the one-sided sweep; the far
    targets that pad the last tile pass nothing on."""
    n = 1025
    args = _inputs(n, 11)
    args[0 if what == "position" else 1][n - 2, 1] = bad
    for op in ("velocity_and_strength_gradients", "strength_gradients_pse"):
        got = _call(op, *args, False)
        ref = _one_sided(threshold, op, *args, False)
        for g, r in zip(got, ref):
            assert torch.equal(torch.isfinite(g), torch.isfinite(r)), op
