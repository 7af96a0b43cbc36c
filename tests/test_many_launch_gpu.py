"""The both-sides sums in several launches (rot_sweep_kernel and rot64_sweep_kernel of
csrc/vpm_rot.cuh), which the planner takes where the partial sums of the one-launch schedules
exceed their budget.  Compact plans (VPM_COMPACT_WORKSPACE) never take those, so the launches run
here at small sizes: two and three tiles, a last tile of one particle, odd and even tile counts,
several diagonals per launch, the diagonal tiles beside on the second stream, and (at the largest
size) in a launch of their own.  FP64 against the one-sided sums (1e-12).  FP32c against the
triangle of tile pairs, which has the same FP32 sums and adds them in FP64 in another order (1e-12),
and past its range against the FP64 sums at the bars of the other both-sides tests.  All bitwise
repeatable."""
import numpy as np
import pytest
import torch

from conftest import normwise

pytestmark = pytest.mark.gpu

# outputs' bars in FP32c against FP64
BARS = {"selfinduced_velocity": (1e-6,), "strength_gradients_pse": (1e-6,),
        "strength_gradients": (), "velocity_and_strength_gradients": (1e-6, 2e-6),
        "les_step_sums": (1e-6, 2e-6, 1e-6, 1e-6), "rhs_vjp": (1e-5,) * 3,
        "rhs_vjp_pse": (1e-5,) * 4}
FORMS = [("fp64", False), ("fp32c", False), ("fp32c", True), ("fp32c_refined", False),
         ("fp32c_refined", True), ("fp64", True)]
CASES = [(op, p, u) for op in BARS for p, u in FORMS
         if not (op == "strength_gradients" and p != "fp64")  # FP32c: one-sided at every size
         and not (op.startswith("rhs_vjp") and u)]  # the adjoint has no uniform-core form


def _inputs(n, seed, uniform):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    rng = np.random.default_rng(n)
    s = np.full(n, 0.05) if uniform else f.radii * 4
    arrays = [f.positions, f.strengths, s, rng.uniform(0.5, 1.5, n) * 1e-3,
              rng.normal(size=(n, 3)), rng.normal(size=(n, 3))]
    arrays = [np.asarray(z, np.float32).astype(np.float64) for z in arrays]
    return [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in arrays]


def _call(op, args, precision, uniform):
    from openonda_b200 import autodiff, kernels

    x, a, s, v, gu, gs = args
    if op.startswith("rhs_vjp"):
        got = autodiff.rhs_vjp(x, a, s, v if op == "rhs_vjp_pse" else None, gu, gs, precision)
        return got[:4 if op == "rhs_vjp_pse" else 3]
    got = getattr(kernels, op)(*((x, a, s, v) if op == "strength_gradients_pse" else (x, a, s)),
                               precision=precision, uniform_core=uniform)
    return got if isinstance(got, tuple) else (got,)


@pytest.fixture
def compact(monkeypatch):
    """Switches the plans of the calls that follow to compact ones and back (False)."""
    from openonda_b200 import _lib

    plain = _lib.precision_code

    def switch(on):
        monkeypatch.setattr(_lib, "precision_code", plain if not on else
                            lambda p, u=False: plain(p, u) | _lib.COMPACT_WORKSPACE)
    switch(True)
    return switch


def _check(op, precision, uniform, n, compact):
    """Compares the many-launch sum of n particles with another schedule's; returns the number
    of launches of diagonal pairs."""
    from openonda_b200 import kernels

    args = _inputs(n, n, uniform)
    same_sums = precision == "fp64" or n <= 150000
    prev = kernels.set_symmetric_min_n(0)
    try:
        plan = kernels.plan_info(op, precision, n, n, uniform)
        launches = kernels.sweep_launches(op, precision, n, n, uniform)
        got = _call(op, args, precision, uniform)
        again = _call(op, args, precision, uniform)
        if precision != "fp64" and same_sums:
            compact(False)
            assert kernels.sweep_launches(op, precision, n, n, uniform) in (4, 5)  # the triangle
            ref = _call(op, args, precision, uniform)
            compact(True)
        else:
            kernels.set_symmetric_min_n(1 << 40)
            assert kernels.sweep_launches(op, "fp64", n, n, uniform) <= 2
            ref = _call(op, args, "fp64", uniform)
    finally:
        kernels.set_symmetric_min_n(prev)
    assert plan["target_blocks"] == -(-n // (plan["threads"] * plan["targets_per_thread"]))
    # zero, diagonal tiles, launches of diagonal pairs, finalize
    assert launches > 3 and plan["target_blocks"] >= 2
    for k, (g, r, h) in enumerate(zip(got, ref, again)):
        e = abs(float(g) - float(r)) / abs(float(r)) if g.dim() == 0 \
            else normwise(g.cpu().numpy(), r.cpu().numpy())
        assert e <= (1e-12 if same_sums else BARS[op][k]), (k, e)
        assert torch.equal(g, h)
    assert kernels.device_errors() == 0
    return launches - 3


@pytest.mark.parametrize("op,precision,uniform", CASES)
@pytest.mark.parametrize("n", [513, 769, 1024, 1536, 1537, 2305, 3001, 4097])
def test_small_sizes(op, precision, uniform, n, compact):
    from openonda_b200 import kernels

    prev = kernels.set_symmetric_min_n(0)
    try:
        p = kernels.plan_info(op, precision, 1 << 16, 1 << 16, uniform)
    finally:
        kernels.set_symmetric_min_n(prev)
    tile = p["threads"] * p["targets_per_thread"]
    _check(op, precision, uniform, n if n > tile else tile + 1, compact)


@pytest.mark.parametrize("op,precision,uniform", CASES)
def test_several_diagonals_per_launch(op, precision, uniform, compact):
    n = 12289  # one particle past 16 tiles of 768, 24 of 512 and 48 of 256
    assert _check(op, precision, uniform, n, compact) < -(-n // 768) // 2


@pytest.mark.parametrize("op,precision,uniform",
                         [c for c in CASES if c[1:] in (("fp64", False), ("fp32c", False),
                                                        ("fp32c", True))])
def test_diagonal_tiles_in_their_own_launch(op, precision, uniform, compact):
    """At 180001 particles the pair launches take more than 64 waves, so the diagonal tiles run
    before them on the caller's stream."""
    assert _check(op, precision, uniform, 180001, compact) >= 2
