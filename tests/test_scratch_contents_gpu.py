"""What the scratch holds before a call reaches no output: every pair sum, on every schedule, gives
the same bits from a workspace of NaN as from one of zeros."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SELF = ("selfinduced_velocity", "strength_gradients", "strength_gradients_pse",
        "velocity_and_strength_gradients", "les_step_sums", "total_kinetic_energy",
        "total_helicity", "total_enstrophy", "rhs_vjp", "rhs_vjp_pse", "kinetic_energy_grad",
        "les_test_filter")


def _run(op, code, n, z, fill):
    from openonda_b200 import _lib

    lib = _lib.load()
    x, a, s, v, g1, g2 = (t.data_ptr() for t in z)
    nb = max(256, lib.vpm_workspace_bytes(_lib.OPS[op], code, n, n))
    ws = torch.full((nb // 8,), fill, dtype=torch.float64, device="cuda")
    o = [torch.zeros((n, 3), dtype=torch.float64, device="cuda") for _ in range(4)]
    p = [t.data_ptr() for t in o]
    st = torch.cuda.current_stream().cuda_stream
    tail = (code, ws.data_ptr(), ws.numel() * 8, st)
    fn = getattr(lib, "vpm_" + ("rhs_vjp" if op == "rhs_vjp_pse" else op))
    if op in ("rhs_vjp", "rhs_vjp_pse"):
        rc = fn(x, a, s, v if op == "rhs_vjp_pse" else None, n, g1, g2, *p, *tail)
    elif op == "kinetic_energy_grad":
        rc = fn(x, a, s, n, *p[:3], *tail)
    elif op == "les_test_filter":
        rc = fn(x, a, s, g1, n, *p[:2], *tail)
    elif op == "les_step_sums":
        rc = fn(x, a, s, n, *p, 1, *tail)
    elif op == "velocity_and_strength_gradients":
        rc = fn(x, a, s, n, *p[:2], *tail)
    elif op == "strength_gradients_pse":
        rc = fn(x, a, s, v, n, p[0], *tail)
    elif op in ("total_helicity", "total_enstrophy"):
        rc = fn(x, a, s, n, 1, p[0], *tail)
    else:
        rc = fn(x, a, s, n, p[0], *tail)
    _lib.check(rc)
    torch.cuda.synchronize()
    return o


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("op", SELF)
def test_scratch_of_nan(op, precision):
    from openonda_b200 import _lib, configs, kernels

    plain = _lib.precision_code(precision)
    prev = kernels.set_symmetric_min_n(24576)
    try:
        # one-sided (and the one launch), the circle, the triangle, several launches
        for n, least, code in ((700, 1 << 40, plain), (5001, 1 << 40, plain), (5001, 24576, plain),
                               (2400, 2400, plain), (2400, 0, plain | _lib.COMPACT_WORKSPACE)):
            f = configs.random_cloud(n, seed=n)
            rng = np.random.default_rng(n)
            arrays = (f.positions, f.strengths, f.radii * 4, f.viscosities,
                      rng.normal(size=(n, 3)), rng.normal(size=(n, 3)))
            z = [torch.from_numpy(np.ascontiguousarray(t)).cuda() for t in arrays]
            kernels.set_symmetric_min_n(least)
            for g, h in zip(_run(op, code, n, z, 0.0), _run(op, code, n, z, float("nan"))):
                assert torch.equal(g, h), (n, least)
                assert torch.isfinite(g).all()
    finally:
        kernels.set_symmetric_min_n(prev)
    assert kernels.device_errors() == 0
