"""Both-sides sums over the triangle of tile pairs (csrc/vpm_triangle.cuh and the FP64 form in
csrc/vpm_circle.cuh), forced on at small sizes: two tiles and more, last tiles of one particle, of
whole and of half units of sources, shares that end inside a list; against the one-sided FP64
sweeps (FP64 1e-12; FP32c the bars of the both-sides sweeps) and bitwise repeatable."""
import numpy as np
import pytest
import torch

from conftest import normwise

pytestmark = pytest.mark.gpu

OPS = ("selfinduced_velocity", "strength_gradients_pse", "velocity_and_strength_gradients",
       "les_step_sums", "rhs_vjp", "rhs_vjp_pse")
# FP32c bars of each output (tests of the both-sides sweeps)
BARS = {"selfinduced_velocity": (1e-6,), "strength_gradients_pse": (1e-6,),
        "velocity_and_strength_gradients": (1e-6, 2e-6), "les_step_sums": (1e-6, 2e-6, 1e-6, 1e-6),
        "rhs_vjp": (1e-5,) * 3, "rhs_vjp_pse": (1e-5,) * 4}


def _inputs(n, seed):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    rng = np.random.default_rng(n)
    arrays = [f.positions, f.strengths, f.radii * 4, rng.uniform(0.5, 1.5, n) * 1e-3,
              rng.normal(size=(n, 3)), rng.normal(size=(n, 3))]
    arrays = [np.asarray(z, np.float32).astype(np.float64) for z in arrays]
    return [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in arrays]


def _call(op, args, precision):
    from openonda_b200 import autodiff, kernels

    x, a, s, v, gu, gs = args
    if op.startswith("rhs_vjp"):
        got = autodiff.rhs_vjp(x, a, s, v if op == "rhs_vjp_pse" else None, gu, gs, precision)
        return got[:4 if op == "rhs_vjp_pse" else 3]
    got = getattr(kernels, op)(*((x, a, s, v) if op == "strength_gradients_pse" else (x, a, s)),
                               precision=precision)
    return got if isinstance(got, tuple) else (got,)


@pytest.mark.parametrize("precision,op", [("fp32c", op) for op in OPS]
                         + [("fp64", op) for op in OPS[:4]])
@pytest.mark.parametrize("n", [769, 1025, 1537, 1568, 1569, 1600, 1601, 2304, 3073])
def test_triangle_vs_one_sided(op, precision, n):
    from openonda_b200 import kernels

    args = _inputs(n, n)
    prev = kernels.set_symmetric_min_n(0)
    try:
        launches = kernels.sweep_launches(op, precision, n, n)
        got = _call(op, args, precision)
        again = _call(op, args, precision)
        kernels.set_symmetric_min_n(1 << 40)
        ref = _call(op, args, "fp64")
    finally:
        kernels.set_symmetric_min_n(prev)
    assert launches == (5 if op == "les_step_sums" else 4)  # zero, own tiles, pairs, finalize
    for k, (g, r, h) in enumerate(zip(got, ref, again)):
        e = abs(float(g) - float(r)) / abs(float(r)) if g.dim() == 0 \
            else normwise(g.cpu().numpy(), r.cpu().numpy())
        assert e <= (1e-12 if precision == "fp64" else BARS[op][k]), (k, e)
        assert torch.equal(g, h)
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
def test_triangle_in_a_graph_and_on_two_streams(precision):
    """The own tiles run on the library's second stream: a captured call replays the same values,
    and calls on two streams keep their own sums."""
    from openonda_b200 import kernels

    prev = kernels.set_symmetric_min_n(0)
    try:
        one, two = _inputs(2100, 1)[:3], _inputs(2300, 2)[:3]
        ref = [kernels.selfinduced_velocity(*z, precision=precision) for z in (one, two)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = kernels.selfinduced_velocity(*one, precision=precision)
        graph.replay()
        assert torch.equal(out, ref[0])
        streams = [torch.cuda.Stream() for _ in range(2)]
        torch.cuda.synchronize()
        for _ in range(4):
            got = []
            for st, z in zip(streams, (one, two)):
                with torch.cuda.stream(st):
                    got.append(kernels.selfinduced_velocity(*z, precision=precision))
            torch.cuda.synchronize()
            for g, r in zip(got, ref):
                assert torch.equal(g, r)
    finally:
        kernels.set_symmetric_min_n(prev)
