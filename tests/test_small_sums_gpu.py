"""Small sums in one launch (csrc/vpm_small.cuh) at the edges of their tiles, windows and range:
against the oracle at the bars of the tiled sweeps (FP64 1e-12; FP32c 1e-6, stretching 2e-6 on the
FP32-rounded inputs that form computes with)."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise

pytestmark = pytest.mark.gpu

TOL = {"fp64": (1e-12, 1e-12), "fp32c": (1e-6, 2e-6)}


def _field(n, seed):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    f.radii *= 4
    return f


def _inputs(f, precision):
    arrays = (f.positions, f.strengths, f.radii, f.viscosities)
    if precision != "fp64":
        arrays = [np.asarray(z, np.float32).astype(np.float64) for z in arrays]
    return arrays, [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in arrays]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 127, 129, 1023, 1024, 1025, 1999])
def test_self_sums_vs_oracle(n, precision):
    from openonda_b200 import kernels

    (x, a, s, v), dev = _inputs(_field(n, n), precision)
    dx, da, ds, dv = dev
    assert kernels.sweep_launches("selfinduced_velocity", precision, n, n) == 1
    o = oracle.gpu
    u, g = kernels.velocity_and_strength_gradients(dx, da, ds, precision=precision)
    got = [(u, o.get_selfinduced_velocity(x, a, s), 0),
           (g, o.get_strength_gradients(x, a, s), 1),
           (kernels.selfinduced_velocity(dx, da, ds, precision=precision),
            o.get_selfinduced_velocity(x, a, s), 0),
           (kernels.strength_gradients(dx, da, ds, precision=precision),
            o.get_strength_gradients(x, a, s), 1),
           (kernels.strength_gradients_pse(dx, da, ds, dv, precision=precision),
            o.get_strength_gradients_PSE(x, a, s, v), 0)]
    for k, (t, ref, bar) in enumerate(got):
        e = normwise(t.cpu().numpy(), ref)
        assert e <= TOL[precision][bar], (k, e)
    again = kernels.velocity_and_strength_gradients(dx, da, ds, precision=precision)
    assert torch.equal(u, again[0]) and torch.equal(g, again[1])
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("m,n", [(1, 500), (33, 1), (70, 129), (2000, 1999), (5000, 33),
                                 (100000, 40), (3000, 4095), (900, 4095), (900, 4096)])
def test_probe_sums_vs_oracle(m, n, precision):
    """Few and many targets, one source, a coincident target (skipped), and both sides of the
    range's ends (fewer than 4096 sources; 6 and 16 million pairs)."""
    from openonda_b200 import kernels

    (x, a, s, _), (dx, da, ds, _) = _inputs(_field(n, n), precision)
    t = np.random.default_rng(m).uniform(-1.1, 1.1, size=(m, 3)).astype(np.float32)
    t = t.astype(np.float64)
    t[m // 2] = x[n // 2]
    dt = torch.from_numpy(t).cuda()
    small = n < 4096 and m * n <= (6000000 if precision == "fp64" else 16000000)
    assert (kernels.sweep_launches("induced_velocity_at", precision, m, n) == 1) == small
    for fn, ref in ((kernels.induced_velocity_at, oracle.gpu.get_induced_velocity_at),
                    (kernels.vorticity_field_at, oracle.gpu.get_vorticity_field_at)):
        got = fn(dt, dx, da, ds, precision=precision).cpu().numpy()
        want = ref(t, x, a, s)[:m]
        if n == 1:
            assert np.max(np.abs(got - want)) <= TOL[precision][0] * np.max(np.abs(want))
        else:
            assert normwise(got, want) <= TOL[precision][0]
    assert kernels.device_errors() == 0


def test_one_particle_views_and_capture():
    """One particle induces nothing on itself; inputs that are views (strided) are taken as
    before; a captured call replays on new values."""
    from openonda_b200 import kernels

    one = torch.tensor([[0.3, 0.1, 0.2]], dtype=torch.float64, device="cuda")
    r = torch.tensor([0.1], dtype=torch.float64, device="cuda")
    u, g = kernels.velocity_and_strength_gradients(one, one, r)
    assert not u.any() and not g.any()
    f = _field(300, 5)
    wide = torch.zeros((300, 8), dtype=torch.float64, device="cuda")
    wide[:, :3] = torch.from_numpy(f.positions).cuda()
    wide[:, 3:6] = torch.from_numpy(f.strengths).cuda()
    wide[:, 6] = torch.from_numpy(f.radii).cuda()
    ref = kernels.selfinduced_velocity(wide[:, :3].clone(), wide[:, 3:6].clone(),
                                       wide[:, 6].clone())
    assert torch.equal(kernels.selfinduced_velocity(wide[:, :3], wide[:, 3:6], wide[:, 6]), ref)
    x, a, s = wide[:, :3].clone(), wide[:, 3:6].clone(), wide[:, 6].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = kernels.selfinduced_velocity(x, a, s)
    graph.replay()
    assert torch.equal(out, ref)
    a.mul_(2.0)
    graph.replay()
    assert torch.equal(out, 2.0 * ref)
