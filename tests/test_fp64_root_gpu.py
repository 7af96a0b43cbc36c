"""The FP64 reciprocal square root (rsqrt_fp64, csrc/vpm_lanes.cuh) over many arguments, through
a sum that takes its fifth power, and the probe sums with a source at infinity."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def test_root_over_mantissas_and_exponents():
    """A source of no core at the origin, strength (0, 0, 1), and targets (d, 0, 0): the velocity is
    d^2 y^5 d / (4 pi) = 1 / (4 pi d^2) with y the root of the rounded square of d.  Relative to
    EPS: the rounding of d^2 counts 5/2 in y^5 and 1 in the factor d^2, against each other, three
    products make y^5, two more the term, three the factor 1/(4 pi) and its product; an error of
    one unit in the last place of y (2 EPS at most) counts five times: 1.5 + 3 + 2 + 3 + 10 < 20."""
    from openonda_b200 import kernels

    rng = np.random.default_rng(7)
    m = 1 << 20
    d = np.ldexp(rng.uniform(1.0, 2.0, m), rng.integers(-13, 190, m))
    d[:64] = np.ldexp(1.0, np.arange(64) - 12)  # powers of two: exact squares and roots
    d[64:128] = np.nextafter(d[:64], 0.0)
    d[128:192] = np.nextafter(d[:64], np.inf)
    t = np.zeros((m, 3))
    t[:, 0] = d
    z = [torch.from_numpy(np.ascontiguousarray(q)).cuda()
         for q in (t, np.zeros((1, 3)), np.array([[0.0, 0.0, 1.0]]), np.zeros(1))]
    got = kernels.induced_velocity_at(*z).cpu().numpy()
    assert not got[:, 0].any() and not got[:, 2].any()
    dl = d.astype(np.longdouble)
    want = 1 / (4 * np.longdouble("3.14159265358979323846264338327950288") * dl * dl)
    err = np.abs(np.abs(got[:, 1]).astype(np.longdouble) - want) / want
    assert err.max() <= 20 * EPS, float(err.max() / EPS)
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [300, 4100])
def test_source_at_infinity(n, precision):
    """A source at infinity is not within the guard radius: its velocity is 0 times infinity (NaN
    for every target), its vorticity is zero times its strength (nothing), in the one launch of
    small sums and in the groups of the tiled sweep."""
    from openonda_b200 import configs, kernels

    f = configs.random_cloud(n, seed=n)
    x, a, s = (np.asarray(q, np.float32).astype(np.float64)
               for q in (f.positions, f.strengths, f.radii * 4))
    x[n - 57, 1] = np.inf
    t = np.concatenate([x[40:48], np.random.default_rng(1).uniform(-1, 1, size=(100, 3))])
    t = np.asarray(t, np.float32).astype(np.float64)
    dev = [torch.from_numpy(np.ascontiguousarray(q)).cuda() for q in (t, x, a, s)]
    u = kernels.induced_velocity_at(*dev, precision=precision).cpu().numpy()
    assert np.isnan(u).all() and np.isnan(oracle.gpu.get_induced_velocity_at(t, x, a, s)).all()
    w = kernels.vorticity_field_at(*dev, precision=precision).cpu().numpy()
    want = oracle.gpu.get_vorticity_field_at(t, x, a, s)[:len(t)]
    assert np.isfinite(want).all()
    assert normwise(w, want) <= (1e-12 if precision == "fp64" else 1e-6)
