"""The FP64 reciprocal square root on the GPU, at the edges of its range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _cuda(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(z, dtype=np.float64)).cuda() for z in arrays]


@pytest.mark.parametrize("exponent", [-150, -60, -8, 0, 8, 60, 150])
def test_enstrophy_of_one_particle_over_the_exponent_range(exponent):
    """One particle alone: r = 0, so the enstrophy is 3.2 s^2 (s^2)^(-3/2) |a|^2 / (8 pi) and the
    reciprocal square root meets s^2 = 4^exponent (1 .. 4).  A dozen roundings of half an ulp,
    the root's own cubed: 16 EPS."""
    from openonda_b200 import kernels

    for f in (1.0, 1.25, 1.7, 1.999):
        s = f * 2.0 ** exponent
        x, a, r = _cuda([[0.0, 0.0, 0.0]], [[1.0, 0.0, 0.0]], [s])
        got = float(kernels.total_enstrophy(x, a, r, ref_extra_4pi=False))
        want = float(np.longdouble(3.2) / np.longdouble(s) / (8 * np.longdouble(np.pi)))
        assert abs(got - want) <= 16 * EPS * want, (s, got, want)


def test_root_of_infinity_and_nan():
    """Outside the normal numbers the sums keep what CUDA's own function gave: an infinite
    distance contributes what inf * 0 makes of it (NaN), a NaN stays NaN, and a probe's skipped
    pair adds nothing even where its root is infinite."""
    from openonda_b200 import kernels

    x, a, s = _cuda([[0.0, 0, 0], [np.inf, 0, 0]], [[1.0, 0, 0], [0, 1.0, 0]], [0.1, 0.1])
    assert torch.isnan(kernels.selfinduced_velocity(x, a, s)).any()
    x[1, 0] = np.nan
    assert torch.isnan(kernels.total_kinetic_energy(x, a, s))
    t, x, a, s = _cuda([[0.0, 0, 0]], [[0.0, 0, 0], [1.0, 0, 0]], [[1.0, 0, 0], [0, 1.0, 0]],
                       [0.0, 0.1])
    assert torch.isfinite(kernels.induced_velocity_at(t, x, a, s)).all()
