"""The guard of the probe sums (pairs with r^2 <= 1e-8 skipped), tested a few sources at a time by
the tiled sweep: coincident and nearby targets at every place of a group, of a carry window and of
the remainders, against the oracle (FP64 1e-12, FP32c 1e-6 on FP32-rounded inputs)."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32c": 1e-6}


def _field(n, seed):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    arrays = [f.positions, f.strengths, f.radii * 4]
    return [np.asarray(z, np.float32).astype(np.float64) for z in arrays]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [4096, 4097, 4098, 4099, 4100, 4127])
def test_skipped_pairs_at_every_place(n, precision):
    from openonda_b200 import kernels

    x, a, s = _field(n, n)
    at = [0, 1, 2, 3, 4, 5, 6, 7, 30, 31, 32, 33, 255, 256, n - 5, n - 4, n - 3, n - 2, n - 1]
    # on the source, inside the guard radius of 1e-4, outside it, and far from all
    t = np.concatenate([x[at], x[at] + [0.5e-4, 0, 0], x[at] + [0, 2e-4, 0],
                        np.random.default_rng(n).uniform(-1, 1, size=(400, 3))])
    t = np.asarray(t, np.float32).astype(np.float64)
    dev = [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in (t, x, a, s)]
    for fn, ref in ((kernels.induced_velocity_at, oracle.gpu.get_induced_velocity_at),
                    (kernels.vorticity_field_at, oracle.gpu.get_vorticity_field_at)):
        got = fn(*dev, precision=precision).cpu().numpy()
        assert normwise(got, ref(t, x, a, s)[:len(t)]) <= TOL[precision]
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_non_finite_source_in_a_group(precision):
    """A NaN or infinite source position is skipped by every target, and its neighbours in the
    group still count; a NaN strength reaches every target but those within the guard radius."""
    from openonda_b200 import kernels

    n = 4100
    x, a, s = _field(n, 3)
    t = np.concatenate([x[40:48], np.random.default_rng(1).uniform(-1, 1, size=(100, 3))])
    t = np.asarray(t, np.float32).astype(np.float64)
    bad = x.copy()
    bad[42, 1] = np.nan
    b = a.copy()
    b[45] = np.nan
    for xs, strengths in ((bad, a), (x, b)):
        dev = [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in (t, xs, strengths, s)]
        for fn, ref in ((kernels.induced_velocity_at, oracle.gpu.get_induced_velocity_at),
                        (kernels.vorticity_field_at, oracle.gpu.get_vorticity_field_at)):
            got = fn(*dev, precision=precision).cpu().numpy()
            assert normwise(got, ref(t, xs, strengths, s)[:len(t)]) <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [259, 4101])
def test_filter_sums_skip_their_own_particle(n, precision):
    """The test-filter sums of the particles over themselves: each particle's own pair is
    skipped, coincident particles skip each other.  Both filters are the vorticity sum of the
    oracle, the second with the fields as strengths."""
    from openonda_b200 import kernels

    x, a, s = _field(n, n)
    x[7] = x[n - 3]
    f = np.random.default_rng(n).normal(size=(n, 3)).astype(np.float32).astype(np.float64)
    dev = [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in (x, a, s, f)]
    w, fh = kernels.les_test_filter(*dev, precision=precision)
    two = f.copy()
    two[:, 2] = 0.0
    for got, strengths in ((w, a), (fh, two)):
        want = oracle.gpu.get_vorticity_field_at(x, x, strengths, s)
        assert normwise(got.cpu().numpy(), want) <= TOL[precision]
