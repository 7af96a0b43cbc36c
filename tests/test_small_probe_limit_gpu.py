"""Probe sums of very many targets and few sources take the tiled sweep: the one launch of small
sums (csrc/vpm_small.cuh) is limited to 3200 blocks of 32 targets in FP64, 4096 of 64 in FP32c."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32c": 1e-6}


@pytest.mark.parametrize("precision,m,n,launches", [
    ("fp64", 102400, 58, 1), ("fp64", 102401, 58, 2), ("fp64", 300000, 10, 2),
    ("fp64", 1000001, 3, 2), ("fp32c", 262144, 61, 1), ("fp32c", 262145, 61, 2),
    ("fp32c", 300000, 40, 2), ("fp32c", 1000001, 5, 2)])
def test_many_targets_few_sources(precision, m, n, launches):
    from openonda_b200 import configs, kernels

    f = configs.random_cloud(n, seed=n)
    x, a, s = (np.asarray(z, np.float32).astype(np.float64)
               for z in (f.positions, f.strengths, f.radii * 4))
    t = np.random.default_rng(m).uniform(-1.1, 1.1, size=(m, 3))
    t = t.astype(np.float32).astype(np.float64)
    t[m - 1] = x[0]
    dev = [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in (t, x, a, s)]
    at = np.r_[0:300, m // 2:m // 2 + 300, m - 300:m]
    for op, ref in (("induced_velocity_at", oracle.gpu.get_induced_velocity_at),
                    ("vorticity_field_at", oracle.gpu.get_vorticity_field_at)):
        assert kernels.sweep_launches(op, precision, m, n) == launches
        got = getattr(kernels, op)(*dev, precision=precision).cpu().numpy()
        want = ref(t[at], x, a, s)[:len(at)]
        assert normwise(got[at], want) <= TOL[precision]
    assert kernels.device_errors() == 0
