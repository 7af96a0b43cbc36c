"""Results are plain tensors, also where the inputs are parameters or of a tensor subclass."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class Tagged(torch.Tensor):
    pass


@pytest.mark.parametrize("wrap", [lambda t: t.as_subclass(Tagged), torch.nn.Parameter])
@pytest.mark.parametrize("n", [200, 5000])
def test_results_are_plain(wrap, n):
    from openonda_b200 import configs, kernels

    f = configs.random_cloud(n, seed=n)
    x, a, s, v = (torch.from_numpy(np.ascontiguousarray(z)).cuda()
                  for z in (f.positions, f.strengths, f.radii, f.viscosities))
    calls = ((kernels.selfinduced_velocity, (x, a, s)), (kernels.strength_gradients, (x, a, s)),
             (kernels.velocity_and_strength_gradients, (x, a, s)),
             (kernels.strength_gradients_pse, (x, a, s, v)),
             (kernels.induced_velocity_at, (x, x, a, s)),
             (kernels.vorticity_field_at, (x, x, a, s)))
    for fn, args in calls:
        got, want = fn(*(wrap(t) for t in args)), fn(*args)
        for g, w in zip(got if isinstance(got, tuple) else (got,),
                        want if isinstance(want, tuple) else (want,)):
            assert type(g) is torch.Tensor and not g.requires_grad
            assert torch.equal(g, w)
