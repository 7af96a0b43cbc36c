"""Plans with little scratch (VPM_COMPACT_WORKSPACE): what they ask for, and that the Python
functions take them where the memory for the plain plan is not free."""
import numpy as np
import pytest
import torch

from conftest import normwise

pytestmark = pytest.mark.gpu

OPS = ("selfinduced_velocity", "strength_gradients", "strength_gradients_pse",
       "velocity_and_strength_gradients", "les_step_sums", "rhs_vjp", "rhs_vjp_pse",
       "kinetic_energy_grad", "les_test_filter", "total_kinetic_energy")


def _bytes(op, code, n):
    from openonda_b200 import _lib

    return int(_lib.load().vpm_workspace_bytes(_lib.OPS[op], code, n, n))


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("op", OPS)
def test_bytes_of_compact_plans(op, precision):
    from openonda_b200 import _lib

    code = _lib.precision_code(precision)
    for n in (1000, 4096, 8192, 24575, 32768, 100003, 131072, 300000, 1 << 20, 1 << 22):
        small = _bytes(op, code | _lib.COMPACT_WORKSPACE, n)
        records = 256 * n  # the widest packed record and the LES step's scalar
        assert 0 < small <= max(256 << 20, 576 * n) + records, (n, small)
        assert small <= _bytes(op, code, n), n


def _field(n, seed):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    rng = np.random.default_rng(n)
    arrays = [f.positions, f.strengths, f.radii * 4, rng.uniform(0.5, 1.5, n) * 1e-3,
              rng.normal(size=(n, 3)), rng.normal(size=(n, 3))]
    return [torch.from_numpy(np.ascontiguousarray(z)).cuda() for z in arrays]


@pytest.mark.parametrize("n", [20000, 50000])
def test_little_free_memory(n):
    """The adjoint and the stretching where the allocator may take no more than the compact
    plans: the plain plan's scratch is refused, the sums are still there."""
    from openonda_b200 import _lib, autodiff, kernels

    x, a, s, v, gu, gs = _field(n, 3)
    want = autodiff.rhs_vjp(x, a, s, v, gu, gs) + (kernels.strength_gradients(x, a, s),)
    plain = _bytes("rhs_vjp_pse", 0, n)
    small = _bytes("rhs_vjp_pse", _lib.COMPACT_WORKSPACE, n)
    assert small < plain // 2
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    room = torch.cuda.memory_reserved() + small + (64 << 20)
    assert room < torch.cuda.memory_reserved() + plain
    torch.cuda.set_per_process_memory_fraction(room / total)
    try:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            torch.empty(plain, dtype=torch.uint8, device="cuda")
        got = autodiff.rhs_vjp(x, a, s, v, gu, gs) + (kernels.strength_gradients(x, a, s),)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for k, (g, w) in enumerate(zip(got, want)):
        assert normwise(g.cpu().numpy(), w.cpu().numpy()) <= 1e-12, k
    assert kernels.device_errors() == 0


@pytest.mark.parametrize("op", ["total_kinetic_energy", "total_helicity", "total_enstrophy"])
def test_bytes_of_the_fp64_scalars(op):
    """The FP64 diagnostics leave two doubles per block: their scratch is the packed records and
    at most 256 splits of the tiles of 128 particles."""
    for n in (1, 2, 1000, 32768, 1 << 20, 1 << 22):
        records = 64 * n
        assert records < _bytes(op, 0, n) <= records + 16 * 256 * -(-n // 128) + 512, n
        assert _bytes(op, 0, n) <= records + (n << 3) + (1 << 20), n


def test_sharded_sweep_in_little_memory():
    """The sweep of one rank keeps its scratch: the compact plan's where the plain one's is not
    free."""
    from openonda_b200 import _lib, kernels
    from openonda_b200.distributed import ShardedVelocityStretching

    n = 60000
    x, a, s, *_ = _field(n, 5)
    want = kernels.velocity_and_strength_gradients(x, a, s)
    op = "velocity_and_strength_gradients"
    plain, small = _bytes(op, 0, n), _bytes(op, _lib.COMPACT_WORKSPACE, n)
    assert small + (64 << 20) < plain
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(
        (torch.cuda.memory_reserved() + small + (64 << 20)) / total)
    try:
        sweep = ShardedVelocityStretching(n, precision="fp64")
        assert sweep.ws_bytes == small and sweep.both_sides
        got = [t.clone() for t in sweep(x, a, s)]
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for g, w in zip(got, want):
        assert normwise(g.cpu().numpy(), w.cpu().numpy()) <= 1e-12
