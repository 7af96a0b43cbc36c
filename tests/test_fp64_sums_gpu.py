"""FP64 reciprocal square root and scalar diagnostics on the GPU, at the edges of their ranges."""
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


def _pair_terms(x, a, s):
    """The three diagnostics' pair terms (kinetic energy, enstrophy, helicity) as n x n arrays."""
    r = x[:, None] - x[None]
    core = 0.5 * (s[:, None] + s[None])
    s2 = core * core
    r2 = (r * r).sum(-1)
    q = r2 + s2
    p1 = a @ a.T
    ra = np.einsum("ijk,ik->ij", r, a)
    rb = np.einsum("ijk,jk->ij", r, a)
    ke = p1 * (q ** -0.5 + s2 * q ** -1.5) + q ** -1.5 * ra * rb
    np.fill_diagonal(ke, 0.0)
    ens = (q + 2.2 * s2) * q ** -1.5 * p1
    hel = (q + 1.5 * s2) * q ** -2.5 * np.einsum("ik,ijk->ij", a, np.cross(r, a[None]))
    size = np.sqrt(np.einsum("ik,ik->i", a, a))
    size = size[:, None] * size[None]
    big = (2 * size * q ** -0.5, 3.2 * size * q ** -0.5, 2.5 * size * np.sqrt(r2) * q ** -1.5)
    return (ke, ens, hel), big


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257, 383, 513, 1025,
                               2047, 3001])
def test_scalar_diagnostics_at_tile_edges(n):
    """Each unordered pair once, on the circle of target tiles: one tile, two (the last of an
    even count meets only half of them), odd counts, pieces and tiles with one record.  Every
    pair term is within 64 roundings of its size, their sum within n more."""
    from openonda_b200 import configs, kernels

    f = configs.random_cloud(n, seed=n)
    f.radii *= 4
    x, a, s = _cuda(f.positions, f.strengths, f.radii)
    got = (kernels.total_kinetic_energy(x, a, s), kernels.total_enstrophy(x, a, s),
           kernels.total_helicity(x, a, s))
    again = (kernels.total_kinetic_energy(x, a, s), kernels.total_enstrophy(x, a, s),
             kernels.total_helicity(x, a, s))
    terms, big = _pair_terms(f.positions, f.strengths, f.radii)
    four_pi = 4 * np.pi
    scales = (1 / (4 * four_pi), 1 / (2 * four_pi) / four_pi, -1 / four_pi / four_pi)
    for g, h, t, b, c in zip(got, again, terms, big, scales):
        bound = (64 + n) * EPS * abs(c) * b.sum()
        assert abs(float(g) - c * t.sum()) <= bound, (n, float(g), c * t.sum(), bound)
        assert torch.equal(g, h)
    assert kernels.device_errors() == 0


def test_scalar_diagnostics_of_records_and_uniform_cores():
    """Packed records of all particles take the same sums; a false claim of equal cores is
    still flagged."""
    from openonda_b200 import _lib, configs, kernels

    n = 700
    f = configs.random_cloud(n, seed=4)
    x, a, s = _cuda(f.positions, f.strengths, f.radii)
    lib = _lib.load()
    rec = torch.empty(n * int(lib.vpm_record_bytes(0)), dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.vpm_pack_records(x.data_ptr(), a.data_ptr(), s.data_ptr(), None, n, 0,
                                    rec.data_ptr(), st))
    for op, fn in (("total_kinetic_energy", kernels.total_kinetic_energy),
                   ("total_enstrophy", kernels.total_enstrophy),
                   ("total_helicity", kernels.total_helicity)):
        out = torch.empty((), dtype=torch.float64, device="cuda")
        nb = kernels.workspace_bytes(op, "fp64", n, n)
        ws = torch.empty(max(nb, 256), dtype=torch.uint8, device="cuda")
        _lib.check(lib.vpm_sweep_records(_lib.OPS[op], rec.data_ptr(), n, 0, n, 1,
                                         out.data_ptr(), None, 0, ws.data_ptr(), ws.numel(), st))
        assert torch.equal(out, fn(x, a, s)), op
    kernels.device_errors()
    kernels.total_enstrophy(x, a, s, uniform_core=True)
    assert kernels.device_errors() & 2
