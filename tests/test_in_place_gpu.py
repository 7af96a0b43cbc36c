"""Outputs that overlap the inputs: every input is read before the first output is written, at
the sizes of the one-launch sums (csrc/vpm_small.cuh, which reads the caller's arrays directly)
and above.  An in-place call packs its inputs first, so it gives the bits of the same sum from
packed records."""
import numpy as np
import pytest
import torch

import oracle
from conftest import normwise

pytestmark = pytest.mark.gpu

OPS = ("selfinduced_velocity", "strength_gradients", "strength_gradients_pse",
       "velocity_and_strength_gradients")


def _arrays(n, seed):
    from openonda_b200 import configs

    f = configs.random_cloud(n, seed=seed)
    f.radii *= 4
    return [torch.from_numpy(np.ascontiguousarray(z)).cuda()
            for z in (f.positions, f.strengths, f.radii, f.viscosities)]


def _from_records(op, x, a, s, v, code):
    """The sum from packed records: pack, sweep, finalize."""
    from openonda_b200 import _lib

    lib, n = _lib.load(), x.shape[0]
    st = torch.cuda.current_stream().cuda_stream
    rec = torch.empty(n * int(lib.vpm_record_bytes(code)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.vpm_pack_records(x.data_ptr(), a.data_ptr(), s.data_ptr(), v.data_ptr(), n,
                                    code, rec.data_ptr(), st))
    out = [torch.empty_like(x) for _ in range(2)]
    nb = lib.vpm_workspace_bytes(_lib.OPS[op], code, n, n)
    ws = torch.empty(max(nb, 256), dtype=torch.uint8, device="cuda")
    _lib.check(lib.vpm_sweep_records(_lib.OPS[op], rec.data_ptr(), n, 0, n, 0, out[0].data_ptr(),
                                     out[1].data_ptr(), code, ws.data_ptr(), ws.numel(), st))
    return out if op == "velocity_and_strength_gradients" else out[:1]


def _abi(op, x, a, s, v, outs, code):
    from openonda_b200 import _lib

    lib, n = _lib.load(), s.shape[0]
    nb = max(256, lib.vpm_workspace_bytes(_lib.OPS[op], code, n, n))
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    nu = [v.data_ptr()] if op == "strength_gradients_pse" else []
    _lib.check(getattr(lib, "vpm_" + op)(
        x.data_ptr(), a.data_ptr(), s.data_ptr(), *nu, n, *(o.data_ptr() for o in outs), code,
        ws.data_ptr(), nb, torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("n", [300, 2000, 4500])
@pytest.mark.parametrize("op", OPS)
def test_outputs_over_inputs(op, n, precision):
    from openonda_b200 import _lib

    code = _lib.precision_code(precision)
    x, a, s, v = _arrays(n, n)
    want = _from_records(op, x, a, s, v, code)
    two = op == "velocity_and_strength_gradients"
    # every input in turn under the first output, and the outputs over both vectors
    for over in range(4 if op == "strength_gradients_pse" else 3):
        buf = torch.zeros(16 * n, dtype=torch.float64, device="cuda")
        at = {0: (0, 3 * n, 6 * n, 7 * n, 0), 1: (0, 3 * n, 6 * n, 7 * n, 3 * n),
              2: (0, 3 * n, 6 * n, 10 * n, 6 * n - 1), 3: (0, 3 * n, 9 * n, 6 * n, 6 * n)}[over]
        z = []
        for t, k in zip((x, a, s, v), at):
            w = buf[k:k + t.numel()].view(t.shape)
            w.copy_(t)
            z.append(w)
        out = buf[at[4]:at[4] + 3 * n].view(n, 3)
        second = [buf[12 * n:15 * n].view(n, 3) if over else buf[3 * n:6 * n].view(n, 3)] * two
        _abi(op, *z, [out, *second], code)
        for g, r in zip([out, *second], want):
            assert torch.equal(g, r), (op, over)


@pytest.mark.parametrize("n", [300, 2000])
def test_outputs_beside_inputs(n):
    """Outputs that only touch the inputs' ends are no overlap: the bits of the one launch."""
    from openonda_b200 import _lib, kernels

    x, a, s, _ = _arrays(n, 5)
    want = kernels.selfinduced_velocity(x, a, s)
    buf = torch.empty(13 * n, dtype=torch.float64, device="cuda")
    z = [buf[k:k + t.numel()].view(t.shape).copy_(t) for t, k in ((x, 3 * n), (a, 9 * n),
                                                                  (s, 12 * n))]
    for k in (0, 6 * n):
        out = buf[k:k + 3 * n].view(n, 3)
        _abi("selfinduced_velocity", *z, None, [out], _lib.precision_code("fp64"))
        assert torch.equal(out, want)


@pytest.mark.parametrize("m,n", [(700, 700), (1500, 900), (300, 3000)])
def test_probe_outputs_over_inputs(m, n):
    """Probe values over the targets, the positions and the strengths."""
    from openonda_b200 import _lib

    x, a, s, _ = _arrays(n, n)
    t = torch.from_numpy(np.random.default_rng(m).uniform(-1, 1, size=(m, 3))).cuda()
    lib = _lib.load()
    for op, ref in (("induced_velocity_at", oracle.gpu.get_induced_velocity_at),
                    ("vorticity_field_at", oracle.gpu.get_vorticity_field_at)):
        want = ref(*(z.cpu().numpy() for z in (t, x, a, s)))[:m]
        for over in range(3):
            buf = torch.zeros(9 * max(m, n), dtype=torch.float64, device="cuda")
            w = [buf[3 * k * max(m, n):][:z.numel()].view(z.shape).copy_(z)
                 for k, z in enumerate((t, x, a))]
            out = buf[3 * over * max(m, n):][:3 * m].view(m, 3)
            nb = max(256, lib.vpm_workspace_bytes(_lib.OPS[op], 0, m, n))
            ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
            _lib.check(getattr(lib, "vpm_" + op)(
                w[0].data_ptr(), m, w[1].data_ptr(), w[2].data_ptr(), s.data_ptr(), n,
                out.data_ptr(), 0, ws.data_ptr(), nb, torch.cuda.current_stream().cuda_stream))
            assert normwise(out.cpu().numpy(), want) <= 1e-12, (op, over)
