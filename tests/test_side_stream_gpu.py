"""The both-sides sums run their diagonal tiles on a second stream of the library.  While a
caller's stream is being captured that stream is part of the capture; a call on another stream
must neither join it nor fail, and the capture must stay whole."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class Call:
    """A self-induced velocity through the C ABI on memory of its own."""

    def __init__(self, n, precision, compact):
        from openonda_b200 import _lib, configs

        f = configs.random_cloud(n, seed=n)
        self.arrays = [torch.from_numpy(np.ascontiguousarray(z)).cuda()
                       for z in (f.positions, f.strengths, f.radii * 4)]
        self.n, self.lib = n, _lib.load()
        self.code = _lib.precision_code(precision) | (_lib.COMPACT_WORKSPACE if compact else 0)
        self.nbytes = self.lib.vpm_workspace_bytes(_lib.OPS["selfinduced_velocity"], self.code,
                                                   n, n)
        self.ws = torch.empty(self.nbytes, dtype=torch.uint8, device="cuda")
        self.out = torch.zeros((n, 3), dtype=torch.float64, device="cuda")

    def __call__(self, stream):
        from openonda_b200 import _lib

        x, a, s = self.arrays
        _lib.check(self.lib.vpm_selfinduced_velocity(
            x.data_ptr(), a.data_ptr(), s.data_ptr(), self.n, self.out.data_ptr(), self.code,
            self.ws.data_ptr(), self.nbytes, stream.cuda_stream))


@pytest.mark.parametrize("compact", [False, True])  # the triangle; several launches
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_call_beside_a_capture(precision, compact):
    from openonda_b200 import kernels

    prev = kernels.set_symmetric_min_n(0)
    try:
        one, two = Call(2100, precision, compact), Call(2300, precision, compact)
        st, other = torch.cuda.Stream(), torch.cuda.Stream()
        refs = []
        torch.cuda.synchronize()
        for c in (one, two):
            c(st)
            torch.cuda.synchronize()
            refs.append(c.out.clone())
            c.out.zero_()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st, capture_error_mode="relaxed"):
            one(torch.cuda.current_stream())
            two(other)  # not captured: runs now
            one(torch.cuda.current_stream())  # the capture goes on
        torch.cuda.synchronize()
        assert torch.equal(two.out, refs[1]) and not one.out.any()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(one.out, refs[0])
        one.out.zero_()
        one(other)  # and the second stream is free again
        torch.cuda.synchronize()
        assert torch.equal(one.out, refs[0])
    finally:
        kernels.set_symmetric_min_n(prev)
    assert kernels.device_errors() == 0
