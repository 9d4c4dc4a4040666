"""The allocation-free derivative in captured graphs: a replay finds its own line length's LU factors whatever calls ran
since the capture, and a call finds its own whatever was captured or replayed before it."""
import ctypes

import pytest
from test_zz_no_alloc_lines import derivative

pytestmark = pytest.mark.gpu


class Lines:
    def __init__(self, lib, nlines, length):
        import numpy as np
        import torch
        self.lib, self.shape = lib, (nlines, length)
        self.x = torch.from_numpy(np.random.default_rng(length).standard_normal(self.shape)).cuda()
        self.y = torch.empty_like(self.x)
        self.expected = derivative(self.x.cpu().numpy())

    def call(self):
        import torch
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert self.lib.ati_deriv_lines_noalloc(self.x.data_ptr(), self.y.data_ptr(), *self.shape, st) == 0

    def clear(self):
        self.y.fill_(float("nan"))

    def right(self):
        import numpy as np
        return np.array_equal(self.y.cpu().numpy(), self.expected)


def test_calls_and_replays_of_different_lengths(ati_lib):
    import torch

    from tandemproject_gb300.solver import load_library
    lib = load_library(ati_lib)
    a, b, c = Lines(lib, 33, 64), Lines(lib, 20, 97), Lines(lib, 7, 130)
    a.call()
    torch.cuda.synchronize()
    graphs = {}
    for name, one in (("same", a), ("new", b)):  # the previous call's length, and a new one
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name]):
            one.call()
    for one in (a, b, c):
        one.clear()
    b.call()  # captured with this length, not run with it
    assert b.right()
    c.call()
    graphs["same"].replay()
    assert c.right() and a.right()
    b.clear()
    c.clear()
    graphs["new"].replay()
    c.call()  # the last call's length, with a replay of another since
    graphs["new"].replay()
    assert b.right() and c.right()
