"""The allocation-free derivative of short lines, around the sizes where one thread a line takes over from the tiles (lines
of up to 2 n + 4 points where a tile holds n lines, 4 to 32 of them), against the numpy restatement: equal bit for bit."""
import ctypes

import numpy as np
import pytest
from test_zz_no_alloc_lines import derivative

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlines", [1, 127, 129, 2432, 2433, 4864, 4865, 9728, 9729, 25000])
@pytest.mark.parametrize("length", [7, 8, 11, 12, 13, 20, 21, 36, 37, 68, 69])
@pytest.mark.parametrize("in_place", [False, True])
def test_short_lines_equal_the_restatement(ati_lib, nlines, length, in_place):
    import torch

    from tandemproject_gb300.solver import load_library
    f = np.random.default_rng(length).standard_normal((nlines, length))
    x = torch.from_numpy(f).cuda()
    y = x if in_place else torch.empty_like(x)
    st = torch.cuda.current_stream()
    assert load_library(ati_lib).ati_deriv_lines_noalloc(x.data_ptr(), y.data_ptr(), nlines, length,
                                                         ctypes.c_void_p(st.cuda_stream)) == 0
    assert np.array_equal(y.cpu().numpy(), derivative(f))
