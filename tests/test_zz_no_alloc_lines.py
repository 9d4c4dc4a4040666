"""The allocation-free derivative at the sizes where its tiling can go wrong, against a numpy restatement in the same
operation order (IEEE double, no contraction: the results are equal bit for bit)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AL, BE = 0.5862704032801503, 0.09549533555017055
AA, AB, AC = 0.6431406736919156, 0.2586011023495066, 0.007140953479797375
ROW = ((-3.456878182643609, 5.839043358834730, 1.015886726041007, -0.2246526470654333, 0.08564940889936562,
        -0.01836710059356763),
       (-0.3177447290722621, -0.02807631929593225, 1.593461635747659, 0.2533027046976367, -0.03619652460174756,
        0.004080281419108407),
       (-0.1219006056449124, -0.6301651351188667, 0.6521195063966084, 0.3938843551210350, 0.01904944407973912,
        -0.001027260523947668))
LHS = ((0, 0, 1, 5.912678614078549, 3.775623951744012),
       (0, 0.08360703307833438, 1, 2.058102869495757, 0.9704052014790193),
       (0.03250008295108466, 0.3998040493524358, 1, 0.7719261277615860, 0.1626635931256900))


def factors(n):
    """penta, src/Subroutineso.f90:15-67: l1, l2, u1, u2 u1, u3 u1 per row."""
    l1, l2, u1, u2, u3 = (np.ones(n) for _ in range(5))
    u2[0], u3[0] = LHS[0][3], LHS[0][4]
    l2[1] = LHS[1][1] * u1[0]
    u1[1] = 1.0 / (1.0 - u2[0] * l2[1])
    u2[1], u3[1] = LHS[1][3] - u3[0] * l2[1], LHS[1][4]
    l1[2] = LHS[2][0] * u1[0]
    l2[2] = (LHS[2][1] - u2[0] * l1[2]) * u1[1]
    u1[2] = 1.0 / (1.0 - u3[0] * l1[2] - u2[1] * l2[2])
    u2[2], u3[2] = LHS[2][3] - u3[1] * l2[2], LHS[2][4]
    for i in range(3, n):
        r = n - 1 - i  # rows of the far end mirror rows 2, 1, 0
        b2, b1, f1, f2 = (BE, AL, AL, BE) if r > 2 else (LHS[r][4], LHS[r][3], LHS[r][1], LHS[r][0])
        l1[i] = b2 * u1[i - 2]
        l2[i] = (b1 - u2[i - 2] * l1[i]) * u1[i - 1]
        u1[i] = 1.0 / (1.0 - u3[i - 2] * l1[i] - u2[i - 1] * l2[i])
        if r > 0:
            u2[i] = f1 - u3[i - 1] * l2[i]
        if r > 1:
            u3[i] = f2
    return l1, l2, u1, u2 * u1, u3 * u1


def derivative(f):
    n, m = f.shape
    g = f.T
    l1, l2, c2, c3, c4 = factors(m)
    s = np.zeros((m, n))
    s[3:m - 3] = AA * (g[4:m - 2] - g[2:m - 4]) + AB * (g[5:m - 1] - g[1:m - 5]) + AC * (g[6:] - g[:m - 6])
    for r in range(3):
        others = [q for q in range(7) if q != r]
        a = b = None
        for w, q in zip(ROW[r], others):
            x, y = w * (g[q] - g[r]), w * (g[m - 1 - r] - g[m - 1 - q])
            a, b = (x, y) if a is None else (a + x, b + y)
        s[r], s[m - 1 - r] = a, b
    s[1] = s[1] - l2[1] * s[0]
    for i in range(2, m):
        s[i] = s[i] - l1[i] * s[i - 2] - l2[i] * s[i - 1]
    s = c2[:, None] * s
    s[m - 2] = s[m - 2] - c3[m - 2] * s[m - 1]
    for i in range(m - 3, -1, -1):
        s[i] = s[i] - c3[i] * s[i + 1] - c4[i] * s[i + 2]
    return np.ascontiguousarray(s.T)


@pytest.mark.parametrize("nlines,length", [(1, 7), (5, 8), (4, 9), (33, 129), (40, 97), (2433, 64), (3327, 601),
                                           (200000, 10), (488, 4096), (1, 4096), (781, 2560)])
@pytest.mark.parametrize("in_place", [False, True])
def test_lines_equal_the_restatement(ati_lib, nlines, length, in_place):
    import torch

    from tandemproject_gb300.solver import load_library
    f = np.random.default_rng(length).standard_normal((nlines, length))
    x = torch.from_numpy(f).cuda()
    y = x if in_place else torch.empty_like(x)
    st = torch.cuda.current_stream()
    assert load_library(ati_lib).ati_deriv_lines_noalloc(x.data_ptr(), y.data_ptr(), nlines, length,
                                                         ctypes.c_void_p(st.cuda_stream)) == 0
    assert np.array_equal(y.cpu().numpy(), derivative(f))
