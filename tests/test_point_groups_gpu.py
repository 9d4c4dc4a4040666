"""Pointwise kernels over groups of points (GB300): where the handle's number of points is even the mixed path takes
pairs, where it is odd single points, and a tile that begins or ends inside a pair stores its own points only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases(precision):
    from tandemproject_gb300.config import small_case
    odd = dict(lxibk=(24, 64, 30), letbk=(16, 15), lzebk=(12,), precision=precision)   # 121 x 33 x 13 points
    even = dict(lxibk=(24, 64, 30), letbk=(16, 16), lzebk=(12,), precision=precision)
    return small_case(**odd), small_case(mach=0.3, aoa_deg=3.0, **odd), small_case(mach=0.25, **even)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("order", [(0, 1), (0, 2), (2, 0, 1), (1, 2, 0, 0)])
def test_pairs_across_odd_cases(ati_lib, precision, order):
    """Cases of odd and even sizes in one handle (pairs, or single points where the sum is odd; blocks and cases that
    begin on odd points) evolve bit for bit as alone."""
    from tandemproject_gb300.solver import setup_batch, setup_case
    base = _cases(precision)
    cfgs = [base[k] for k in order]
    b = setup_batch(cfgs)
    b.step(6)
    for cs, cfg in enumerate(cfgs):
        a = setup_case(cfg)
        a.step(6)
        for mb, q in enumerate(b.case_state(cs)):
            np.testing.assert_array_equal(q, a.get_state(mb))
        a.close()
    b.close()
