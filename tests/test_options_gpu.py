"""Kernel options that no kernel reads any more cost nothing (GB300)."""
import pytest

pytestmark = pytest.mark.gpu


def test_stress_option_adds_no_launches(ati_lib):
    """The FP64 path's viscous fluxes take the stresses at the point whatever ATI_OPT_STRESS_AT_POINT says: without it a
    step must not write stress planes that nothing reads."""
    from tandemproject_gb300.config import FP64, small_case
    from tandemproject_gb300.solver import setup_case
    h = setup_case(small_case(precision=FP64))
    launches = {}
    for on in (True, False):
        assert h.set_options(stress_at_point=on)["stress_at_point"] is on
        h.step(2)  # (captures the step graphs again)
        before = h.launch_count()
        h.step(2)
        launches[on] = h.launch_count() - before
    h.close()
    assert launches[True] == launches[False] > 0, launches
