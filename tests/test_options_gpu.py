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


def test_eta_tiles_are_timed_where_fp64_sweeps_remain(ati_lib):
    """Lines of under 13 and over 800 points stay with the FP64 eta sweeps, whose lines a CTA ati_init times on the handle's
    own grid: lines of 851 or 901 points leave shared memory at the default of 128, and fewer lines a CTA are faster by
    more than the 3 % that a candidate has to be."""
    from tandemproject_gb300.config import FP64, CaseConfig
    from tandemproject_gb300.solver import Case
    import numpy as np
    from tandemproject_gb300.grid import aerofoil_grid
    eta = []
    for lxibk, letbk, lzebk in (((24, 64, 24), (850, 850), (40,)), ((60, 120, 60), (10, 900), (12,))):
        cfg = CaseConfig(lxibk=lxibk, letbk=letbk, lzebk=lzebk, precision=FP64)
        h = Case(cfg)
        for mb, xyz in enumerate(aerofoil_grid(cfg)):
            h.set_grid(mb, np.ascontiguousarray(xyz))
        h.init()
        eta.append(h.tiles()[1])
        h.close()
    assert any(n != 128 for n in eta), eta
