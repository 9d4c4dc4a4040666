"""The FP64 fast path's fixed-point fluxes (csrc/ati_fixed_flux.h), compiled for the host, against extended precision.

Errors are taken per component and point, in units of the sum of the magnitudes of the terms that make the component up,
so a component of a small velocity or along a direction of small metrics counts as much as the largest one.  They may be
no larger than the FP64 arithmetic's on the same inputs, in the root mean square over 20,000 points.  The limit is
1 + 2^-8: where a component is one product the FP64 result is correctly rounded, and the integers' own error of some 2^-57
of the result adds that part to the one rounding both share.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tandemproject_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("flux") / "fixed_flux_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "fixed_flux_host.cpp")], check=True)
    return exe


# log2 of: the spread of the directions' metrics, u over w, the spread of the derivatives, the pressure's scale
@pytest.mark.parametrize("spread", [(0, 0, 0, 0), (5, 2, 3, 0), (10, 0, 0, 0), (8, 10, 5, 0), (3, 0, 0, -8), (6, 40, 20, 0),
                                    (0, 12, 0, 5), (20, 100, 60, 30)])
@pytest.mark.parametrize("viscous", [1, 0])
def test_errors_no_larger_than_fp64(program, viscous, spread):
    out = subprocess.run([program, str(viscous), *map(str, spread), "1"], check=True, capture_output=True, text=True)
    ratios = [float(line.split()[3]) for line in out.stdout.splitlines()]
    assert len(ratios) == 15 and max(ratios) <= 1 + 2.0 ** -8, ratios
