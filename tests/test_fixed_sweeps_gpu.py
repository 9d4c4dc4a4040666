"""The fixed-point line sweeps (csrc/ati_fixed.cu) and fluxes (csrc/ati_fixed_flux.h) of the FP64 fast path against the
CPU restatement.

Line lengths sit at the edges of the kernel's segments (48 points a segment, tiles of 32 lines, lines of 13 to 800
points; others take the FP64 sweeps).  The tolerances are those of the FP64 fast build: a filter step adds a
correction rounded well below an ulp of the state (1e-14 of each variable's norm), a stage's right-hand side nearly
cancels, so the state after two steps is held to 1e-12 and a stage's right-hand side to 1e-9 of its largest value.
"""
import numpy as np
import pytest

from conftest import rel_err
from tandemproject_gb300.config import small_case
from tandemproject_gb300.grid import aerofoil_grid

pytestmark = pytest.mark.gpu

# last indices of the blocks' lines: segment edges along xi and eta, ragged tiles; zeta lines of 13, 48, 49 and 97 points
SIZES = [
    ((47, 95, 48), (16, 17), (12,)),
    ((96, 120, 51), (48, 47), (13,)),
    ((24, 64, 31), (16, 95), (48,)),
    ((30, 66, 24), (11, 12), (96,)),
    ((24, 200, 24), (39, 39), (47,)),
    ((799, 800, 60), (17, 16), (12,)),
]


def pair(cfg):
    from oracle.oracle import OracleCase
    from tandemproject_gb300.solver import Case
    g = aerofoil_grid(cfg)
    gpu, orc = Case(cfg), OracleCase(cfg)
    for mb in range(cfg.nblocks):
        gpu.set_grid(mb, g[mb])
        orc.set_grid(mb, g[mb])
    gpu.init()
    orc.init()
    return gpu, orc, g


def smooth_state(xyz, seed):
    """rho, rho u, rho v, rho w, rho E near the freestream, a smooth function of the position (period 0.1 along z)."""
    rng = np.random.default_rng(seed)
    x, y, z = xyz.reshape(3, -1)

    def wave(a):
        k = rng.uniform(-4, 4, 2)
        return a * np.sin(k[0] * x + k[1] * y + 2 * np.pi * z / 0.1 + rng.uniform(0, 6))
    rho, u, v, w = 1 + wave(0.02), wave(0.05), wave(0.05), wave(0.02)
    p = (1 + wave(0.02)) / 1.4
    return np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)])


@pytest.mark.parametrize("lxibk,letbk,lzebk", SIZES)
def test_filter_and_steps_match_oracle(ati_lib, oracle_lib, lxibk, letbk, lzebk):
    cfg = small_case(lxibk=lxibk, letbk=letbk, lzebk=lzebk)
    gpu, orc, g = pair(cfg)
    for mb in range(cfg.nblocks):
        q = smooth_state(g[mb], 7)
        gpu.set_state(mb, q)
        orc.set_state(mb, q)
    gpu.filter_step()
    orc.filter_step()
    for mb in range(cfg.nblocks):
        a, b = gpu.get_state(mb), orc.get_state(mb).reshape(5, -1)
        for m in range(5):
            assert rel_err(a[m], b[m]) < 1e-14, (mb, m)
    gpu.step(2)
    orc.step(2)
    for mb in range(cfg.nblocks):
        a, b = gpu.get_state(mb), orc.get_state(mb).reshape(5, -1)
        for m in range(5):
            assert rel_err(a[m], b[m]) < 1e-12, (mb, m)
    gpu.close()


@pytest.mark.parametrize("scale", [0.0, 1e-300, 1e-160, 1e290])
def test_filter_of_extreme_scales(ati_lib, oracle_lib, scale):
    """Lines of zeros, of values near the ends of the exponent range, and of one value against tiny ones."""
    cfg = small_case(lxibk=(60, 100, 24), letbk=(17, 50), lzebk=(12,))
    gpu, orc, g = pair(cfg)
    for mb in range(cfg.nblocks):
        q = smooth_state(g[mb], 3)
        q[1] *= scale
        q[2] = 1.0
        q[3] = np.where(np.arange(q.shape[1]) % 97 == 5, 1.0, 1e-12 * q[3])
        gpu.set_state(mb, q)
        orc.set_state(mb, q)
    gpu.filter_step()
    orc.filter_step()
    for mb in range(cfg.nblocks):
        a, b = gpu.get_state(mb), orc.get_state(mb).reshape(5, -1)
        for m in range(5):
            assert rel_err(a[m] / max(scale, 1e-307) if m == 1 and scale else a[m],
                           b[m] / max(scale, 1e-307) if m == 1 and scale else b[m]) < 1e-13, (mb, m)
        assert scale or not a[1].any()
    gpu.close()


def test_filter_spreads_a_nan_as_the_oracle_does(ati_lib, oracle_lib):
    cfg = small_case(lxibk=(60, 100, 24), letbk=(17, 50), lzebk=(12,))
    gpu, orc, g = pair(cfg)
    for mb in range(cfg.nblocks):
        q = smooth_state(g[mb], 5)
        if mb == 1:
            q[0, 12345] = np.nan
            q[4, 4321] = np.inf
        gpu.set_state(mb, q)
        orc.set_state(mb, q)
    gpu.filter_step()
    orc.filter_step()
    for mb in range(cfg.nblocks):
        a, b = gpu.get_state(mb), orc.get_state(mb).reshape(5, -1)
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        ok = np.isfinite(b)
        assert rel_err(a[ok], b[ok]) < 1e-14
    gpu.close()


@pytest.mark.parametrize("viscous", [1, 0])
@pytest.mark.parametrize("pressure,speed", [(1.0, 1.0), (1.0, 0.0), (1e-40, 1e-20), (1e66, 1e33)])
def test_right_hand_side_matches_oracle(ati_lib, oracle_lib, viscous, pressure, speed):
    """One stage (dt = 0 before the first step: the state stays) of flows at all scales: within the fixed-point
    fluxes' exponent range, at rest, near its lower end, and beyond the upper one (the FP64 operations)."""
    from tandemproject_gb300.solver import F_DE
    cfg = small_case(lxibk=(30, 70, 24), letbk=(17, 20), lzebk=(12,), nviscous=viscous)
    gpu, orc, g = pair(cfg)
    for mb in range(cfg.nblocks):
        q = smooth_state(g[mb], 11)
        kinetic = 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) / q[0]
        q[4] = (q[4] - kinetic) * pressure + kinetic * speed ** 2
        q[1:4] *= speed
        gpu.set_state(mb, q)
        orc.set_state(mb, q)
    gpu.rk_stage(1)
    orc.rk_stage(1)
    for mb in range(cfg.nblocks):
        a, b = gpu.get_field(mb, F_DE), orc.get_field(mb, F_DE).reshape(5, -1)
        for m in range(5):
            assert rel_err(a[m], b[m]) < 1e-9, (mb, m)
    gpu.close()


@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e25, 1e70])
def test_pressure_matches_oracle_pointwise(ati_lib, oracle_lib, scale):
    """The fixed-point primitives, and the FP64 ones beyond their range (1e70), point by point: p is (gamma - 1) times
    the energy less the kinetic one, 2 to 5 units in the last place with the cancellation of these states."""
    from tandemproject_gb300.solver import F_P
    cfg = small_case(lxibk=(30, 70, 24), letbk=(17, 20), lzebk=(12,))
    gpu, orc, g = pair(cfg)
    for mb in range(cfg.nblocks):
        q = smooth_state(g[mb], 2)
        q[1:4] *= scale ** 0.5
        q[4] *= scale
        gpu.set_state(mb, q)
        orc.set_state(mb, q)
    gpu.rk_stage(1)
    orc.rk_stage(1)
    for mb in range(cfg.nblocks):
        a, b = gpu.get_field(mb, F_P), orc.get_field(mb, F_P).reshape(1, -1)
        assert np.max(np.abs(a / b - 1)) < 1e-14, mb
    gpu.close()


def test_negative_pressure_is_flagged(ati_lib):
    from tandemproject_gb300.solver import ATI_ENONFINITE, AtiError, Case
    cfg = small_case(lxibk=(30, 70, 24), letbk=(17, 20), lzebk=(12,))
    g = aerofoil_grid(cfg)
    gpu = Case(cfg)
    for mb in range(cfg.nblocks):
        gpu.set_grid(mb, g[mb])
    gpu.init()
    q = smooth_state(g[2], 2)
    q[4, 777] = 0.5 * (q[1, 777] ** 2) / q[0, 777] * 0.5
    gpu.set_state(2, q)
    gpu.rk_stage(1)
    with pytest.raises(AtiError) as err:
        gpu.check()
    assert err.value.code == ATI_ENONFINITE
    gpu.close()
