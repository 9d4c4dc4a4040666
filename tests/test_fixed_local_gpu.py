"""The FP64 fast path's fixed-point filter sweeps (GB300) where a field falls along its lines: every point as accurate as its
neighbourhood allows, not only the line's largest values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lxibk,letbk", [((47, 120, 60), (16, 17)), ((200, 96, 30), (48, 24)), ((24, 64, 31), (95, 60))])
@pytest.mark.parametrize("along", [1, 2])
def test_filter_of_falling_fields(ati_lib, oracle_lib, lxibk, letbk, along):
    """Momentum components that fall by a third of a bit a row along xi or eta, to 2^-40: filtered, they agree with the CPU
    restatement to 64 units in the last place of the largest value within six rows.  (Both round a handful of times in
    each of the three directions; a third of a bit a row is a factor of 4 over six rows.)"""
    from oracle.oracle import OracleCase
    from tandemproject_gb300.config import small_case
    from tandemproject_gb300.grid import aerofoil_grid
    from tandemproject_gb300.solver import Case
    cfg = small_case(lxibk=lxibk, letbk=letbk, lzebk=(12,))
    g = aerofoil_grid(cfg)
    gpu, orc = Case(cfg), OracleCase(cfg)
    for mb in range(cfg.nblocks):
        gpu.set_grid(mb, g[mb])
        orc.set_grid(mb, g[mb])
    gpu.init()
    orc.init()
    rng = np.random.default_rng(1)
    local = {}
    for mb in range(cfg.nblocks):
        nx, ny, nz = (v + 1 for v in gpu.dims[mb][:3])
        i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
        row = i if along == 1 else j
        q = np.ones((5, nz, ny, nx))
        for m, down in ((1, row), (2, row.max() - row), (3, np.abs(row - row.max() // 2))):
            amp = np.exp2(-np.minimum(down, 120) / 3.0)
            wave = 1 + 0.2 * np.sin(0.3 * i + rng.uniform(0, 6)) * np.sin(0.2 * j + rng.uniform(0, 6))
            q[m] = (amp * wave + 0.0 * k).transpose(2, 1, 0)
        gpu.set_state(mb, q.reshape(5, -1))
        orc.set_state(mb, q.reshape(5, -1))
        near = np.abs(q)
        axis = 3 if along == 1 else 2
        wide = near.copy()
        for d in range(1, 7):
            lo, hi = [slice(None)] * 4, [slice(None)] * 4
            lo[axis], hi[axis] = slice(None, -d), slice(d, None)
            wide[tuple(lo)] = np.maximum(wide[tuple(lo)], near[tuple(hi)])
            wide[tuple(hi)] = np.maximum(wide[tuple(hi)], near[tuple(lo)])
        local[mb] = wide.reshape(5, -1)
    gpu.filter_step()
    orc.filter_step()
    for mb in range(cfg.nblocks):
        a, b = gpu.get_state(mb), orc.get_state(mb).reshape(5, -1)
        worst = np.max(np.abs(a - b) / local[mb], axis=1)
        assert np.all(worst < 64 * 2.0 ** -53), (mb, worst * 2.0 ** 53)
    gpu.close()
