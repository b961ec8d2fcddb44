"""Bricks in which staged and crowded cells alternate, so that the force pass changes between its two kinds
of unit many times, also from brick to brick: against the restatement, and bit for bit the same for
every brick width."""
import numpy as np
import pytest

import oracle
from fluid_helpers import RTOL, make_fluid, pos_err, rel_err, sorted_outputs, state
from libcl_gb300 import OK, OPT_BRICK_WIDTH
from libcl_gb300.scenes import Scene3D, fluid_params

pytestmark = pytest.mark.gpu

H = 0.02


# crowd: particles of a crowded cell. 800: its neighbours' windows and its own exceed the force pass's
# staging (768) and not the density pass's; 1100: both. period: a crowded cell every so many along x
@pytest.mark.parametrize("crowd", [800, 1100])
@pytest.mark.parametrize("period,first", [(4, 0), (5, 2), (9, 8), (16, 3), (40, 39)])
def test_alternating_units(cuda, crowd, period, first):
    grid = (40, 4, 4)
    rng = np.random.default_rng(crowd + period)
    cells = np.stack(np.meshgrid(*[np.arange(g) for g in grid], indexing="ij"), -1).reshape(-1, 3)
    cells = np.repeat(cells, rng.integers(0, 4, len(cells)), axis=0)
    crowds = np.array([(x, 1, 2) for x in range(first, grid[0], period)])
    cells = np.concatenate([cells, np.repeat(crowds, crowd, axis=0)])
    pos = np.zeros((len(cells), 4), np.float32)
    pos[:, :3] = (cells + rng.uniform(0.02, 0.98, cells.shape)) * H
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(size=cells.shape) * 0.2
    p = fluid_params(H, 0.01, 1e-5, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0), tuple(H * g for g in grid), grid)
    sc = Scene3D("mixed", pos, vel, p)
    f = make_fluid(sc, vel=vel)
    f.compute()
    g, gs = sorted_outputs(f, oracle.table_cells(p)), state(f)
    assert f.sync_status() == OK
    x, v, frc = pos.copy(), vel.copy(), np.zeros_like(pos)
    r = oracle.step(x, v, frc, p)
    np.testing.assert_array_equal(g["index"], r.index)
    assert rel_err(g["spos"][:, 3], r.spos[:, 3]) < RTOL
    assert rel_err(gs["vel"][:, :3], v[:, :3]) < RTOL
    assert pos_err(gs["pos"][:, :3], x[:, :3], pos[:, :3]) <= 1.0
    np.testing.assert_array_equal(gs["force"], frc)
    for bw in (1, 3, 16):
        b = make_fluid(sc, vel=vel)
        b.set_option(OPT_BRICK_WIDTH, bw)
        b.compute()
        sb = state(b)
        for k in gs:
            np.testing.assert_array_equal(gs[k].view(np.uint32), sb[k].view(np.uint32), err_msg=f"{k}, brick width {bw}")
