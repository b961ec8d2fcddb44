"""The reference-order kernels where a particle has about as many neighbours as its list holds (64), and
one and two lists more: bit for bit the oracle's, for few particles (the warp adds such a particle's
terms up together) and for many (a thread each)."""
import numpy as np
import pytest

import oracle
from fluid_helpers import hash_block, make_fluid, sorted_outputs, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beside", [0, 40000])
@pytest.mark.parametrize("crowd", [65, 66, 67, 96, 97, 98, 128, 129, 130, 161, 193, 194, 257])
def test_lists_about_full(cuda, crowd, beside):
    sc = hash_block(4)
    h = float(sc.params.cellSize)
    rng = np.random.default_rng(crowd)
    n = crowd + beside
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.uniform(-0.9, 0.9, (n, 3))
    pos[:crowd, :3] = (np.array([3, -2, 5]) + rng.uniform(0.25, 0.8, (crowd, 3))) * h  # all in reach of one another
    pos[crowd // 3:crowd // 2, 0] += 0.6 * h  # some of them in the next cell
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.uniform(-1, 1, (n, 3))
    sc.pos, sc.vel = pos, vel
    f = make_fluid(sc, vel=vel)
    f.compute()
    out, st = sorted_outputs(f, 262144), state(f)
    p, v, force = pos.copy(), vel.copy(), np.zeros_like(vel)
    r = oracle.step(p, v, force, sc.params, ref_sort=True)
    for got, want in ((out["spos"], r.spos), (out["svel"], r.svel), (st["pos"], p), (st["vel"], v), (st["force"], force)):
        np.testing.assert_array_equal(got.view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
