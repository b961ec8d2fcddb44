"""The fused step's counting sort at the edges of its tiles and of the rule that chooses it, against
the stable sort of the oracle's keys: sorted keys, permutation and cell bounds, over several steps
(the counts and the table are cleared for the next one by the step itself)."""
import numpy as np
import pytest

import oracle
from fluid_helpers import make_fluid, sorted_outputs, state
from libcl_gb300 import BUF_FORCE, BUF_POSITION, BUF_VELOCITY, KEY_REFERENCE_HASH, OK, Batch3D, SceneDesc
from libcl_gb300.scenes import Scene3D, fluid_params

pytestmark = pytest.mark.gpu

H = 0.02


def cell_keys(pos, params):
    r = oracle.hash(pos, params)
    return np.asarray(r[0] if isinstance(r, tuple) else r).astype(np.int64)


def scattered(n, grid, seed, clump=0):
    """n particles in no order over the grid (some beyond it), `clump` of them in one cell."""
    rng = np.random.default_rng(seed)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(-0.02, 1.02, size=(n, 3)) * np.array(grid) * H
    pos[rng.permutation(n)[:clump], :3] = (np.array(grid) // 2 + 0.5) * H
    p = fluid_params(H, 0.01, 1e-3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0), tuple(H * g for g in grid), tuple(grid))
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(size=(n, 3)) * 200  # half a cell a step: other cells every time
    return Scene3D("scattered", pos, vel, p)


# grids around a tile of 1,024 cells, SCAN_DIRECT (65,536), 2^18 (always taken), 2^20 (larger tiles),
# and 32 cells per particle (beyond: the radix sort)
@pytest.mark.parametrize("n,grid,clump", [(1, (1, 1, 1), 0), (257, (32, 32, 1), 0), (300, (41, 5, 5), 100), (5000, (64, 32, 32), 900),
                                          (5000, (65, 32, 32), 0), (7, (64, 64, 64), 3), (8400, (65, 64, 64), 0), (8100, (65, 64, 64), 0),
                                          (40000, (103, 101, 101), 3000), (600000, (128, 128, 100), 0)])
def test_linear_grid(cuda, n, grid, clump):
    sc = scattered(n, grid, n, clump)
    f = make_fluid(sc, vel=sc.vel)
    cells = oracle.table_cells(sc.params)
    for _ in range(3):  # eager, captured, replayed
        before = state(f)["pos"]
        f.compute()
        g = sorted_outputs(f, cells)
        key = cell_keys(before, sc.params)
        order = np.argsort(key, kind="stable")
        np.testing.assert_array_equal(g["cell"], key[order])
        np.testing.assert_array_equal(g["index"], order)
        start = np.searchsorted(g["cell"], np.arange(cells)).astype(np.uint32)
        end = np.searchsorted(g["cell"], np.arange(cells), side="right").astype(np.uint32)
        empty = start == end
        start[empty] = end[empty] = 0xFFFFFFFF
        np.testing.assert_array_equal(g["cell_start"], start)
        np.testing.assert_array_equal(g["cell_end"], end)
        np.testing.assert_array_equal(g["spos"][:, :3], before[order, :3])
        assert f.sync_status() == OK


@pytest.mark.parametrize("n", [1, 255, 3000, 530000])
def test_hashed_keys(cuda, n):
    sc = scattered(n, (50, 50, 50), n, n // 10 if n < 10000 else 0)
    sc.params.keyMode = KEY_REFERENCE_HASH
    f = make_fluid(sc, vel=sc.vel)
    for _ in range(3):
        before = state(f)["pos"]
        f.compute()
        g = sorted_outputs(f, 262144)
        key = cell_keys(before, sc.params)
        order = np.argsort(key, kind="stable")
        np.testing.assert_array_equal(g["index"], order)
        start = np.searchsorted(key[order], np.arange(262144)).astype(np.uint32)
        empty = start == np.searchsorted(key[order], np.arange(262144), side="right")
        start[empty] = 0xFFFFFFFF
        np.testing.assert_array_equal(g["cell_start"], start)
        assert f.sync_status() == OK


def test_both_key_modes_and_grids_on_one_handle(cuda):
    """Changing the key mode and the grid between steps leaves no stale counts or cells behind."""
    sc = scattered(3000, (30, 20, 10), 5)
    f = make_fluid(sc, vel=sc.vel)
    for mode, grid in ((1, (30, 20, 10)), (0, None), (1, (30, 20, 10)), (1, (200, 200, 50)), (1, (12, 9, 8)), (0, None), (1, (30, 20, 10))):
        p = f.getParameters()
        p.keyMode = mode
        for i in range(3):
            if grid:
                p.gridDim[i] = grid[i]
        for _ in range(2):
            before = state(f)["pos"]
            f.compute()
            key = cell_keys(before, p)
            np.testing.assert_array_equal(f.getIndexBuffer().cpu().numpy().view(np.uint32), np.argsort(key, kind="stable"))
            assert f.sync_status() == OK


def test_batch_beyond_the_rule_equals_its_scenes(cuda):
    """A batch with more than 32 cells per particle (radix sort) and one with fewer, bit for bit alike."""
    import torch
    sc = scattered(400, (10, 10, 10), 3)
    out = []
    for grid in ((10, 10, 10), (10, 10, 4000)):  # the same cells occupied, the second grid far longer
        d = SceneDesc()
        d.n_particles, d.stiffness, d.viscosity = 400, 3.0, 0.05
        for i in range(3):
            d.boxMin[i], d.boxMax[i], d.gridOrigin[i], d.gridDim[i] = 0.0, sc.params.boxMax[i], 0.0, grid[i]
        b = Batch3D()
        b.set_scenes(sc.params, [d])
        b.buffer(BUF_POSITION).copy_(torch.from_numpy(np.minimum(sc.pos, np.float32(9.9 * H))))
        b.buffer(BUF_VELOCITY).zero_()
        b.buffer(BUF_FORCE).zero_()
        for _ in range(3):
            b.compute()
        assert b.sync_status() == OK
        out.append([b.buffer(w).cpu().numpy().view(np.uint32) for w in (BUF_POSITION, BUF_VELOCITY, 5)])
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
