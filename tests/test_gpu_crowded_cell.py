"""A cell so crowded that its pairs keep a CTA busy for longer than any wait of the neighbour passes may
last: the step is slow, but complete and without an error."""
import numpy as np
import pytest

from fluid_helpers import make_fluid, sorted_outputs, state
from libcl_gb300 import OK
from libcl_gb300.scenes import Scene3D, fluid_params

pytestmark = pytest.mark.gpu

H = 0.02
GRID = (24, 9, 9)
CROWDED = (9, 4, 4)  # the second cell of a brick of 8: the brick goes on behind it
EPS = 2.0 ** -24


def scene(n_crowd):
    """Four particles a cell, none of them in the crowded cell, and n_crowd there."""
    rng = np.random.default_rng(8)
    cells = np.stack(np.meshgrid(*[np.arange(g) for g in GRID], indexing="ij"), -1).reshape(-1, 3)
    cells = np.repeat(cells[np.any(cells != CROWDED, axis=1)], 4, axis=0)
    base = len(cells)
    pos = np.zeros((base + n_crowd, 4), np.float32)
    pos[:base, :3] = (cells + rng.uniform(0.02, 0.98, (base, 3))) * H
    pos[base:, :3] = (np.array(CROWDED) + rng.uniform(0.02, 0.98, (n_crowd, 3))) * H
    vel = np.zeros_like(pos)
    vel[:, :3] = np.random.default_rng(9).normal(size=(base + 60000, 3))[:len(pos)]
    p = fluid_params(H, 0.01, 1e-3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0), tuple(H * g for g in GRID), GRID,
                     velocity_limit=1e15)
    return Scene3D("crowded", pos, vel, p), base


def test_crowded_cell_is_slow_but_complete(cuda):
    import torch
    sc, base = scene(60000)
    f = make_fluid(sc, vel=sc.vel)
    f.compute()
    assert f.sync_status() == OK
    s = state(f)
    g = sorted_outputs(f, int(np.prod(GRID)))
    p = sc.params

    # three cells and more away nothing tells that the crowded cell is there
    quiet, _ = scene(0)
    q = make_fluid(quiet, vel=quiet.vel)
    q.compute()
    sq = state(q)
    far = np.any(np.abs(np.floor(quiet.pos[:, :3] / np.float32(H)) - np.array(CROWDED)) >= 4, axis=1)
    assert far.sum() > 2000
    for k in ("pos", "vel"):
        np.testing.assert_array_equal(s[k][:base][far].view(np.uint32), sq[k][far].view(np.uint32), err_msg=k)

    # some of the crowd, and some of its neighbours, against 64 bits: densities from the positions,
    # forces from the densities that the step computed. A lane adds up a quarter of the
    # candidates one after the other; a term has some 16 roundings, and its distance to the
    # support radius h is off by as many of h's.
    spos, svel = torch.from_numpy(g["spos"]).cuda().double(), torch.from_numpy(g["svel"]).cuda().double()
    orig = g["index"].astype(np.int64)
    near = np.abs(sc.pos[orig, :3] / H - (np.array(CROWDED) + 0.5)).max(1) < 1.4
    rows = np.nonzero(near)[0]
    rows = np.concatenate([rows[orig[rows] < base][:20], rows[orig[rows] >= base][::1500]])
    adds = len(orig) / 4 + 16
    v0 = torch.from_numpy(sc.vel).cuda().double()[torch.from_numpy(orig).cuda()]
    for i in rows:
        d = spos[i, :3] - spos[:, :3]
        r2 = (d * d).sum(1)
        near_i = (r2 < float(np.float32(H)) ** 2) & (r2 > 0)
        d, r2 = d[near_i], r2[near_i]
        h = float(p.cellSize)
        t = h * h - r2
        rho = p.mass * p.kernelConstant * (t ** 3).sum()
        err = p.mass * p.kernelConstant * (t ** 3 * (adds + 16 * h * h / t)).sum() + p.mass * p.kernelConstant * h ** 6 * 16
        assert abs(float(rho) - g["spos"][i, 3]) <= EPS * float(err), (i, float(rho), g["spos"][i, 3])
        r = r2.sqrt()
        hr, rr = h - r, spos[i, 3] * spos[near_i, 3]
        a = ((svel[i, 3] + svel[near_i, 3]) / rr * hr * hr / r)[:, None] * d * p.pressureConstant
        b = (v0[near_i, :3] - v0[i, :3]) * (hr / rr)[:, None] * p.viscosityConstant
        dv = p.mass * float(p.deltaTime) * (a + b).sum(0)
        tol = p.mass * float(p.deltaTime) * ((a.abs() + b.abs()) * (adds + 32 * h / hr)[:, None]).sum(0)
        got = torch.from_numpy(s["vel"][orig[i], :3]).cuda().double()
        off = (got - (v0[i, :3] + dv)).abs()
        assert bool((off <= EPS * (tol + 8 * got.abs() + 8 * v0[i, :3].abs())).all()), (i, off, tol * EPS)
