"""The reference-order density and force kernels where their work is cut: warps whose targets
lie in many cells or in one, candidate batches that fill and overflow what a warp holds, lists at
and beyond their capacity, and both numbers of targets per warp. The sums run in the reference's
order, so every output is the oracle's bit for bit."""
import numpy as np
import pytest

import oracle
from fluid_helpers import hash_block, make_fluid, sorted_outputs, state

pytestmark = pytest.mark.gpu
BUCKETS = 262144


def positions(kind, n, h, rng):
    p = np.ones((n, 4), np.float32)
    if kind == "sparse":            # a cell each, most without any neighbour
        p[:, :3] = rng.uniform(-0.9, 0.9, (n, 3))
    elif kind == "one cell":        # every particle a candidate of every other, all lists overflow
        p[:, :3] = rng.uniform(0.1 * h, 0.9 * h, (n, 3))
    elif kind == "wide cell":       # many candidates of one cell, few of them in range
        p[:, 0] = rng.uniform(0.0, 0.99 * h, n)
        p[:, 1:3] = rng.choice([0.01, 0.99], (n, 2)) * h
    else:                           # "mixed": clumps of 1 to 70 in one cell each, single particles between
        k = 0
        while k < n:
            m = min(n - k, int(rng.integers(1, 71)))
            c = np.floor(rng.uniform(-0.8, 0.8, 3) / h)
            p[k:k + m, :3] = (c + rng.uniform(0.02, 0.98, (m, 3))) * h
            k += m
        p[::9, :3] = rng.uniform(-0.9, 0.9, (len(p[::9]), 3))
    return p


@pytest.mark.parametrize("dims", [3, 2])
@pytest.mark.parametrize("kind", ["sparse", "one cell", "wide cell", "mixed"])
@pytest.mark.parametrize("n", [3, 31, 33, 129, 700, 8193, 32769, 49153])
def test_reference_order_kernels(cuda, kind, n, dims):
    if n > 1000 and kind in ("one cell", "wide cell"):
        pytest.skip("all pairs of one cell")
    sc = hash_block(4)
    sc.params.dims = dims
    h = float(sc.params.cellSize)
    rng = np.random.default_rng(n + dims)
    sc.pos = positions(kind, n, h, rng)
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.uniform(-1, 1, (n, 3))
    sc.vel = vel
    f = make_fluid(sc, fused=True, vel=vel)
    g = make_fluid(sc, fused=False, vel=vel)
    f.compute()
    g.compute()
    pos, v, force = sc.pos.copy(), vel.copy(), np.zeros_like(vel)
    r = oracle.step(pos, v, force, sc.params, ref_sort=True)
    for fl in (f, g):
        out, st = sorted_outputs(fl, BUCKETS), state(fl)
        for name, want in (("spos", r.spos), ("svel", r.svel)):
            assert np.array_equal(out[name].view(np.uint32), want.view(np.uint32)), name
        for name, want in (("pos", pos), ("vel", v), ("force", force)):
            assert np.array_equal(st[name].view(np.uint32), want.view(np.uint32)), name


@pytest.mark.parametrize("n", [31, 5000, 40000])
def test_forces_left_to_a_hook(cuda, n):
    """With an integrate hook the fused step leaves the force before clipping: as the staged step's."""
    sc = hash_block(4)
    rng = np.random.default_rng(n)
    sc.pos = positions("mixed", n, float(sc.params.cellSize), rng)
    vel = np.zeros((n, 4), np.float32)
    vel[:, :3] = rng.uniform(-1, 1, (n, 3))
    sc.vel = vel
    force = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    out = []
    for fused in (True, False):
        f = make_fluid(sc, fused=fused, vel=vel, force=force)
        f.addEventHandler(lambda fluid, stream: 0)
        f.compute()
        out.append(state(f))
    for name in ("pos", "vel", "force"):
        assert np.array_equal(out[0][name].view(np.uint32), out[1][name].view(np.uint32)), name
    assert not np.array_equal(out[0]["force"], force)
