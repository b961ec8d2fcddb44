"""The 2D model's neighbour search and sort where their work is cut: warps whose targets lie in one
cell or in many, lists at and beyond their capacity, particles beyond the grid, both numbers of
targets per warp, and both sorts (few cells per particle or many). The sums run in the
reference's order, so every output is the oracle's bit for bit."""
import numpy as np
import pytest

import oracle
from libcl_gb300 import (BUF2D_CELL, BUF2D_INDEX, BUF2D_PRESSURE, BUF2D_RELAXED, BUF2D_SORTED_STATE, BUF2D_STATE, Fluid2D)
from scenes2d import box_mask

pytestmark = pytest.mark.gpu


def scatter(kind, n, p, rng):
    st = np.zeros((n, 6), np.float32)
    st[:, 4] = 0.7
    st[:, 2:4] = rng.uniform(-1, 1, (n, 2))
    lim = np.array([p.containerW, p.containerH])
    st[:, :2] = rng.uniform(0.02, 0.98, (n, 2)) * lim
    if kind == "clumps":       # up to 150 within a cell, single particles between
        k = 0
        while k < n:
            m = min(n - k, int(rng.integers(1, 151)))
            c = np.floor(rng.uniform(0.1, 0.9, 2) * lim / p.cellSize)
            st[k:k + m, :2] = (c + rng.uniform(0.02, 0.98, (m, 2))) * p.cellSize
            k += m
        st[::7, :2] = rng.uniform(0.02, 0.98, (len(st[::7]), 2)) * lim
    elif kind == "pile":       # all within half the radius of one another
        st[:, :2] = 5.0 + rng.uniform(0, 0.3, (n, 2)) * p.h
    elif kind == "beyond":     # a border of one cell and more around the grid
        st[:, :2] = rng.uniform(-0.05, 1.05, (n, 2)) * lim
    return st


@pytest.mark.parametrize("kind,n,cells", [
    ("even", 2, None), ("even", 33, None), ("even", 5000, None), ("even", 70001, None),
    ("clumps", 3000, None), ("clumps", 66000, None), ("pile", 90, None), ("pile", 300, None),
    ("beyond", 1000, None), ("clumps", 1000, (1024, 512)), ("even", 3000, (300, 250))])
def test_search_and_sort(cuda, kind, n, cells):
    import torch
    f = Fluid2D()
    f.compile()
    p = f.getParameters()
    if cells:
        p.cellCountX, p.cellCountY = cells
    f.setParticleCount(n)
    st = scatter(kind, n, p, np.random.default_rng(n))
    mask = box_mask()
    f.computeBorder(torch.from_numpy(mask).cuda())
    f.getStateBuffer().copy_(torch.from_numpy(st))
    vec, bst = oracle.compute_border_2d(mask, p)
    table = oracle.table_size_2d(p)
    host = st.copy()
    for step in range(2):
        f.compute()
        r = oracle.step_2d(host, p, bst, vec)
        cs, ce = f.cell_bounds(table)
        for got, want in ((f.buffer(BUF2D_CELL), r.cell), (f.buffer(BUF2D_INDEX), r.index), (cs, r.cell_start), (ce, r.cell_end),
                          (f.buffer(BUF2D_SORTED_STATE), r.sorted), (f.buffer(BUF2D_PRESSURE), r.pstate),
                          (f.buffer(BUF2D_RELAXED), r.relaxed), (f.buffer(BUF2D_STATE), host)):
            g = np.ascontiguousarray(got.cpu().numpy()).view(np.uint32).ravel()
            assert np.array_equal(g, np.ascontiguousarray(want).view(np.uint32).ravel()), (step, kind)
    assert f.sync_status() == 0
