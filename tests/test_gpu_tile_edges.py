"""Sizes at which the counting sort's scan and the BVH's tree kernel change their way: one tile of 1,024
cells, 16,384 cells (sums of tiles from there on), both with more particles than the comparison
sort takes, and one, two and three blocks of 128 leaves."""
import numpy as np
import pytest

import oracle
from fluid_helpers import make_fluid, sorted_outputs, state
from libcl_gb300 import BUF2D_CELL, BUF2D_INDEX, BUF2D_STATE, OK, BvhLines, Fluid2D
from scenes2d import box_mask
from test_gpu_bvh_tree import check, test_triangles as tree_of_triangles
from test_gpu_count_sort import cell_keys, scattered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(33, 31, 1), (32, 32, 1), (41, 25, 1), (129, 127, 1), (128, 128, 1), (145, 113, 1)])
@pytest.mark.parametrize("n,clump", [(2049, 0), (4000, 900)])
def test_counting_sort_on_a_grid(cuda, n, clump, grid):
    sc = scattered(n, grid, n, clump)
    f = make_fluid(sc, vel=sc.vel)
    cells = oracle.table_cells(sc.params)
    for _ in range(3):  # eager, captured, replayed
        before = state(f)["pos"]
        f.compute()
        g = sorted_outputs(f, cells)
        key = cell_keys(before, sc.params)
        order = np.argsort(key, kind="stable")
        np.testing.assert_array_equal(g["index"], order)
        start = np.searchsorted(key[order], np.arange(cells)).astype(np.uint32)
        end = np.searchsorted(key[order], np.arange(cells), side="right").astype(np.uint32)
        empty = start == end
        start[empty] = end[empty] = 0xFFFFFFFF
        np.testing.assert_array_equal(g["cell_start"], start)
        np.testing.assert_array_equal(g["cell_end"], end)
        assert f.sync_status() == OK


@pytest.mark.parametrize("cells", [(128, 127), (128, 128), (129, 128)])  # tables of 16,384, 16,640 and 16,640 words
def test_counting_sort_in_2d(cuda, cells):
    import torch
    n = 3000
    f = Fluid2D()
    f.compile()
    p = f.getParameters()
    p.cellCountX, p.cellCountY = cells
    f.setParticleCount(n)
    rng = np.random.default_rng(cells[0])
    st = np.zeros((n, 6), np.float32)
    st[:, 4] = 0.7
    st[:, :2] = rng.uniform(0.02, 0.98, (n, 2)) * np.array([p.containerW, p.containerH])
    mask = box_mask()
    f.computeBorder(torch.from_numpy(mask).cuda())
    f.getStateBuffer().copy_(torch.from_numpy(st))
    vec, bst = oracle.compute_border_2d(mask, p)
    host = st.copy()
    for _ in range(2):
        f.compute()
        r = oracle.step_2d(host, p, bst, vec)
        cs, ce = f.cell_bounds(oracle.table_size_2d(p))
        for got, want in ((f.buffer(BUF2D_CELL), r.cell), (f.buffer(BUF2D_INDEX), r.index), (cs, r.cell_start), (ce, r.cell_end),
                          (f.buffer(BUF2D_STATE), host)):
            g = np.ascontiguousarray(got.cpu().numpy()).view(np.uint32).ravel()
            assert np.array_equal(g, np.ascontiguousarray(want).view(np.uint32).ravel())
    assert f.sync_status() == OK


LEAVES = (127, 128, 129, 130, 255, 256, 257, 383, 384, 385)


@pytest.mark.parametrize("size", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("n", LEAVES)
def test_trees_of_triangles(cuda, n, size):
    tree_of_triangles(cuda, n, size)


@pytest.mark.parametrize("run", [2, 3, 40, 200])
@pytest.mark.parametrize("n", LEAVES)
def test_repeated_keys_across_the_blocks_edge(cuda, n, run):
    """Runs of `run` equal keys, one of them over each block's edge."""
    import torch
    rng = np.random.default_rng(n + run)
    at = (np.arange(n) + run // 2) // run * 3 + 10
    mid = np.stack([at, at], 1).astype(np.float32)
    d = rng.uniform(-4, 4, size=(n, 2)).astype(np.float32)
    perm = rng.permutation(n)
    v = np.stack([mid - d, mid + d], 1)[perm].reshape(2 * n, 2)
    b = BvhLines()
    b.compute(torch.from_numpy(v).cuda())
    assert b.sync_status() == OK
    o, root, _, _ = oracle.bvh_lines_build(v, 0)
    check(b.getNodeBuffer().cpu().numpy().view(oracle.BVH2D_NODE_DTYPE).ravel(), o, b.getRootNode(), root, n, 3)
