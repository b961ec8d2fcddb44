"""The tree kernel of both BVHs around the edges of its 256-leaf blocks, with distinct and with
repeated Morton keys: links, split bits, primitives and root as in the oracle's sequential run,
and every reachable node's box the union of its children's, bit for bit."""
import numpy as np
import pytest

import oracle
from libcl_gb300 import BvhLines, BvhTrimesh

pytestmark = pytest.mark.gpu

SIZES = (2, 3, 255, 256, 257, 258, 511, 513, 1500)


def check(g, o, root, want_root, n, trav):
    for f in ("left", "right", "bit"):
        np.testing.assert_array_equal(g[f], o[f], err_msg=f)
    assert root == want_root
    todo, seen = [root], 0
    while todo:
        i = todo.pop()
        seen += 1
        if i >= n - 1:
            continue
        l, r = int(g["left"][i]), int(g["right"][i])
        np.testing.assert_array_equal(g["bbMin"][i], np.minimum(g["bbMin"][l], g["bbMin"][r]))
        np.testing.assert_array_equal(g["bbMax"][i], np.maximum(g["bbMax"][l], g["bbMax"][r]))
        assert g["trav"][i] == trav
        todo += [l, r]
    assert seen >= 2
    return seen


@pytest.mark.parametrize("spread", [1, 2, 12, 30000])
@pytest.mark.parametrize("n", SIZES)
def test_lines(cuda, n, spread):
    import torch
    rng = np.random.default_rng(n * 31 + spread)
    mid = rng.integers(0, spread, size=(n, 2)).astype(np.float32) + 8
    d = rng.uniform(-4, 4, size=(n, 2)).astype(np.float32)
    v = np.stack([mid - d, mid + d], 1).reshape(2 * n, 2)
    b = BvhLines()
    b.compute(torch.from_numpy(v).cuda())
    assert b.sync_status() == 0
    o, root, sk, _ = oracle.bvh_lines_build(v, 0)
    g = b.getNodeBuffer().cpu().numpy().view(oracle.BVH2D_NODE_DTYPE).ravel()
    seen = check(g, o, b.getRootNode(), root, n, 3)
    for k in range(n):
        s = int(g["bit"][n - 1 + k])
        np.testing.assert_array_equal(g["bbMin"][n - 1 + k], v[2 * s:2 * s + 2].min(0))
        np.testing.assert_array_equal(g["bbMax"][n - 1 + k], v[2 * s:2 * s + 2].max(0))
    if len(np.unique(sk)) == n:
        assert seen == 2 * n - 1


@pytest.mark.parametrize("size", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("n", SIZES)
def test_triangles(cuda, n, size):
    """size 0: all triangles in one spot next to a far one, 0.02: many to a Morton cell."""
    import torch
    rng = np.random.default_rng(n * 7 + int(size * 100))
    c = rng.uniform(0, max(size, 1e-4), size=(n, 1, 3))
    c[0] = 1.0
    v = np.zeros((3 * n, 4), np.float32)
    v[:, :3] = (c + rng.uniform(-0.001, 0.001, size=(n, 3, 3))).reshape(3 * n, 3)
    idx = np.arange(3 * n, dtype=np.uint32)
    b = BvhTrimesh()
    b.compute(torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda())
    assert b.sync_status() == 0
    o, root, sk, _ = oracle.bvh_build(v, idx, np.zeros(8, np.float32), 0)
    g = b.getNodeBuffer().cpu().numpy().view(oracle.BVH_NODE_DTYPE).ravel()
    seen = check(g, o, b.getRootNode(), root, n, 2)
    for k in range(n):
        t = int(g["bit"][n - 1 + k])
        np.testing.assert_array_equal(g["bbMin"][n - 1 + k], v[3 * t:3 * t + 3].min(0))
        np.testing.assert_array_equal(g["bbMax"][n - 1 + k], v[3 * t:3 * t + 3].max(0))
    if len(np.unique(sk)) == n:
        assert seen == 2 * n - 1
