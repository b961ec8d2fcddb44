"""The 2D model's search on either side of the particle counts at which a warp's targets change (one, two,
four), with targets at and beyond their lists' capacity: bit for bit the oracle's."""
import numpy as np
import pytest

import oracle
from libcl_gb300 import BUF2D_PRESSURE, BUF2D_RELAXED, BUF2D_STATE, Fluid2D
from scenes2d import box_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 131, 4095, 4096, 4097, 8191, 8192, 8193])
@pytest.mark.parametrize("crowd", [0, 33, 64, 65, 66, 97, 130])
def test_targets_per_warp(cuda, n, crowd):
    import torch
    if crowd >= n:
        pytest.skip("more in the crowd than particles")
    f = Fluid2D()
    f.compile()
    p = f.getParameters()
    f.setParticleCount(n)
    rng = np.random.default_rng(n + crowd)
    st = np.zeros((n, 6), np.float32)
    st[:, 4] = 0.7
    st[:, 2:4] = rng.uniform(-1, 1, (n, 2))
    st[:, :2] = rng.uniform(0.02, 0.98, (n, 2)) * np.array([p.containerW, p.containerH])
    st[:crowd, :2] = 6.0 + rng.uniform(0, 0.6, (crowd, 2)) * p.h  # about all of one another's neighbours
    st = st[rng.permutation(n)]
    mask = box_mask()
    f.computeBorder(torch.from_numpy(mask).cuda())
    f.getStateBuffer().copy_(torch.from_numpy(st))
    vec, bst = oracle.compute_border_2d(mask, p)
    f.compute()
    host = st.copy()
    r = oracle.step_2d(host, p, bst, vec)
    for got, want in ((f.buffer(BUF2D_PRESSURE), r.pstate), (f.buffer(BUF2D_RELAXED), r.relaxed), (f.buffer(BUF2D_STATE), host)):
        g = np.ascontiguousarray(got.cpu().numpy()).view(np.uint32).ravel()
        assert np.array_equal(g, np.ascontiguousarray(want).view(np.uint32).ravel())
    assert f.sync_status() == 0
