"""clCollideBVH where its 256-entry ring of nodes wraps, and for rays the fast box test is not made
for: bit for bit as the oracle's sequential traversal."""
import numpy as np
import pytest

import oracle
from libcl_gb300 import BvhTrimesh, default_params
from libcl_gb300.scenes import triangle_soup

pytestmark = pytest.mark.gpu


# size 0.4: most boxes overlap, so a ray's front outgrows the ring; 0.02: it does not
@pytest.mark.parametrize("n,size", [(3000, 0.4), (700, 0.4), (3000, 0.02), (2, 0.4)])
def test_collide_matches_the_sequential_queue(cuda, n, size):
    import torch
    v, idx = triangle_soup(n, seed=5, extent=1.0, size=size)
    b = BvhTrimesh()
    dv, di = torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    b.compute(dv, di)
    nodes = b.getNodeBuffer().cpu().numpy().view(oracle.BVH_NODE_DTYPE).ravel()
    rng = np.random.default_rng(n)
    m = 4001  # not a multiple of the particles per block
    pos, vel, frc = (np.zeros((m, 4), np.float32) for _ in range(3))
    pos[:, :3] = rng.uniform(-0.2, 1.2, size=(m, 3))
    vel[:, :3] = rng.normal(size=(m, 3)) * 2
    vel[:600, 0] = 0  # infinite inverse directions, some from the boxes' own planes (0 * inf)
    vel[600:900, 1:3] = 0
    vel[900:1000] = 0
    pos[:300, 0] = v[rng.integers(0, 3 * n, 300), 0]
    vel[1000:1010, 0] = np.nan
    pos[1010:1020, 1] = np.inf
    frc[:, 2] = -9.8
    p = default_params()
    got = [torch.from_numpy(a.copy()).cuda() for a in (pos, vel, frc)]
    b.collide(p, *got, dv, di)
    assert b.sync_status() == 0
    want = [a.copy() for a in (pos, vel, frc)]
    oracle.bvh_collide(p, *want, nodes, b.getRootNode(), idx, v)
    for g, w, name in zip(got, want, ("position", "velocity", "force")):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), w.view(np.uint32), err_msg=name)
    if n > 2:
        assert np.any(want[1] != vel)
