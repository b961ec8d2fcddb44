"""clCollideBVH with trees of few nodes, which take fewer lanes a particle and a smaller ring: on either
side of the node and particle counts where that changes, bit for bit the oracle's traversal."""
import numpy as np
import pytest

import oracle
from libcl_gb300 import BvhTrimesh, default_params
from libcl_gb300.scenes import triangle_soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 131, 65535, 65536, 65537])
@pytest.mark.parametrize("n", [2, 3, 8, 9, 33, 63, 64, 65])
def test_collide_with_few_triangles(cuda, n, m):
    import torch
    v, idx = triangle_soup(n, seed=n, extent=1.0, size=0.6)
    b = BvhTrimesh()
    dv, di = torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    b.compute(dv, di)
    nodes = b.getNodeBuffer().cpu().numpy().view(oracle.BVH_NODE_DTYPE).ravel()
    rng = np.random.default_rng(n + m)
    pos, vel, frc = (np.zeros((m, 4), np.float32) for _ in range(3))
    pos[:, :3] = rng.uniform(-0.2, 1.2, size=(m, 3))
    vel[:, :3] = rng.normal(size=(m, 3)) * 2
    vel[::17] = 0
    vel[5::19, 0] = 0
    frc[:, 2] = -9.8
    p = default_params()
    got = [torch.from_numpy(a.copy()).cuda() for a in (pos, vel, frc)]
    b.collide(p, *got, dv, di)
    assert b.sync_status() == 0
    want = [a.copy() for a in (pos, vel, frc)]
    oracle.bvh_collide(p, *want, nodes, b.getRootNode(), idx, v)
    for g, w, name in zip(got, want, ("position", "velocity", "force")):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint32), w.view(np.uint32), err_msg=name)
    if m > 60000 and n > 2:
        assert np.any(want[1] != vel)
