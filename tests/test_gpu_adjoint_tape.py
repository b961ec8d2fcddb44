"""The adjoint's tape: gradients from the steps forward() recorded and from recomputed ones are the
same bit for bit, whatever the number of segments, also when the fluid has moved on in between."""
import numpy as np
import pytest

from libcl_gb300 import Adjoint3D
from libcl_gb300.scenes import differentiable_block, perturbed_velocities

from fluid_helpers import make_fluid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,every", [(1, 1), (4, 4), (5, 2), (3, 8), (6, 3)])
def test_recorded_and_recomputed_steps(cuda, steps, every):
    import torch
    sc = differentiable_block(16, 9, 11)
    f = make_fluid(sc, vel=perturbed_velocities(sc.vel))
    adj = Adjoint3D(f, steps, every)
    adj.forward()
    pos, vel = f.getPositionBuffer().clone(), f.getVelocityBuffer().clone()
    g = torch.zeros_like(pos)
    g[:, :3] = pos[:, :3] - 0.1
    first = adj.backward(g, vel)       # the last segment as forward() left it
    again = adj.backward(g, vel)       # recomputed, unless it is the only one
    for _ in range(2):
        f.compute()                    # the fluid's own buffers hold another step now
    f.getPositionBuffer().copy_(pos)
    f.getVelocityBuffer().copy_(vel)
    third = adj.backward(g, vel)
    # the oracle for the tape itself: the same steps, each a segment of its own, so that all but
    # the last are recomputed from checkpoints
    h = make_fluid(sc, vel=perturbed_velocities(sc.vel))
    single = Adjoint3D(h, steps, 1)
    single.forward()
    assert torch.equal(h.getPositionBuffer(), pos) and torch.equal(h.getVelocityBuffer(), vel)
    other = single.backward(g, vel)
    for k in range(3):
        a = first[k].cpu().numpy()
        assert np.isfinite(a).all() and np.abs(a).max() > 0
        for r in (again, third, other):
            assert np.array_equal(a, r[k].cpu().numpy()), k


@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 70000])
def test_parameter_sums(cuda, n):
    """The parameters' gradients, per-particle terms summed in shares: repeatable and independent
    of the checkpoints at every number of shares."""
    import torch
    sc = differentiable_block(70, 25, 40)
    sc.pos, sc.vel = sc.pos[:n].copy(), sc.vel[:n].copy()
    out = []
    for every in (1, 2):
        f = make_fluid(sc, vel=perturbed_velocities(sc.vel))
        adj = Adjoint3D(f, 2, every)
        adj.forward()
        g = torch.ones_like(f.getPositionBuffer())
        out += [adj.backward(g)[2].cpu().numpy() for _ in range(2)]
    for o in out:
        assert np.isfinite(o).all() and np.array_equal(o, out[0])
