"""Forces of targets whose candidates do not fit the staging: reciprocals of the densities are
correctly rounded there."""
import numpy as np
import pytest

import oracle
from fluid_helpers import make_fluid, sorted_outputs, state
from libcl_gb300 import OK
from libcl_gb300.scenes import Scene3D, fluid_params

pytestmark = pytest.mark.gpu

H = 0.02
f32 = np.float32


@pytest.mark.parametrize("na", [1024, 800])
def test_reciprocals_of_unstaged_targets_are_correctly_rounded(cuda, na):
    """A pile of coincident particles at rest, and d = 2^-7 along x, in the same cell, four at speed
    (0, 1, 0): one for each of the lanes that share a target. All pairs that count are alike, so
    the pile's viscosity along y, restated in float32 with 1 / rho correctly rounded, is met to
    the bit. The one thing unknown is the approximate root of r^2 = 2^-14, the same in every
    run: 2^7 within 4 units in the last place."""
    n, d = na + 4, 2.0 ** -7
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = 0.0625
    pos[na:, 0] += d
    vel = np.zeros_like(pos)
    vel[na:, 1] = 1.0
    r2 = 2.0 ** -14
    roots = {f32(2.0 ** 7) + f32(j) * np.spacing(f32(2.0 ** 7)) / (f32(2) if j < 0 else f32(1)) for j in range(-8, 5)}
    p = fluid_params(H, 0.01, 1e-3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0), (0.16, 0.16, 0.16), (8, 8, 8))
    f = make_fluid(Scene3D("piles", pos, vel, p), vel=vel)
    f.addEventHandler(lambda fluid, stream: 0)  # leaves the forces as the force pass wrote them
    for k in range(50):
        mass = f32(1e-3 * 1.0173 ** k)
        f.getParameters().mass = mass
        f.getForceBuffer().zero_()
        f.compute()
        assert f.sync_status() == OK
        rho = sorted_outputs(f, oracle.table_cells(p))["spos"][:, 3]
        force = state(f)["force"]
        assert len(np.unique(rho[:na])) == 1 and len(np.unique(rho[na:])) == 1 and len(np.unique(force[:na, 1])) == 1
        a = f32(1) / rho[0] * (f32(1) / rho[na])
        met = set()
        for inv in roots:
            cv = f32(np.float64(f32(p.cellSize)) - r2 * np.float64(inv)) * a
            if f32(4) * (f32(p.viscosityConstant) * cv) * mass == force[0, 1]:
                met.add(inv)
        roots = met
        assert roots, (mass, force[0, 1], rho[0], rho[na])
