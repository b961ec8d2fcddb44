"""The brick passes where a brick is cut into units and where lists and staging overflow: lattices
from sparse to far too dense, against the restatement and bitwise across brick widths."""
import numpy as np
import pytest

import oracle
from fluid_helpers import RTOL, make_fluid, perturbed, pos_err, rel_err, sorted_outputs, state
from libcl_gb300 import OK, OPT_BRICK_WIDTH
from libcl_gb300.scenes import Scene3D, fluid_params, lattice

pytestmark = pytest.mark.gpu

H = 0.02


def block(n, per_h, dims, seed=31):
    """n[0] x n[1] x n[2] particles, about per_h to a cell side, jittered by 0.2 spacings so that
    odd and even cells occur."""
    sp = H / per_h
    pos = lattice(*n, sp, (0.3 * sp,) * 3, 0.2 * sp, seed)
    if dims == 2:
        pos[:, 2] = 0.0
    grid = [int(np.ceil(2 * k * sp / H)) + 1 for k in n]
    box = [g * H for g in grid]
    p = fluid_params(H, sp, 1000.0 * sp ** dims, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, -1.0 if dims == 2 else 0.0),
                     tuple(box), tuple(grid[:dims] + [1] * (3 - dims)), dims=dims)
    return Scene3D("units", pos, np.zeros_like(pos), p)


# per_h 0.8: mostly empty cells, single particles. 2: the lattice the units are sized for (cut only
# at the brick's end). 2.2 - 2.9: units cut short, pairs with more than 128 in reach. 3.2: windows
# of about 880 candidates, staged by the density pass (1,024) and not by the force pass (768).
# 3.6: staged by neither. 2D: 2.0 and a list that overflows (7).
@pytest.mark.parametrize("n,per_h,dims", [((9, 7, 5), 0.8, 3), ((2, 1, 1), 2.0, 3), ((1, 1, 3), 2.0, 3), ((37, 11, 9), 2.0, 3),
                                          ((41, 12, 11), 2.2, 3), ((31, 13, 12), 2.6, 3), ((25, 15, 11), 2.9, 3),
                                          ((27, 14, 13), 3.2, 3), ((26, 14, 15), 3.6, 3), ((45, 33, 1), 2.0, 2), ((90, 40, 1), 7.0, 2)])
def test_units_match_the_restatement_and_any_brick_width(cuda, n, per_h, dims):
    sc = block(n, per_h, dims)
    vel = perturbed(sc, sigma=0.2)
    if dims == 2:
        vel[:, 2] = 0.0
    f = make_fluid(sc, vel=vel)
    f.compute()
    g, gs = sorted_outputs(f, oracle.table_cells(sc.params)), state(f)
    assert f.sync_status() == OK
    pos, v, frc = sc.pos.copy(), vel.copy(), np.zeros_like(sc.pos)
    r = oracle.step(pos, v, frc, sc.params)
    np.testing.assert_array_equal(g["index"], r.index)
    assert rel_err(g["spos"][:, 3], r.spos[:, 3]) < RTOL
    assert rel_err(gs["vel"][:, :3], v[:, :3]) < RTOL
    assert pos_err(gs["pos"][:, :3], pos[:, :3], sc.pos[:, :3]) <= 1.0
    np.testing.assert_array_equal(gs["force"], frc)
    for bw in (1, 3, 16):
        b = make_fluid(sc, vel=vel)
        b.set_option(OPT_BRICK_WIDTH, bw)
        b.compute()
        sb = state(b)
        for k in gs:
            np.testing.assert_array_equal(gs[k].view(np.uint32), sb[k].view(np.uint32), err_msg=f"{k}, brick width {bw}")


def test_particles_that_are_not_numbers_stay_alone(cuda):
    """A NaN particle is nobody's neighbour: with five of them every other particle moves bit for
    bit as with five particles far outside the grid, which lie in the same (lowest) cell."""
    sc = block((16, 8, 8), 2.0, 3)
    vel = perturbed(sc, sigma=0.2)
    out = []
    for x in (-1e6, np.nan):
        p = sc.pos.copy()
        p[:5, :3] = x
        f = make_fluid(Scene3D("nan", p, sc.vel, sc.params), vel=vel)
        f.compute()
        assert f.sync_status() == OK
        out.append((state(f), sorted_outputs(f, oracle.table_cells(sc.params))["cell"]))
    np.testing.assert_array_equal(out[0][1], out[1][1])
    for k in ("pos", "vel", "force"):
        np.testing.assert_array_equal(out[0][0][k][5:].view(np.uint32), out[1][0][k][5:].view(np.uint32), err_msg=k)
