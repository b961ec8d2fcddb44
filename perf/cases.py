"""The workloads the library is timed on: SPH steps (3D and 2D, linear-grid and reference-hash
keys, device- and host-resident), the radix sort, the mesh BVH with collisions, batched scenes,
the differentiable rollout and the reference's 2D relaxation model.

`listed()` names them, `draw(rng)` gives others of the same ranges, `prepare` makes a case's
inputs and handles on the GPU from a seed, `run` is one pass through the public entry points,
`work` the bytes and operations a pass cannot do without, and `exact` the same results in
64-bit arithmetic, written here in plain torch.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import libcl_gb300 as gb
from libcl_gb300.scenes import fluid_params

H3, SP3 = 0.02, 0.01      # 3D scenes: cell size (= support radius) and lattice spacing
H2, SP2 = 0.01, 0.005     # 2D dam break
SMOKE_SIDE = 1.0          # the reference's test cloud fills [-0.5, 0.5]^3


def listed():
    return [
        # the reference's own test program: 256 particles, its default parameters and hash keys;
        # a frame of 8 sub-steps. The smallest call there is: launches and host time.
        {"name": "smoke_hash_256", "kind": "cloud", "n": 256, "steps": 8},
        # 2D dam break (16,384 particles, poly6/spiky, the 3D step with dims = 2): an interactive
        # scene, far too small to fill the GPU.
        {"name": "dam_break_2d_16k", "kind": "step", "keys": "linear", "dims": 2, "nx": 128, "ny": 128, "nz": 1,
         "disorder": 0.0, "steps": 8, "io": "device"},
        # the headline: 3D block collapse, 1,048,576 particles, from the start of the collapse.
        {"name": "collapse_1m", "kind": "step", "keys": "linear", "dims": 3, "nx": 128, "ny": 64, "nz": 128,
         "disorder": 0.0, "steps": 4, "io": "device"},
        # a fluid some way into its motion (uneven cells, compressed bottom, particles moving),
        # odd sizes; every array a renderer or an analysis reads afterwards comes back.
        {"name": "splash_530k", "kind": "step", "keys": "linear", "dims": 3, "nx": 100, "ny": 57, "nz": 93,
         "disorder": 0.8, "steps": 1, "io": "device"},
        # the same step for a program that keeps its particles on the host (pinned arrays in and
        # out on every step).
        {"name": "host_1m", "kind": "step", "keys": "linear", "dims": 3, "nx": 128, "ny": 64, "nz": 128,
         "disorder": 0.4, "steps": 1, "io": "host"},
        # the reference's default keys (262,144 hash buckets, its summation order) at full size.
        {"name": "collapse_hash_1m", "kind": "step", "keys": "hash", "dims": 3, "nx": 128, "ny": 64, "nz": 128,
         "disorder": 0.2, "steps": 2, "io": "device"},
        # the sort on its own, at the size of the sort benchmark: uniform 32-bit keys.
        {"name": "sort_uniform_16m", "kind": "sort", "n": 1 << 24, "keys": "uniform", "bits": 32, "bounds": False},
        # sorting particles into Morton cells and extracting the cells' ranges, an odd count.
        {"name": "sort_cells_1m5", "kind": "sort", "n": 1500001, "keys": "cells", "bits": 24, "bounds": True},
        # a deforming obstacle: its BVH rebuilt each frame (1.05M triangles), then the particles
        # near it collided with it.
        {"name": "obstacle_1m", "kind": "mesh", "nlat": 513, "nlon": 1024, "particles": 262144},
        # an ensemble of independent scenes of 4,096 to 262,144 particles (17M in all).
        {"name": "batch_256", "kind": "batch", "scenes": 256, "n_min": 4096, "n_max": 262144, "steps": 2},
        # gradients through a rollout (loss on the final state, to the initial state and the
        # fluid's gas constant and viscosity).
        {"name": "rollout_grad_64k", "kind": "grad", "nx": 64, "ny": 32, "nz": 32, "steps": 20, "every": 10},
        # the reference's 2D relaxation model at its default size, with walls (two steps: its
        # trajectories part within a few more).
        {"name": "relax_2d_16k", "kind": "relax", "nx": 128, "ny": 128, "steps": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "hash", "host", "sort", "sort", "mesh", "batch", "grad", "relax", "cloud"])
    if kind == "cloud":
        return {"kind": "cloud", "n": _log(rng, 200, 20000), "steps": rng.choice([1, 4, 8])}
    if kind in ("step", "hash", "host"):
        dims = 2 if kind == "step" and rng.random() < 0.3 else 3
        # particle count 1,000 to 1,048,576 with uneven sides
        n = _log(rng, 1000, 1000000)
        if dims == 2:
            nx = max(8, int(math.sqrt(min(n, 200000)) * rng.uniform(0.6, 1.6)))
            ny, nz = max(8, min(n, 200000) // nx), 1
        else:
            side = n ** (1 / 3)
            nx = max(4, int(side * rng.uniform(0.7, 1.5)))
            ny = max(4, int(side * rng.uniform(0.5, 1.1)))
            nz = max(4, n // (nx * ny))
        while nx * ny * nz > 1048576:
            nz -= 1
        return {"kind": "step", "keys": "hash" if kind == "hash" else "linear", "dims": dims, "nx": nx, "ny": ny,
                "nz": nz, "disorder": round(rng.uniform(0.0, 1.0), 3), "steps": 1 if kind == "host" else rng.randint(1, 4),
                "io": "host" if kind == "host" else "device"}
    if kind == "sort":
        keys = rng.choice(["uniform", "cells"])
        n = _log(rng, 3000, 1 << 24)
        return {"kind": "sort", "n": n, "keys": keys, "bits": rng.choice([16, 24, 28, 32]) if keys == "uniform" else 24,
                "bounds": keys == "cells"}
    if kind == "mesh":
        nlat = _log(rng, 17, 513)
        return {"kind": "mesh", "nlat": nlat, "nlon": max(8, int(nlat * rng.uniform(1.2, 2.0))),
                "particles": _log(rng, 2000, 262144)}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 64), "n_min": _log(rng, 300, 5000),
                "n_max": _log(rng, 20000, 200000), "steps": rng.randint(1, 2)}
    if kind == "grad":
        side = _log(rng, 8, 32)
        steps = rng.randint(3, 20)
        return {"kind": "grad", "nx": int(side * rng.uniform(1, 2)), "ny": side, "nz": max(6, int(side * rng.uniform(0.5, 1))),
                "steps": steps, "every": rng.randint(2, 10)}
    nx = rng.randint(20, 200)
    return {"kind": "relax", "nx": nx, "ny": rng.randint(20, min(160, 30000 // nx)), "steps": rng.choice([1, 2])}


# ---- scenes ---------------------------------------------------------------------------------

def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _f32(x):
    return float(np.float32(x))


def _block(nx, ny, nz, sp, disorder, seed, dims=3, salt=0):
    """Jittered lattice at the lower corner of the box, float32 [n, 4] positions and velocities
    (x fastest). `disorder` 0: at rest, jittered by 0.1 spacing, as the collapse starts; up to 1:
    half a spacing of jitter, compressed towards the floor, falling and eddying."""
    n = nx * ny * nz
    g = _gen(seed, salt)
    i = torch.arange(n, device="cuda")
    p = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1).double()
    u = torch.rand((n, 3), device="cuda", generator=g, dtype=torch.float64)
    p = (p + 0.5 + (2 * u - 1) * (0.1 + 0.4 * disorder)) * sp
    ext = torch.tensor([nx, ny, nz], device="cuda", dtype=torch.float64) * sp
    rel = p / ext
    p[:, 1] *= 1 - 0.12 * disorder * (1 - rel[:, 1])
    v = torch.zeros((n, 3), device="cuda", dtype=torch.float64)
    if disorder > 0:
        noise = torch.randn((n, 3), device="cuda", generator=g, dtype=torch.float64)
        v = 0.1 * disorder * noise
        v[:, 0] += 0.8 * disorder * torch.sin(6.0 * rel[:, 1]) * torch.cos(4.0 * rel[:, 0])
        v[:, 1] -= disorder * rel[:, 1]
    if dims == 2:
        p[:, 2], v[:, 2] = 0, 0
    pos = torch.zeros((n, 4), device="cuda")
    vel = torch.zeros((n, 4), device="cuda")
    pos[:, :3], vel[:, :3] = p.float(), v.float()
    return pos, vel


def _box3(nx, ny, nz, factor=3.125):
    """Box of `factor` times the block (the collapse: 1.28 x 0.64 x 1.28 in 4 x 2 x 4) and its cells."""
    box = [max(factor * k * SP3, 2 * H3) for k in (nx, ny, nz)]
    return box, [int(math.ceil(b / H3 - 1e-9)) for b in box]


def _step_params(c):
    if c["dims"] == 2:
        box = [max(1.5625 * k * SP2, 2 * H2) for k in (c["nx"], c["ny"])]
        p = fluid_params(H2, SP2, 1000.0 * SP2 ** 2, 1000.0, 3.0, 0.1, 1e-4, (0.0, -9.81, 0.0), (0.0, 0.0, -1.0),
                         (box[0], box[1], 1.0), (int(math.ceil(box[0] / H2 - 1e-9)), int(math.ceil(box[1] / H2 - 1e-9)), 1),
                         dims=2)
    else:
        box, grid = _box3(c["nx"], c["ny"], c["nz"])
        p = fluid_params(H3, SP3, 1000.0 * SP3 ** 3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0),
                         tuple(box), tuple(grid))
    p.keyMode = gb.KEY_REFERENCE_HASH if c["keys"] == "hash" else gb.KEY_LINEAR_GRID
    return p


def _set(dst, src):
    ctypes.memmove(ctypes.byref(dst), ctypes.byref(src), ctypes.sizeof(gb.Fluid3DParams))


def _gravity(p):
    return torch.tensor([float(np.float32(g)) for g in p.gravity], dtype=torch.float32, device="cuda")


def _cloud(c, seed):
    """The reference's test scene: particles uniform in a cube, at rest."""
    u = torch.rand((c["n"], 3), device="cuda", generator=_gen(seed), dtype=torch.float64)
    pos = torch.zeros((c["n"], 4), device="cuda")
    pos[:, :3] = ((u - 0.5) * SMOKE_SIDE).float()
    return pos, torch.zeros_like(pos)


def _fluid(params, n):
    f = gb.Fluid3D()
    f.compile()
    f.setParticleCount(n)
    if params is not None:
        _set(f.getParameters(), params)
    return f


def _batch_scenes(c, seed):
    """Near-cubic blocks of log-uniform size, each in its own box of twice its extent."""
    rng = np.random.default_rng(int(seed) + 5)
    shared = fluid_params(H3, SP3, 1000.0 * SP3 ** 3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0),
                          (1.0, 1.0, 1.0), (1, 1, 1))
    # the sizes are the case's, the same for every seed: another seed moves the particles and
    # changes the fluids
    sizes = np.exp(np.random.default_rng(17).uniform(math.log(c["n_min"]), math.log(c["n_max"]), c["scenes"]))
    descs, dims = [], []
    for s, size in enumerate(sizes):
        side = max(2, int(round(size ** (1 / 3))))
        nx, ny, nz = side, side, max(1, int(round(size / (side * side))))
        box, grid = _box3(nx, ny, nz, 2.0)
        d = gb.SceneDesc()
        d.n_particles = nx * ny * nz
        d.stiffness, d.viscosity = float(rng.uniform(1, 5)), float(rng.uniform(0.01, 0.2))
        for i in range(3):
            d.boxMin[i], d.boxMax[i], d.gridOrigin[i], d.gridDim[i] = 0.0, float(box[i]), 0.0, grid[i]
        descs.append(d)
        dims.append((nx, ny, nz))
    return shared, descs, dims


def _batch_state(c, seed, dims):
    parts = [_block(*d, SP3, 0.0, seed, salt=s + 1) for s, d in enumerate(dims)]
    return torch.cat([p for p, _ in parts]), torch.cat([v for _, v in parts])


def _mesh(c, seed):
    """A bumpy UV sphere around (1, 1, 1): shared vertices, 2 * nlon * (nlat - 1) triangles."""
    nlat, nlon = c["nlat"], c["nlon"]
    ph = torch.rand(6, generator=torch.Generator().manual_seed(int(seed)), dtype=torch.float64) * 6.28
    i = torch.arange((nlat - 1) * nlon, device="cuda")
    th = math.pi * (i // nlon + 1).double() / nlat
    ps = 2 * math.pi * (i % nlon).double() / nlon
    r = 0.5 + 0.03 * (torch.sin(3 * th + ph[0]) * torch.cos(4 * ps + ph[1]) + torch.sin(7 * th + ph[2]) * torch.cos(9 * ps + ph[3]))
    xyz = torch.stack([r * torch.sin(th) * torch.cos(ps), r * torch.sin(th) * torch.sin(ps), r * torch.cos(th)], 1)
    pole = torch.tensor([[0.0, 0.0, 0.5]], device="cuda", dtype=torch.float64)
    v = torch.zeros(((nlat - 1) * nlon + 2, 4), device="cuda")
    v[:, :3] = (torch.cat([pole, xyz, -pole]) + 1.0).float()
    j = torch.arange(nlon, device="cuda")
    jn = (j + 1) % nlon
    north = torch.stack([torch.zeros_like(j), 1 + j, 1 + jn], 1)
    a = (1 + torch.arange(nlat - 2, device="cuda") * nlon)[:, None]
    quads = torch.stack([torch.stack([a + j, a + nlon + j, a + nlon + jn], 2),
                         torch.stack([a + j, a + nlon + jn, a + jn], 2)], 2).reshape(-1, 3)
    last, south = 1 + (nlat - 2) * nlon, v.shape[0] - 1
    cap = torch.stack([last + j, torch.full_like(j, south), last + jn], 1)
    return v, torch.cat([north, quads, cap]).reshape(-1).int()


def _spread(x, bits):
    out = torch.zeros_like(x)
    for b in range(bits):
        out |= ((x >> b) & 1) << (3 * b)
    return out


def _cell_bits(n):
    """Morton bits per axis so that about 8 keys fall into each cell."""
    return max(1, math.ceil(math.log2(max(2.0, n / 8)) / 3))


BORDER = 8  # wall pixels around the 2D container


def _relax_state(c, seed):
    n = c["nx"] * c["ny"]
    i = torch.arange(n, device="cuda")
    u = torch.rand((n, 2), device="cuda", generator=_gen(seed), dtype=torch.float64)
    st = torch.zeros((n, 6), device="cuda")
    st[:, 0] = (1.0 + (i % c["nx"]) * 0.06 + (u[:, 0] - 0.5) * 0.03).float()
    st[:, 1] = (0.6 + (i // c["nx"]) * 0.06 + (u[:, 1] - 0.5) * 0.03).float()
    st[:, 4] = _f32(0.7)
    mask = torch.zeros((256, 256, 4), device="cuda")
    mask[:BORDER, :, 3] = mask[-BORDER:, :, 3] = mask[:, :BORDER, 3] = mask[:, -BORDER:, 3] = 1
    return st, mask


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("step", "cloud"):
        if kind == "cloud":
            p, (pos, vel) = None, _cloud(c, seed)
        else:
            p = _step_params(c)
            pos, vel = _block(c["nx"], c["ny"], c["nz"], SP2 if c["dims"] == 2 else SP3, c["disorder"], seed, c["dims"])
        f = _fluid(p, pos.shape[0])
        g = _gravity(f.getParameters())
        f.getForceBuffer().copy_(g.expand_as(pos))
        s = {"case": c, "fluid": f, "pos0": pos, "vel0": vel, "pos": f.getPositionBuffer(), "vel": f.getVelocityBuffer()}
        if c.get("io") == "host":
            s["in"] = [t.cpu().pin_memory() for t in (pos, vel, g.expand_as(pos).contiguous())]
            s["out"] = [torch.empty_like(t).pin_memory() for t in s["in"]]
        return s
    if kind == "sort":
        n, g = c["n"], _gen(seed)
        if c["keys"] == "uniform":
            keys = torch.randint(0, 1 << c["bits"], (n,), device="cuda", generator=g)
            cells = 0
        else:
            b = _cell_bits(n)
            x = torch.randint(0, 1 << b, (3, n), device="cuda", generator=g)
            keys = _spread(x[0], b) | (_spread(x[1], b) << 1) | (_spread(x[2], b) << 2)
            cells = 1 << (3 * b)
        keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).int()
        s = {"case": c, "sort": gb.RadixSort(), "keys0": keys, "vals0": torch.arange(n, device="cuda", dtype=torch.int32)}
        s["keys"], s["vals"] = torch.empty_like(keys), torch.empty_like(keys)
        if c["bounds"]:
            s["start"] = torch.empty(cells, dtype=torch.int32, device="cuda")
            s["end"] = torch.empty(cells, dtype=torch.int32, device="cuda")
        return s
    if kind == "mesh":
        v, idx = _mesh(c, seed)
        n, g = c["particles"], _gen(seed, 3)
        d = torch.randn((n, 3), device="cuda", generator=g, dtype=torch.float64)
        d /= d.norm(dim=1, keepdim=True)
        u = torch.rand((n, 2), device="cuda", generator=g, dtype=torch.float64)
        pos, vel, frc = (torch.zeros((n, 4), device="cuda") for _ in range(3))
        # most particles close to the surface and moving towards it, a quarter elsewhere, some at rest
        pos[:, :3] = (1.0 + d * (0.44 + 0.13 * u[:, :1])).float()
        vel[:, :3] = (-d * (1.0 + 2.0 * u[:, 1:])).float()
        k = n // 4
        pos[:k, :3] = torch.rand((k, 3), device="cuda", generator=g) * 2
        vel[:k, :3] = torch.randn((k, 3), device="cuda", generator=g)
        vel[:k // 4] = 0
        frc[:, 2] = _f32(-9.8)
        return {"case": c, "bvh": gb.BvhTrimesh(), "params": gb.default_params(), "vertex": v, "index": idx,
                "state0": (pos, vel, frc), "state": tuple(torch.empty_like(pos) for _ in range(3))}
    if kind == "batch":
        shared, descs, dims = _batch_scenes(c, seed)
        b = gb.Batch3D()
        b.set_scenes(shared, descs)
        b.set_option(gb.OPT_BRICK_WIDTH, 16)  # what the autotuner picks for ensembles of this kind
        pos, vel = _batch_state(c, seed, dims)
        b.buffer(gb.BUF_FORCE).copy_(_gravity(shared).expand_as(pos))
        return {"case": c, "batch": b, "pos0": pos, "vel0": vel, "pos": b.buffer(gb.BUF_POSITION),
                "vel": b.buffer(gb.BUF_VELOCITY)}
    if kind == "grad":
        pos, vel, tpos, tvel = _grad_inputs(c, seed)
        box, grid = _box3(c["nx"], c["ny"], c["nz"], 2.0)
        p = fluid_params(H3, SP3, 1000.0 * SP3 ** 3, 1000.0, 3.0, 0.05, 5e-5, (0.0, -9.81, 0.0), (0.0, 0.0, 0.0),
                         tuple(box), tuple(grid))
        f = _fluid(p, pos.shape[0])
        leaves = [pos.requires_grad_(), vel.requires_grad_(), torch.tensor(_f32(3.0), requires_grad=True),
                  torch.tensor(_f32(0.05), requires_grad=True)]
        return {"case": c, "adj": gb.Adjoint3D(f, c["steps"], min(c["every"], c["steps"])), "fluid": f, "leaves": leaves,
                "target": (tpos, tvel)}
    st, mask = _relax_state(c, seed)
    f = gb.Fluid2D()
    f.compile()
    f.setParticleCount(st.shape[0])
    f.computeBorder(mask)
    return {"case": c, "fluid": f, "state0": st, "state": f.getStateBuffer()}


def _grad_inputs(c, seed):
    """The block at rest with small random velocities; the target a state near its future one."""
    pos, vel = _block(c["nx"], c["ny"], c["nz"], SP3, 0.0, seed)
    n, g = pos.shape[0], _gen(seed, 9)
    vel[:, :3] = 0.1 * torch.randn((n, 3), device="cuda", generator=g)
    tvel = vel.clone()
    tvel[:, :3] += 0.1 * torch.randn((n, 3), device="cuda", generator=g)
    return pos, vel, pos + 5e-5 * c["steps"] * tvel, tvel


def _loss(pos, vel, target, n):
    return ((vel - target[1]) ** 2).sum() * (0.5 / n) + ((pos - target[0]) ** 2).sum() * (5e3 / n)


class _Outputs(dict):
    """run()'s answer: views of the library's buffers among it, which live as long as their handle."""

    def __init__(self, state, values):
        super().__init__(values)
        self.owner = state


def run(s):
    return _Outputs(s, _run(s))


def _run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind in ("step", "cloud"):
        f = s["fluid"]
        if c.get("io") == "host":
            f.compute_host(*s["in"], *s["out"])
            return {"position": s["out"][0], "velocity": s["out"][1], "force": s["out"][2]}
        s["pos"].copy_(s["pos0"])
        s["vel"].copy_(s["vel0"])
        for _ in range(c["steps"]):
            f.compute()
        out = {"position": s["pos"], "velocity": s["vel"], "force": f.getForceBuffer()}
        if c["steps"] == 1:
            out.update(sorted_position=f.getSortedPositionBuffer(), sorted_velocity=f.getSortedVelocityBuffer(),
                       index=f.getIndexBuffer(), cell=f.getCellBuffer())
        return out
    if kind == "sort":
        s["keys"].copy_(s["keys0"])
        s["vals"].copy_(s["vals0"])
        s["sort"].compute(s["keys"], s["vals"], 0, c["bits"])
        out = {"keys": s["keys"], "values": s["vals"]}
        if c["bounds"]:
            s["sort"].cell_bounds(s["keys"], s["start"], s["end"])
            out.update(start=s["start"], end=s["end"])
        return out
    if kind == "mesh":
        s["bvh"].compute(s["vertex"], s["index"])
        for dst, src in zip(s["state"], s["state0"]):
            dst.copy_(src)
        s["bvh"].collide(s["params"], *s["state"], s["vertex"], s["index"])
        return {"nodes": s["bvh"].getNodeBuffer(), "position": s["state"][0], "velocity": s["state"][1], "force": s["state"][2]}
    if kind == "batch":
        s["pos"].copy_(s["pos0"])
        s["vel"].copy_(s["vel0"])
        for _ in range(c["steps"]):
            s["batch"].compute()
        return {"position": s["pos"], "velocity": s["vel"]}
    if kind == "grad":
        from libcl_gb300.autograd import rollout
        pos, vel = rollout(s["adj"], *s["leaves"])
        grads = torch.autograd.grad(_loss(pos, vel, s["target"], pos.shape[0]), s["leaves"])
        return {"position": pos.detach(), "velocity": vel.detach(), "d_position": grads[0], "d_velocity": grads[1],
                "d_stiffness": grads[2], "d_viscosity": grads[3]}
    s["state"].copy_(s["state0"])
    for _ in range(c["steps"]):
        s["fluid"].compute()
    out = {"state": s["state"]}
    if c["steps"] == 1:
        out["pressure"] = s["fluid"].buffer(gb.BUF2D_PRESSURE)
    return out


def _particles(c):
    if c["kind"] == "cloud":
        return c["n"]
    if c["kind"] == "batch":
        return sum(d.n_particles for d in _batch_scenes(c, 0)[1])
    if c["kind"] == "relax":
        return c["nx"] * c["ny"]
    return c["nx"] * c["ny"] * c["nz"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "sort":
        n = c["n"]
        cells = 1 << (3 * _cell_bits(n)) if c["bounds"] else 0
        return {"bytes": 16.0 * n + 8 * cells, "flops": 0}  # pairs in, pairs out; the two tables
    if kind == "mesh":
        v, t = (c["nlat"] - 1) * c["nlon"] + 2, 2 * c["nlon"] * (c["nlat"] - 1)
        # vertices, indices, 48-byte nodes; three float4 in and out per particle; a root-to-leaf
        # path of two box tests (about 40 operations each) per particle
        return {"bytes": 16.0 * v + 12 * t + 48 * (2 * t - 1) + 96 * c["particles"],
                "flops": 80.0 * c["particles"] * math.log2(t) + 40.0 * t}
    n, steps = _particles(c), c["steps"]
    if kind == "relax":  # 24-byte state in and out, 16-byte pressures out; about 34 neighbours, two passes
        return {"bytes": 64.0 * n * steps, "flops": 34.0 * 45 * n * steps}
    # position, velocity, force in and out; density (30) and force (60) operations for each
    # neighbour in range: 33 in 3D and 12 in 2D at the lattice's spacing, hardly any in the cloud
    near = 12 if c.get("dims") == 2 else 1 if kind == "cloud" else 33
    w = {"bytes": 96.0 * n * steps, "flops": 90.0 * near * n * steps}
    if kind == "grad":  # the recomputed and the reversed step beside the forward one
        w = {"bytes": 3 * w["bytes"], "flops": w["flops"] * 2 + 120.0 * near * n * steps}
    return w


# ---- the same in 64 bits --------------------------------------------------------------------

class _Sys:
    """Constants of a step (float32 inputs, 64-bit arithmetic); stiff, cvisc and the box may be
    per-particle tensors."""

    def __init__(self, h, radius, mass, stiff, visc, dt, gravity, lo, hi, grid=None, dims=3, vlimit=500.0, rho0=1000.0):
        self.h, self.radius, self.mass, self.rho0 = _f32(h), _f32(radius), _f32(mass), rho0
        self.stiff, self.dt, self.vlimit, self.dims, self.grid = stiff, _f32(dt), vlimit, dims, grid
        self.g = torch.tensor([_f32(x) for x in gravity], dtype=torch.float64, device="cuda")
        self.lo = lo if torch.is_tensor(lo) else torch.tensor([_f32(x) for x in lo], dtype=torch.float64, device="cuda")
        self.hi = hi if torch.is_tensor(hi) else torch.tensor([_f32(x) for x in hi], dtype=torch.float64, device="cuda")
        hh = self.h
        if dims == 2:
            self.k, self.cp, self.cv = 4 / (math.pi * hh ** 8), 30 / (math.pi * hh ** 5), visc * 40 / (math.pi * hh ** 5)
        else:
            self.k, self.cp = 315 / (64 * math.pi * hh ** 9), 45 / (math.pi * hh ** 6)
            self.cv = visc * self.cp


def _cells64(x, sys, first=0):
    """Integer cell coordinates [n, 3] (float32 division, as the key is defined)."""
    h = torch.tensor(sys.h, dtype=torch.float32, device="cuda")
    c = torch.floor(x.detach().float() / h).long()
    if sys.dims == 2:
        c[:, 2] = 0
    if sys.grid is not None:
        c = torch.minimum(c.clamp(min=0), torch.as_tensor(sys.grid, device="cuda").long() - 1)
    return c


def _hash(c):
    m = 0xFFFFFFFF
    return (((73856093 * c[:, 0]) & m) ^ ((19349663 * c[:, 1]) & m) ^ ((83492791 * c[:, 2]) & m)) % 262144


def _neighbours(x, sys, offset=None):
    """(key, iterator): the iterator gives (j, valid) for every neighbour cell and every place in
    it, j a candidate of each particle. `offset`: per-particle first cell of its scene's table."""
    c = _cells64(x, sys)
    n = x.shape[0]
    me = torch.arange(n, device="cuda")
    grid = None if sys.grid is None else torch.as_tensor(sys.grid, device="cuda").long().expand(n, 3)

    def key_of(q):
        if grid is None:
            return _hash(q), torch.ones(n, dtype=torch.bool, device="cuda")
        ok = ((q >= 0) & (q < grid)).all(1)
        k = q[:, 0] + grid[:, 0] * (q[:, 1] + grid[:, 1] * q[:, 2])
        return torch.where(ok, k if offset is None else k + offset, 0), ok

    key, _ = key_of(c)
    order = torch.sort(key, stable=True)[1]
    count = torch.bincount(key)
    start = torch.cumsum(count, 0) - count

    def each():
        for dz in ((0,) if sys.dims == 2 else (-1, 0, 1)):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    k, ok = key_of(c + torch.tensor([dx, dy, dz], device="cuda"))
                    ok &= k < count.numel()
                    k = k.clamp(max=count.numel() - 1)
                    ln = torch.where(ok, count[k], 0)
                    st = start[k]
                    for m in range(int(ln.max())):
                        j = order[(st + m).clamp(max=n - 1)]
                        yield j, (m < ln) & (j != me)

    return key, order, each


def _post64(x, v, f, sys):
    """Walls, clamp, integration: (x', v')."""
    for a in (0, 1) if sys.dims == 2 else (0, 1, 2):
        for sign, d in ((1.0, x[:, a] - sys.lo[..., a]), (-1.0, sys.hi[..., a] - x[:, a])):
            diff = sys.radius - d
            wall = torch.where(diff > 1e-5, sign * (2000 * diff - 256 * sign * v[:, a]), 0.0)
            f = f + torch.nn.functional.one_hot(torch.tensor(a), 3).to(f) * wall[:, None]
    speed = f.norm(dim=1, keepdim=True)
    f = torch.where(speed > sys.vlimit, f * (sys.vlimit / speed.clamp(min=1e-30)), f)
    v = v + f * sys.dt
    return x + v * sys.dt, v


def _rho64(s, cnt, sys):
    rho = torch.where(cnt > 2, (sys.mass * sys.k * s).clamp(min=1.0), sys.rho0)
    return rho, torch.where(cnt > 2, sys.stiff * (rho - sys.rho0), 0.0)


def _step64(x, v, sys, offset=None):
    """One step: (x', v', key, order, rho, p), x and v [n, 3] in float64; the force on entry is gravity."""
    key, order, each = _neighbours(x, sys, offset)
    n, h2 = x.shape[0], sys.h * sys.h
    s = torch.zeros(n, dtype=torch.float64, device="cuda")
    cnt = torch.zeros(n, dtype=torch.float64, device="cuda")
    for j, ok in each():
        r2 = ((x - x[j]) ** 2).sum(1)
        ok = ok & (r2 < h2)
        t = torch.where(ok, h2 - r2, 0.0)
        s += t * t * t
        cnt += ok
    rho, p = _rho64(s, cnt, sys)
    fp, fv = torch.zeros_like(x), torch.zeros_like(x)
    for j, ok in each():
        d = x - x[j]
        r2 = (d * d).sum(1)
        ok = ok & (r2 < h2) & (r2 > 0)
        r = torch.sqrt(torch.where(ok, r2, 1.0))
        q = torch.where(ok, 1.0 / (rho * rho[j]), 0.0)
        fp += d * ((p + p[j]) * q * (sys.h - r) ** 2 / r)[:, None]
        fv += (v[j] - v) * (q * (sys.h - r))[:, None]
    cv = sys.cv if not torch.is_tensor(sys.cv) else sys.cv[:, None]
    f = sys.g[:3] + sys.mass * (sys.cp * fp + cv * fv)
    x1, v1 = _post64(x, v, f, sys)
    return x1, v1, key, order, rho, p


def _four(x, w=None):
    return torch.cat([x, torch.zeros_like(x[:, :1]) if w is None else w[:, None]], 1)


def _exact_step(c, seed):
    if c["kind"] == "cloud":
        pos, vel = _cloud(c, seed)
        spacing = _f32(0.87 * float(np.float32(_f32(0.006) / 1000) ** np.float32(1 / 3)))
        sys = _Sys(2 * spacing, 0.5 * spacing, 0.006, 1.0, 6.0, 0.005, (0, 0, -9.8, 0), (-1, -1, -1), (1, 1, 1))
    else:
        d2 = c["dims"] == 2
        sp = SP2 if d2 else SP3
        pos, vel = _block(c["nx"], c["ny"], c["nz"], sp, c["disorder"], seed, c["dims"])
        if d2:
            hi = [max(1.5625 * k * SP2, 2 * H2) for k in (c["nx"], c["ny"])] + [1.0]
            grid = [int(math.ceil(b / H2 - 1e-9)) for b in hi[:2]] + [1]
        else:
            hi, grid = _box3(c["nx"], c["ny"], c["nz"])
        sys = _Sys(H2 if d2 else H3, 0.5 * sp, 1000.0 * sp ** (2 if d2 else 3), 3.0, _f32(0.1 if d2 else 0.05),
                   1e-4 if d2 else 5e-5, (0, -9.81, 0, 0), (0, 0, -1) if d2 else (0, 0, 0), hi,
                   None if c["keys"] == "hash" else grid, c["dims"])
    x, v = pos[:, :3].double(), vel[:, :3].double()
    for _ in range(c["steps"]):
        x0, v0 = x, v
        x, v, key, order, rho, p = _step64(x, v, sys)
    out = {"position": _four(x), "velocity": _four(v), "force": sys.g.expand(x.shape[0], 4)}
    if c["steps"] == 1 and c.get("io") != "host":
        out.update(sorted_position=_four(x0[order], rho[order]), sorted_velocity=_four(v0[order], p[order]), index=None, cell=None)
    return out


def _exact_batch(c, seed):
    _, descs, dims = _batch_scenes(c, seed)
    pos, vel = _batch_state(c, seed, dims)
    cnt = torch.tensor([d.n_particles for d in descs], device="cuda")

    def per(values):
        return torch.tensor(values, device="cuda", dtype=torch.float64).repeat_interleave(cnt, 0)

    cells = np.cumsum([0] + [int(np.prod([d.gridDim[i] for i in range(3)])) for d in descs])
    sys = _Sys(H3, 0.5 * SP3, 1000.0 * SP3 ** 3, per([d.stiffness for d in descs]), per([d.viscosity for d in descs]), 5e-5,
               (0, -9.81, 0, 0), (0, 0, 0), per([[d.boxMax[i] for i in range(3)] for d in descs]),
               per([[d.gridDim[i] for i in range(3)] for d in descs]))
    offset = per([float(k) for k in cells[:-1]]).long()
    x, v = pos[:, :3].double(), vel[:, :3].double()
    for _ in range(c["steps"]):
        x, v = _step64(x, v, sys, offset)[:2]
    return {"position": _four(x), "velocity": _four(v)}


def _exact_grad(c, seed):
    """Autograd through the steps, each over its list of pairs in range."""
    pos, vel, tpos, tvel = _grad_inputs(c, seed)
    n = pos.shape[0]
    hi, grid = _box3(c["nx"], c["ny"], c["nz"], 2.0)
    x0, v0 = pos[:, :3].double().requires_grad_(), vel[:, :3].double().requires_grad_()
    k = torch.tensor(_f32(3.0), dtype=torch.float64, device="cuda", requires_grad=True)
    mu = torch.tensor(_f32(0.05), dtype=torch.float64, device="cuda", requires_grad=True)
    sys = _Sys(H3, 0.5 * SP3, 1000.0 * SP3 ** 3, k, mu, 5e-5, (0, -9.81, 0, 0), (0, 0, 0), hi, grid)
    h2, x, v = sys.h * sys.h, x0, v0
    for _ in range(c["steps"]):
        with torch.no_grad():
            pi, pj = [], []
            for j, ok in _neighbours(x, sys)[2]():
                ok = ok & (((x - x[j]) ** 2).sum(1) < h2)
                i = ok.nonzero()[:, 0]
                pi.append(i)
                pj.append(j[i])
            i, j = torch.cat(pi), torch.cat(pj)
        d = x[i] - x[j]
        r2 = (d * d).sum(1)
        zero = torch.zeros(n, dtype=torch.float64, device="cuda")
        rho, p = _rho64(zero.index_add(0, i, (h2 - r2) ** 3), zero.index_add(0, i, torch.ones_like(r2)), sys)
        r, q = torch.sqrt(r2), 1.0 / (rho[i] * rho[j])
        pair = sys.cp * d * ((p[i] + p[j]) * q * (sys.h - r) ** 2 / r)[:, None] + sys.cv * (v[j] - v[i]) * (q * (sys.h - r))[:, None]
        f = sys.g[:3] + sys.mass * torch.zeros_like(x).index_add(0, i, pair)
        x, v = _post64(x, v, f, sys)
    grads = torch.autograd.grad(_loss(x, v, (tpos[:, :3].double(), tvel[:, :3].double()), n), [x0, v0, k, mu])
    return {"position": _four(x.detach()), "velocity": _four(v.detach()), "d_position": _four(grads[0]),
            "d_velocity": _four(grads[1]), "d_stiffness": grads[2], "d_viscosity": grads[3]}


class _Relax:
    """oclFluid2D's constants (libCL/phys/oclFluid2D.cl:121-151)."""
    h = _f32(22 * 0.05 / 5)
    dt, m, cw, ch, psize = _f32(0.00433333333), _f32(0.7), _f32(17.68), _f32(15.76), _f32(0.01)
    stiff, near_stiff, tension, rest = _f32(0.08), _f32(0.1), _f32(21.00035), 82.0
    kn, knn = 20 / (2 * math.pi * h * h), 30 / (2 * math.pi * h * h)


def _wall_images(mask, k):
    """The wall field (clComputeBorder): (density, near, pressure, near pressure) and (normal, distance), as half floats."""
    hh, w = mask.shape[:2]
    wall = mask[..., 3] == 1
    dw, dh = int(w * k.h / k.cw + 0.5), int(hh * k.h / k.ch + 0.5)
    dx, dy = k.cw / w, k.ch / hh
    s = dx * dy / (2 * math.pi * k.psize * k.psize)
    yy, xx = torch.meshgrid(torch.arange(hh, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    den = torch.where(wall, 112 * k.m * k.kn, 0.0).double()
    near = torch.where(wall, 112 * k.m * k.knn, 0.0).double()
    best = torch.full((hh, w), 10000.0, dtype=torch.float64, device="cuda")
    vec = torch.zeros((hh, w, 3), dtype=torch.float64, device="cuda")
    for i in range(-dw, dw):
        for j in range(-dh, dh):
            x, y = xx + i, yy + j
            inside = (x >= 0) & (x < w) & (y >= 0) & (y < hh)
            other = wall[y.clamp(0, hh - 1), x.clamp(0, w - 1)]
            r = math.hypot(i * dx, j * dy)
            hit = inside & (other != wall) & (wall | (r < k.h))
            a = 1 - r / k.h
            den += torch.where(hit & ~wall, s * k.m * a ** 3 * k.kn, 0.0)
            near += torch.where(hit & ~wall, s * k.m * a ** 4 * k.knn, 0.0)
            closer = hit & (r < best)
            sign = torch.where(wall, 1.0, -1.0).double()
            for q, t in enumerate((i * dx, j * dy)):
                vec[..., q] = torch.where(closer, sign * t / max(r, 1e-30), vec[..., q])
            vec[..., 2] = torch.where(closer, r, vec[..., 2])
            best = torch.where(closer, r, best)
    img = torch.stack([den, near, k.stiff * (den - k.m * k.rest), k.near_stiff * near], 2)
    return img.half().double(), vec.half().double()


def _sample(img, s, t):
    """Bilinear, normalised coordinates, clamped to the edge."""
    h, w = img.shape[:2]
    u, v = s * w - 0.5, t * h - 0.5
    a, b = (u - u.floor())[:, None], (v - v.floor())[:, None]
    i, j = u.floor().long(), v.floor().long()
    i0, i1, j0, j1 = i.clamp(0, w - 1), (i + 1).clamp(0, w - 1), j.clamp(0, h - 1), (j + 1).clamp(0, h - 1)
    return (1 - a) * (1 - b) * img[j0, i0] + a * (1 - b) * img[j0, i1] + (1 - a) * b * img[j1, i0] + a * b * img[j1, i1]


def _exact_relax(c, seed):
    st, mask = _relax_state(c, seed)
    k = _Relax
    img, vec = _wall_images(mask, k)
    pos, vel = st[:, :2].double(), st[:, 2:4].double()
    # cells of 2h, 40 x 36 of them; the sweep below visits the 3 x 3 around a particle
    sys = _Sys(2 * k.h, 0, 1, 0.0, 0.0, 0, (0,), (0,), (0,), [40, 36, 1], dims=2)
    for _ in range(c["steps"]):
        prev = pos
        vel = vel + torch.tensor([0.0, _f32(-9.81)], dtype=torch.float64, device="cuda") * k.dt
        pos = pos + vel * k.dt
        key, order, each = _neighbours(torch.cat([pos, torch.zeros_like(pos[:, :1])], 1), sys)
        wall = _sample(img, pos[:, 0] / k.cw, pos[:, 1] / k.ch)
        den = torch.where(wall[:, 0] != 0, wall[:, 0], 0.0)
        near = torch.where(wall[:, 0] != 0, wall[:, 1], 0.0)

        def pairs():
            for j, ok in each():
                d = pos[j] - pos
                r = d.norm(dim=1)
                ok = ok & (r > 1e-7) & (r < k.h)
                yield j, d, torch.where(ok, r, 1.0), torch.where(ok, 1 - r / k.h, 0.0)

        for j, d, r, a in pairs():
            den = den + k.m * a ** 3 * k.kn
            near = near + k.m * a ** 4 * k.knn
        pr, prn = k.stiff * (den - k.m * k.rest), k.near_stiff * near
        x, dt2 = pos.clone(), k.dt * k.dt
        for j, d, r, a in pairs():
            push = dt2 * ((prn + prn[j]) * a ** 3 * k.knn + (pr + pr[j]) * a * a * k.kn) / 2
            surf = dt2 * k.tension * (a ** 3 * k.knn + a * a * k.kn) / 2
            x += d * (surf - push / (r * k.m))[:, None]
        wall = _sample(img, x[:, 0] / k.cw, x[:, 1] / k.ch)
        nrm = _sample(vec, x[:, 0] / k.cw, x[:, 1] / k.ch)
        a = 1 - nrm[:, 2] / k.h
        push = dt2 * ((prn + wall[:, 3]) * a ** 3 * k.knn + (pr + wall[:, 2]) * a * a * k.kn) / 2
        x = torch.where((wall[:, 0] != 0)[:, None], x + nrm[:, :2] * (push / k.m)[:, None], x)
        d = x - prev
        l = d.norm(dim=1, keepdim=True)
        d = d * (l.clamp(max=4 * k.psize) / l)
        vel, pos = d / k.dt, prev + d
    out = {"state": torch.cat([pos, vel, st[:, 4:].double()], 1)}
    if c["steps"] == 1:
        out["pressure"] = torch.stack([den, near, pr, prn], 1)[order]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "cloud"):
        return _exact_step(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "relax":
        return _exact_relax(case, seed)
    return None  # sorted pairs, and a tree with the first triangle a particle meets: nothing that 64 bits define
