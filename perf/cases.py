"""The work that users of the framework have it do, as measurable cases.

One pass is one call, or a short run of calls, through the public entry points: a frame of a running
simulation (`Fluid.step`), the first frames of a scene that is started again (`Fluid.reset`, then frames, with
the bodies' coupling loop where the scene has bodies), a batch of simulations stepped together (`Batch.step`),
and the forward and backward pass of the warm start's network (`UNet.gradients`).

Scenes follow `bevy_eulerian_fluid_b200/scenes.py`: water at rest that collapses (a one-shot box source at the
bottom or the side), length unit 10, rho 99.7, 1/60 s frames, walls on all sides.  The seed moves the water's
shape, the bodies, the sources and the droplets.  A frame's outputs are the fields a program reads afterwards
(both velocity components, the level set and the pressure, as views of the device planes), the forces on the
bodies where there are any and the particle counts where there are particles.

Frames have no 64-bit values to be held to: the level set's signs decide which cells are water, so an f32 and a
64-bit run part at single cells after one frame (`exact` gives None).  The network's gradients have.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from bevy_eulerian_fluid_b200 import _capi as capi
from bevy_eulerian_fluid_b200 import learned, scenes
from bevy_eulerian_fluid_b200.plugin import (Collider, FastIterativeMethodConfig, FluidPlugin, FluidSettings,
                                             FluidSource, FluidSourceMode, FluidSourceShape, FluidSourceVelocity,
                                             ForceToFluid, GaussSeidelConfig, ParticleLevelsetTwoLayersPlugin,
                                             ProjectionMethod, ReinitializeMethod, RigidBody, RigidBodyKind,
                                             pack_obstacles)
from bevy_eulerian_fluid_b200.rigid import RigidWorld, device_bodies

DT, RHO, LENGTH_UNIT = scenes.DT, scenes.RHO, scenes.LENGTH_UNIT

FRAMES = {"kind": "frames", "solver": "gauss-seidel", "tolerance": 0.0, "reinit": "fim", "bodies": 0,
          "coupling": "none", "forces": 0, "inflow": False, "particles": False, "frames": 1}


def frames(name, nx, ny, **kw):
    c = dict(FRAMES, nx=nx, ny=ny, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest grid in use (the tests' scenes): default settings, one frame; latency and launches.
        frames("frame 64x64", 64, 64, inflow=True),
        # A ragged grid (no multiple of 64) with the Jacobi projection, jump flooding, a few bodies driven by the
        # host and local forces from user input: an interactive toy with every component in use.
        frames("frame 200x136 jacobi", 200, 136, solver="jacobi", reinit="jfa", bodies=4, coupling="host", forces=8),
        # The reference's example scene (water_surface: 256^2, 20 red-black iterations, fast iterative method).
        frames("frame 256x256", 256, 256, inflow=True),
        # The multigrid projection at its defaults (one V-cycle a frame) on a wide window.
        frames("frame 768x512 multigrid", 768, 512, solver="multigrid", inflow=True),
        # Default settings on a large grid: every stage is a pass over memory.
        frames("frame 2048x2048", 2048, 2048, bodies=1, coupling="static", inflow=True),
        # The two-way coupled scene (the benchmark's): 24 bodies, jump flooding, red-black to 1e-5, the host's
        # rigid-body loop between the frames.
        frames("coupled 512x512", 512, 512, tolerance=1e-5, reinit="jfa", bodies=24, coupling="host", frames=4),
        # The same scene with multigrid-preconditioned conjugate gradients, its bodies integrated on the device.
        frames("coupled 512x512 mgpcg", 512, 512, solver="mgpcg", tolerance=1e-5, reinit="jfa", bodies=24,
               coupling="device", frames=8),
        # The large dam break around a static circle, solved to 1e-5: the largest work.
        frames("dam break 4096x4096 mgpcg", 4096, 4096, solver="mgpcg", tolerance=1e-5, bodies=1, coupling="static",
               frames=4),
        # Iterated multigrid V-cycles to 1e-5, the offline setting at 2048^2.
        frames("dam break 2048x2048 v-cycles", 2048, 2048, solver="multigrid", tolerance=1e-5, bodies=1,
               coupling="static", frames=4),
        # A frame with the two-layer particle level set (about 2.7 million particles).
        frames("frame 512x512 particles", 512, 512, particles=True, inflow=True),
        # Many pools of different sizes stepped together (examples/multiple.rs spawns several fluids).
        {"name": "batch of 32 pools", "kind": "batch", "pools": 32, "smallest": 128, "largest": 768, "frames": 2},
        # Training of the learned warm start on a caller's own samples: forward, loss and every gradient.
        {"name": "network gradients 256x256", "kind": "network", "nx": 256, "ny": 256},
    ]


def _log(rng, lo, hi, multiple):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng: random.Random):
    pick = rng.randrange(8)
    if pick <= 1:  # a frame at default settings, any size the grid rule allows (multiples of 8)
        solver = rng.choice(["gauss-seidel", "gauss-seidel", "jacobi"])
        top = 2048 if solver == "gauss-seidel" else 768
        return frames(None, _log(rng, 48, top, 8), _log(rng, 48, top, 8), solver=solver,
                      reinit=rng.choice(["fim", "jfa"]), bodies=rng.choice([0, 0, 3, 12]), coupling="static",
                      forces=rng.choice([0, 0, 5]), inflow=rng.random() < 0.5)
    if pick == 2:  # one V-cycle a frame
        return frames(None, _log(rng, 128, 2048, 64), _log(rng, 128, 2048, 64), solver="multigrid",
                      reinit=rng.choice(["fim", "jfa"]), inflow=True)
    if pick == 3:  # coupled scenes, red-black to a tolerance
        n = _log(rng, 96, 640, 32)
        return frames(None, n, max(96, _log(rng, 0.6 * n, n, 8)), tolerance=rng.choice([1e-4, 1e-5]),
                      reinit=rng.choice(["fim", "jfa"]), bodies=rng.randrange(2, 25),
                      coupling=rng.choice(["host", "device"]), frames=rng.randrange(2, 5))
    if pick == 4:  # conjugate gradients to a tolerance
        n = _log(rng, 256, 4096, 64)
        return frames(None, n, _log(rng, max(192, n // 2), n, 64), solver="mgpcg", tolerance=1e-5,
                      reinit=rng.choice(["fim", "jfa"]), bodies=rng.randrange(1, 13), coupling="device",
                      frames=rng.randrange(2, 5))
    if pick == 5:
        return frames(None, _log(rng, 96, 768, 8), _log(rng, 96, 768, 8), particles=True,
                      reinit=rng.choice(["fim", "jfa"]), inflow=rng.random() < 0.5)
    if pick == 6:
        return {"kind": "batch", "pools": _log(rng, 4, 32, 1), "smallest": rng.choice([64, 128]),
                "largest": rng.choice([256, 512, 768]), "frames": 2}
    return {"kind": "network", "nx": _log(rng, 64, 384, 8), "ny": _log(rng, 64, 384, 8)}


# ---------------------------------------------------------------------------
# What a program has in hand

class _Plane:
    """A field's device plane as torch reads it in place (__cuda_array_interface__).  The tensor keeps this object,
    and this object the handle that owns the memory, so a result may outlive the program's own reference."""

    def __init__(self, owner, ptr, pitch, w, h):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (h, w), "strides": (pitch, 4), "typestr": "<f4",
                                         "data": (ptr, False), "version": 3}


FIELDS = {"u": capi.FIELD_U, "v": capi.FIELD_V, "level_set": capi.FIELD_LEVELSET_AIR, "pressure": capi.FIELD_PRESSURE}


def _views(owner, sim, kept):
    out = {}
    for name, f in FIELDS.items():
        ptr, pitch = sim.device_ptr(f)
        if (name, ptr) not in kept:
            w, h, _ = sim.field_shape(f)
            kept[name, ptr] = torch.as_tensor(_Plane(owner, ptr, pitch, w, h), device="cuda")
        out[name] = kept[name, ptr]
    return out


def _projection(case):
    kw = {"tolerance": case["tolerance"]}
    if case["solver"] == "jacobi":
        return ProjectionMethod.Jacobi()
    if case["solver"] == "multigrid":
        return ProjectionMethod.MultiGrid(max_iterations=60, **kw)
    if case["solver"] == "mgpcg":
        return ProjectionMethod(capi.PROJECTION_MGPCG, max_iterations=60, **kw)
    return ProjectionMethod.GaussSeidel(GaussSeidelConfig(20), **kw)


def _bodies(case, rng):
    nx, ny, n = case["nx"], case["ny"], case["bodies"]
    if case["coupling"] == "static" and n == 1:  # the large scenes' obstacle
        return [RigidBody(Collider.circle(min(nx, ny) / 16.0), (0.0, 0.0), kind=RigidBodyKind.Static, density=RHO)]
    s = min(nx, ny) / 512.0
    kind = RigidBodyKind.Static if case["coupling"] == "static" else RigidBodyKind.Dynamic
    out = []
    for i in range(n):
        if i % 4 == 0:
            col = Collider.circle(s * rng.uniform(8, 32))
        elif i % 4 == 1:
            col = Collider.rectangle(2 * s * rng.uniform(6, 30), 2 * s * rng.uniform(6, 30))
        elif i % 4 == 2:
            col = Collider.capsule(s * rng.uniform(5, 15), 2 * s * rng.uniform(10, 30))
        else:
            ang = sorted(rng.uniform(0, 2 * math.pi) for _ in range(3))
            col = Collider.triangle(*[(s * r * math.cos(a), s * r * math.sin(a))
                                      for a, r in zip(ang, [rng.uniform(10, 30) for _ in range(3)])])
        pos = (rng.uniform(-0.42 * nx, 0.42 * nx), rng.uniform(0.08 * ny, 0.42 * ny))
        out.append(RigidBody(col, pos, rng.uniform(0, 2 * math.pi), kind=kind, density=rng.uniform(0.5, 2.0) * RHO))
    return out


def _prepare_frames(case, seed):
    rng = random.Random(seed * 7919 + 17)
    nx, ny = case["nx"], case["ny"]
    plugin = FluidPlugin(LENGTH_UNIT)
    if case["particles"]:
        plugin.add_plugins(ParticleLevelsetTwoLayersPlugin())
    reinit = (ReinitializeMethod.JumpFlooding() if case["reinit"] == "jfa"
              else ReinitializeMethod.FastIterative(FastIterativeMethodConfig(10)))
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # the recommendation of multiples of 64
        fluid = plugin.spawn(FluidSettings(RHO, (0.0, 9.8), (nx, ny)), projection=_projection(case),
                             reinitialize=reinit)
    if case["bodies"] and case["coupling"] in ("host", "device"):  # the coupled scenes: a pool under the bodies
        depth = rng.uniform(0.35, 0.45) * ny
        fluid.add_source(FluidSource(), FluidSourceShape.Aabb((0.5 * nx, 0.5 * depth)),
                         (0.0, -0.5 * ny + 0.5 * depth), oneshot=True)
    else:  # the dam break: a column of water against the left wall
        w, h = rng.uniform(0.4, 0.7) * nx, rng.uniform(0.5, 0.7) * ny
        fluid.add_source(FluidSource(), FluidSourceShape.Aabb((0.5 * w, 0.5 * h)),
                         (-0.5 * nx + 0.5 * w, -0.5 * ny + 0.5 * h), oneshot=True)
    if case["inflow"]:  # a jet that keeps the water moving, and a drain
        r = 0.04 * min(nx, ny)
        fluid.add_source(FluidSource(), FluidSourceShape.Circle(r), (rng.uniform(-0.2, 0.3) * nx, 0.3 * ny),
                         FluidSourceVelocity((rng.uniform(-40.0, 40.0), 60.0)))
        fluid.add_source(FluidSource(mode=FluidSourceMode.Sink), FluidSourceShape.Circle(1.5 * r),
                         (0.45 * nx, -0.45 * ny))
    bodies = _bodies(case, rng)
    if bodies:
        fluid.set_rigid_bodies(bodies)
    forces = [ForceToFluid((rng.uniform(-40, 40), rng.uniform(-40, 40)),
                           (float(rng.randrange(nx)), float(rng.randrange(ny)))) for _ in range(case["forces"])]
    state = {"case": case, "fluid": fluid, "bodies": bodies, "forces": forces, "world": None, "views": {}}
    _start(state)
    if not case["tolerance"]:  # a running simulation, a few frames in
        for _ in range(3):
            _frame(state)
    return state


def _copies(bodies):
    return [RigidBody(b.collider, b.position, b.rotation, b.linear_velocity, b.angular_velocity, b.kind, b.density)
            for b in bodies]


def _start(state):
    """The scene from its first frame: the init sequence, the bodies where they begin."""
    case, fluid = state["case"], state["fluid"]
    fluid.reset()
    if case["coupling"] == "host":
        state["world"] = RigidWorld(_copies(state["bodies"]), (case["nx"], case["ny"]), gravity=9.8 * LENGTH_UNIT,
                                    grid_length=1.0 / LENGTH_UNIT)
        fluid.set_rigid_bodies(state["world"].bodies)
    elif case["coupling"] == "device":
        fluid.sim.set_obstacles(pack_obstacles(state["bodies"]))
        fluid.sim.set_rigid_bodies(device_bodies(state["bodies"]), 9.8 * LENGTH_UNIT, 1.0 / LENGTH_UNIT)
    fluid.step(DT)


def _frame(state):
    fluid = state["fluid"]
    if state["forces"]:
        fluid.forces_to_fluid.forces.extend(state["forces"])
    fluid.step(DT)
    if state["world"] is not None:  # two-way coupling on the host
        forces = fluid.sim.solid_forces()[:len(state["bodies"])]
        state["world"].apply_fluid_forces(forces, DT)
        state["world"].step(DT)
        fluid.set_rigid_bodies(state["world"].bodies)
        return forces
    return None


def _run_frames(state):
    case, fluid = state["case"], state["fluid"]
    if case["tolerance"]:
        _start(state)
    forces = None
    for _ in range(case["frames"]):
        forces = _frame(state)
    out = _views(fluid.sim, fluid.sim, state["views"])
    if forces is not None:
        out["forces"] = forces
    if case["coupling"] == "device":
        n = len(state["bodies"])
        out["bodies"] = np.array([[b.position[0], b.position[1], b.rotation] for b in fluid.sim.get_rigid_bodies(n)])
    if case["particles"]:
        (a, b), _ = fluid.sim.particle_counts()
        out["particles"] = [a, b]
    return out


def _prepare_batch(case, seed):
    lo, hi = case["smallest"], case["largest"]
    shapes = [s for s in [(64, 64), (96, 64)] + scenes.BATCH_SHAPES if lo <= max(s) <= hi and min(s) >= min(lo, 64)]
    rng = random.Random(case["pools"] * 131 + lo + hi)  # the sizes belong to the case, the water to the seed
    sizes = [rng.choice(shapes) for _ in range(case["pools"])]
    scs = [scenes.batch(1, seed=seed * 1009 + i, shapes=[s]).scenes[0] for i, s in enumerate(sizes)]
    bs = scenes.BatchScene("pools", scs, seed)
    batch = capi.Batch(capi.load(), bs.configs())
    bs.setup(batch.sims)
    state = {"case": case, "batch": batch, "scene": bs, "views": [{} for _ in scs]}
    for _ in range(5):  # the init sequence and the solver's choice of tiles
        batch.step(DT)
    return state


def _run_batch(state):
    batch = state["batch"]
    for sim in batch.sims:
        sim.reset()
    batch.step(DT)
    for k in range(state["case"]["frames"]):
        if k == 1:  # a gust over every pool
            for i, sim in enumerate(batch.sims):
                sim.set_local_forces(state["scene"].forces(i, 30))
        batch.step(DT)
    batch.sims[0].synchronize()
    views = [_views(batch, sim, kept) for sim, kept in zip(batch.sims, state["views"])]
    return {f: torch.cat([v[f].reshape(-1) for v in views]) for f in FIELDS}


def _sample(case, seed):
    """A training sample as the recorder makes it: normalised residual, fractions, level set, counted cells; the
    target is a smooth correction."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(seed * 31 + 5)
    y, x = np.mgrid[0:ny, 0:nx].astype(np.float32)
    surface = ny * (0.45 + 0.08 * np.sin(x * (2 * np.pi / nx) * rng.integers(1, 5) + rng.uniform(0, 6)))
    phi = (surface - y).astype(np.float32)
    mask = phi < 0
    smooth = sum(rng.normal() * np.cos(np.pi * (i * x / nx + j * y / ny) + rng.uniform(0, 6))
                 for i in range(4) for j in range(4)).astype(np.float32)
    res = rng.standard_normal((ny, nx)).astype(np.float32) + 0.5 * smooth
    feats = np.zeros((ny, nx, 16), np.float32)
    feats[..., 0] = np.where(mask, res / np.sqrt(np.mean(res[mask] ** 2)), 0.0)
    feats[..., 1] = feats[..., 2] = 1.0
    feats[:, [0, -1], 1] = feats[[0, -1], :, 2] = 0.5
    feats[..., 3] = np.clip(phi / ny, -1, 1)
    feats[..., 4] = mask
    target = np.where(mask, 20.0 * smooth, 0.0).astype(np.float32)
    return feats, target, mask.astype(np.uint8)


def _prepare_network(case, seed):
    n = max(case["nx"], case["ny"])
    net = learned.load_weights(capi.load(), n, n)
    return {"case": case, "net": net, "sample": _sample(case, seed)}


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    if case["kind"] == "network":
        return _prepare_network(case, seed)
    return _prepare_frames(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "batch":
        return _run_batch(state)
    if kind == "network":
        loss, grads = state["net"].gradients(*state["sample"])
        return {"loss": np.float32(loss), "gradients": grads}
    return _run_frames(state)


def work(case):
    if case["kind"] == "network":
        n = case["nx"] * case["ny"]
        params = sum(9 * ci * co + co for ci, co, _ in learned.UNET_CONVS)
        flops = learned.forward_flops(case["nx"], case["ny"])
        return {"bytes": n * (16 * 4 + 4 + 1) + 2 * 4 * params, "flops": 3 * flops}
    if case["kind"] == "batch":
        rng = random.Random(case["pools"] * 131 + case["smallest"] + case["largest"])
        lo, hi = case["smallest"], case["largest"]
        shapes = [s for s in [(64, 64), (96, 64)] + scenes.BATCH_SHAPES
                  if lo <= max(s) <= hi and min(s) >= min(lo, 64)]
        cells = sum(w * h for w, h in (rng.choice(shapes) for _ in range(case["pools"])))
    else:
        cells = case["nx"] * case["ny"]
    # A frame reads and writes both velocity components, the level set and the pressure (f32) once, and computes
    # about 500 operations a cell outside the projection; a red-black or Jacobi iteration is 13 more.
    per_cell = 500.0
    if case["kind"] == "frames" and not case["tolerance"]:
        per_cell += {"gauss-seidel": 20, "jacobi": 100, "multigrid": 8}[case["solver"]] * 13.0
    return {"bytes": 32.0 * cells * case["frames"], "flops": per_cell * cells * case["frames"]}


# ---------------------------------------------------------------------------
# The network in 64 bits

def exact(case, seed):
    if case["kind"] != "network":
        return None
    params = torch.tensor(np.load(learned.WEIGHTS_PATH)["params"], dtype=torch.float64, requires_grad=True)
    feats, target, mask = _sample(case, seed)
    F = torch.nn.functional
    convs, off = [], 0
    for i, (ci, co, _) in enumerate(learned.UNET_CONVS):
        w = params[off:off + 9 * ci * co].reshape(3, 3, co, ci).permute(2, 3, 0, 1)
        off += 9 * ci * co
        convs.append((w, params[off:off + co], i + 1 < len(learned.UNET_CONVS)))
        off += co

    def conv(i, x):
        w, b, relu = convs[i]
        y = F.conv2d(x, w, b, padding=1)
        return F.relu(y) if relu else y

    def up(x):
        return F.interpolate(x, scale_factor=2, mode="nearest")

    x = torch.tensor(feats, dtype=torch.float64).permute(2, 0, 1)[None]
    s0 = conv(1, conv(0, x))
    s1 = conv(3, conv(2, F.avg_pool2d(s0, 2)))
    s2 = conv(5, conv(4, F.avg_pool2d(s1, 2)))
    u = conv(7, conv(6, F.avg_pool2d(s2, 2)))
    u = conv(9, conv(8, torch.cat([up(u), s2], 1)))
    u = conv(11, conv(10, torch.cat([up(u), s1], 1)))
    u = conv(13, conv(12, torch.cat([up(u), s0], 1)))
    pred = conv(14, u)[0, 0]
    m = torch.tensor(mask != 0)
    t = torch.tensor(target, dtype=torch.float64)
    loss = ((pred - t)[m] ** 2).sum() / (t[m] ** 2).sum()
    loss.backward()
    return {"loss": loss.detach().numpy(), "gradients": params.grad.numpy()}
