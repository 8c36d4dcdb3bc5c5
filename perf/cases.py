"""The work a user of this framework has it do, as cases that can be timed and compared.

Each case goes through the public entry points (`VbdSolver`, `OgcWorld`, `Mlp`):
physics steps from a three-row patch to a 640 x 640 sheet, with each arithmetic,
initial guess and stopping rule, one collision detection through host arrays, and the
learned guess's network forward and backward. `listed()` holds the fixed cases,
`draw(rng)` gives others of the same ranges.

A step case starts every pass from the same state and runs `frames` steps, as a program
that simulates a few frames from a state it holds: `frames` > 1 makes the later steps
start from the history and the candidate cache that the earlier ones left.
"""
from __future__ import annotations

import dataclasses
import functools
import math
import os

import numpy as np
import torch

import clothcraft_b200
from clothcraft_b200 import scenes
from clothcraft_b200.learned import Mlp
from clothcraft_b200.profile_fold import FOLD_STATE
from clothcraft_b200.vbd import OgcWorld, VbdSolver

WEIGHTS = os.path.join(os.path.dirname(clothcraft_b200.__file__), "data", "fold_init_mlp.npz")
LANES32 = 8 | 4 << 8  # one FP32 sweep variant: FP32 sums of another lane count differ in their last bits


def _step(scene, **more):
    case = {"kind": "step", "scene": scene, "iterations": 20, "frames": 1, "tolerance": 0.0, "acceleration": 0.0,
            "learned": False, "precision": 0}
    case.update(more)
    return case


def listed():
    return [
        # the smallest interactive call: the reference's 3 x 3-cell patch of the default fabric
        # (compression law on) resting on a floor, default dt and 16 iterations
        _step("patch", name="patch_rest", cells=3, iterations=16),
        # the CPU-runnable scene: a 64 x 64 sheet on a sphere, two corners pinned, 20 iterations
        _step("sheet", name="sheet64", side=64, frames=2),
        # the benchmark's step: the 256 x 256 self-contact fold to a 1e-3 residual, learned guess,
        # Chebyshev acceleration
        _step("fold", name="fold256_learned", iterations=200, tolerance=1e-3, acceleration=0.95, learned=True,
              frames=2),
        # the reference's own step on the fold: 30 fixed iterations in FP64
        _step("fold", name="fold256_fixed30", iterations=30, frames=2),
        # the same with FP32 element assembly
        _step("fold", name="fold256_fp32", iterations=30, precision=1),
        # the sewn garment: two irregular panels of ~20k vertices around a capsule
        _step("garment", name="garment40k", spacing=0.0036),
        # dense layered self-contact on an odd, oblong sheet: a roll of cloth
        _step("roll", name="roll201x311", nx=201, ny=311, iterations=20),
        # the scale run: a crumpling sheet with driven corners, 40 iterations
        _step("crumple", name="crumple640", side=640, iterations=40),
        # uneven independent instances stepped as one solver
        _step("batch", name="batch16", count=16, lo=32, hi=160),
        # collision detection alone, host arrays in and the whole contact set out
        {"kind": "detect", "name": "detect_fold", "scene": "fold", "radius_factor": 3.0},
        # the learned guess's inference on a fold's vertices (FP16 tensor cores)
        {"kind": "mlp", "name": "mlp_forward_fp16", "rows": 65536, "precision": 1},
        # one minibatch's loss and gradients (FP32), train_init's batch size
        {"kind": "mlp_grad", "name": "mlp_gradients", "rows": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["patch", "sheet", "sheet", "fold", "roll", "roll", "crumple", "garment", "batch", "detect", "mlp",
                       "mlp_grad"])
    if kind == "detect":
        return {"kind": "detect", "scene": "roll", "nx": _log(rng, 24, 300), "ny": _log(rng, 24, 300),
                "radius_factor": round(rng.uniform(2.0, 4.0), 3)}
    if kind == "mlp":
        return {"kind": "mlp", "rows": _log(rng, 100, 400000), "precision": rng.choice([0, 1])}
    if kind == "mlp_grad":
        return {"kind": "mlp_grad", "rows": _log(rng, 100, 60000)}
    case = _step(kind, iterations=rng.randint(10, 30), frames=rng.randint(1, 2))
    if kind == "patch":
        case["cells"] = rng.randint(2, 24)
    elif kind == "sheet":
        case["side"] = _log(rng, 20, 160)
    elif kind == "roll":
        case["nx"], case["ny"] = _log(rng, 32, 280), _log(rng, 32, 280)
    elif kind == "crumple":
        case["side"] = _log(rng, 96, 400)
    elif kind == "garment":
        case["spacing"] = round(rng.uniform(0.006, 0.02), 5)
    elif kind == "batch":
        case["count"], case["lo"], case["hi"] = rng.randint(2, 12), 24, _log(rng, 40, 120)
    option = rng.choice(["fixed", "fixed", "target", "learned", "fp32"])
    if kind in ("fold", "sheet", "roll") and option != "fixed":
        if option == "fp32":
            case["precision"], case["frames"] = 1, 1
        else:
            case.update(iterations=60, tolerance=1e-3, acceleration=rng.choice([0.0, 0.9, 0.95]),
                        learned=option == "learned")
    return case


# ------------------------------------------------------------------ scenes
# Meshes depend on the case alone and are kept; positions and velocities on the seed.
@functools.lru_cache(maxsize=4)
def _fold_scene():
    with np.load(FOLD_STATE) as z:
        return scenes.config1(), z["x"].astype(np.float64), z["v"].astype(np.float64), float(z["time"])


@functools.lru_cache(maxsize=4)
def _garment_scene(spacing):
    return scenes.config3(spacing=spacing)


@functools.lru_cache(maxsize=4)
def _crumple_scene(side):
    return scenes.config4(n_side=side)


SPACING = 0.004  # vertex spacing of the rolls, the fold's


@functools.lru_cache(maxsize=4)
def _roll_mesh(nx, ny):
    return scenes.build_mesh(scenes.grid_uv(nx, ny, SPACING * (nx - 1), SPACING * (ny - 1)),
                             scenes.grid_triangles(nx, ny, alternate=False), scenes.Material.stvk_mapped())


def _pinned(mesh, pins, x):
    """The mesh with these vertices pinned where they are."""
    flags = np.zeros(mesh.n, np.uint8)
    flags[list(pins)] = 1
    where = np.zeros((mesh.n, 3))
    where[list(pins)] = x[list(pins)]
    return dataclasses.replace(mesh, pinned=flags, pin_positions=where)


def _turn(rng):
    a = rng.uniform(0.0, 2.0 * math.pi)
    return np.array([[math.cos(a), 0.0, math.sin(a)], [0.0, 1.0, 0.0], [-math.sin(a), 0.0, math.cos(a)]])


def _breeze(x, rng, speed):
    """A smooth velocity field (three waves of ~20 cm) of about `speed` m/s."""
    v = np.zeros_like(x)
    for _ in range(3):
        k = rng.normal(size=3)
        k *= 30.0 / np.linalg.norm(k)
        v += np.sin(x @ k + rng.uniform(0.0, 6.28))[:, None] * rng.normal(size=3) * (speed / 2.0)
    return v


def _scene(case, seed):
    """(scene, x, v, time) of a case: what the program holds before the call."""
    rng = np.random.default_rng(seed)
    kind = case["scene"]
    if kind == "fold":  # the committed fold-phase state, turned about the vertical with its sphere
        sc, x, v, t = _fold_scene()
        R = _turn(rng)
        obstacle = scenes.Obstacle(np.ascontiguousarray(sc.obstacle.vertices @ R.T), sc.obstacle.triangles)
        x = np.ascontiguousarray(x @ R.T)
        v = np.ascontiguousarray(v @ R.T) + _breeze(x, rng, 0.01)
        return dataclasses.replace(sc, obstacle=obstacle, x0=x, v0=v), x, v, t
    if kind == "garment":
        sc = _garment_scene(case["spacing"])
        R = _turn(rng)
        obstacle = scenes.Obstacle(np.ascontiguousarray(sc.obstacle.vertices @ R.T), sc.obstacle.triangles)
        x = np.ascontiguousarray(sc.x0 @ R.T)
        v = _breeze(x, rng, 0.1)
        return dataclasses.replace(sc, obstacle=obstacle, x0=x, v0=v), x, v, 0.0
    if kind == "crumple":
        sc = _crumple_scene(case["side"])
        x = sc.x0 + rng.uniform(-1e-5, 1e-5, sc.x0.shape)
        sc = dataclasses.replace(sc, mesh=_pinned(sc.mesh, np.nonzero(sc.mesh.pinned)[0], x), x0=x,
                                 v0=_breeze(x, rng, 0.02))
        return sc, scenes.driven_corners(sc, x, sc.settings.dt), sc.v0, 0.0
    if kind == "patch":  # resting_patch's layout with `cells` cells of 4 cm a side
        c = case["cells"]
        size = 0.04 * c
        mesh = scenes.pattern_build(size, size, c, c, scenes.Material())
        x = np.stack([mesh.uv[:, 0] - 0.5 * size, np.full(mesh.n, 0.00305), mesh.uv[:, 1] - 0.5 * size], axis=1)
        x[:, 1] += rng.uniform(0.0, 1e-4, mesh.n)
        floor = scenes.Obstacle(np.array([[-2.0, 0.0, -2.0], [2.0, 0.0, -2.0], [0.0, 0.0, 3.0]]),
                                np.array([[0, 2, 1]], dtype=np.uint32))
        v = rng.normal(0.0, 0.005, x.shape)
        sc = scenes.Scene("patch", mesh, floor, x, v, scenes.StepSettings(), 1)
        return sc, x, v, 0.0
    if kind == "sheet":  # config 0's sheet as it meets the sphere
        n = case["side"]
        side = (n - 1) * (0.5 / 63)
        mesh, x = scenes.sheet(n, side, 0.0, scenes.Material.stvk_mapped(), jitter=1e-4, seed=seed)
        ball = scenes.icosphere(3, 0.2 * side + 0.02)
        x[:, 1] += 0.2 * side + 0.02 + 0.0025
        v = _breeze(x, rng, 0.05) - np.array([0.0, 0.2, 0.0])
        mesh = _pinned(mesh, (0, n - 1), x)
        v[[0, n - 1]] = 0.0
        sc = scenes.Scene("sheet", mesh, ball, x, v, scenes.config0(n_side=4).settings, 1)
        return sc, x, v, 0.0
    # a roll: the sheet wound into a spiral whose turns lie 1.5 contact radii apart
    nx, ny = case["nx"], case["ny"]
    mesh = _roll_mesh(nx, ny)
    radius = 0.25 * SPACING
    pitch, r0 = 1.5 * radius, 0.035
    th = np.linspace(0.0, 2.0 + SPACING * nx / r0, 40 * nx + 2000)
    rr = r0 + pitch * th / (2.0 * math.pi)
    ds = np.hypot(np.diff(rr), 0.5 * (rr[1:] + rr[:-1]) * np.diff(th))
    a = np.interp(mesh.uv[:, 0], np.concatenate([[0.0], np.cumsum(ds)]), th)
    r = r0 + pitch * a / (2.0 * math.pi)
    x = np.stack([r * np.cos(a), r * np.sin(a), mesh.uv[:, 1]], axis=1)
    x = (x + np.random.default_rng(nx * 1000 + ny).uniform(-1e-5, 1e-5, x.shape)) @ _turn(rng).T
    v = _breeze(x, rng, 0.05)
    mesh = _pinned(mesh, (nx - 1, nx * ny - 1), x)  # the outer end's corners
    v[[nx - 1, nx * ny - 1]] = 0.0
    s = scenes.StepSettings(dt=1 / 60, iterations=20, damping=1.5, radius=radius, stiffness=1e4)
    return scenes.Scene("roll", mesh, None, np.ascontiguousarray(x), v, s, 1), x, v, 0.0


def _settings(case, base):
    s = dataclasses.replace(base, iterations=case["iterations"], sweep_precision=case["precision"])
    if case["tolerance"] > 0.0:
        s = dataclasses.replace(s, residual_tolerance=case["tolerance"], residual_check_every=2, stall_refresh=2,
                                acceleration=case["acceleration"], init_mode=1 if case["learned"] else 0)
    return s


# ------------------------------------------------------------------ network
def _features(rows, seed):
    """Features as a step makes them: displacements of a few units, a unit normal, strains, distances."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.randn((rows, 24), generator=g, device="cuda")
    f[:, 6:12] *= 0.3
    f[:, 12:15] /= f[:, 12:15].norm(dim=1, keepdim=True)
    f[:, 15:18] = f[:, 15:18].abs() * 0.5
    f[:, 18:20] = torch.rand((rows, 2), generator=g, device="cuda") * torch.tensor([1.0, 4.0], device="cuda")
    f[:, 23] = 0.0
    return f.contiguous(), (0.5 * torch.randn((rows, 3), generator=g, device="cuda")).contiguous()


def _layers64():
    with np.load(WEIGHTS) as z:
        p = torch.from_numpy(z["params"].astype(np.float64)).cuda()
    out, at = [], 0
    for outs, ins in ((64, 24), (64, 64), (64, 64), (3, 64)):
        out.append((p[at:at + outs * ins].reshape(outs, ins), p[at + outs * ins:at + outs * ins + outs]))
        at += outs * ins + outs
    return out


def _forward64(f, layers):
    h = f.double()
    for k, (W, b) in enumerate(layers):
        h = h @ W.T + b
        if k < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    return h


# --------------------------------------------------------------------- cases
class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    if case["kind"] in ("mlp", "mlp_grad"):
        s.net = Mlp.load(WEIGHTS)
        s.features, s.targets = _features(case["rows"], seed)
        return s
    if case["kind"] == "detect":
        sc, x, _, _ = _scene(case, seed)
        solver_x = x if sc.obstacle is None else np.concatenate([x, sc.obstacle.vertices])
        tri = sc.mesh.triangles
        if sc.obstacle is not None:
            tri = np.concatenate([tri, sc.obstacle.triangles + np.uint32(sc.n)])
        s.world = OgcWorld(solver_x, tri, sc.n)
        # two frames' positions in turn, further apart than the candidate skin: the broad phase runs on
        # each, as it does on a moving cloth
        moved = np.array(solver_x)
        moved[:sc.n, 1] += 1.5 * sc.settings.radius
        s.x = [np.ascontiguousarray(solver_x), moved]
        s.settings = sc.settings
        s.rq = case["radius_factor"] * sc.settings.radius
        return s
    if case["scene"] == "batch":
        rng = np.random.default_rng(seed)
        insts = []
        for k, n in enumerate(_sides(case)):  # the sizes are the case's, the materials and positions the seed's
            one, x, v, _ = _scene({"scene": "sheet", "side": int(n)}, seed * 64 + k)
            shift = np.array([3.0 * (k % 10), 0.0, 3.0 * (k // 10)])
            x = x + shift
            obstacle = scenes.Obstacle(one.obstacle.vertices + shift, one.obstacle.triangles)
            scale = float(rng.uniform(0.5, 2.0))
            mesh = dataclasses.replace(_pinned(one.mesh, np.nonzero(one.mesh.pinned)[0], x),
                                       materials=[scenes.Material.stvk_mapped(mu=1e4 * scale, lam=2e4 * scale)])
            insts.append(dataclasses.replace(one, mesh=mesh, obstacle=obstacle, x0=x, v0=v))
        s.solver = VbdSolver.batch(insts)
        s.x, s.v = (np.concatenate([np.asarray(getattr(i, f)) for i in insts]) for f in ("x0", "v0"))
        s.t, base = 0.0, insts[0].settings
    else:
        sc, s.x, s.v, s.t = _scene(case, seed)
        s.solver = VbdSolver(sc)
        base = sc.settings
    if case["precision"]:
        s.solver.set_lanes32(LANES32)
    if case["learned"]:
        s.solver.set_mlp(Mlp.load(WEIGHTS), 1)
    s.settings = _settings(case, base)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "mlp":
        return s.net.forward(s.features, s.case["precision"])
    if kind == "mlp_grad":
        g, loss = s.net.gradients(s.features, s.targets)
        return {"gradient": g, "loss": np.float32(loss)}
    if kind == "detect":
        out = []
        for x in s.x:
            r = s.world.detect(x, s.rq, s.settings)
            out.append({"kinds": r["kinds"], "vertices": r["vertices"], "epsilon": r["epsilon"], "radii": r["radii"],
                        "offsets": r["incident_offsets"], "incident": r["incident"], "active": r["active_contacts"],
                        "minimum_distance": r["minimum_distance"]})
        return out
    c = s.settings.to_c()
    if s.solver.n <= 16384:  # interactive: the caller's own arrays go in and come back every frame
        x, v, t = s.x, s.v, s.t
        for _ in range(s.case["frames"]):
            x, v, t, m = s.solver.step(x, v, t, c)
    else:  # the state stays on the GPU between frames and is read at the end
        s.solver.set_state(s.x, s.v, s.t)
        for _ in range(s.case["frames"]):
            m = s.solver.step_resident(c)
        x, v, t = s.solver.get_state()
    # v is (x - x_old) / dt: x in full says what it is, and v in the 32 bits in which states are stored
    # (tests/golden); its last FP64 digits are x's last digits times 60 to 240
    return {"x": x, "v": v.astype(np.float32), "time": t, "iterations": int(m["iterations"]), "contact_terms": int(m["contact_terms"]),
            "colors": int(m["colors"]), "minimum_distance": float(m["minimum_distance_m"])}


def exact(case, seed):
    """Plain 64-bit results of the network; a step's result is an iterate that has none."""
    if case["kind"] not in ("mlp", "mlp_grad"):
        return None
    f, t = _features(case["rows"], seed)
    layers = _layers64()
    if case["kind"] == "mlp":
        return _forward64(f, layers)
    layers = [(W.clone().requires_grad_(True), b.clone().requires_grad_(True)) for W, b in layers]
    loss = (_forward64(f, layers) - t.double()).square().sum(dim=1).mean()
    loss.backward()
    g = torch.cat([torch.cat([W.grad.reshape(-1), b.grad.reshape(-1)]) for W, b in layers])
    return {"gradient": g.cpu().numpy(), "loss": loss.detach().cpu().numpy()}


def _sides(case):
    return np.linspace(case["lo"], case["hi"], case["count"]).astype(int)


def _vertices(case):
    kind = case["scene"]
    if kind == "patch":
        return (case["cells"] + 1) ** 2
    if kind in ("sheet", "crumple"):
        return case["side"] ** 2
    if kind == "roll":
        return case["nx"] * case["ny"]
    if kind == "fold":
        return 65536
    if kind == "garment":  # two 0.6 x 0.7 m panels; a Poisson-disk sample has ~0.63 points per spacing squared
        return int(2 * 0.42 * 0.63 / case["spacing"] ** 2)
    return int((_sides(case) ** 2).sum())


def work(case):
    """One pass, each array once. A vertex has 2 triangles and 3 hinges of its own: ids, rest shape and
    stiffness 2 x 56 + 3 x 24 bytes, mass, target and state ~150. A local solve evaluates 6 triangles and 12
    hinges with derivatives and once more for the line search, ~4,000 FP64 operations."""
    if case["kind"] == "mlp":
        return {"bytes": case["rows"] * 4 * 27 + 4 * 10115, "flops": case["rows"] * 2 * 9920}
    if case["kind"] == "mlp_grad":
        return {"bytes": case["rows"] * 4 * 27 + 8 * 10115, "flops": case["rows"] * 6 * 9920}
    n = _vertices(case)
    if case["kind"] == "detect":
        # positions, triangles, edges and their pairs (~20 candidates a vertex of ~60 operations), the contact set
        return {"bytes": 2 * n * (24 + 24 + 24 + 20 * 8 + 60), "flops": 2 * n * 20 * 60}
    its = case["iterations"] if case["tolerance"] == 0.0 else min(case["iterations"], 20)
    return {"bytes": case["frames"] * n * (184 + 150 + 20 * 8), "flops": case["frames"] * n * (its * 4000 + 2000)}
