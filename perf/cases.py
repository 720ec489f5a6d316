"""Performance cases of the framework: what its users have it do, through its public entry points.

A case is one of four kinds:

* ``stepper`` -- one engine object stepped by the drop-in ``GpuStepper`` (host state in and out every step);
* ``world``   -- one or many scenes resident in a ``DeviceWorld``: the state uploaded, a number of time steps
                 (``step``, or replays of a captured CUDA graph), the state read back;
* ``serve``   -- a ``Server`` that takes a stream of scene requests of different sizes and horizons to their end;
* ``grids``   -- the signed distance grids of many shapes (scene set-up).

Scenes are moving: ``prepare`` steps them in FP64 until their bodies have met, and a pass starts from the state
reached there, with no carried impulses, so that every pass does the same work.  A case fixes its bodies, shapes and
requests; the seed gives the bodies' places, turns and speeds.  Step outputs have no value of their own in 64 bits
short of the whole step restated (contact search, solver and all), so ``exact`` answers for the grids alone; FP64
steps are reproducible to the bit.
"""
import math

import numpy as np
import torch

from rainbow_b200 import api, engine_io, geometry, scenes, serving, types
from rainbow_b200 import world as W
from rainbow_b200.stepper import GpuStepper

DEVICE = "cuda:0"
GROUND = 24.0


def listed():
    return [
        # the smallest call: a handful of boxes in a user's own loop, bound by launches and host work
        dict(name="stack of 5, drop-in", kind="stepper", scene="tower", bodies=5, resolution=32,
             scheme="rigid_gauss_seidel", ordering="serial", stabilise=False),
        # the reference's CPU-sized scene through the drop-in stepper, coloured proximal Gauss-Seidel
        dict(name="64 boxes, drop-in", kind="stepper", scene="boxes", bodies=64, resolution=32,
             scheme="parallel_gauss_seidel", ordering="serial", stabilise=False),
        # the mass-ratio tower: one scene alone in FP64 and in FP32 with FP64 refinement
        dict(name="tower of 32, FP64", kind="world", scene="tower", bodies=32, scenes=1, resolution=32, steps=4,
             precision="fp64", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=100, graph=False),
        dict(name="tower of 32, FP32", kind="world", scene="tower", bodies=32, scenes=1, resolution=32, steps=4,
             precision="fp32_refine", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=100,
             graph=False),
        # one large scene: 4096 boxes and spheres in contact, in FP64 and in the fast mode
        dict(name="lattice of 4096, FP64", kind="world", scene="lattice", bodies=4096, scenes=1, resolution=64,
             steps=1, precision="fp64", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=100, graph=False),
        dict(name="lattice of 4096, FP32", kind="world", scene="lattice", bodies=4096, scenes=1, resolution=64,
             steps=2, precision="fp32_refine", termination="residual_fixed_r", scheme="rigid_gauss_seidel",
             sweeps=100, graph=False),
        # a pile too large for the shared memory of one multiprocessor, as the serving stream has them
        dict(name="pile of 1500, FP32", kind="world", scene="pile", bodies=1500, scenes=1, resolution=32, steps=2,
             precision="fp32_refine", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=400,
             graph=False),
        # many uneven scenes in one step, a shape and grid per body: the batched workload at its sweep limit,
        # at equal residual, and in FP64
        dict(name="batch of 512, FP32", kind="world", scene="pile", bodies=256, scenes=512, resolution=32, steps=4,
             precision="fp32_refine", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=100,
             graph=True),
        dict(name="batch of 128, equal residual", kind="world", scene="pile", bodies=256, scenes=128, resolution=32,
             steps=2, precision="fp32_refine", termination="residual_fixed_r", scheme="rigid_gauss_seidel",
             sweeps=4000, graph=True),
        dict(name="batch of 64, FP64", kind="world", scene="pile", bodies=256, scenes=64, resolution=32, steps=2,
             precision="fp64", termination="residual_fixed_r", scheme="rigid_gauss_seidel", sweeps=100, graph=False),
        # continuous batching: scenes join and leave, the batch is laid out anew on the device
        dict(name="serving 24 requests", kind="serve", requests=24, bodies=384, horizon=8, resolution=32,
             precision="fp32_refine", sweeps=100, resident=2048),
        # scene set-up: a grid for every one of 96 boxes and spheres
        dict(name="96 grids of 32^3", kind="grids", shapes=96, resolution=32),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["stepper", "stepper", "tower", "lattice", "pile", "batch", "batch", "serve", "grids"])
    scheme = rng.choice(["rigid_gauss_seidel", "rigid_gauss_seidel", "rigid_gauss_seidel", "parallel_gauss_seidel",
                         "parallel_jacobi_hybrid"])
    if kind == "stepper":
        return dict(kind="stepper", scene=rng.choice(["tower", "boxes"]), bodies=_spread(rng, 2, 64),
                    resolution=rng.randint(16, 40), scheme=rng.choice(["rigid_gauss_seidel", "parallel_gauss_seidel"]),
                    ordering=rng.choice(["serial", "coloured"]), stabilise=rng.random() < 0.3)
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(6, 24), bodies=_spread(rng, 48, 384),
                    horizon=rng.randint(3, 8), resolution=32, precision=rng.choice(["fp32_refine", "fp64"]),
                    sweeps=_spread(rng, 30, 100), resident=_spread(rng, 512, 2048))
    if kind == "grids":
        return dict(kind="grids", shapes=_spread(rng, 3, 96), resolution=rng.randint(17, 32))
    case = dict(kind="world", scene=kind if kind != "batch" else "pile", scenes=1, resolution=32, scheme=scheme,
                precision=rng.choice(["fp32_refine", "fp32_refine", "fp64", "fp32"]),
                termination="residual_fixed_r", steps=rng.randint(1, 2), sweeps=_spread(rng, 25, 100),
                graph=rng.random() < 0.5)
    if case["precision"] == "fp64":
        case["termination"] = rng.choice(["residual_fixed_r", "residual", "merit"])
    if kind == "tower":
        case["bodies"] = _spread(rng, 2, 48)
    elif kind == "lattice":
        case["bodies"] = rng.randint(3, 13) ** 3
    elif kind == "pile":
        case["bodies"] = _spread(rng, 100, 1500)
    else:
        case["bodies"] = _spread(rng, 12, 256)
        case["scenes"] = _spread(rng, 4, 256)
    return case


# ------------------------------------------------------------------------------------------------------------
# scenes
# ------------------------------------------------------------------------------------------------------------
def _engine(case, seed):
    """An engine object with a tower, or a lattice of unit boxes or of boxes and spheres."""
    rng = np.random.default_rng(seed)
    n = case["bodies"]
    if case["scene"] == "lattice":
        engine = scenes.mixed_lattice(n=round(n ** (1.0 / 3.0)), resolution=case["resolution"], seed=seed,
                                      device=DEVICE)
        return engine
    engine = scenes.box_tower(n, resolution=case["resolution"], device=DEVICE)
    side = math.ceil(n ** (1.0 / 3.0))
    for k in range(n):   # a little askew, and each box a little into the one below
        if case["scene"] == "tower":
            r = np.array([0.0, 0.498 + 0.998 * k, 0.0])
        else:
            i, j, l = k % side, k // (side * side), (k // side) % side
            r = np.array([1.05 * (i - 0.5 * (side - 1)), 0.498 + 0.998 * j, 1.05 * (l - 0.5 * (side - 1))])
        turn = geometry.quat_axis_angle(rng.uniform(-0.05, 0.05), np.array([0.0, 1.0, 0.0]))
        api.set_position(engine, "t%d" % k, r + rng.uniform(-0.02, 0.02, 3) * [1.0, 0.02, 1.0], True)
        api.set_orientation(engine, "t%d" % k, turn, True)
        if case["scene"] == "boxes":
            api.set_mass_properties(engine, "t%d" % k, 1.0)
    if case["scene"] == "boxes":
        engine.params.time_step = 0.01
    return engine


def _scatter(arrays, rng):
    """New places, turns and speeds for the bodies of these scenes (the ground, body 0, stays)."""
    for s in arrays:
        n = len(s["body_mass"]) - 1
        turn = rng.normal(size=(n, 4))
        for name, moved in (("body_q", turn / np.linalg.norm(turn, axis=1, keepdims=True)),
                            ("body_r", s["body_r"][1:] + rng.uniform(-0.1, 0.1, (n, 3))),
                            ("body_v", rng.uniform(-0.5, 0.5, (n, 3)) - [0.0, 2.0, 0.0]),
                            ("body_w", rng.uniform(-1.0, 1.0, (n, 3)))):
            s[name] = np.concatenate([s[name][:1], moved])
    return arrays


def _scene_list(case, seed):
    if case["scene"] != "pile":
        return [engine_io.scene_arrays(_engine(case, seed))]
    n = case["bodies"]
    lo = n if case["scenes"] == 1 else min(n, 8)
    arrays = scenes.batch_arrays_per_body(case["scenes"], seed=n + case["scenes"], body_range=(lo, n),
                                          resolution=case["resolution"], device=DEVICE,
                                          ground=max(GROUND, 2.3 * math.ceil(n ** (1.0 / 3.0)) + 8.0))[0]
    return _scatter(arrays, np.random.default_rng(seed))


def _pre_roll(world, params, scene):
    """FP64 steps until the bodies are in contact."""
    steps, dt = {"tower": (60, 0.01), "lattice": (24, None), "pile": (30, 0.02)}[scene]
    rp = W.make_rb_params(params, dt=dt, termination="residual_fixed_r", residual_interval=4, warm_start=True)
    rp.max_iterations = 30
    for _ in range(steps):
        world.step(rp)


# ------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"stepper": _prepare_stepper, "world": _prepare_world, "serve": _prepare_serve,
            "grids": _prepare_grids}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_stepper(case, seed):
    engine = _engine(case, seed)
    engine.params.proximal_solver = case["scheme"]
    engine.params.contact_ordering = case["ordering"]
    engine.params.use_pre_stabilization = engine.params.use_post_stabilization = case["stabilise"]
    engine.stepper = GpuStepper(DEVICE)
    dt = engine.params.time_step
    for _ in range(48):
        engine.stepper.step(0.01, engine, False)
    start = [(b, b.r, b.q, b.v, b.w) for b in engine.bodies.values()]
    return dict(run=_run_stepper, engine=engine, start=start, dt=dt)


def _run_stepper(state):
    engine = state["engine"]
    for b, r, q, v, w in state["start"]:
        b.r, b.q, b.v, b.w = r, q, v, w
    engine.stepper.step(state["dt"], engine, False)
    bodies = engine.bodies.values()
    ids, p, n, g = engine.contact_points.arrays()
    contacts = np.full((24 * len(bodies), 9), -1.0)   # one size for every seed's contacts
    contacts[:len(g)] = np.concatenate([ids, p, n, g[:, None]], axis=1)
    return dict(r=np.array([b.r for b in bodies]), q=np.array([b.q for b in bodies]),
                v=np.array([b.v for b in bodies]), w=np.array([b.w for b in bodies]), contacts=contacts)


def _prepare_world(case, seed):
    arrays = _scene_list(case, seed)
    params = W.params_from_vector(arrays[0]["params"])
    world = W.DeviceWorld(arrays, device=DEVICE, max_iterations=max(100, case["sweeps"]))
    _pre_roll(world, params, case["scene"])
    x, u = world.state()
    rp = W.make_rb_params(params, scheme=case["scheme"], termination=case["termination"],
                          precision=case["precision"], residual_interval=4, warm_start=True)
    rp.max_iterations = case["sweeps"]
    state = dict(run=_run_world, world=world, rp=rp, x=x, u=u, steps=case["steps"], graph=None)
    if case["graph"]:   # a captured step needs work lists that hold every step's contacts
        sizing = W.make_rb_params(params, termination="residual_fixed_r", residual_interval=4, warm_start=True)
        sizing.max_iterations = 30
        for _ in range(case["steps"] + 2):
            world.step(sizing)
        state["graph"] = world.capture(rp)
    return state


def _run_world(state):
    world = state["world"]
    world.set_state(state["x"], state["u"])
    world.reset_warm_start()
    for _ in range(state["steps"]):
        if state["graph"] is not None:
            state["graph"].replay()
        else:
            world.step(state["rp"])
    x, u = world.state()
    return dict(x=x, u=u, contacts=world.n_contacts_total())


def _prepare_serve(case, seed):
    rng, fixed = np.random.default_rng(seed), np.random.default_rng(case["requests"])
    arrays, params = scenes.batch_arrays(n_scenes=12, seed=case["requests"], pool=6, body_range=(16, case["bodies"]),
                                         resolution=case["resolution"], device=DEVICE, ground=GROUND)
    requests = []
    for k in range(case["requests"]):   # a pile already close to the ground: its bodies meet within a few steps
        scene = _scatter([dict(arrays[int(fixed.integers(len(arrays)))])], rng)[0]
        scene["body_v"][1:, 1] += rng.uniform(-20.0, -8.0)
        requests.append((scene, int(fixed.integers(2, case["horizon"] + 1))))
    rp = W.make_rb_params(params, termination="residual_fixed_r", precision=case["precision"], residual_interval=4,
                          warm_start=True)
    rp.max_iterations = case["sweeps"]
    server = serving.Server(rp, device=DEVICE, max_iterations=case["sweeps"], max_active_bodies=case["resident"])
    return dict(run=_run_serve, server=server, requests=requests)


def _run_serve(state):
    server = state["server"]
    uids = [server.submit(scene, horizon) for scene, horizon in state["requests"]]
    server.run()
    done = {r.uid: r.result for r in server.finished}
    server.finished.clear()
    return dict(x=np.concatenate([done[k][0] for k in uids]), u=np.concatenate([done[k][1] for k in uids]))


def _prepare_grids(case, seed):
    rng = np.random.default_rng(seed)
    V, T, metas = [], [], []
    n = case["resolution"]
    for k in range(case["shapes"]):   # boxes and 16 x 16 spheres by turns, each of a size of its own
        if k % 2 == 0:
            v, t = geometry.create_box(*rng.uniform(0.5, 2.0, 3))
        else:
            v, t = geometry.create_sphere(rng.uniform(0.25, 1.0), 16, 16)
        margin = 0.1 * float((v.max(axis=0) - v.min(axis=0)).max())
        V.append(v)
        T.append(np.asarray(t, np.int32))
        metas.append(types.Grid(v.min(axis=0) - margin, v.max(axis=0) + margin, n, n, n).meta())
    return dict(run=_run_grids, V=V, T=T, metas=metas)


def _run_grids(state):
    return geometry.signed_distance_grids(state["V"], state["T"], state["metas"], device=DEVICE)[0]


# ------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------
def work(case):
    """Body state and statics, the bodies' vertices and one update of one contact per body and sweep bound are
    not known before the step; counted are what every step must touch: 104 B of state read and written and 80 B
    of statics per body, each body's mesh once (24 B a vertex, 12 B a triangle), and per body the transform of
    its vertices (36 flops each) and one sweep over one contact (four rows of 12 products each way, ~220 flops)."""
    if case["kind"] == "grids":
        nodes = case["resolution"] ** 3 * case["shapes"]
        return {"bytes": 8.0 * nodes, "flops": 200.0 * nodes * 0.5 * (12 + 448)}
    if case["kind"] == "serve":
        bodies = case["requests"] * (case["bodies"] - 16.0) / math.log(case["bodies"] / 16.0)
        steps = 0.5 * (2 + case["horizon"])
    else:
        n = case["bodies"]
        many = case.get("scenes", 1)
        bodies = n if many == 1 else many * ((n - 8.0) / math.log(n / 8.0) if n > 8 else n)
        steps = case.get("steps", 1)
    round_ = 0.0 if case.get("scene") in ("tower", "boxes") else 0.5   # share of spheres
    vertices, triangles = 8 + round_ * (226 - 8), 12 + round_ * (448 - 12)
    return {"bytes": steps * bodies * (2 * 104.0 + 80.0 + 24.0 * vertices + 12.0 * triangles),
            "flops": steps * bodies * (36.0 * vertices + 220.0)}


# ------------------------------------------------------------------------------------------------------------
# the same in 64 bits, without the framework's own code
# ------------------------------------------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "grids":
        return None
    s = _prepare_grids(case, seed)
    return torch.cat([_signed_distance(torch.from_numpy(np.asarray(v, np.float64)[t]).to(DEVICE), m)
                      for v, t, m in zip(s["V"], s["T"], s["metas"])])


def _signed_distance(tri, meta):
    """Distance of every grid node (i fastest) to the triangles, negative where the winding number is over 1/2:
    the nearer of each triangle's three edge segments, or its plane where the foot point lies inside."""
    n = [int(v) for v in meta[9:12]]
    at = [meta[a] + meta[6 + a] * torch.arange(n[a], dtype=torch.float64, device=DEVICE) for a in range(3)]
    k, j, i = torch.meshgrid(at[2], at[1], at[0], indexing="ij")
    nodes = torch.stack([i, j, k], dim=-1).reshape(-1, 3)
    corner = [tri[:, c][None] for c in range(3)]
    normal = torch.linalg.cross(corner[1] - corner[0], corner[2] - corner[0])
    unit = normal / normal.norm(dim=-1, keepdim=True)
    out = []
    for p in nodes.split(8192):
        p = p[:, None]
        away = [p - c for c in corner]
        height = (away[0] * unit).sum(-1)
        inside = torch.ones_like(height, dtype=torch.bool)
        nearest = torch.full_like(height, math.inf)
        for c in range(3):
            edge = corner[(c + 1) % 3] - corner[c]
            along = ((away[c] * edge).sum(-1) / (edge * edge).sum(-1)).clamp(0.0, 1.0)
            nearest = torch.minimum(nearest, (away[c] - along[..., None] * edge).norm(dim=-1))
            inside &= (torch.linalg.cross(edge.expand_as(away[c]), away[c]) * unit).sum(-1) >= 0.0
        nearest = torch.where(inside, height.abs(), nearest).amin(dim=1)
        a, b, c = away
        la, lb, lc = (v.norm(dim=-1) for v in away)
        solid = torch.atan2((a * torch.linalg.cross(b, c)).sum(-1),
                            la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb)
        winding = 2.0 * solid.sum(dim=1).abs() / (4.0 * math.pi)
        out.append(torch.where(winding > 0.5, -nearest, nearest))
    return torch.cat(out)
