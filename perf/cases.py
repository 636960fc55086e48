"""The work that programs have this framework do, as cases for timing it.

A case is a dict of plain values.  Its "kind" names the way of calling:

  frame    a game loop on one small world: update_world, then read the bodies
  run      runEngine on a scene of host objects: create, step, read, close
           (the reference's own benchmark, runWorld on Stacks.makeScene)
  rollout  one handle: the state is set, stepped n times and read back (a
           planner or a simulation environment); "scene" says which worlds
  io       several handles stepped together with the state in pinned host
           memory (step_many_io: state in, one step, state out)
  collide  contact queries of one large world between frames that the host
           moves: set_bodies, collide, contacts into pinned host memory (the
           whole buffer is the output: what no pass wrote stays zero)
  noalloc  shapes_collide_noalloc on the caller's own device buffers
  learned  a rollout with the learned warm start and its judge
  net      the network itself: predictions and the loss gradient

Sizes follow the workload definitions in shapes_gb300/scenes.py, the tests
and the benchmark: single worlds of tens to 65,536 bodies, batches of 4096
worlds, 2 to 8 sweeps, hulls of 3 to 8 vertices, circles.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from shapes_gb300 import _lib, engine, scenes

STEP_FIELDS = _lib.BODY_FIELDS[:6]  # what a step writes


def listed():
    return [
        # the smallest call: one frame of a small demo scene, reference defaults (2 sweeps, grid below its size)
        dict(name="frame_21", kind="frame", cols=5, rows=4, sweeps=2),
        # the reference's benchmark: a scene of 901 bodies made, stepped ten times, read and dropped
        dict(name="run_stacks_901", kind="run", cols=30, rows=30, steps=10),
        # one world of a 20 x 20 box stack, the single-world workload: a chain of dependent contacts
        dict(name="boxes_401", kind="rollout", scene="boxes", worlds=1, bodies=401, sweeps=4, settle=60, steps=5),
        # many columns of very different heights, the batched workload, default packing
        dict(name="columns_4096", kind="rollout", scene="columns", worlds=4096, bodies=512, sweeps=8, settle=60,
             steps=3),
        # 1024 piles of mixed boxes and polygons, the headline workload, with the packing the autotuner gives there
        dict(name="mixed_1024", kind="rollout", scene="mixed", worlds=1024, bodies=256, sweeps=8, settle=200,
             steps=3, packed=True),
        # an odd, middling batch of the same with the reference's two sweeps and default packing
        dict(name="mixed_75", kind="rollout", scene="mixed", worlds=75, bodies=121, sweeps=2, settle=150, steps=4),
        # circles and polygons in containers, stepped through pinned host memory by eight handles
        dict(name="balls_1024_io", kind="io", scene="balls", worlds=1024, bodies=128, sweeps=8, settle=90, handles=8),
        # one large world in a container: the order-preserving solve, then the coloured sweep
        dict(name="pile_32771", kind="rollout", scene="pile", worlds=1, bodies=32771, sweeps=4, settle=140, steps=2),
        dict(name="pile_65539_coloured", kind="rollout", scene="pile", worlds=1, bodies=65539, sweeps=4, settle=140,
             steps=2, coloured=True),
        # contact queries only: the 65,536-polygon workload between moving frames, and a plugin's small world
        dict(name="field_65536", kind="collide", bodies=65536),
        dict(name="noalloc_2001", kind="noalloc", bodies=2001),
        # the network: a batch of samples forward and backward
        dict(name="net_100003", kind="net", rows=100003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "run", "rollout", "rollout", "rollout", "io", "collide", "noalloc", "learned", "net"])
    if kind == "frame":
        return dict(kind=kind, cols=rng.randint(1, 8), rows=rng.randint(1, 8), sweeps=rng.randint(1, 8))
    if kind == "run":
        return dict(kind=kind, cols=rng.randint(2, 30), rows=rng.randint(2, 30), steps=rng.randint(1, 10))
    if kind == "collide":
        return dict(kind=kind, bodies=_log(rng, 500, 65536))
    if kind == "noalloc":
        return dict(kind=kind, bodies=_log(rng, 20, 4096))
    if kind == "net":
        return dict(kind=kind, rows=_log(rng, 100, 100003))
    if kind == "learned":
        return dict(kind=kind, scene="mixed", worlds=_log(rng, 2, 200), bodies=rng.randint(40, 256),
                    sweeps=rng.randint(2, 8), settle=60, steps=2)
    scene = rng.choice(["boxes", "columns", "mixed", "mixed", "balls", "pile"]) if kind == "rollout" else \
        rng.choice(["columns", "mixed", "balls"])
    c = dict(kind=kind, scene=scene, sweeps=rng.randint(2, 8))
    if scene == "boxes":
        n = rng.randint(5, 25)
        c.update(worlds=1, bodies=n * rng.randint(5, 25) + 1, settle=60, steps=rng.randint(1, 5))
    elif scene == "columns":
        c.update(worlds=_log(rng, 16, 2048), bodies=rng.randint(40, 512), settle=60, steps=rng.randint(1, 3))
    elif scene == "mixed":
        c.update(worlds=_log(rng, 2, 700), bodies=rng.randint(33, 256), settle=120, steps=rng.randint(1, 3),
                 packed=rng.random() < 0.5)
    elif scene == "balls":
        c.update(worlds=_log(rng, 2, 700), bodies=rng.randint(20, 160), settle=80, steps=rng.randint(1, 3))
    else:
        c.update(worlds=1, bodies=_log(rng, 4200, 32771), sweeps=4, settle=120, steps=rng.randint(1, 2),
                 coloured=rng.random() < 0.3)
    if kind == "io":
        c.update(handles=rng.choice([2, 4, 8]), worlds=max(c["worlds"], 16), steps=1, packed=False)
    return c


# ---------------------------------------------------------------------------------------------------------------------
# scenes


def _pile(seed, n, sweeps):
    """One container of n bodies, four times as wide as high, close enough that
    most touch once the settling steps have run: boxes of nearly the grid's
    pitch and, two in five, polygons of 3 to 8 vertices."""
    rng = np.random.default_rng(seed)
    nb, pitch = n - 3, 1.5
    xy, nvs, area, inertia = scenes.polygons_arrays(rng, nb, 0.48 * pitch, 0.52 * pitch)
    side, box = rng.uniform(0.93, 0.99, nb) * pitch, np.arange(nb) % 5 < 3
    hulls = np.split(xy, np.cumsum(nvs)[:-1])
    for k in np.flatnonzero(box):
        hulls[k] = scenes.rectangle_vertices(side[k], side[k])
    nvs = np.where(box, 4, nvs)
    area, inertia = np.where(box, side ** 2, area), np.where(box, side ** 4 / 6.0, inertia)
    cols = max(4, int(math.sqrt(4.0 * nb)))
    width = cols * pitch + 0.5
    high = (nb // cols + 2) * pitch + 40.0
    walls = [scenes.rectangle_vertices(width + 4.0, 2.0), scenes.rectangle_vertices(2.0, high),
             scenes.rectangle_vertices(2.0, high)]
    f = {k: np.zeros(n) for k in _lib.BODY_FIELDS}
    k = np.arange(nb)
    f["pos_x"][3:] = (k % cols - (cols - 1) / 2.0) * pitch
    f["pos_y"][3:] = (k // cols + 0.51) * pitch
    f["rot"][3:] = np.where(box, rng.uniform(-0.02, 0.02, nb), rng.uniform(0.0, 2.0 * np.pi, nb))
    f["inv_mass_lin"][3:], f["inv_mass_rot"][3:] = 1.0 / area, 1.0 / inertia
    f["mu"][:] = scenes.DEFAULT_MU
    f["pos_y"][0] = -1.0
    f["pos_x"][1:3] = -(width / 2.0 + 1.0), width / 2.0 + 1.0
    f["pos_y"][1:3] = high / 2.0 - 2.0
    return scenes.assemble([n], f, np.concatenate(walls + hulls), np.concatenate([[4, 4, 4], nvs]), dt=1.0 / 120.0,
                           baumgarte=scenes.DEFAULT_BAUMGARTE, slop=scenes.DEFAULT_SLOP, accel=(0.0, -9.8),
                           iterations=sweeps, steps=1)


def _boxes(seed, n, sweeps):
    rows = max(1, int(math.sqrt(n - 1)))
    s = scenes.single_world_boxes(seed=seed, cols=max(1, (n - 1) // rows), rows=rows)
    s["config"]["iterations"] = sweeps
    return s


def _scene(case, seed):
    kind, n, sweeps = case["scene"], case["bodies"], case["sweeps"]
    if kind == "boxes":
        return _boxes(seed, n, sweeps)
    if kind == "pile":
        return _pile(seed, n, sweeps)
    if kind == "columns":  # world sizes from the case alone, so that every seed has as many bodies
        s = scenes.batched_columns(seed=n, n_worlds=case["worlds"], nmin=8, nmax=n)
        rng, moves = np.random.default_rng(seed), s["bodies"]["inv_mass_lin"] != 0.0
        for f, by in (("pos_x", 0.05), ("rot", 0.02)):
            s["bodies"][f][moves] += rng.uniform(-by, by, int(moves.sum()))
    elif kind == "mixed":
        s = scenes.batched_mixed(seed=seed, n_worlds=case["worlds"], n_bodies=n)
    else:
        s = scenes.batched_balls(seed=seed, n_worlds=case["worlds"], n_bodies=n)
    s["config"]["iterations"] = sweeps
    return s


def _batch(s):
    return _lib.Batch(s["world_body_offsets"], s["bodies"], s["vert_offsets"], s["local_xy"], s.get("shape_kind"))


def _config(s, **flags):
    c = s["config"]
    return _lib.make_config(c["dt"], c["baumgarte"], c["slop"], c["accel"], c["iterations"], **flags)


def _shard(s, worlds):
    """The scene of the given worlds alone."""
    off, vo = s["world_body_offsets"], s["vert_offsets"]
    body = np.concatenate([np.arange(off[w], off[w + 1]) for w in worlds])
    vert = np.concatenate([np.arange(vo[off[w]], vo[off[w + 1]]) for w in worlds])
    out = scenes.assemble([off[w + 1] - off[w] for w in worlds], {k: v[body] for k, v in s["bodies"].items()},
                          s["local_xy"][vert], np.diff(vo)[body], **s["config"])
    if "shape_kind" in s:
        out["shape_kind"] = s["shape_kind"][body]
    return out


def _pinned(bodies):
    """(tensor [10, n] of the body state in pinned memory, the Bodies struct over it)."""
    t = torch.empty((len(_lib.BODY_FIELDS), len(bodies["pos_x"])), dtype=torch.float64, pin_memory=True)
    for k, name in enumerate(_lib.BODY_FIELDS):
        t[k] = torch.from_numpy(bodies[name])
    return t, _lib.Bodies(*[ctypes.cast(t[k].data_ptr(), _lib._dp) for k in range(len(_lib.BODY_FIELDS))])


def _engine_scene(b, accel):
    """The flat scene arrays as the engine API's objects, as a Haskell-style caller builds them."""
    objs = []
    vo, f = b["vert_offsets"], b["bodies"]
    for k in range(len(vo) - 1):
        masses = [1.0 / m if m else 0.0 for m in (f["inv_mass_lin"][k], f["inv_mass_rot"][k])]
        p = engine.make_physical_obj((f["vel_x"][k], f["vel_y"][k]), f["rot_vel"][k],
                                     (f["pos_x"][k], f["pos_y"][k]), f["rot"][k], masses)
        objs.append(engine.make_world_obj(p, f["mu"][k], f["bounce"][k],
                                          engine.make_hull(b["local_xy"][vo[k]:vo[k + 1]])))
    c = b["config"]
    return engine.Scene(engine.make_world(objs), engine.make_constant_accel(accel),
                        engine.ContactBehavior(c["baumgarte"], c["slop"]))


def _stacks(case, seed):
    """Stacks.makeScene with its boxes moved sideways by a seeded hair's breadth."""
    s = scenes.stacks_make_scene((case["cols"], case["rows"]))
    rng = np.random.default_rng(seed)
    s["bodies"]["pos_x"][1:] += rng.uniform(-0.01, 0.01, len(s["bodies"]["pos_x"]) - 1)
    return s


def _frame(case, seed):
    return scenes.single_world_boxes(seed=seed, cols=case["cols"], rows=case["rows"])


FRAME_SETTLE = 30


# ---------------------------------------------------------------------------------------------------------------------
# the network's samples


def _samples(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((case["rows"], _lib.SHAPES_MLP_FEATURES)).astype(np.float32)
    y = np.stack([np.maximum(x[:, 0] - 0.5 * x[:, 2], 0) + 0.3 * x[:, 5], 0.4 * x[:, 1] - 0.2 * x[:, 9]], 1)
    return x, y.astype(np.float32)


def _net_params(seed):
    rng = np.random.default_rng(seed + 1)
    layers = [(64, 16), (64, 64), (64, 64), (2, 64)]
    p = np.concatenate([np.concatenate([rng.uniform(-1, 1, o * i) * math.sqrt(6.0 / i), rng.uniform(-0.1, 0.1, o)])
                        for o, i in layers])
    norm = np.concatenate([rng.uniform(-0.2, 0.2, 16), rng.uniform(0.8, 1.2, 16), [0.1, -0.1], [1.5, 0.7]])
    return p.astype(np.float32), norm.astype(np.float32)


# ---------------------------------------------------------------------------------------------------------------------
# prepare and run


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        s = _frame(case, seed)
        sc = _engine_scene(s, s["config"]["accel"])
        st = engine.init_engine(sc)
        cfg = engine.EngineConfig(s["config"]["dt"], sc.contact_beh, case["sweeps"])
        engine.step_world(st, cfg, FRAME_SETTLE)
        return dict(kind=kind, state=st, cfg=cfg)
    if kind == "run":
        s = _stacks(case, seed)
        return dict(kind=kind, scene=_engine_scene(s, s["config"]["accel"]), dt=s["config"]["dt"],
                    steps=case["steps"])
    if kind == "net":
        x, y = _samples(case, seed)
        net = _lib.Mlp(seed=seed)
        net.set_params(*_net_params(seed))
        return dict(kind=kind, net=net, x=x, y=y)
    if kind in ("collide", "noalloc"):
        s = scenes.polygon_field(seed=seed, n=case["bodies"], extent=2.0 * math.sqrt(case["bodies"]))
        return _prepare_collide(s, seed) if kind == "collide" else _prepare_noalloc(s)
    s = _scene(case, seed)
    if kind == "io":
        w = case["worlds"]
        shards = [_shard(s, range(k, w, case["handles"])) for k in range(case["handles"])]
        batches, cfg = [_batch(q) for q in shards], _config(s)
        _lib.step_many(batches, cfg, case["settle"])
        ins = [_pinned(b.get_bodies()) for b in batches]
        outs = [_pinned(b.get_bodies()) for b in batches]
        return dict(kind=kind, batches=batches, cfg=cfg, ins=ins, outs=outs)
    b, plain = _batch(s), _config(s)
    if case.get("packed"):  # worlds per group, threads, warps per group: what the autotuner gives the headline scene
        b.set_launch_groups(2, 128, 4)
    if kind == "learned":
        net = _lib.Mlp(seed=seed)
        net.set_params(_net_params(seed)[0] * np.float32(0.3))
        b.step(plain, case["settle"])
        b.set_mlp(net)
        n = case["worlds"]
        b.set_judge(np.full(n, 2.0), np.full(n, 1.0))
        cfg = _config(s, learned=True, residual=True)
        return dict(kind=kind, batch=b, net=net, cfg=cfg, start=b.get_bodies(), steps=case["steps"])
    if case["scene"] == "pile":  # settles at twice the time step
        plain.dt *= 2.0
    b.step(plain, case["settle"])
    return dict(kind=kind, batch=b, cfg=_config(s, coloured=bool(case.get("coloured"))), start=b.get_bodies(),
                steps=case["steps"])


def _prepare_collide(s, seed):
    """Two frames of a field whose bodies drift by up to a tenth of a unit."""
    b = _batch(s)
    rng = np.random.default_rng(seed + 1)
    n = len(s["bodies"]["pos_x"])
    moved = dict(s["bodies"])
    for f in ("pos_x", "pos_y", "rot"):
        moved[f] = moved[f] + rng.uniform(-0.1, 0.1, n)
    cap = 4 * n + 1024
    keys = torch.zeros((cap, 5), dtype=torch.int32, pin_memory=True)
    vals = torch.zeros((cap, 5), dtype=torch.float64, pin_memory=True)
    return dict(kind="collide", batch=b, frames=[_pinned(s["bodies"]), _pinned(moved)], at=0, cap=cap, keys=keys,
                vals=vals)


def _prepare_noalloc(s):
    dev = torch.device("cuda", torch.cuda.current_device())
    f = {k: torch.from_numpy(s["bodies"][k]).to(dev) for k in
         ("pos_x", "pos_y", "rot", "inv_mass_lin", "inv_mass_rot")}
    n, nv = len(s["bodies"]["pos_x"]), int(s["vert_offsets"][-1])
    cap_p, cap_c = 8 * n + 64, 8 * n + 64
    return dict(kind="noalloc", f=f, n=n, nv=nv, vo=torch.from_numpy(s["vert_offsets"]).to(dev),
                xy=torch.from_numpy(s["local_xy"].reshape(-1)).to(dev), cap_p=cap_p, cap_c=cap_c,
                pairs=torch.zeros((cap_p, 2), dtype=torch.int32, device=dev),
                keys=torch.zeros((cap_c, 5), dtype=torch.int32, device=dev),
                vals=torch.zeros((cap_c, 5), dtype=torch.float64, device=dev), stream=torch.cuda.current_stream())


def run(state):
    kind = state["kind"]
    if kind == "frame":
        engine.update_world(state["state"], state["cfg"])
        return state["state"].batch.get_bodies()
    if kind == "run":
        def action(st, cfg):
            engine.step_world(st, cfg, state["steps"])
            return st.batch.get_bodies()

        return engine.run_engine(state["dt"], state["scene"], action)
    if kind == "rollout":
        b = state["batch"]
        b.set_bodies(state["start"])
        b.step(state["cfg"], state["steps"])
        return b.get_bodies()
    if kind == "learned":
        b = state["batch"]
        b.set_bodies(state["start"])
        b.step(state["cfg"], state["steps"])
        out = b.get_bodies()
        out["residual"], out["depth"] = b.world_metrics()
        return out
    if kind == "io":
        rc = _lib.step_many_io(state["batches"], state["cfg"], [b for _, b in state["ins"]],
                               [b for _, b in state["outs"]])
        _lib.check(rc, "step_many_io")
        return [t for t, _ in state["outs"]]
    if kind == "net":
        grad, loss = state["net"].gradient(state["x"], state["y"])
        return dict(out=state["net"].forward(state["x"]), grad=grad, loss=loss)
    return _run_collide(state) if kind == "collide" else _run_noalloc(state)


def _run_collide(state):
    b, L = state["batch"], _lib.lib()
    _, bodies = state["frames"][state["at"]]
    state["at"] = 1 - state["at"]
    _lib.check(L.shapes_batch_set_bodies(b.handle, ctypes.byref(bodies)), "set_bodies")
    b.collide()
    n = b.stats()["contacts"]
    wc = np.zeros(1, dtype=np.int32)
    _lib.check(L.shapes_batch_get_contacts(b.handle, ctypes.cast(state["keys"].data_ptr(), _lib._ip),
                                           ctypes.cast(state["vals"].data_ptr(), _lib._dp), state["cap"],
                                           wc.ctypes.data_as(_lib._ip)), "get_contacts")
    return dict(n=n, keys=state["keys"], vals=state["vals"])


def _run_noalloc(s):
    n_p, n_c = ctypes.c_int64(), ctypes.c_int64()
    f = s["f"]
    rc = _lib.lib().shapes_collide_noalloc(
        s["n"], f["pos_x"].data_ptr(), f["pos_y"].data_ptr(), f["rot"].data_ptr(), f["inv_mass_lin"].data_ptr(),
        f["inv_mass_rot"].data_ptr(), s["vo"].data_ptr(), s["xy"].data_ptr(), s["nv"], s["pairs"].data_ptr(),
        s["cap_p"], s["keys"].data_ptr(), s["vals"].data_ptr(), s["cap_c"], s["stream"].cuda_stream or None,
        ctypes.byref(n_p), ctypes.byref(n_c))
    _lib.check(rc, "shapes_collide_noalloc")
    return dict(n_pairs=n_p.value, n_contacts=n_c.value, pairs=s["pairs"], keys=s["keys"], vals=s["vals"])


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    """Bytes: the state in and out, and shapes; operations: the pose (about 330 binary64 operations a body), and in a
    settled pile about two contacts a body at some 125 for finding and building one and 67 for each sweep's update."""
    kind = case["kind"]
    if kind == "net":
        r = case["rows"]
        macs = 16 * 64 + 2 * 64 * 64 + 64 * 2
        return dict(bytes=2 * r * 72 + r * 8 + 4 * 9538 * 3, flops=2 * r * macs * 4)
    steps, sweeps = case.get("steps", 1), case.get("sweeps", 2)
    if kind in ("collide", "noalloc"):
        n = case["bodies"]
        return dict(bytes=n * (80 if kind == "collide" else 40) + 5.5 * 20 * n + 60 * n, flops=n * (330 + 250))
    if kind in ("frame", "run"):
        n = case["cols"] * case["rows"] + 1
    elif case["scene"] == "columns":
        n = case["worlds"] * (case["bodies"] - 8) / math.log(case["bodies"] / 8.0)
    else:
        n = case["worlds"] * case["bodies"]
    return dict(bytes=n * (80 + 80 + 4.5 * 16), flops=steps * n * (330 + 2 * (125 + 67 * (sweeps + 1))))


# ---------------------------------------------------------------------------------------------------------------------
# the same in plain 64-bit Python and numpy


def exact(case, seed):
    """The network in float64; contact queries and whole steps of small worlds by an interpreter-speed restatement.
    Larger worlds would take minutes."""
    kind = case["kind"]
    if kind == "net":
        return _exact_net(case, seed)
    if kind == "noalloc" and case["bodies"] <= 2500:
        s = scenes.polygon_field(seed=seed, n=case["bodies"], extent=2.0 * math.sqrt(case["bodies"]))
        pairs, contacts = _World(s).collide()
        cap = 8 * case["bodies"] + 64
        out = dict(n_pairs=len(pairs), n_contacts=len(contacts), pairs=np.zeros((cap, 2), dtype=np.int32),
                   keys=np.zeros((cap, 5), dtype=np.int32), vals=np.zeros((cap, 5)))
        for k, ij in enumerate(pairs):
            out["pairs"][k] = ij
        for k, (key, flip, v) in enumerate(contacts):
            out["keys"][k], out["vals"][k] = key + (int(flip),), v
        return out
    if kind == "frame":
        s = _frame(case, seed)
        steps = FRAME_SETTLE + 1
    elif kind == "run":
        s = _stacks(case, seed)
        steps = case["steps"]
    else:
        return None
    sweeps = case.get("sweeps", 2)
    if len(s["bodies"]["pos_x"]) * steps > 10000:
        return None
    w = _World(s)
    for _ in range(steps):
        w.step(s["config"], sweeps)
    state = np.array([v + p + [r] for v, p, r in zip(w.vel, w.pos, w.rot)])
    out = {f: state[:, k] for k, f in enumerate(STEP_FIELDS)}
    return out | {f: s["bodies"][f] for f in _lib.BODY_FIELDS[6:]}


def _exact_net(case, seed):
    p, norm = (a.astype(np.float64) for a in _net_params(seed))
    x, y = (a.astype(np.float64) for a in _samples(case, seed))
    layers, at = [], 0
    for o, i in [(64, 16), (64, 64), (64, 64), (2, 64)]:
        layers.append((p[at:at + o * i].reshape(o, i), p[at + o * i:at + o * i + o]))
        at += o * i + o
    h = [np.clip((x - norm[:16]) * norm[16:32], -8.0, 8.0)]
    for k, (w, b) in enumerate(layers):
        z = h[-1] @ w.T + b
        h.append(np.maximum(z, 0.0) if k < 3 else z)
    mean, scale = norm[32:34], norm[34:36]
    err = h[-1] - (y - mean) / scale
    rows, d, grads = len(x), 2.0 / len(x) * err, []
    for k in (3, 2, 1, 0):
        grads = [(d.T @ h[k]).reshape(-1), d.sum(0)] + grads
        if k:
            d = (d @ layers[k][0]) * (h[k] > 0)
    return dict(out=h[-1] * scale + mean, grad=np.concatenate(grads), loss=float((err * err).sum() / rows))


class _World:
    """One world of hulls, stepped in plain Python floats."""

    def __init__(self, s):
        f, vo = s["bodies"], s["vert_offsets"]
        self.local = [s["local_xy"][vo[k]:vo[k + 1]].tolist() for k in range(len(vo) - 1)]
        col = {k: v.tolist() for k, v in f.items()}
        self.vel = [list(t) for t in zip(col["vel_x"], col["vel_y"], col["rot_vel"])]
        self.pos = [list(t) for t in zip(col["pos_x"], col["pos_y"])]
        self.rot, self.mu, self.bounce = col["rot"], col["mu"], col["bounce"]
        self.inv = list(zip(col["inv_mass_lin"], col["inv_mass_rot"]))
        self.cache = {}
        self.unit = [[_unit(a, b) for a, b in zip(v, v[1:] + v[:1])] for v in self.local]
        self.ext = [[_extent(v, n) for n in u] for v, u in zip(self.local, self.unit)]
        self.pose()

    def pose(self):
        self.pts, self.nrm, self.box = [], [], []
        for v, (px, py), th in zip(self.local, self.pos, self.rot):
            c, s = math.cos(th), math.sin(th)
            w = [((c * x - s * y) + px, (s * x + c * y) + py) for x, y in v]
            self.pts.append(w)
            self.nrm.append([_unit(a, b) for a, b in zip(w, w[1:] + w[:1])])
            xs, ys = [p[0] for p in w], [p[1] for p in w]
            self.box.append((min(xs), max(xs), min(ys), max(ys)))

    def pairs(self):
        box = np.array(self.box)
        x0, x1, y0, y1 = box.T
        still = np.array([m == (0.0, 0.0) for m in self.inv])
        out = []
        for i in range(len(box) - 1, 0, -1):
            j = slice(0, i)
            hit = (x0[j] <= x1[i]) & (x1[j] >= x0[i]) & (y0[j] <= y1[i]) & (y1[j] >= y0[i]) & ~(still[j] & still[i])
            out += [(i, int(k)) for k in np.flatnonzero(hit)[::-1]]
        return out

    def overlap(self, a, b):
        """(depth, edge of a, penetrating vertex of b) of a's axis of least overlap, None if one separates."""
        best = None
        for e, (nx, ny) in enumerate(self.nrm[a]):
            lo, hi = ((self.pts[a][k][0] * nx + self.pts[a][k][1] * ny) for k in self.ext[a][e])
            t = [x * nx + y * ny for x, y in self.pts[b]]
            least, most = min(t), max(t)
            if hi < least or most < lo:
                return None
            if best is None or hi - least < best[0]:
                best = (hi - least, e, t.index(least))
        return best

    def manifold(self, a, e, b, pen):
        """The points of b's edge at `pen` clipped to a's edge e: [(vertex of b, x, y)], descending."""
        p, q, n = self.pts[a][e], self.pts[a][(e + 1) % len(self.pts[a])], self.nrm[a][e]
        w = self.pts[b]
        before, after = (pen - 1) % len(w), (pen + 1) % len(w)
        span = lambda s, t: abs((w[t][0] - w[s][0]) * n[0] + (w[t][1] - w[s][1]) * n[1])  # noqa: E731
        first = (pen, after) if span(pen, after) < span(before, pen) else (before, pen)
        pts = [(k,) + w[k] for k in first]
        (_, cx, cy), (_, dx, dy) = pts
        line = ((cx, cy), (dy - cy, -(dx - cx)))
        for at, normal in ((p, (q[0] - p[0], q[1] - p[1])), (q, (p[0] - q[0], p[1] - q[1])), (p, (-n[0], -n[1]))):
            x = _meet(at, normal, line[0], line[1])
            limit = x[0] * normal[0] + x[1] * normal[1]
            out = [t[1] * normal[0] + t[2] * normal[1] < limit for t in pts]
            if all(out):
                return []
            if normal == (-n[0], -n[1]):
                pts = [t for t, o in zip(pts, out) if not o]
            else:
                pts = [(t[0],) + x if o else t for t, o in zip(pts, out)]
        return sorted(pts, reverse=True)

    def collide(self):
        """(pairs, contacts [((i, j, feature i, feature j), flipped, (normal x, y, point x, y, depth))]), descending."""
        pairs, out = self.pairs(), []
        for i, j in pairs:
            ij = self.overlap(i, j)
            ji = ij and self.overlap(j, i)
            if not ji:
                continue
            flip = not ij[0] < ji[0]
            a, b, (_, e, pen) = (j, i, ji) if flip else (i, j, ij)
            nx, ny = self.nrm[a][e]
            top = self.pts[a][e][0] * nx + self.pts[a][e][1] * ny
            for k, x, y in self.manifold(a, e, b, pen):
                key = (i, j, k, e) if flip else (i, j, e, k)
                out.append((key, flip, (nx, ny, x, y, top - (x * nx + y * ny))))
        return pairs, out

    def constraint(self, c, cfg):
        (i, j, _, _), flip, (nx, ny, x, y, depth) = c
        a, b = (self.pos[j], self.pos[i]) if flip else (self.pos[i], self.pos[j])
        tx, ty = ny, -nx
        jn = [-nx, -ny, _cross(a[0] - x, a[1] - y, nx, ny), nx, ny, _cross(x - b[0], y - b[1], nx, ny)]
        jf = [-tx, -ty, _cross(x - a[0], y - a[1], -tx, -ty), tx, ty, _cross(x - b[0], y - b[1], tx, ty)]
        if flip:
            jn, jf = jn[3:] + jn[:3], jf[3:] + jf[:3]
        m = [self.inv[i][0]] * 2 + [self.inv[i][1]] + [self.inv[j][0]] * 2 + [self.inv[j][1]]
        mass = [sum((g * k) * g for g, k in zip(row, m)) for row in (jn, jf)]
        bias = cfg["baumgarte"] / cfg["dt"] * (cfg["slop"] - depth) if depth > cfg["slop"] else 0.0
        sign = -1.0 if flip else 1.0
        arms = [x - self.pos[i][0], y - self.pos[i][1], x - self.pos[j][0], y - self.pos[j][1], sign * nx, sign * ny]
        return jn, jf, m, mass, bias, arms, (self.mu[i] + self.mu[j]) / 2.0, min(self.bounce[i], self.bounce[j])

    def apply(self, i, j, row, m, amount):
        for body, o in ((i, 0), (j, 3)):
            if self.inv[body] != (0.0, 0.0):
                self.vel[body] = [v + (row[o + k] * amount) * m[o + k] for k, v in enumerate(self.vel[body])]

    def step(self, cfg, sweeps):
        _, contacts = self.collide()
        cons = [self.constraint(c, cfg) for c in contacts]
        dt = cfg["dt"]
        for v, m in zip(self.vel, self.inv):
            if m[0] != 0.0:
                v[0] += cfg["accel"][0] * dt
                v[1] += cfg["accel"][1] * dt
        lam = [self.cache.get(c[0]) for c in contacts]
        for c, k, start in zip(contacts, cons, lam):
            if start:
                self.apply(c[0][0], c[0][1], k[0], k[2], start[0])
                self.apply(c[0][0], c[0][1], k[1], k[2], start[1])
        lam = [start or (0.0, 0.0) for start in lam]
        for _ in range(sweeps):
            for at, ((i, j, _, _), _, _) in enumerate(contacts):
                jn, jf, m, mass, bias, r, mu, bounce = cons[at]
                v = self.vel[i] + self.vel[j]
                cx = ((-v[0] + v[2] * r[1]) + v[3]) - v[5] * r[3]
                cy = ((-v[1] - v[2] * r[0]) + v[4]) + v[5] * r[2]
                bias += min(0.0, bounce * (cx * r[4] + cy * r[5]))
                normal = -(sum(g * u for g, u in zip(jn, v)) + bias) / mass[0]
                slide = -sum(g * u for g, u in zip(jf, v)) / mass[1]
                normal = max(normal, -lam[at][0])
                total = lam[at][0] + normal
                held = min(max(lam[at][1] + slide, -(total * mu)), total * mu)
                self.apply(i, j, jn, m, normal)
                self.apply(i, j, jf, m, held - lam[at][1])
                lam[at] = (total, held)
        self.cache = {c[0]: k for c, k in zip(contacts, lam)}
        for k, v in enumerate(self.vel):
            self.pos[k] = [v[0] * dt + self.pos[k][0], v[1] * dt + self.pos[k][1]]
            self.rot[k] = dt * v[2] + self.rot[k]
        self.pose()


def _unit(a, b):
    x, y = b[1] - a[1], -(b[0] - a[0])
    n = math.sqrt(x * x + y * y)
    return (x / n, y / n)


def _extent(pts, n):
    t = [x * n[0] + y * n[1] for x, y in pts]
    return t.index(min(t)), t.index(max(t))


def _cross(ax, ay, bx, by):
    return ax * by - ay * bx


def _meet(p, n, q, m):
    """Where the line through p with normal n crosses the one through q with normal m."""
    b0, b1 = p[0] * n[0] + p[1] * n[1], q[0] * m[0] + q[1] * m[1]
    det = n[0] * m[1] - n[1] * m[0]
    inv = 1.0 / det if det else math.copysign(math.inf, det)
    return (m[1] * inv) * b0 + (-n[1] * inv) * b1, (-m[0] * inv) * b0 + (n[0] * inv) * b1
