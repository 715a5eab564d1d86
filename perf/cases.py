"""Performance cases: the calls a user of csdecomp_b200 makes, over the sizes they make them at.

``listed()`` are the standing cases, ``draw(rng)`` gives further ones of the same
ranges. A case is a dict of plain values; ``prepare(case, seed)`` makes what a
program has in hand before the call (inputs from the seed, the uploaded plant,
the inflator or surrogate handle it keeps), ``run(state)`` is one pass through
the public entry points, ``work(case)`` the bytes and FLOPs of a pass that any
implementation needs, ``exact(case, seed)`` the outputs in 64 bits where they
have such a value.

Robots and worlds are the repository's own (csdecomp_b200/scenes.py):

  table  7-DOF arm, 40 spheres; 20 boxes
  cell   7-DOF arm, 80 spheres + 4 capsules; 100 boxes + 100 spheres, 0.8 m keep-out around the base
  dual   14-DOF two-arm plant, 80 spheres + 4 capsules; 50 to 400 boxes and spheres
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import csdecomp_b200 as csd
from csdecomp_b200 import _capi as C
from csdecomp_b200 import scenes
from csdecomp_b200.surrogate import CollisionSurrogate

EDGE_MODES = {"l2": csd.CSD_EDGE_L2_REF, "linf": csd.CSD_EDGE_LINF, "vg": csd.CSD_EDGE_VG}
HIDDEN, PADDED = 256, 16  # layers of the surrogate's nets: dim (padded to 16) -> 256 -> 256 -> 256 -> 1


# ---------------------------------------------------------------------- cases
def listed():
    return [
        # a planner asks about the waypoints of one path: launch and copy latency
        {"name": "check_path", "op": "check", "scene": "table", "n": 33, "device": False},
        # a roadmap batch from host memory
        {"name": "check_10k", "op": "check", "scene": "table", "n": 10000, "device": False},
        # dense coverage sampling of a cluttered cell, configurations already on the GPU
        {"name": "check_1m", "op": "check", "scene": "cell", "n": 1000003, "device": True},
        # sensor voxels against the arm, configurations and voxels on the GPU
        {"name": "voxels", "op": "voxels", "scene": "cell", "n": 262147, "voxels": 10000},
        # link poses of a trajectory batch
        {"name": "fk", "op": "fk", "scene": "cell", "n": 100003},
        # local connections of a roadmap
        {"name": "edges", "op": "edges", "scene": "cell", "n": 40009, "mode": "l2"},
        # all pairs of a set of free configurations
        {"name": "visibility", "op": "visibility", "scene": "cell", "nodes": 501},
        # samples of finished regions, for coverage and trajectory seeds
        {"name": "sample", "op": "sample", "polytopes": 16, "dim": 7, "faces": 67, "samples": 1000, "mixing": 40},
        # one edge grown into a region, as a program does between two plans
        {"name": "inflate_one", "op": "inflate", "scene": "cell", "particles": 2000, "mixing": 50},
        # a whole cover: many edges in many worlds, one- and two-arm plants
        {"name": "inflate_batch", "op": "batch", "slots": 128, "particles": 2000, "mixing": 50},
        # regions cut back after new collisions were seen in them
        {"name": "edit", "op": "edit", "scene": "cell", "regions": 64, "collisions": 512},
        # the collision surrogates of a cover's worlds, one net per world, trained on labelled configurations
        {"name": "surrogate_train", "op": "train", "nets": 64, "dim": 14, "rows": 2048, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["check", "check", "voxels", "fk", "edges", "visibility", "sample", "inflate", "batch", "edit",
                     "train", "gradients", "logits"])
    scene = rng.choice(["table", "cell", "dual"])
    if op == "check":
        return {"op": op, "scene": scene, "n": _log_int(rng, 24, 1 << 20), "device": rng.random() < 0.5}
    if op == "voxels":
        return {"op": op, "scene": scene, "n": _log_int(rng, 64, 1 << 18), "voxels": _log_int(rng, 16, 10000)}
    if op == "fk":
        return {"op": op, "scene": scene, "n": _log_int(rng, 4, 200000)}
    if op == "edges":
        return {"op": op, "scene": scene, "n": _log_int(rng, 16, 100000), "mode": rng.choice(sorted(EDGE_MODES))}
    if op == "visibility":
        return {"op": op, "scene": scene, "nodes": _log_int(rng, 16, 600)}
    if op == "sample":
        return {"op": op, "polytopes": _log_int(rng, 1, 48), "dim": rng.choice([2, 3, 6, 7, 14]),
                "faces": _log_int(rng, 8, 400), "samples": _log_int(rng, 16, 4096), "mixing": rng.randint(10, 50)}
    if op == "inflate":
        return {"op": op, "scene": scene, "particles": _log_int(rng, 500, 2000), "mixing": rng.randint(20, 50)}
    if op == "batch":
        return {"op": op, "slots": _log_int(rng, 2, 96), "particles": _log_int(rng, 500, 2000),
                "mixing": rng.randint(20, 50)}
    if op == "edit":
        return {"op": op, "scene": scene, "regions": _log_int(rng, 1, 64), "collisions": _log_int(rng, 8, 512)}
    if op == "train":
        return {"op": op, "nets": _log_int(rng, 1, 64), "dim": rng.choice([7, 14]), "rows": 512 * rng.randint(1, 8),
                "steps": rng.randint(1, 16)}
    rows = _log_int(rng, 4, 64) * 32
    return {"op": op, "nets": _log_int(rng, 1, 64), "dim": rng.choice([7, 14]),
            "rows": rows if op == "gradients" else rows + rng.randint(1, 31)}


# --------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _scene(name):
    if name == "table":
        return scenes.point_check_scene()
    if name == "cell":
        return scenes.edge_check_scene(keepout=0.8)
    return _batch_scene(1)


@functools.lru_cache(maxsize=None)
def _batch_scene(i):
    return scenes.batch_scene(i, scenes.batch_scene_seeds(i + 1)[i])


def _box(sc):
    d = csd.HPolyhedron()
    d.MakeBox(sc.lower(), sc.upper())
    return d


def _seed_edges(sc, count, seed, length=(0.05, 1.0)):
    return scenes.seed_edges(sc, count, seed, lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant),
                             lambda a, b: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant), length=length)


def _free(sc, n, rng):
    """n collision-free configurations of the scene."""
    got = np.zeros((0, sc.dim), np.float32)
    while len(got) < n:
        q = sc.random_configs(max(4096, 4 * n), int(rng.integers(1 << 30)))
        got = np.concatenate([got, q[csd.CheckCollisionFreeCuda(q.T, sc.plant) == 1]])
    return got[:n]


def _eizo_options(case):
    return csd.EizoOptions(num_particles=case["particles"], mixing_steps=case["mixing"], bisection_steps=9,
                           max_hyperplanes_per_iteration=10, epsilon=0.01, delta=0.05, tau=0.5, max_iterations=500,
                           configuration_margin=0.01, seed=1337)


def _random_polytope(rng, dim, faces):
    """A region as inflation leaves one: the joint-limit box and cuts around a centre."""
    n = max(faces - 2 * dim, 0)
    a = rng.normal(size=(n, dim))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    c = rng.uniform(-1.0, 1.0, dim)
    A = np.concatenate([np.kron(np.eye(dim), [[-1.0], [1.0]]), a]).astype(np.float32)
    b = np.concatenate([np.full(2 * dim, math.pi), a @ c + rng.uniform(0.2, 1.5, n)]).astype(np.float32)
    return csd.HPolyhedron(A, b), c.astype(np.float32)


def _surrogate_data(case, seed):
    rng = np.random.default_rng(seed)
    nets, dim, rows = case["nets"], case["dim"], case["rows"]
    w1 = np.zeros((nets, HIDDEN, PADDED), np.float32)
    w1[:, :, :dim] = rng.uniform(-1, 1, (nets, HIDDEN, dim)) * math.sqrt(6.0 / dim)
    w2, w3 = (rng.uniform(-1, 1, (nets, HIDDEN, HIDDEN)).astype(np.float32) * np.float32(math.sqrt(6.0 / HIDDEN))
              for _ in range(2))
    w4 = rng.uniform(-1, 1, (nets, HIDDEN)).astype(np.float32) * np.float32(math.sqrt(3.0 / HIDDEN))
    b1, b2, b3 = (rng.uniform(-0.1, 0.1, (nets, HIDDEN)).astype(np.float32) for _ in range(3))
    b4 = np.zeros((nets, 1), np.float32)
    params = np.concatenate([x.reshape(nets, -1) for x in (w1, b1, w2, b2, w3, b3, w4, b4)], axis=1)
    x = rng.uniform(-math.pi, math.pi, (nets, rows, dim)).astype(np.float32)
    y = (np.linalg.norm(x, axis=2) < 1.8 * math.sqrt(dim)).astype(np.uint8)
    return params, x, y


def prepare(case, seed):
    op = case["op"]
    rng = np.random.default_rng(seed)
    s = {"op": op, "case": case}
    if op == "sample":
        made = [_random_polytope(rng, case["dim"], case["faces"] + int(rng.integers(0, 9))) for _ in
                range(case["polytopes"])]
        s["polytopes"] = [p for p, _ in made]
        s["starts"] = np.stack([c for _, c in made], 1)
        s["seed"] = int(rng.integers(1 << 30))
        return s
    if op in ("train", "gradients", "logits"):
        params, x, y = _surrogate_data(case, seed)
        s["bank"] = CollisionSurrogate([case["dim"]] * case["nets"], seed=0)
        s["bank"].set_params(params)
        s["x"], s["y"] = list(x), list(y)
        return s
    if op == "batch":
        worlds = [_batch_scene(i) for i in range(case["slots"])]
        slot_plant, starts, ends = [], [], []
        while len(starts) < case["slots"]:  # a world where no free seed edge turns up is passed over
            for i, sc in enumerate(worlds[:case["slots"] - len(starts)]):
                e = _seed_edges(sc, 1, int(rng.integers(1 << 30)))
                if e:
                    slot_plant.append(i)
                    starts.append(e[0][0])
                    ends.append(e[0][1])
        s["args"] = (slot_plant, starts, ends, [_box(worlds[i]) for i in slot_plant])
        _region_buffers(s, 1000 * (case["slots"] + 4), 14)
        s["inflator"] = csd.BatchedEdgeInflator([sc.plant for sc in worlds], _eizo_options(case),
                                                max_slots=case["slots"])
        return s
    sc = _scene(case["scene"])
    s["plant"] = sc.plant
    s["handle"] = csd.plant_handle(sc.plant)
    if op == "inflate":
        s["edge"] = _seed_edges(sc, 1, int(rng.integers(1 << 30)), (0.1, 0.5))[0]
        s["inflator"] = csd.CudaEdgeInflator(sc.plant, sc.inspector.robot_geometry_ids, _eizo_options(case), _box(sc))
        _region_buffers(s, csd.MAX_NUM_FACES, sc.dim)
        return s
    if op == "edit":
        return _prepare_edit(s, sc, case, rng)
    if op == "visibility":
        s["q"] = np.asfortranarray(_free(sc, case["nodes"], rng).T)
        s["indices"] = np.zeros(case["nodes"] * (case["nodes"] - 1) // 2, np.int32)
        return s
    n = case["n"]
    if op == "edges":  # from free configurations, 0.05 to 1 rad in any direction, inside the joint limits
        q0 = _free(sc, n, rng)
        d = rng.normal(size=q0.shape)
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        q1 = np.clip(q0 + rng.uniform(0.05, 1.0, (n, 1)) * d, sc.lower(), sc.upper()).astype(np.float32)
        s["q0"], s["q1"] = np.asfortranarray(q0.T), np.asfortranarray(q1.T)
        return s
    q = sc.random_configs(n, seed)
    if op == "check" and not case["device"]:
        s["q"] = np.asfortranarray(q.T)
        return s
    s["q"] = torch.from_numpy(q).cuda()
    if op == "fk":
        s["out"] = torch.zeros((n, s["handle"].num_links, 16), dtype=torch.float32, device="cuda")
        return s
    s["out"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    if op == "voxels":  # around the robot, clear of its base
        v = rng.uniform([-1.5, -1.5, 0.0], [1.5, 1.5, 1.5], (4 * case["voxels"] + 64, 3)).astype(np.float32)
        v = v[np.linalg.norm(v, axis=1) > 0.9][:case["voxels"]]
        s["voxels"] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
        s["ids"] = np.ascontiguousarray(np.asarray(list(sc.inspector.robot_geometry_ids), np.int32))
    return s


def _region_buffers(s, rows, dim):
    s["A"], s["b"] = np.zeros(rows * dim, np.float32), np.zeros(rows, np.float32)


def _prepare_edit(s, sc, case, rng):
    edges = []
    while len(edges) < case["regions"]:
        edges += _seed_edges(sc, case["regions"] - len(edges), int(rng.integers(1 << 30)), (0.1, 0.5))
    lo, hi = sc.lower(), sc.upper()
    regions, cols, segs = [], [], []
    for r, (q0, q1) in enumerate(edges):
        blo = np.maximum(lo, np.minimum(q0, q1) - 1.2).astype(np.float32)
        bhi = np.minimum(hi, np.maximum(q0, q1) + 1.2).astype(np.float32)
        box = csd.HPolyhedron()
        box.MakeBox(blo, bhi)
        regions.append(box)
        got = np.zeros((0, sc.dim), np.float32)
        while len(got) < case["collisions"]:
            q = (blo + (bhi - blo) * rng.random((8 * case["collisions"], sc.dim))).astype(np.float32)
            got = np.concatenate([got, q[csd.CheckCollisionFreeCuda(q.T, sc.plant) == 0]])
        cols.append(got[:case["collisions"]])
        segs.append(np.full(len(cols[-1]), r))
    _region_buffers(s, case["regions"] * (2 * sc.dim + case["collisions"]), sc.dim)
    s["args"] = (np.asfortranarray(np.concatenate(cols).T), np.concatenate(segs),
                 np.stack([e[0] for e in edges], 1).astype(np.float32),
                 np.stack([e[1] for e in edges], 1).astype(np.float32), regions, sc.plant,
                 sc.inspector.robot_geometry_ids, csd.Voxels(), 0.01, csd.EditRegionsOptions())
    return s


# ----------------------------------------------------------------------- pass
def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _filled(buffer, values):
    """The values at the front of a buffer of the program's own (zeros after them: how many there are varies)."""
    buffer[:values.size] = values.reshape(-1)
    return buffer


def _regions(s, regions):
    return {"A": _filled(s["A"], np.concatenate([r.A().reshape(-1) for r in regions])),
            "b": _filled(s["b"], np.concatenate([r.b() for r in regions])),
            "faces": np.asarray([r.b().size for r in regions])}


def run(s):
    op, case = s["op"], s["case"]
    if op == "check":
        if not case["device"]:
            return csd.CheckCollisionFreeCuda(s["q"], s["plant"])
        C.check(C.lib().csd_check_points(s["handle"].handle, C.ptr(s["q"].data_ptr()), ctypes.c_int64(case["n"]), None,
                                         0, ctypes.c_float(0), None, 0, C.ptr(s["out"].data_ptr()), C.CSD_PTR_DEVICE,
                                         _stream()))
        return s["out"]
    if op == "voxels":
        C.check(C.lib().csd_check_points(s["handle"].handle, C.ptr(s["q"].data_ptr()), ctypes.c_int64(case["n"]),
                                         C.ptr(s["voxels"].data_ptr()), case["voxels"], ctypes.c_float(0.02),
                                         C.ptr(s["ids"]), s["ids"].size, C.ptr(s["out"].data_ptr()), C.CSD_PTR_DEVICE,
                                         _stream()))
        return s["out"]
    if op == "fk":
        C.check(C.lib().csd_fk(s["handle"].handle, C.ptr(s["q"].data_ptr()), ctypes.c_int64(case["n"]),
                               C.ptr(s["out"].data_ptr()), C.CSD_PTR_DEVICE, _stream()))
        return s["out"]
    if op == "edges":
        return csd.CheckEdgesCollisionFreeCuda(s["q0"], s["q1"], s["plant"], 0.01, EDGE_MODES[case["mode"]])
    if op == "visibility":
        g = csd.VisibilityGraph(s["q"], s["plant"], 0.01)
        return g.indptr, _filled(s["indices"], g.indices)
    if op == "sample":
        return csd.UniformSampleInHPolyhedraCuda(s["polytopes"], s["starts"], case["samples"], case["mixing"],
                                                 seed=s["seed"])
    if op == "inflate":
        p = s["inflator"].inflateEdge(s["edge"][0], s["edge"][1], None, 0.0, verbose=False)
        return _regions(s, [p])
    if op == "batch":
        regions = s["inflator"].inflate(*s["args"])
        return {**_regions(s, regions), "iterations": s["inflator"].last_iterations}
    if op == "edit":
        regions, (projections, optimized) = csd.EditRegionsCuda(*s["args"])
        return {**_regions(s, regions), "projections": projections, "optimized": optimized}
    if op == "train":
        loss = s["bank"].train(s["x"], s["y"], batch=512, epochs=case["steps"] * 512 / case["rows"], lr=1e-3, seed=0)
        return {"params": s["bank"].params(), "loss": loss}
    if op == "gradients":
        grads, loss = s["bank"].gradients(s["x"], s["y"])
        return {"gradients": grads, "loss": loss}
    return {"logits": np.concatenate(s["bank"].logits(list(enumerate(s["x"]))))}


# ----------------------------------------------------------------------- work
def _config_flops(sc):
    """FLOPs of one configuration that no culling removes: every moving joint and geometry placed (FMA = 2)."""
    types = sc.plant.arrays()["geom_type"]
    moving = len(sc.inspector.robot_geometry_ids)
    capsules = int((types == int(csd.ShapePrimitive.CAPSULE)).sum())
    return 99.0 * sc.dim + 18.0 * (moving - capsules) + 33.0 * capsules


def _inflation_flops(sc, case):
    """One inflation, with the iterations and faces that these plants take on average."""
    d = sc.dim
    iterations, samples = (6, 3600) if d <= 7 else (24, 5000)
    faces = 2 * d + 5 * iterations
    per_sample = case["mixing"] * (2.0 * d + 4.0) * faces + _config_flops(sc)
    return iterations * (max(samples, case["particles"]) * per_sample + case["particles"] * 9 * _config_flops(sc))


def work(case):
    op = case["op"]
    if op == "sample":
        d, f, chains = case["dim"], case["faces"], case["polytopes"] * case["samples"]
        return {"bytes": 4.0 * (chains * d + case["polytopes"] * (f * (d + 1) + d)),
                "flops": chains * case["mixing"] * f * (2.0 * d + 4.0)}
    if op in ("train", "gradients", "logits"):
        weights = HIDDEN * case["dim"] + 2 * HIDDEN * HIDDEN + HIDDEN
        rows, nets = case["nets"] * case["rows"], case["nets"]
        seen = nets * 512 * case["steps"] if op == "train" else rows
        out = rows if op == "logits" else nets * (HIDDEN * PADDED + 2 * HIDDEN * HIDDEN + 4 * HIDDEN + 1)
        return {"bytes": 4.0 * (rows * case["dim"] + nets * weights + out),
                "flops": (2.0 if op == "logits" else 6.0) * seen * weights}
    if op == "batch":
        plants = [_batch_scene(i) for i in range(case["slots"])]
        return {"bytes": sum(4.0 * 400 * (sc.dim + 1) for sc in plants),
                "flops": sum(_inflation_flops(sc, case) for sc in plants)}
    sc = _scene(case["scene"])
    d, per = sc.dim, _config_flops(sc)
    if op == "inflate":
        return {"bytes": 4.0 * 67 * (d + 1), "flops": _inflation_flops(sc, case)}
    if op == "edit":
        n = case["regions"] * case["collisions"]
        return {"bytes": n * 4.0 * (3 * d + 1), "flops": 9.0 * n * per}
    if op == "visibility":
        pairs = case["nodes"] * (case["nodes"] - 1) // 2
        return {"bytes": 4.0 * case["nodes"] * d + pairs, "flops": pairs * per}
    n = case["n"]
    if op == "edges":
        return {"bytes": n * (8.0 * d + 1), "flops": n * per}
    if op == "fk":
        links = sc.plant.kin_tree.num_links
        return {"bytes": 4.0 * n * (d + 16 * links), "flops": 99.0 * n * d}
    return {"bytes": n * (4.0 * d + 1) + 12.0 * case.get("voxels", 0), "flops": n * per}


# ---------------------------------------------------------------------- exact
def exact(case, seed):
    """Verdicts are bytes and have none. A sampled chain, an inflated or an edited region follows from thousands of
    32-bit verdicts and draws before it and has no 64-bit value of its own; the projections onto the segments do."""
    op = case["op"]
    if op == "fk":
        return _exact_fk(_scene(case["scene"]), _scene(case["scene"]).random_configs(case["n"], seed))
    if op in ("train", "gradients", "logits"):
        return _exact_surrogate(case, seed)
    if op == "edit":
        q, seg, start, end = prepare(case, seed)["args"][:4]
        q, a, d = q.astype(np.float64), start.astype(np.float64)[:, seg], (end.astype(np.float64) - start)[:, seg]
        t = np.clip(((q - a) * d).sum(0) / (d * d).sum(0), 0.0, 1.0)
        return {"A": None, "b": None, "faces": None, "projections": (1.0 - t) * a + t * (a + d), "optimized": None}
    return None


def _exact_fk(sc, q):
    t = sc.plant.arrays()
    links = sc.plant.kin_tree.num_links
    q = torch.from_numpy(q).double()
    X = [None] * links
    X[0] = torch.eye(4, dtype=torch.float64).expand(len(q), 4, 4)
    for j in t["joint_traversal_sequence"].tolist():
        fixed = torch.from_numpy(t["joint_X_PL_J"].reshape(-1, 4, 4)[j].astype(np.float64).T.copy())
        local = torch.eye(4, dtype=torch.float64).repeat(len(q), 1, 1)
        if t["joint_type"][j] == 1:  # revolute: Rodrigues' formula about the unit axis
            k = torch.from_numpy(t["joint_axis"].reshape(-1, 3)[j].astype(np.float64))
            K = torch.tensor([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]], dtype=torch.float64)
            a = q[:, int(t["joint_idx_to_config_idx"][j])].reshape(-1, 1, 1)
            local[:, :3, :3] += torch.sin(a) * K + (1.0 - torch.cos(a)) * (K @ K)
        X[int(t["joint_child_link"][j])] = X[int(t["joint_parent_link"][j])] @ (fixed @ local)
    return torch.stack(X, 1).transpose(2, 3).reshape(len(q), links, 16)  # each 4x4 column-major


def _exact_surrogate(case, seed):
    params, x, y = _surrogate_data(case, seed)
    p = torch.from_numpy(params).cuda().double()
    x, y = torch.from_numpy(x).cuda().double(), torch.from_numpy(y).cuda().double()
    if case["op"] == "logits":
        return {"logits": _net_pass(p, x, y)[0].reshape(-1)}
    if case["op"] == "gradients":
        _, grads, loss = _net_pass(p, x, y)
        return {"gradients": grads, "loss": loss}
    # Adam (Kingma & Ba 2015) over batches of 512 of the rows in the order that train() shuffles them into
    rng = np.random.default_rng(0)
    order = [torch.from_numpy(rng.permutation(case["rows"])).cuda() for _ in range(case["nets"])]
    x, y = torch.stack([a[o] for a, o in zip(x, order)]), torch.stack([a[o] for a, o in zip(y, order)])
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for t in range(case["steps"]):
        at = t * 512 % case["rows"]
        _, g, loss = _net_pass(p, x[:, at:at + 512], y[:, at:at + 512])
        losses.append(loss.mean())
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** (t + 1))) / (torch.sqrt(v / (1 - 0.999 ** (t + 1))) + 1e-8)
    return {"params": p, "loss": torch.stack(losses)}


def _net_pass(p, x, y):
    """(logits, gradients of the mean loss, mean loss) of every net."""
    nets, rows, dim = x.shape
    cut = np.cumsum([0, HIDDEN * PADDED, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN, 1])
    w1, b1, w2, b2, w3, b3, w4, b4 = (p[:, cut[i]:cut[i + 1]] for i in range(8))
    w1, w2, w3 = (w.reshape(nets, HIDDEN, -1) for w in (w1, w2, w3))
    h0 = torch.nn.functional.pad(x / math.pi, (0, PADDED - dim))
    h1 = torch.relu(h0 @ w1.transpose(1, 2) + b1[:, None])
    h2 = torch.relu(h1 @ w2.transpose(1, 2) + b2[:, None])
    h3 = torch.relu(h2 @ w3.transpose(1, 2) + b3[:, None])
    z = (h3 * w4[:, None]).sum(2) + b4
    loss = torch.nn.functional.binary_cross_entropy_with_logits(z, y, reduction="none").mean(1)
    dz = (torch.sigmoid(z) - y) / rows
    d3 = dz[:, :, None] * w4[:, None] * (h3 > 0)
    d2 = (d3 @ w3) * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grads = [d1.transpose(1, 2) @ h0, d1.sum(1), d2.transpose(1, 2) @ h1, d2.sum(1), d3.transpose(1, 2) @ h2, d3.sum(1),
             (dz[:, :, None] * h3).sum(1), dz.sum(1, keepdim=True)]
    return z, torch.cat([g.reshape(nets, -1) for g in grads], 1), loss
