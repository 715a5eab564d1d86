"""The EI-ZO samplers against the oracle's replay, bit for bit, where they switch: the register sampler's region sizes
(rows of 32 face pairs over 1, 2, 4 or 8 warps, two to four per lane), and the domains on which the packed quotients
hand over to one IEEE division per face."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OPT = dict(num_particles=300, mixing_steps=12, bisection_steps=9, max_hyperplanes_per_iteration=10, epsilon=0.05,
           delta=0.05, tau=0.5, max_iterations=3, configuration_margin=0.01, seed=91)


def scene(d):
    return scenes.arm_scene(700 + d, num_spheres=2 * d, num_world_boxes=12, num_world_spheres=12, dof_per_arm=d,
                            keepout=0.6)


def seed_edge(sc):
    edges = scenes.seed_edges(sc, 1, 900, lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant),
                              lambda a, b: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant))
    assert edges
    return edges[0]


def box(sc):
    p = csd.HPolyhedron()
    p.MakeBox(sc.lower(), sc.upper())
    return p


def compare(sc, q0, q1, dom, capacity, single=True):
    opt = csd.EizoOptions(**OPT)
    cp = lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant)  # noqa: E731
    A, b, iters = O.eizo(sc.plant, q0, q1, dom.A(), dom.b(), opt, sc.inspector.robot_geometry_ids, capacity=capacity,
                         checker=cp)
    batch = csd.BatchedEdgeInflator([sc.plant], opt, max_slots=1, face_capacity=capacity, autotune_iterations=0)
    got = batch.inflate([0], [q0], [q1], [dom])[0]
    np.testing.assert_array_equal(got.A(), A)
    np.testing.assert_array_equal(got.b(), b)
    assert int(batch.last_iterations[0]) == len(iters)
    if single:
        inf = csd.CudaEdgeInflator(sc.plant, sc.inspector.robot_geometry_ids, opt, dom, face_capacity=capacity)
        one = inf.inflateEdge(q0, q1, None, 0.0, verbose=False)
        np.testing.assert_array_equal(one.A(), A)
        np.testing.assert_array_equal(one.b(), b)
    return A.shape[0]


# faces: pairs 64 | 65; 96 | 97; 128 | 129; 256 | 257; 512 | 513; 1024 | 1025; odd counts leave a repeated half
@pytest.mark.parametrize("dim", [9, 14, 15, 16])
@pytest.mark.parametrize("faces", [128, 129, 131, 193, 255, 257, 400, 513, 1025, 1999, 2048, 2049])
def test_region_sizes_equal_oracle_replay(dim, faces):
    sc = scene(dim)
    q0, q1 = seed_edge(sc)
    rng = np.random.default_rng(1000 * dim + faces)
    n = faces - 2 * dim
    a = rng.normal(size=(n, dim))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    off = np.maximum(a @ q0, a @ q1) + rng.uniform(0.4, 4.0, n)
    dom = box(sc)
    dom = csd.HPolyhedron(np.concatenate([dom.A(), a]).astype(np.float32),
                          np.concatenate([dom.b(), off]).astype(np.float32))
    assert dom.b().size == faces
    assert compare(sc, q0, q1, dom, 2400, single=faces == 257) > faces


@pytest.mark.parametrize("dim", [3, 7, 14])
@pytest.mark.parametrize("faces", [0, 200])
@pytest.mark.parametrize("case", ["scaled up", "scaled down", "mixed scales", "huge box", "start on faces",
                                  "start outside by a rounding", "unbounded"])
def test_odd_domains_equal_oracle_replay(dim, faces, case):
    sc = scene(dim)
    q0, q1 = seed_edge(sc)
    rng = np.random.default_rng(dim)
    a = rng.normal(size=(faces, dim))
    a /= np.maximum(np.linalg.norm(a, axis=1, keepdims=True), 1e-9)
    off = np.maximum(a @ q0, a @ q1) + rng.uniform(0.4, 4.0, faces)
    A = np.concatenate([box(sc).A(), a]).astype(np.float32)
    b = np.concatenate([box(sc).b(), off]).astype(np.float32)
    scale = np.ones(len(b))
    if case == "scaled up":
        scale[:] = 2.0 ** 80
    elif case == "scaled down":
        scale[:] = 2.0 ** -80
    elif case == "mixed scales":
        scale = 2.0 ** rng.integers(-100, 100, len(b))
    elif case == "huge box":
        b[:2 * dim] = 1e12
    elif case in ("start on faces", "start outside by a rounding"):
        b[0] = -q0[0]  # the face -x_0 <= -q0_0 holds the start
        b[3] = q0[1]
        q1 = q1.copy()
        q1[0], q1[1] = max(q1[0], q0[0]), min(q1[1], q0[1])
        if case == "start outside by a rounding":
            b[3] = np.nextafter(b[3], np.float32(-10))
            if not q0[1] <= b[3] + np.float32(1e-9):
                b[3] = q0[1]  # the containment test refuses more than its tolerance
    elif case == "unbounded":
        A, b, scale = np.delete(A, [0, 2], 0), np.delete(b, [0, 2]), np.delete(scale, [0, 2])
    dom = csd.HPolyhedron((A * scale[:, None]).astype(np.float32), (b * scale).astype(np.float32))
    compare(sc, q0, q1, dom, 800)


# lanes per chain 32, 16, 8; one chain to several rounds per block; faces below, at and beyond a lane each, odd
# counts, and past the staging buffer (48 KB: 1,228 faces at up to 8 dimensions, 682 above)
@pytest.mark.parametrize("dim", [1, 2, 3, 7, 8, 9, 14, 16])
@pytest.mark.parametrize("samples,polytopes", [(1, 1), (33, 3), (1000, 5), (9001, 2), (21000, 1)])
def test_uniform_samples_equal_oracle(dim, samples, polytopes):
    rng = np.random.default_rng(100 * dim + samples)
    polys, starts = [], []
    for i in range(polytopes):
        n = int(rng.choice([0, 1, 2, 15, 16, 17, 64, 333])) if samples > 33 else [3, 1300, 700][i]
        a = rng.normal(size=(n, dim))
        a /= np.linalg.norm(a, axis=1, keepdims=True)
        c = rng.uniform(-0.5, 0.5, dim)
        A = np.concatenate([np.kron(np.eye(dim), [[-1.0], [1.0]]), a]).astype(np.float32)
        b = np.concatenate([np.full(2 * dim, 1.0), a @ c + rng.uniform(0.0, 1.0, n)]).astype(np.float32)
        if i == 1:  # a start on a face: its slack is too small for the packed quotients
            b[1] = np.float32(c[0])
        polys.append(csd.HPolyhedron(A, b))
        starts.append(c.astype(np.float32))
    mixing = 3 if samples > 5000 else 12
    got = csd.UniformSampleInHPolyhedraCuda(polys, np.stack(starts, 1), samples, mixing, seed=dim)
    for i, (p, x) in enumerate(zip(polys, starts)):
        ref, _ = O.hit_and_run(p.A(), p.b(), x, samples, mixing, seed=dim, stream=i)
        np.testing.assert_array_equal(got[i].T, ref)
