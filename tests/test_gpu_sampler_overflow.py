"""Faces whose a . dir overflows to infinity still bound the chain: the quotient is 0 (one IEEE division), so the chain
stays where it is, as in the oracle's replay. Coefficients near the largest float, alone or among ordinary faces."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def huge_faces(rng, q0, q1, dim, count, scale):
    """`count` faces +-scale x_k <= scale c, c a little beyond the segment on the coordinate, every product finite."""
    k = int(np.argmin(np.maximum(np.abs(q0), np.abs(q1))))
    assert max(abs(q0[k]), abs(q1[k])) < 0.7
    A, b = np.zeros((count, dim)), np.zeros(count)
    for i in range(count):
        s = 1.0 if i % 2 else -1.0
        A[i, k] = s * scale
        b[i] = scale * (max(s * q0[k], s * q1[k]) + rng.uniform(0.05, 0.25))
    return A.astype(np.float32), b.astype(np.float32)


# faces in all: one lane's few, several pairs per lane, the register sampler's rows (130 on, above 8 dimensions)
@pytest.mark.parametrize("dim", [2, 7, 14, 16])
@pytest.mark.parametrize("plain", [0, 120, 420])
@pytest.mark.parametrize("huge,scale", [(1, 2.0 ** 127), (2, 2.0 ** 127), (3, 3.4e38), (4, 2.0 ** 126), (2, 2.0 ** 101)])
def test_regions_with_huge_coefficients_equal_oracle_replay(dim, plain, huge, scale):
    sc = scenes.arm_scene(700 + dim, num_spheres=2 * dim, num_world_boxes=12, num_world_spheres=12, dof_per_arm=dim,
                          keepout=0.6)
    edges = scenes.seed_edges(sc, 60, 900, lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant),
                              lambda a, b: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant), length=(0.05, 0.3))
    q0, q1 = min(edges, key=lambda e: np.abs(np.stack(e)).max(0).min())
    rng = np.random.default_rng(1000 * dim + plain)
    box = csd.HPolyhedron()
    box.MakeBox(sc.lower(), sc.upper())
    a = rng.normal(size=(plain, dim))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    off = np.maximum(a @ q0, a @ q1) + rng.uniform(0.4, 4.0, plain)
    Ah, bh = huge_faces(rng, q0, q1, dim, huge, scale)
    A = np.concatenate([box.A(), a, Ah]).astype(np.float32)
    b = np.concatenate([box.b(), off, bh]).astype(np.float32)
    assert np.isfinite(A).all() and np.isfinite(b).all()
    order = rng.permutation(len(b))
    dom = csd.HPolyhedron(A[order], b[order])
    opt = csd.EizoOptions(num_particles=300, mixing_steps=12, bisection_steps=9, epsilon=0.05, max_iterations=3, seed=91)
    A, b, iters = O.eizo(sc.plant, q0, q1, dom.A(), dom.b(), opt, sc.inspector.robot_geometry_ids, capacity=800,
                         checker=lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant))
    got = csd.BatchedEdgeInflator([sc.plant], opt, max_slots=1, face_capacity=800,
                                  autotune_iterations=0).inflate([0], [q0], [q1], [dom])[0]
    np.testing.assert_array_equal(got.A(), A)
    np.testing.assert_array_equal(got.b(), b)
    one = csd.CudaEdgeInflator(sc.plant, sc.inspector.robot_geometry_ids, opt, dom,
                               face_capacity=800).inflateEdge(q0, q1, None, 0.0, verbose=False)
    np.testing.assert_array_equal(one.A(), A)
    np.testing.assert_array_equal(one.b(), b)


# the second polytope's coefficients overflow, the others' do not; staged rows and rows read from global memory
@pytest.mark.parametrize("dim", [1, 2, 3, 7, 8, 9, 14, 16])
@pytest.mark.parametrize("samples", [200, 6000])
@pytest.mark.parametrize("plain", [5, 60, 1300])
@pytest.mark.parametrize("scale", [2.0 ** 101, 2.0 ** 126, 2.0 ** 127, 3.4e38])
def test_uniform_samples_with_huge_coefficients_equal_oracle(dim, samples, plain, scale):
    rng = np.random.default_rng(dim + plain)
    polys, starts = [], []
    for i in range(3):
        x = rng.uniform(-0.3, 0.3, dim).astype(np.float32)
        a = rng.normal(size=(plain, dim))
        a /= np.linalg.norm(a, axis=1, keepdims=True)
        A = np.concatenate([np.kron(np.eye(dim), [[-1.0], [1.0]]), a]).astype(np.float32)
        b = np.concatenate([np.full(2 * dim, 1.0), a @ x + rng.uniform(0.05, 1.0, plain)]).astype(np.float32)
        if i == 1:
            Ah, bh = huge_faces(rng, x, x, dim, 3, scale)
            A, b = np.concatenate([A, Ah]), np.concatenate([b, bh])
        polys.append(csd.HPolyhedron(A, b))
        starts.append(x)
    mixing = 12 if samples * plain < 200000 else 3
    got = csd.UniformSampleInHPolyhedraCuda(polys, np.stack(starts, 1), samples, mixing, seed=dim)
    for i, (p, x) in enumerate(zip(polys, starts)):
        ref, _ = O.hit_and_run(p.A(), p.b(), x, samples, mixing, seed=dim, stream=i)
        np.testing.assert_array_equal(got[i].T, ref)
