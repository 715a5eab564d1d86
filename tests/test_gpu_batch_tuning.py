"""The batch autotuner times the staged samplers only on iterations that run one: beside the register sampler alone they
would find nothing to do, and the least of five empty launches would be kept."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes

pytestmark = pytest.mark.gpu


def scene(d):
    sc = scenes.arm_scene(700 + d, num_spheres=2 * d, num_world_boxes=12, num_world_spheres=12, dof_per_arm=d, keepout=0.6)
    e = scenes.seed_edges(sc, 1, 900, lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant),
                          lambda a, b: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant))
    return sc, e[0]


def box(sc):
    p = csd.HPolyhedron()
    p.MakeBox(sc.lower(), sc.upper())
    return p


def test_sampler_variants_wait_for_an_iteration_that_runs_one():
    sc, (q0, q1) = scene(12)
    rng = np.random.default_rng(2)
    a = rng.normal(size=(200, 12))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    off = np.maximum(a @ q0, a @ q1) + rng.uniform(0.4, 4.0, 200)
    many = csd.HPolyhedron(np.concatenate([box(sc).A(), a]).astype(np.float32),
                           np.concatenate([box(sc).b(), off]).astype(np.float32))  # sampled from registers throughout
    opt = csd.EizoOptions(num_particles=300, mixing_steps=12, epsilon=0.05, max_iterations=6, seed=91)
    b = csd.BatchedEdgeInflator([sc.plant], opt, max_slots=2, face_capacity=1200, autotune_iterations=2)
    plain = csd.BatchedEdgeInflator([sc.plant], opt, max_slots=2, face_capacity=1200, autotune_iterations=0)
    args = ([0, 0], [q0, q0], [q1, q1])
    got = b.inflate(*args, [many, many])
    t = b.tuning()
    assert all(v == 0.0 for v in t["sample_ms"].values()), t
    assert all(v > 0.0 for v in t["check_ms"].values()), t
    for P, R in zip(got, plain.inflate(*args, [many, many])):
        np.testing.assert_array_equal(P.A(), R.A())
    got = b.inflate(*args, [box(sc), box(sc)])  # 24 faces to start with: the staged sampler
    t = b.tuning()
    assert all(v > 0.0 for v in t["sample_ms"].values()), t
    assert t["sample_variant"] == min(t["sample_ms"], key=t["sample_ms"].get)
    for P, R in zip(got, plain.inflate(*args, [box(sc), box(sc)])):
        np.testing.assert_array_equal(P.A(), R.A())
