"""One batch handle used again after its surrogate changed gives what a fresh handle gives: no captured iteration keeps
an earlier stop probability, bank or round schedule."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from csdecomp_b200.surrogate import CollisionSurrogate, training_set

pytestmark = pytest.mark.gpu

OPT = dict(num_particles=600, mixing_steps=20, max_iterations=30)
SLOTS = [0, 1] * 4  # over 3 slots: later inflations start in slots that finished


@pytest.fixture(scope="module")
def world():
    scs = [scenes.arm_scene(41, num_spheres=40, num_capsules=2, num_world_boxes=40, num_world_spheres=40, keepout=0.8),
           scenes.arm_scene(42, num_spheres=40, num_capsules=2, num_world_boxes=30, num_world_spheres=30, arms=2,
                            keepout=0.9, arm_spacing=1.4)]
    edges, doms = [], []
    for i, sc in enumerate(scs):
        edges.append(scenes.seed_edges(sc, 4, 50 + i, lambda q, sc=sc: csd.CheckCollisionFreeCuda(q.T, sc.plant),
                                       lambda a, b, sc=sc: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant),
                                       length=(0.2, 0.6)))
        d = csd.HPolyhedron()
        d.MakeBox(sc.lower(), sc.upper())
        doms.append(d)
    banks = []
    for seed, epochs in ((7, 4), (8, 1)):
        bank = CollisionSurrogate([sc.dim for sc in scs], seed=seed)
        data = [training_set(sc, e, 8192, seed=100 + i) for i, (sc, e) in enumerate(zip(scs, edges))]
        bank.train([x for x, _ in data], [y for _, y in data], batch=512, epochs=epochs, lr=2e-3)
        banks.append(bank)
    return scs, edges, doms, banks


def handle(world):
    return csd.BatchedEdgeInflator([sc.plant for sc in world[0]], csd.EizoOptions(**OPT), max_slots=3,
                                   face_capacity=400, autotune_iterations=0)


def inflate(world, b, setting):
    _, edges, doms, banks = world
    bank, stop, rounds = setting
    b.set_surrogate(banks[bank] if bank is not None else None, stop)
    if rounds:
        b.set_surrogate_rounds(*rounds)
    regs = b.inflate(SLOTS, [edges[p][k // 2][0] for k, p in enumerate(SLOTS)],
                     [edges[p][k // 2][1] for k, p in enumerate(SLOTS)], [doms[p] for p in SLOTS])
    return regs, b.last_configs_checked.copy(), b.last_iterations.copy()


@pytest.mark.parametrize("first,second", [
    ((0, 0.5, None), (0, 1e-30, None)),
    ((0, 1e-30, None), (0, 0.5, None)),
    ((0, 0.5, None), (1, 0.5, None)),
    ((0, 0.5, None), (None, 0.5, None)),
    ((0, 0.5, (3, 1024)), (0, 0.5, (2, 64))),
], ids=["stop lower", "stop higher", "other bank", "off", "rounds"])
def test_handle_follows_its_surrogate(world, first, second):
    b = handle(world)
    before = inflate(world, b, first)
    again = inflate(world, b, second)
    fresh = inflate(world, handle(world), second)
    assert not np.array_equal(before[1], fresh[1])  # the change matters here
    np.testing.assert_array_equal(again[1], fresh[1])
    np.testing.assert_array_equal(again[2], fresh[2])
    for P, R in zip(again[0], fresh[0]):
        np.testing.assert_array_equal(P.A(), R.A())
        np.testing.assert_array_equal(P.b(), R.b())
