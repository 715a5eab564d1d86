"""Plants that the field path's tables are not made for keep the pair sweep, and creating them returns: numbers that
are not finite, sizes and distances at which FP32 rounding is not small against the tables' margins."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from csdecomp_b200.plant import (CollisionGeometry, Joint, JointType, KinematicTree, Link, ShapePrimitive, build_plant,
                                 make_transform)

pytestmark = pytest.mark.gpu
S, B, C = ShapePrimitive.SPHERE, ShapePrimitive.BOX, ShapePrimitive.CAPSULE


def shape(kind, link, centre, *dims):
    return CollisionGeometry(type=kind, dimensions=np.asarray((list(dims) + [-1, -1])[:3], np.float32), link_index=link,
                             X_L_B=make_transform(np.eye(3), centre))


def arm(statics, prismatic=False, moving=(), base=(0, 0, 0)):
    """Three joints (the first prismatic along x, or revolute) with a sphere each, `moving` more on the last link."""
    rng = np.random.default_rng(3)
    tree = KinematicTree()
    tree.add_link(Link(name="world"))
    parent, geoms = 0, []
    for i in range(3):
        link = tree.add_link(Link(name=f"l{i}"))
        first = i == 0
        kind = JointType.PRISMATIC if first and prismatic else JointType.REVOLUTE
        X = make_transform(np.eye(3) if first else scenes.random_rotation(rng), base if first else (0.2, 0.1, 0.3))
        tree.add_joint(Joint(name=f"j{i}", type=kind, parent_link=parent, child_link=link, X_PL_J=X,
                             axis=np.array([1, 0, 0] if first else [0, 0, 1], np.float32), position_lower_limit=-3.0,
                             position_upper_limit=3.0))
        geoms.append(shape(S, link, (0.1, 0.0, 0.15), 0.06))
        parent = link
    geoms += [shape(kind, parent, c, *dims) for kind, c, *dims in moving]
    world = tree.add_link(Link(name="w"))
    tree.add_joint(Joint(name="weld", type=JointType.FIXED, parent_link=0, child_link=world))
    geoms += [shape(kind, world, c, *dims) for kind, c, *dims in statics]
    tree.finalize()
    return build_plant(tree, geoms)[0]


def on_off(plant, q):
    h = csd.plant_handle(plant)
    on = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(False)
    off = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(True)
    return on, off


ORDINARY = [(S, (0.5, 0.2, 0.4), 0.1), (B, (-0.5, 0.3, 0.2), 0.2, 0.3, 0.2), (C, (0.1, -0.6, 0.3), 0.05, 0.4)]


@pytest.mark.parametrize("prismatic", [False, True])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e38])
@pytest.mark.parametrize("kind", [S, B, C])
@pytest.mark.parametrize("where", ["centre", "size", "only static", "moving centre", "moving size"])
def test_creation_returns_for_any_numbers(prismatic, bad, kind, where):
    sizes = {S: (0.1,), B: (0.1, 0.2, 0.1), C: (0.1, 0.2)}[kind]
    odd = (kind, (bad if "centre" in where or where == "only static" else 0.3, 0.0, 0.2),
           *((bad if "size" in where else sizes[0]),), *sizes[1:])
    if where.startswith("moving"):
        plant = arm(ORDINARY, prismatic, moving=[odd])
    else:
        plant = arm([odd] if where == "only static" else ORDINARY + [odd], prismatic)
    q = np.random.default_rng(1).uniform(-3, 3, (300, 3)).astype(np.float32)
    on, off = on_off(plant, q)
    assert set(np.unique(on)) <= {0, 1}
    if where == "size" and bad == np.inf and kind == S:
        assert not on.any() and not off.any()  # an infinite ball


def test_verdicts_beside_a_ground_of_any_extent():
    """Spheres within a rounding of contact with boxes of 20 m to 200 km, revolute arms and a rail."""
    mixed = 0
    for prismatic in (False, True):
        for half in (10.0, 200.0, 300.0, 5e3, 5e4, 1e5):
            top = -0.1
            plant = arm(ORDINARY + [(B, (0.0, 0.0, top - half), 2 * half, 2 * half, 2 * half)], prismatic)
            rng = np.random.default_rng(int(half))
            q = rng.uniform(-3, 3, (200003, 3)).astype(np.float32)
            on, off = on_off(plant, q)
            np.testing.assert_array_equal(on, off)
            mixed += 0 < off.mean() < 1
    assert mixed >= 6


@pytest.mark.parametrize("prismatic", [False, True])
@pytest.mark.parametrize("base", [(40.0, 0, 0), (63.0, 1, 0), (70.0, 0, 0), (-90.0, 100.0, -60.0), (120.0, 0, 0), (127.5, 0, 0), (0, 200.0, 0)])
def test_verdicts_far_from_the_origin(prismatic, base):
    statics = [(k, tuple(np.add(c, base)), *d) for k, c, *d in ORDINARY + [(S, (0.1, 0.15, 0.0), 0.05)]]
    plant = arm(statics, prismatic, base=base)
    q = np.random.default_rng(7).uniform(-3, 3, (100003, 3)).astype(np.float32)
    if prismatic:
        q[::3, 0] *= 30  # beyond the grid on a rail
    on, off = on_off(plant, q)
    np.testing.assert_array_equal(on, off)
    assert 0 < off.mean() < 1


# a block's eight warps hold the poses of up to some 1,780 moving spheres; the field path's batch of configurations
# shrinks, and ends in the pair sweep, before they stop fitting
@pytest.mark.parametrize("spheres", [1200, 1500, 1560, 1600, 1640, 1700, 1750])
def test_plants_up_to_the_shared_memory_limit(spheres):
    rng = np.random.default_rng(spheres)
    more = [(S, tuple(rng.uniform(-0.1, 0.1, 3)), rng.uniform(0.01, 0.03)) for _ in range(spheres)]
    plant = arm(ORDINARY[:2], moving=more)
    pairs = plant.collision_pair_matrix()
    assert plant.num_scene_geometries == spheres + 5
    q = rng.uniform(-3, 3, (3001, 3)).astype(np.float32)
    on, off = on_off(plant, q)
    np.testing.assert_array_equal(on, off)
    assert 0 < on.mean() < 1 and pairs.shape[1] > spheres
    h = csd.plant_handle(plant)
    s, e = np.ascontiguousarray(q[:64].T), np.ascontiguousarray(np.roll(q, 1, 0)[:64].T)
    on = csd.CheckEdgesCollisionFreeCuda(s, e, plant, 0.05)
    h.set_culling(False)
    np.testing.assert_array_equal(on, csd.CheckEdgesCollisionFreeCuda(s, e, plant, 0.05))
