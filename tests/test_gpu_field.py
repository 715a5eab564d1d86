"""The field path (grid over the statics, link capsules: csrc/check_field.cuh) only prunes: its verdicts equal the full
pair sweep's (broad phase off) bit for bit, whatever the tree, the statics and the pair list."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from csdecomp_b200.plant import (CollisionGeometry, Joint, JointType, KinematicTree, Link, ShapePrimitive, build_plant,
                                 make_transform)

pytestmark = pytest.mark.gpu


def geometry(rng, kind, link, spread, size):
    X = make_transform(scenes.random_rotation(rng), rng.uniform(-spread, spread, 3))
    if kind == ShapePrimitive.SPHERE:
        dims = [size * rng.uniform(0.5, 1.5), -1, -1]
    elif kind == ShapePrimitive.CAPSULE:
        dims = [size * rng.uniform(0.3, 1.0), size * rng.uniform(0.0, 6.0), 0]
    else:
        dims = size * rng.uniform(0.5, 3.0, 3)
    return CollisionGeometry(type=kind, dimensions=np.asarray(dims, np.float32), link_index=link, X_L_B=X)


def random_plant(rng, joints, branching, prismatic, spheres, capsules, statics, world_extent, static_size, base):
    """A random tree: joint i hangs off a random earlier link with probability `branching`, else off the last one."""
    tree = KinematicTree()
    tree.add_link(Link(name="world"))
    base_link = tree.add_link(Link(name="base"))
    tree.add_joint(Joint(name="base_weld", type=JointType.FIXED, parent_link=0, child_link=base_link))
    links = [base_link]
    for i in range(joints):
        li = tree.add_link(Link(name=f"l{i}"))
        parent = int(rng.choice(links)) if rng.random() < branching else links[-1]
        kind = JointType.PRISMATIC if rng.random() < prismatic else JointType.REVOLUTE
        axis = rng.normal(size=3)
        tree.add_joint(Joint(name=f"j{i}", type=kind, parent_link=parent, child_link=li,
                             X_PL_J=make_transform(scenes.random_rotation(rng), rng.uniform(0.05, 0.35, 3)),
                             axis=(axis / np.linalg.norm(axis)).astype(np.float32), position_lower_limit=-2.0,
                             position_upper_limit=2.0))
        links.append(li)
    geoms = []
    for kind, count in ((ShapePrimitive.SPHERE, spheres), (ShapePrimitive.CAPSULE, capsules)):
        for _ in range(count):
            geoms.append(geometry(rng, kind, int(rng.choice(links[1:])), 0.15, 0.06))
    for _ in range(base):  # robot geometry welded to the world: a static the first link does not pair with
        geoms.append(geometry(rng, ShapePrimitive.SPHERE, base_link, 0.1, 0.1))
    obstacles = tree.add_link(Link(name="obstacles"))
    tree.add_joint(Joint(name="weld", type=JointType.FIXED, parent_link=0, child_link=obstacles))
    kinds = [ShapePrimitive.SPHERE, ShapePrimitive.BOX, ShapePrimitive.CAPSULE]
    for _ in range(statics):
        geoms.append(geometry(rng, kinds[int(rng.integers(3))], obstacles, world_extent, static_size))
        if rng.random() < 0.5:
            geoms[-1].X_L_B[:3, :3] = np.eye(3)
    tree.finalize()
    return build_plant(tree, geoms)[0], tree


def both(plant, q):
    h = csd.plant_handle(plant)
    on = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(False)
    off = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(True)
    return on, off


TREES = {  # joints, branching, prismatic, spheres, capsules, statics, world extent, static size, base geometries
    "arm": (7, 0.0, 0.0, 20, 2, 60, 1.2, 0.08, 0),
    "one joint": (1, 0.0, 0.0, 3, 0, 5, 0.6, 0.1, 0),
    "no statics": (6, 0.0, 0.0, 18, 3, 0, 1.0, 0.1, 0),
    "capsules only": (5, 0.2, 0.0, 0, 9, 40, 1.2, 0.08, 0),
    "branches": (14, 0.5, 0.0, 21, 3, 40, 1.8, 0.06, 2),
    "prismatic": (6, 0.2, 0.4, 9, 2, 12, 2.0, 0.08, 1),
    "crowded cells": (6, 0.0, 0.0, 12, 2, 900, 0.9, 0.02, 0),
    "tiny statics": (6, 0.0, 0.0, 43, 1, 300, 1.2, 0.005, 0),
    "one far wall": (7, 0.0, 0.0, 31, 1, 1, 9.0, 3.0, 0),
    "32 spheres": (4, 0.0, 0.0, 32, 0, 33, 1.0, 0.1, 0),
}


@pytest.mark.parametrize("name", sorted(TREES))
def test_field_matches_pair_sweep(name):
    rng = np.random.default_rng(sorted(TREES).index(name))
    mixed = 0
    for _ in range(4):
        plant, tree = random_plant(rng, *TREES[name])
        dim = tree.numConfigurationVariables()
        q = rng.uniform(-2.0, 2.0, (4099, dim)).astype(np.float32)
        on, off = both(plant, q)
        np.testing.assert_array_equal(on, off)
        mixed += 0 < on.mean() < 1
        # a pair list that leaves out half of the pairs: the field's hits are looked up in it
        pairs = plant.collision_pair_matrix()
        if pairs.shape[1]:
            plant.set_collision_pairs_from_matrix(pairs[:, rng.random(pairs.shape[1]) < 0.5])
            on, off = both(plant, q)
            np.testing.assert_array_equal(on, off)
    assert mixed >= 1 or name in ("one joint", "one far wall", "no statics", "crowded cells", "tiny statics")


@pytest.mark.parametrize("i", range(6))
def test_field_matches_pair_sweep_on_cover_scenes(i):
    sc = scenes.batch_scene(i, scenes.batch_scene_seeds(i + 1)[i])
    on, off = both(sc.plant, sc.random_configs(60001, i))
    np.testing.assert_array_equal(on, off)
    assert 0 < on.mean() < 1


def test_field_odd_configurations():
    """NaN and infinite coordinates: as the pair sweep decides them."""
    rng = np.random.default_rng(5)
    for name in ("arm", "prismatic", "branches", "no statics"):
        plant, tree = random_plant(rng, *TREES[name])
        dim = tree.numConfigurationVariables()
        q = rng.uniform(-2.0, 2.0, (512, dim)).astype(np.float32)
        for k, bad in enumerate((np.nan, np.inf, -np.inf, 3e38)):
            q[64 * k:64 * k + 64][np.arange(64), rng.integers(0, dim, 64)] = bad
        on, off = both(plant, q)
        np.testing.assert_array_equal(on, off)
