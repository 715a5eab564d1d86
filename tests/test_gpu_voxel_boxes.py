"""Geometry large against the cells: its query box covers many columns of the voxels' grid. Few voxels are then tested one
by one; verdicts are the full sweep's, and the check costs no more than it."""
import time

import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from csdecomp_b200.plant import (CollisionGeometry, Joint, JointType, KinematicTree, Link, ShapePrimitive, build_plant,
                                 make_transform)

pytestmark = pytest.mark.gpu


def plant(large, count, capsules=0):
    rng = np.random.default_rng(1)
    tree = KinematicTree()
    tree.add_link(Link(name="world"))
    links = []
    for i in range(3):
        links.append(tree.add_link(Link(name=f"l{i}")))
        tree.add_joint(Joint(name=f"j{i}", type=JointType.REVOLUTE, parent_link=links[i - 1] if i else 0,
                             child_link=links[i], X_PL_J=make_transform(scenes.random_rotation(rng), [0.1, 0.1, 0.2]),
                             axis=np.array([0, 0, 1], np.float32), position_lower_limit=-3.0, position_upper_limit=3.0))
    geoms = []
    for k in range(20 + count + capsules):
        kind = ShapePrimitive.CAPSULE if k >= 20 + count else ShapePrimitive.SPHERE
        r = 0.02 if k < 20 else large
        geoms.append(CollisionGeometry(type=kind, dimensions=np.array([r, 0.3, -1], np.float32), link_index=links[k % 3],
                                       X_L_B=make_transform(scenes.random_rotation(rng), rng.uniform(-0.05, 0.05, 3))))
    tree.finalize()
    p, insp = build_plant(tree, geoms)
    p.set_collision_pairs_from_matrix(np.zeros((2, 0), np.int32))
    return p, insp.robot_geometry_ids


def both(p, ids, q, v, radius=0.02):
    h = csd.plant_handle(p)
    on = csd.CheckCollisionFreeVoxelsCuda(q.T, v, radius, p, ids)
    h.set_voxel_grid(False)
    off = csd.CheckCollisionFreeVoxelsCuda(q.T, v, radius, p, ids)
    h.set_voxel_grid(True)
    return on, off


@pytest.mark.parametrize("large,count,capsules", [(0.1, 3, 0), (0.3, 12, 2), (0.6, 1, 1), (1.5, 1, 0)])
@pytest.mark.parametrize("voxels", [64, 65, 67, 300, 1000, 1601, 5003])
@pytest.mark.parametrize("n", [300, 6000])
def test_large_geometry_equals_full_sweep(large, count, capsules, voxels, n):
    p, ids = plant(large, count, capsules)
    rng = np.random.default_rng(voxels)
    v = rng.normal(size=(3, voxels))
    v *= rng.uniform(large + 0.3, large + 1.5, voxels) / np.linalg.norm(v, axis=0)
    v = v.astype(np.float32)
    q = rng.uniform(-3, 3, (n, 3)).astype(np.float32)
    q[::50, 1] = np.nan
    keep = rng.random(voxels) < 20.0 / voxels  # some verdicts each way
    for vv in (v, np.concatenate([v[:, keep], np.tile(v[:, :1] * 30, 70)], 1)):
        on, off = both(p, ids, q, np.ascontiguousarray(vv))
        np.testing.assert_array_equal(on, off)


def test_large_geometry_costs_no_more_than_the_full_sweep():
    """12 spheres of 0.3 m among 20 small ones, voxels out of reach: a check of 20,000 configurations with 64 voxels took
    0.9 ms through the grid's columns, 0.15 ms voxel by voxel."""
    p, ids = plant(0.3, 12)
    h = csd.plant_handle(p)
    rng = np.random.default_rng(2)
    q = rng.uniform(-2, 2, (20000, 3)).astype(np.float32)
    for voxels in (64, 300, 1000, 5000):
        v = rng.normal(size=(3, voxels))
        v = (2.0 * v / np.linalg.norm(v, axis=0)).astype(np.float32)
        least = []
        for grid in (True, False):
            h.set_voxel_grid(grid)
            t = []
            for _ in range(8):
                t0 = time.perf_counter()
                csd.CheckCollisionFreeVoxelsCuda(q.T, v, 0.02, p, ids)
                t.append(time.perf_counter() - t0)
            least.append(1e6 * min(t))
        h.set_voxel_grid(True)
        assert least[0] < 1.3 * least[1] + 100, (voxels, least)
