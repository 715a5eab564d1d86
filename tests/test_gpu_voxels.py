"""Voxel checks through the hash grid where its parts have edges: the buckets'
scan (one block per 1,024 buckets), runs of cells that wrap around the last
bucket, large query boxes, capsules found through their probe spheres. The
grid only prunes, so verdicts equal the every-voxel sweep's, bit for bit."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes

pytestmark = pytest.mark.gpu


def verdicts(plant, q, vox, vr, rids, grid):
    h = csd.plant_handle(plant)
    h.set_voxel_grid(grid)
    try:
        return csd.CheckCollisionFreeVoxelsCuda(q.T, csd.Voxels(vox.T), vr, plant, rids)
    finally:
        h.set_voxel_grid(True)


def around(rng, n, spread):
    """n voxels off the robot's base, where every configuration would collide."""
    v = rng.uniform(-spread, spread, (8 * n + 64, 3))
    return v[np.linalg.norm(v, axis=1) > 0.8][:n]


@pytest.fixture(scope="module")
def scene():
    return scenes.arm_scene(71, num_spheres=45, num_capsules=5, num_world_spheres=2, keepout=0.9)


# buckets of cells' own voxels: 256 up to 128 voxels, 1,024 up to 512, 2,048 from 513 (two blocks of the scan);
# more than 65,536 voxels are never listed around cells
@pytest.mark.parametrize("nv", [64, 65, 128, 129, 512, 513, 1025, 20011, 65536, 65537])
@pytest.mark.parametrize("vr", [0.004, 0.03])
@pytest.mark.parametrize("n", [3001, 4097])  # cells' own voxels, and from 4,096 configurations those around them too
def test_counts(scene, nv, vr, n):
    rng = np.random.default_rng(nv)
    q = scene.random_configs(n, 2)
    spread = max(0.9, 0.16 * nv ** (1 / 3))
    vox = around(rng, nv, spread).astype(np.float32)
    ids = scene.inspector.robot_geometry_ids
    on, off = (verdicts(scene.plant, q, vox, vr, ids, g) for g in (True, False))
    np.testing.assert_array_equal(on, off)


@pytest.mark.parametrize("shape", ["cell", "column", "plane", "far", "large_voxels", "duplicates"])
@pytest.mark.parametrize("n", [2500, 4500])
def test_shapes(scene, shape, n):
    rng = np.random.default_rng(5)
    m, vr = 700, 0.02
    v = around(rng, m, 1.0)
    if shape == "cell":  # one bucket holds everything
        v = np.array([0.5, 0.1, 0.4]) + 0.01 * v
    elif shape == "column":  # longer than the table of 256 buckets: the runs wrap
        v = np.stack([np.full(100, 0.4), np.full(100, 0.1), np.linspace(-30, 30, 100)], 1)
    elif shape == "plane":
        v[:, 2] = 0.3
    elif shape == "far":
        v[::2] += 1e6
    elif shape == "large_voxels":  # boxes of more cells than a query walks
        vr = 0.6
        v = v * 0.5 + np.array([1.4, 0.0, 0.4])
    else:
        v = np.repeat(v[:70], 10, 0)
    q = np.concatenate([scene.random_configs(n, 6), np.full((2, scene.dim), np.nan, np.float32)])
    vox = v.astype(np.float32)
    ids = scene.inspector.robot_geometry_ids
    on, off = (verdicts(scene.plant, q, vox, vr, ids, g) for g in (True, False))
    np.testing.assert_array_equal(on, off)
    assert not on[-2:].any()


@pytest.mark.parametrize("keep", ["spheres", "capsules", "one_capsule", "repeated", "every_third"])
@pytest.mark.parametrize("n", [3000, 5000])
def test_robot_geometry_subsets(scene, keep, n):
    """Only the listed robot geometries are tested against voxels, repeated ids or not."""
    rng = np.random.default_rng(9)
    ids = list(scene.inspector.robot_geometry_ids)
    caps = [i for i in ids if scene.plant.scene_collision_geometries[i].type == csd.ShapePrimitive.CAPSULE]
    rest = [i for i in ids if i not in caps]
    assert len(caps) == 5
    sub = {"spheres": rest, "capsules": caps, "one_capsule": caps[-1:], "repeated": ids[:9] + caps[:2] * 3,
           "every_third": ids[::3]}[keep]
    q = scene.random_configs(n, 12)
    vox = around(rng, 1200, 1.4).astype(np.float32)
    on, off = (verdicts(scene.plant, q, vox, 0.01, sub, g) for g in (True, False))
    np.testing.assert_array_equal(on, off)
    assert 0 < on.mean() < 1
