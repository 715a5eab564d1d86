"""Cells that list many statics: every entry of a list decides some verdict, and a probe much larger than the others,
which makes every list long, neither changes verdicts nor sends the small ones through all statics."""
import ctypes

import numpy as np
import pytest
import torch

import csdecomp_b200 as csd
from csdecomp_b200 import _capi, scenes
from csdecomp_b200.plant import (CollisionGeometry, Joint, JointType, KinematicTree, Link, ShapePrimitive, build_plant,
                                 make_transform)

pytestmark = pytest.mark.gpu
S, B, C = ShapePrimitive.SPHERE, ShapePrimitive.BOX, ShapePrimitive.CAPSULE


def shape(kind, link, X, *dims):
    return CollisionGeometry(type=kind, dimensions=np.asarray((list(dims) + [-1, -1])[:3], np.float32), link_index=link,
                             X_L_B=X)


def build(rng, statics, big=0.0, capsules=0):
    """A 5-joint arm (30 spheres of 3 to 6 cm, `capsules`, a sphere of radius `big` on the first link) and `statics`
    (kind, transform, dims), paired with the small moving geometry only: no self pairs, none of the large sphere's."""
    tree = KinematicTree()
    tree.add_link(Link(name="world"))
    links, parent = [], 0
    for i in range(5):
        link = tree.add_link(Link(name=f"l{i}"))
        tree.add_joint(Joint(name=f"j{i}", type=JointType.REVOLUTE, parent_link=parent, child_link=link,
                             X_PL_J=make_transform(scenes.random_rotation(rng), rng.uniform(0.1, 0.25, 3)),
                             axis=np.array([0, 0, 1], np.float32), position_lower_limit=-3.0, position_upper_limit=3.0))
        links.append(link)
        parent = link
    at = lambda s: make_transform(scenes.random_rotation(rng), rng.uniform(-s, s, 3))  # noqa: E731
    geoms = [shape(S, links[i % 5], at(0.12), rng.uniform(0.03, 0.06)) for i in range(30)]
    geoms += [shape(C, links[1 + i % 4], at(0.1), 0.04, 0.3) for i in range(capsules)]
    small = len(geoms)
    if big:
        geoms.append(shape(S, links[0], np.eye(4, dtype=np.float32), big))
    world = tree.add_link(Link(name="w"))
    tree.add_joint(Joint(name="weld", type=JointType.FIXED, parent_link=0, child_link=world))
    geoms += [shape(kind, world, X, *dims) for kind, X, *dims in statics]
    tree.finalize()
    plant = build_plant(tree, geoms)[0]
    return plant, small, len(geoms) - len(statics)


def pair_up(plant, small, first, keep):
    """Pairs the moving geometries 0 .. small with the statics s where keep(s)."""
    order = np.arange(plant.num_scene_geometries)
    statics = [g for g in order[first:] if keep(g - first)]
    a, b = np.meshgrid(order[:small], statics, indexing="ij")
    plant.set_collision_pairs_from_matrix(np.stack([a.ravel(), b.ravel()]).astype(np.int32))


def both(plant, q):
    h = csd.plant_handle(plant)
    on = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(False)
    off = csd.CheckCollisionFreeCuda(q.T, plant)
    h.set_culling(True)
    return on, off


# clusters of 5 to 40 small statics, each cell near a cluster listing all of it (up to six are held in the cell)
@pytest.mark.parametrize("per", [5, 6, 7, 13, 40])
@pytest.mark.parametrize("capsules", [0, 3])
def test_every_entry_of_a_list_decides(per, capsules):
    rng = np.random.default_rng(per)
    statics = []
    for _ in range(20):
        c = rng.normal(size=3)
        c *= rng.uniform(0.4, 0.9) / np.linalg.norm(c)
        for j in range(per):
            kind = (S, B, C)[j % 3]
            X = make_transform(np.eye(3) if j % 2 else scenes.random_rotation(rng), c + rng.uniform(-0.02, 0.02, 3))
            statics.append((kind, X, *{S: (0.01,), B: (0.02, 0.03, 0.02), C: (0.008, 0.03)}[kind]))
    plant, small, first = build(rng, statics, capsules=capsules)
    q = rng.uniform(-3, 3, (20011, 5)).astype(np.float32)
    for t in range(per):
        pair_up(plant, small, first, lambda s: s % per == t)
        on, off = both(plant, q)
        np.testing.assert_array_equal(on, off)
        assert 100 < (off == 0).sum() < len(q) - 100


@pytest.mark.parametrize("big", [0.0, 0.3, 0.6, 1.0])
@pytest.mark.parametrize("count,size", [(900, 0.01), (300, 0.03), (1024, 0.002)])
def test_one_large_sphere(big, count, size):
    rng = np.random.default_rng(count)
    statics = [((S, B)[i % 2], make_transform(np.eye(3), rng.uniform(-0.9, 0.9, 3)), *((size,) * (1 + 2 * (i % 2))))
               for i in range(count)]
    plant, small, first = build(rng, statics, big=big, capsules=2)
    q = rng.uniform(-3, 3, (30011, 5)).astype(np.float32)
    for part in (1, 7):  # every static, every seventh
        pair_up(plant, small, first, lambda s: s % part == 0)
        on, off = both(plant, q)
        np.testing.assert_array_equal(on, off)
        assert 0 < off.mean() < 1


def check_ms(plant, q):
    """Device time of one check of the device configurations q (least of eight)."""
    h = csd.plant_handle(plant)
    out = torch.zeros(len(q), dtype=torch.uint8, device="cuda")
    times = []
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        _capi.check(_capi.lib().csd_check_points(
            h.handle, ctypes.c_void_p(q.data_ptr()), ctypes.c_int64(len(q)), None, 0, ctypes.c_float(0), None, 0,
            ctypes.c_void_p(out.data_ptr()), _capi.CSD_PTR_DEVICE,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        e[1].record()
        e[1].synchronize()
        times.append(e[0].elapsed_time(e[1]))
    return min(times)


def scene(big, extent):
    rng = np.random.default_rng(5)
    statics = [(S, make_transform(np.eye(3), rng.uniform(-extent, extent, 3)), 0.01) for _ in range(900)]
    plant, small, first = build(rng, statics, big=big)
    pair_up(plant, small, first, lambda s: True)
    return plant, torch.as_tensor(rng.uniform(-3, 3, (1 << 17, 5)).astype(np.float32)).cuda()


def test_one_large_sphere_does_not_slow_the_others():
    """Among 900 small statics, a sphere of 0.4 m: several times the check without it, 40 times when the cells' lists did
    not fit and each cell tested every static."""
    without, with_big = (check_ms(*scene(big, 1.2)) for big in (0.0, 0.4))
    assert with_big < 10 * without + 0.1, (without, with_big)


def test_lists_of_most_statics_leave_the_check_to_the_sweep():
    """A sphere of 1 m in the middle of 900 statics: every cell lists most of them, and the check may not cost more than
    the sweep over every pair."""
    plant, q = scene(1.0, 0.9)
    on = check_ms(plant, q)
    csd.plant_handle(plant).set_culling(False)
    off = check_ms(plant, q)
    csd.plant_handle(plant).set_culling(True)
    assert on < 1.2 * off + 0.1, (on, off)
