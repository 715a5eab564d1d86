"""Forward kinematics of any tree and batch: the two kernels agree bit for bit, trees of thousands of links are accepted,
and a few configurations of a large tree do not pay for the tables of many."""
import ctypes

import numpy as np
import pytest
import torch

import csdecomp_b200 as csd
from csdecomp_b200 import _capi, scenes
from csdecomp_b200.plant import Joint, JointType, KinematicTree, Link, MinimalPlant, make_transform

pytestmark = pytest.mark.gpu


def tree_plant(links, branching=0.0, seed=1, joints=7):
    """A tree of `links` links: `joints` moving ones, the rest welded to random earlier links, some to the world."""
    rng = np.random.default_rng(seed)
    tree = KinematicTree()
    tree.add_link(Link(name="world"))
    moving = set(rng.choice(np.arange(1, links), min(joints, links - 1), replace=False).tolist())
    last = 0
    for i in range(1, links):
        link = tree.add_link(Link(name=f"l{i}"))
        kind = JointType.FIXED
        if i in moving:
            kind = JointType.PRISMATIC if rng.random() < 0.3 else JointType.REVOLUTE
        parent = int(rng.integers(0, i)) if kind == JointType.FIXED or rng.random() < branching else last
        tree.add_joint(Joint(name=f"j{i}", type=kind, parent_link=parent, child_link=link,
                             X_PL_J=make_transform(scenes.random_rotation(rng), rng.uniform(-0.2, 0.2, 3)),
                             axis=np.array([0, 0, 1], np.float32), position_lower_limit=-3.0, position_upper_limit=3.0))
        if kind != JointType.FIXED:
            last = link
    tree.finalize()
    return MinimalPlant(tree.get_minimal_kinematic_tree(), [], np.zeros((2, 0), np.int32)), tree


@pytest.mark.parametrize("links,branching", [(2, 0.0), (9, 0.0), (15, 0.5), (40, 1.0), (300, 0.3), (700, 0.0)])
def test_small_and_large_batches_agree(links, branching):
    plant, tree = tree_plant(links, branching, joints=12)
    n = 6144 + 64 * links + 33  # just past the line
    q = np.random.default_rng(2).uniform(-3, 3, (min(n, 16384 + 33), tree.numConfigurationVariables())).astype(np.float32)
    many = csd.ComputeForwardKinematicsCuda(q.T, plant)
    for i0, i1 in ((0, 1), (31, 64), (1000, 3001), (len(q) - 5, len(q))):
        np.testing.assert_array_equal(csd.ComputeForwardKinematicsCuda(q[i0:i1].T, plant), many[i0:i1])


@pytest.mark.parametrize("links", [3000, 5000, 9000])
@pytest.mark.parametrize("n", [3, 16500])
def test_trees_of_thousands_of_links(links, n):
    if n > 3 and links > 5000:
        n = 4000  # (the transforms are 64 bytes each)
    plant, tree = tree_plant(links)
    rng = np.random.default_rng(links)
    q = rng.uniform(-3, 3, (n, tree.numConfigurationVariables())).astype(np.float32)
    h = csd.plant_handle(plant)
    assert h.num_links == links
    qd = torch.as_tensor(q).cuda()
    out = torch.zeros((n, links, 4, 4), dtype=torch.float32, device="cuda")
    _capi.check(_capi.lib().csd_fk(h.handle, ctypes.c_void_p(qd.data_ptr()), ctypes.c_int64(n),
                                   ctypes.c_void_p(out.data_ptr()), _capi.CSD_PTR_DEVICE, None))
    torch.cuda.synchronize()
    for i in (0, n - 1):
        ref = np.stack(tree.compute_link_frame_to_world_transforms(q[i]))
        np.testing.assert_allclose(out[i].cpu().numpy().transpose(0, 2, 1), ref, rtol=0, atol=2e-4)


def test_one_configuration_of_a_large_tree():
    """2,101 links: 33 us; 766 us when every call staged and ranked all links."""
    us = []
    for links in (9, 2101):
        plant, tree = tree_plant(links)
        h = csd.plant_handle(plant)
        q = torch.zeros(tree.numConfigurationVariables(), device="cuda")
        out = torch.zeros(links * 16, device="cuda")
        times = []
        for _ in range(10):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            _capi.check(_capi.lib().csd_fk(h.handle, ctypes.c_void_p(q.data_ptr()), ctypes.c_int64(1),
                                           ctypes.c_void_p(out.data_ptr()), _capi.CSD_PTR_DEVICE,
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            e[1].record()
            e[1].synchronize()
            times.append(1e3 * e[0].elapsed_time(e[1]))
        us.append(min(times))
    assert us[1] < 10 * us[0] + 100, us
