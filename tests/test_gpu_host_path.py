"""Calls whose host work depends on their size or history: point checks on
mapped host memory up to 16,384 configurations and through copies beyond, call
scratch kept between calls (several threads, growing and shrinking sizes), the
staging status read only where the pair sweep may have run."""
import threading

import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 16383, 16384, 16385])
def test_small_point_checks(n):
    sc = scenes.arm_scene(81, num_spheres=40, num_capsules=2, num_world_spheres=20, keepout=0.6)
    q = sc.random_configs(17700, 3)
    whole = csd.CheckCollisionFreeCuda(q.T, sc.plant)
    assert 0 < whole.mean() < 1
    for k in (0, 1300):
        np.testing.assert_array_equal(csd.CheckCollisionFreeCuda(q[k:k + n].T, sc.plant), whole[k:k + n])


def test_uniform_sampling_from_several_threads():
    """Calls of different sizes at once equal the same calls one after the other."""
    rng = np.random.default_rng(4)
    boxes = []
    for d, s in [(2, 40), (7, 3000), (3, 700), (7, 12), (14, 900), (6, 5000)]:
        p = csd.HPolyhedron()
        p.MakeBox(-rng.uniform(0.5, 1.0, d), rng.uniform(0.5, 1.0, d))
        boxes.append((p, np.zeros((d, 1), np.float32), s))
    run = lambda p, x, s: csd.UniformSampleInHPolyhedraCuda([p], x, s, 20, 11)[0]  # noqa: E731
    want = [run(*b) for b in boxes]
    got = [[None] * len(boxes) for _ in range(6)]

    def work(t):
        for r in range(4):
            for i in range(len(boxes)):
                j = (i + t + r) % len(boxes)
                got[t][j] = run(*boxes[j])

    threads = [threading.Thread(target=work, args=(t,)) for t in range(len(got))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for row in got:
        for a, b in zip(row, want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind", ["int64", "uint32", "uint64", "list"])
def test_edit_segment_index_types(kind):
    sc = scenes.arm_scene(82, num_spheres=24, num_world_spheres=20, keepout=0.5)
    lo, hi = sc.lower(), sc.upper()
    q = sc.random_configs(1500, 3)
    q = q[csd.CheckCollisionFreeCuda(q.T, sc.plant) == 0][:300]
    seg = np.arange(q.shape[0]) % 3
    mid, w = (lo + hi) / 2, (hi - lo) * 0.02
    ls = np.tile((mid - w)[:, None], (1, 3)).astype(np.float32)
    le = np.tile((mid + w)[:, None], (1, 3)).astype(np.float32)
    dom = csd.HPolyhedron()
    dom.MakeBox(lo, hi)
    opt = csd.EditRegionsOptions()
    idx = list(seg) if kind == "list" else seg.astype(kind)
    out, _ = csd.EditRegionsCuda(q.T, idx, ls, le, [dom] * 3, sc.plant, sc.inspector.robot_geometry_ids, csd.Voxels(),
                                 0.03, opt)
    ref, _, _ = O.edit_regions(sc.plant, q, seg, ls.T, le.T, [(dom.A(), dom.b())] * 3, sc.inspector.robot_geometry_ids,
                               None, 0.03, opt.configuration_margin, opt.bisection_steps,
                               checker=lambda x: csd.CheckCollisionFreeCuda(x.T, sc.plant))
    for e, (A, b) in zip(out, ref):
        np.testing.assert_array_equal(e.A(), A)
        np.testing.assert_array_equal(e.b(), b)
    with pytest.raises(IndexError):
        csd.EditRegionsCuda(q.T, np.full(q.shape[0], 3), ls, le, [dom] * 3, sc.plant,
                            sc.inspector.robot_geometry_ids, csd.Voxels(), 0.03, opt)
