"""Face placement (place_faces) at the edges of what a thread keeps in
registers: two candidates a thread, 512 for region editing's 256 threads and
2,048 for an inflation's 1,024, the rest in global memory. Every face is
decided by the oracle with the GPU's verdicts, bit for bit (the arithmetic is
the oracle's, so there is no tolerance)."""
import numpy as np
import pytest

import csdecomp_b200 as csd
from csdecomp_b200 import scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def box(lo, hi):
    p = csd.HPolyhedron()
    p.MakeBox(lo, hi)
    return p


@pytest.mark.parametrize("dof", [2, 7])
def test_edit_candidates_per_region(dof):
    sc = scenes.arm_scene(310 + dof, num_spheres=max(8, 3 * dof), num_world_boxes=30, num_world_spheres=20,
                          dof_per_arm=dof, keepout=0.5)
    d, rids = sc.dim, sc.inspector.robot_geometry_ids
    lo, hi = sc.lower(), sc.upper()
    chk = lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant)  # noqa: E731
    counts = [1, 31, 255, 256, 257, 511, 512, 513, 1300]
    mid = ((lo + hi) / 2).astype(np.float32)
    w = ((hi - lo) * 0.02).astype(np.float32)
    m = len(counts)
    ls = np.tile((mid - w)[:, None], (1, m)).astype(np.float32)
    le = np.tile((mid + w)[:, None], (1, m)).astype(np.float32)
    regions = [box(lo, hi)] * m
    q = sc.random_configs(200000, 5)
    q = q[chk(q) == 0]
    assert q.shape[0] >= sum(counts)
    col = q[:sum(counts)]
    col[1::7] = col[::7][:col[1::7].shape[0]]  # equal distances: the lower index wins
    seg = np.repeat(np.arange(m), counts)
    opt = csd.EditRegionsOptions()
    edited, (proj, best) = csd.EditRegionsCuda(col.T, seg, ls, le, regions, sc.plant, rids, csd.Voxels(), 0.03, opt)
    ref, rproj, rbest = O.edit_regions(sc.plant, col, seg, ls.T, le.T, [(r.A(), r.b()) for r in regions], rids, None,
                                       0.03, opt.configuration_margin, opt.bisection_steps, checker=chk)
    np.testing.assert_array_equal(proj.T, rproj)
    np.testing.assert_array_equal(best.T, rbest)
    for e, (A, b), n in zip(edited, ref, counts):
        np.testing.assert_array_equal(e.A(), A, err_msg=f"{n} candidates")
        np.testing.assert_array_equal(e.b(), b, err_msg=f"{n} candidates")


@pytest.mark.parametrize("particles", [1023, 2048, 2049, 4000])
def test_inflation_candidates(particles):
    sc = scenes.arm_scene(321, num_spheres=14, num_world_boxes=40, num_world_spheres=40, dof_per_arm=5, keepout=0.4)
    chk = lambda q: csd.CheckCollisionFreeCuda(q.T, sc.plant)  # noqa: E731
    ce = lambda a, b: csd.CheckEdgesCollisionFreeCuda(a.T, b.T, sc.plant)  # noqa: E731
    q0, q1 = scenes.seed_edges(sc, 1, 17, chk, ce)[0]
    opt = csd.EizoOptions(num_particles=particles, mixing_steps=6, bisection_steps=7,
                          max_hyperplanes_per_iteration=10, epsilon=0.01, delta=0.05, tau=0.5, max_iterations=3,
                          configuration_margin=0.01, seed=5)
    dom = box(sc.lower(), sc.upper())
    A, b, _ = O.eizo(sc.plant, q0, q1, dom.A(), dom.b(), opt, sc.inspector.robot_geometry_ids, capacity=200,
                     checker=chk)
    inf = csd.CudaEdgeInflator(sc.plant, sc.inspector.robot_geometry_ids, opt, dom, face_capacity=200)
    got = inf.inflateEdge(q0, q1, None, 0.0, verbose=False)
    assert A.shape[0] > 2 * sc.dim  # faces were placed beyond the box
    np.testing.assert_array_equal(got.A(), A)
    np.testing.assert_array_equal(got.b(), b)
