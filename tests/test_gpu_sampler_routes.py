"""Uniform sampling on both sides of the line between a thread and a group of lanes per chain: the samples are the
oracle's either way, from host and from device arrays, with polytopes of both kinds in one call."""
import ctypes

import numpy as np
import pytest
import torch

import csdecomp_b200 as csd
from csdecomp_b200 import _capi
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def polytope(rng, dim, faces):
    """`faces` faces around a start: the box first, the rest cutting it."""
    c = rng.uniform(-0.5, 0.5, dim)
    A = np.kron(np.eye(dim), [[-1.0], [1.0]])[:faces]
    b = np.full(len(A), 1.0)
    n = faces - len(A)
    a = rng.normal(size=(n, dim))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.concatenate([b, a @ c + rng.uniform(0.01, 1.0, n)])
    return np.concatenate([A, a]).astype(np.float32), b.astype(np.float32), c.astype(np.float32)


def device_samples(A, b, off, dim, starts, samples, mixing, seed):
    put = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    P = len(off) - 1
    t = [put(A), put(b), put(np.asarray(off, np.int32)), put(starts)]
    out = torch.zeros((P, samples, dim), dtype=torch.float32, device="cuda")
    failed = ctypes.c_int32(-1)
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    _capi.check(_capi.lib().csd_uniform_sample_hpolyhedra(p(t[0]), p(t[1]), p(t[2]), P, dim, p(t[3]), samples, mixing,
                                                          ctypes.c_uint64(seed), p(out), ctypes.byref(failed),
                                                          _capi.CSD_PTR_DEVICE, None))
    torch.cuda.synchronize()
    return out.cpu().numpy(), failed.value


# faces on both sides of 44 and 58, chains on both sides of 12,000 + 1,500 per face and of 60,000; odd chain counts
@pytest.mark.parametrize("dim", [1, 2, 3, 5, 7, 8, 9, 14, 16])
@pytest.mark.parametrize("faces", [(2,), (6, 44, 45), (30, 58, 59, 300)])
@pytest.mark.parametrize("chains", [11999, 21001, 70003])
def test_routes_equal_oracle(dim, faces, chains):
    rng = np.random.default_rng(1000 * dim + chains + len(faces))
    polys = [polytope(rng, dim, f) for f in faces]
    samples, mixing = chains // len(faces) + 1, 3
    starts = np.stack([c for _, _, c in polys])
    got = csd.UniformSampleInHPolyhedraCuda([csd.HPolyhedron(A, b) for A, b, _ in polys], starts.T, samples, mixing, seed=dim)
    off = np.cumsum([0] + [len(b) for _, b, _ in polys])
    dev, failed = device_samples(np.concatenate([A for A, _, _ in polys]), np.concatenate([b for _, b, _ in polys]), off,
                                 dim, starts, samples, mixing, dim)
    for i, (A, b, c) in enumerate(polys):
        ref, _ = O.hit_and_run(A, b, c, samples, mixing, seed=dim, stream=i)
        np.testing.assert_array_equal(got[i].T, ref)
        np.testing.assert_array_equal(dev[i], ref)
    assert failed == sum(int(np.isnan(d[:, 0]).sum()) for d in dev)


# rows beyond the staging buffer, chains on both sides of 80,000
@pytest.mark.parametrize("dim,faces", [(2, 2100), (7, 1300), (14, 700), (14, 1100)])
@pytest.mark.parametrize("chains", [30000, 90001])
def test_unstaged_polytopes_equal_oracle(dim, faces, chains):
    rng = np.random.default_rng(faces + chains)
    A, b, c = polytope(rng, dim, faces)
    got = csd.UniformSampleInHPolyhedraCuda([csd.HPolyhedron(A, b)], c[:, None], chains, 1, seed=3)[0]
    ref, _ = O.hit_and_run(A, b, c, chains, 1, seed=3, stream=0)
    np.testing.assert_array_equal(got.T, ref)


def test_failed_chains_and_no_faces():
    """An empty polytope's chains are NaN and counted, whichever kernel runs them; no faces bound nothing."""
    A = np.array([[1.0, 0.0], [-1.0, 0.0]], np.float32)
    b = np.array([-2.0, -2.0], np.float32)
    off = [0, 2, 2]
    starts = np.zeros((2, 2), np.float32)
    for samples in (100, 40000):
        out, failed = device_samples(A, b, off, 2, starts, samples, 2, 1)
        assert np.isnan(out[0]).all() and failed == samples
        ref, _ = O.hit_and_run(np.zeros((0, 2), np.float32), np.zeros(0, np.float32), starts[1], samples, 2, seed=1, stream=1)
        np.testing.assert_array_equal(out[1], ref)


def test_many_chains_in_small_polytopes():
    """1.6 million chains of ten steps, 12 faces in two dimensions: 0.42 ms, 0.99 ms with eight lanes on each chain."""
    rng = np.random.default_rng(0)
    A, b, c = polytope(rng, 2, 12)
    put = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()  # noqa: E731
    t = [put(np.tile(A, (4, 1))), put(np.tile(b, 4)), put(np.arange(5, dtype=np.int32) * 12), put(np.tile(c, 4))]
    out = torch.zeros(4 * 400000 * 2, device="cuda")
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    times = []
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        _capi.check(_capi.lib().csd_uniform_sample_hpolyhedra(p(t[0]), p(t[1]), p(t[2]), 4, 2, p(t[3]), 400000, 10,
                                                              ctypes.c_uint64(1), p(out), None, _capi.CSD_PTR_DEVICE,
                                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        e[1].record()
        e[1].synchronize()
        times.append(e[0].elapsed_time(e[1]))
    assert min(times) < 0.7, times
