"""GPU: one octree walked by several host threads at a time, as the reference's
parallel loops over update_velocity do.  Every thread must get the bits that the
same calls give one after another."""
import ctypes as C
import threading

import numpy as np
import pytest

from openvort_b200 import geometry as G
from openvort_b200._lib import Vec3d
from openvort_b200.tangle import Params

pytestmark = pytest.mark.gpu

D, THREADS = 0.1, 4
P = Params(kappa=9.97e-4, core_a=1e-8, dl_max=1e-3, use_bh=1, bh_theta=0.5)


@pytest.fixture(scope="module")
def ov():
    import openvort_b200 as ov
    lib = ov.load()
    assert lib.ov_init(0) == 0, lib.ov_last_error_message()
    yield ov
    ov.configure(P, ov.OV_PREC_FP64)


def in_threads(work):
    """work(i) for every thread number i, all at once; their results"""
    out, errors = [None] * THREADS, []
    gate = threading.Barrier(THREADS)

    def body(i):
        try:
            gate.wait(60)
            out[i] = work(i)
        except Exception as e:
            errors.append(e)

    ts = [threading.Thread(target=body, args=(i,)) for i in range(THREADS)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    return out


@pytest.mark.parametrize("precision", [0, 1])
def test_one_tree_many_threads(ov, precision):
    lib = ov.load()
    ov.configure(P, precision)
    t = G.random_ring_tangle(11, 30, D, boundary="periodic-26")
    ov.update_tangle(t, 0.0)
    tree = lib.octree_build(t.ptr(), 0)
    ov.check(lib)
    copies = [t.copy() for _ in range(THREADS)]
    for h in copies:
        h.set_images_from_library(lib)
        h.tangents[:], h.normals[:] = t.tangents, t.normals

    def nodes(i):
        h = copies[i]
        h.vels[:] = 0
        for k in range(i, t.n, t.n // 10):
            lib.update_velocity(h.ptr(), k, 0.0, tree)
            ov.check(lib)
        return h.vels.copy()

    def points(i):
        out = []
        for x in np.random.default_rng(i).uniform(0, D, size=(20, 3)):
            res = Vec3d()
            lib.octree_get_vs(tree, C.byref(Vec3d((C.c_double * 3)(*x))), P.bh_theta, C.byref(res), i)
            ov.check(lib)
            out.append(res.p[:])
        return np.array(out)

    def everything(i):
        for _ in range(3):
            lib.update_velocities(copies[i].ptr(), 0.0, tree)
            ov.check(lib)
        return copies[i].vels.copy()

    def mixture(i):
        return points(i) if i % 2 else nodes(i)

    for work in (nodes, points, everything, mixture):
        want = [work(i) for i in range(THREADS)]
        assert all(np.any(w != 0) for w in want)
        for got, w in zip(in_threads(work), want):
            assert np.array_equal(got, w), work.__name__
    lib.octree_destroy(tree)
