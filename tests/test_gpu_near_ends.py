"""GPU: FP64 sums at targets very near the ends of segments keep the precision
of the formula: R' is formed from the target and the segment's end themselves,
not through its start.

The reference is the segment formula in 80-bit arithmetic on the same inputs.
At 1e-7 from a node the two segments there are all but the whole sum (800 cm/s
against under 1), and R and R' are exact differences or right to an ulp of
their own, so the formula carries some tens of roundings: 1e-14 relative, where
an R' of R + (r2 - r1) is off by 1e-12 of itself."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from openvort_b200 import geometry as G
from openvort_b200._lib import Vec3d
from openvort_b200.tangle import Params

pytestmark = pytest.mark.gpu

P = Params(kappa=9.97e-4, core_a=1e-8, use_mf=0, hyperfriction=0, dl_max=1e-2, bh_theta=1e-3)
H, TOL = 1e-7, 1e-14


@pytest.fixture(scope="module")
def ov():
    import openvort_b200 as ov
    lib = ov.load()
    assert lib.ov_init(0) == 0, lib.ov_last_error_message()
    yield ov
    ov.configure(P, ov.OV_PREC_FP64)


def exact(t, pts, segments=None):
    """the sum over the segments (slots) in 80 bits, open boundaries"""
    x = t.pos.astype(np.longdouble)
    m = np.nonzero(t.active)[0] if segments is None else segments
    f = np.longdouble(P.kappa) / (4 * np.longdouble("3.14159265358979323846264338327950288"))
    out = np.zeros((len(pts), 3), np.longdouble)
    for i, r in enumerate(pts.astype(np.longdouble)):
        R, Rp = x[m] - r, x[t.links[m, 0]] - r
        a, b = np.sqrt((R * R).sum(1)), np.sqrt((Rp * Rp).sum(1))
        out[i] = (f * ((a + b) / (a * b * (a * b + (R * Rp).sum(1))))[:, None] * np.cross(R, Rp)).sum(0)
    return out


def rel(a, b):
    return float(np.max(np.linalg.norm((a - b).astype(float), axis=1) / np.linalg.norm(b.astype(float), axis=1)))


def coarse_ring():
    """segments of 2.5e-3, so R at the far end is 25000 times R'; tilted and off
    the middle of the box, where a tree drops the nodes on its mid-planes"""
    r = G.ring_points(np.array([1.3e-3, -0.7e-3, 0.9e-3]), (0.3, 0.2, 0.9), 1e-2, 25)
    return G.rings_to_tangle([r], (-0.05,) * 3, (0.05,) * 3, "open")


def near_nodes(t, rng):
    """points at H from some nodes, off the line there"""
    k = np.array([0, 1, 7, 24])
    u = rng.normal(size=(len(k), 3))
    return t.pos[k] + H * u / np.linalg.norm(u, axis=1)[:, None]


def test_points(ov):
    """Direct sums in chain order (with the ring's closing segment, which does
    not chain), of a node list, through the tree at its theta (the multi-image
    walk) and at another (the walk per image); at these no cell is accepted."""
    t = coarse_ring()
    pts = near_nodes(t, np.random.default_rng(1))
    want = exact(t, pts)
    lib = ov.load()
    ov.configure(P, 0)
    st = ov.DeviceState(t.copy())
    assert rel(st.eval_points(pts, method=0), want) < TOL
    assert rel(st.eval_points(pts, method=1), want) < TOL
    st.close()
    only = np.array([0, 6, 23, 24], np.int32)   # the segments that end at a node with a point
    want_only = exact(t, pts, only)
    zero = Vec3d((C.c_double * 3)(0, 0, 0))
    tree = lib.octree_build(t.ptr(), 0)
    for i, x in enumerate(pts):
        p = Vec3d((C.c_double * 3)(*x))
        v = lib.calculate_vs_shift(t.ptr(), p, -1, C.byref(zero), only.ctypes.data_as(C.POINTER(C.c_int)), len(only))
        assert rel(np.array(v.p[:])[None], want_only[i:i + 1]) < TOL, i
        for theta in (P.bh_theta, 2e-3):
            res = Vec3d()
            lib.octree_get_vs(tree, C.byref(p), theta, C.byref(res), -1)
            assert rel(np.array(res.p[:])[None], want[i:i + 1]) < TOL, (i, theta)
    lib.octree_destroy(tree)


def test_ensemble_and_nodes(ov):
    """Nodes of a second loop at H from nodes of the first: velocities less those
    of the second loop alone, as a tangle and as an ensemble of one system."""
    a = coarse_ring()
    pts = near_nodes(a, np.random.default_rng(2))
    far = pts + np.array([0.0, 0.0, 3e-3])
    loop = np.concatenate([np.stack([p, q]) for p, q in zip(pts, far)])
    box = ((-0.05,) * 3, (0.05,) * 3, "open")
    t = G.rings_to_tangle([a.pos, loop], *box)
    at = a.n + 2 * np.arange(len(pts))
    ov.configure(P, 0)
    both, alone = t.copy(), G.rings_to_tangle([loop], *box)
    ov.update_tangle(both, 0.0)
    ov.update_tangle(alone, 0.0)
    want = exact(a, t.pos[at])
    # the second loop's part is below 1 % of the difference, which keeps its digits
    assert np.linalg.norm(alone.vs, axis=1).max() < 1e-2 * np.linalg.norm(want.astype(float), axis=1).min()
    assert rel(both.vs[at] - alone.vs[2 * np.arange(len(pts))], want) < TOL
    b = ov.DeviceBatch(t.copy(), [0, t.n])
    b.update(0.0)
    b.download()
    assert rel(b.t.vs[at] - alone.vs[2 * np.arange(len(pts))], want) < TOL
    b.close()
