"""GPU: a NaN in an input that the host does not check (probe points, the
adjoint's positions) comes out as NaN, whichever sign it has: the distance
cut-off, which drops a segment with an end at the target, must not take it for
a distance of zero."""
import ctypes as C

import numpy as np
import pytest

from openvort_b200 import geometry as G
from openvort_b200._lib import Vec3d
from openvort_b200.tangle import Flow, Params

pytestmark = pytest.mark.gpu

PARAMS = dict(kappa=9.97e-4, core_a=1e-8, alpha=0.098, alpha_p=0.016, use_mf=1, dl_max=1e-3, bh_theta=0.5,
              vn=Flow("simple", {"external_v": (0.5, 0, 0)}))
NANS = [np.uint64(0x7ff8000000000000).view(np.float64), np.uint64(0xfff8000000000000).view(np.float64)]


@pytest.fixture(scope="module")
def ov():
    import openvort_b200 as ov
    lib = ov.load()
    assert lib.ov_init(0) == 0, lib.ov_last_error_message()
    yield ov
    ov.configure(Params(**PARAMS), ov.OV_PREC_FP64)


@pytest.mark.parametrize("nan", NANS, ids=["plus", "minus"])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("boundary", ["open", "periodic-26"])
def test_points(ov, boundary, precision, nan):
    t = G.random_ring_tangle(3, 8, 0.1, boundary=boundary)
    pts = np.random.default_rng(3).uniform(0, 0.1, size=(40, 3))
    pts[[0, 7, 39], [0, 1, 2]] = nan
    bad = np.isnan(pts).any(axis=1)
    lib = ov.load()
    for use_bh in (0, 1):
        ov.configure(Params(use_bh=use_bh, **PARAMS), precision)
        st = ov.DeviceState(t.copy())
        for method in (0, 1):
            v = st.eval_points(pts, method=method)
            assert np.isnan(v[bad]).any(axis=1).all() and np.isfinite(v[~bad]).all(), (use_bh, method)
        st.close()
    tree = lib.octree_build(t.ptr(), 0)
    for i in np.nonzero(bad)[0]:
        x = Vec3d((C.c_double * 3)(*pts[i]))
        assert np.isnan(lib.calculate_vs(t.ptr(), x, -1).p[:]).any()
        # a node list: the segment-table kernel
        only = np.arange(5, dtype=np.int32)
        zero = Vec3d((C.c_double * 3)(0, 0, 0))
        v = lib.calculate_vs_shift(t.ptr(), x, -1, C.byref(zero), only.ctypes.data_as(C.POINTER(C.c_int)), 5)
        assert np.isnan(v.p[:]).any()
        res = Vec3d()
        lib.octree_get_vs(tree, C.byref(x), 0.5, C.byref(res), -1)
        assert np.isnan(res.p[:]).any()
    lib.octree_destroy(tree)


@pytest.mark.parametrize("nan", NANS, ids=["plus", "minus"])
def test_adjoint_positions(ov, nan):
    """A NaN node makes every live node's gradient NaN, as each node is a target
    of that node's segments."""
    from openvort_b200.adjoint import Adjoint
    ov.configure(Params(**PARAMS), ov.OV_PREC_FP64)
    t = G.single_ring(40, 1e-2)
    a = Adjoint(t)
    x = t.pos.copy()
    x[5] = nan
    x_bar, _ = a.velocity_vjp(x, np.random.default_rng(5).normal(size=x.shape), np.zeros(3))
    assert np.isnan(x_bar).any(axis=1).all()
    a.close()
