"""GPU: EMPTY slots may hold anything.

A tangle grows by realloc, so the position of an EMPTY slot can be any bit
pattern.  Every entry point must give the live nodes the same values whatever
the EMPTY slots hold: each call with NaN (of either sign), an infinity or 1e300
in the holes against the same call with the box centre.  FP64 bit for bit;
the mixed sums in slot order add their unchained segments in no fixed order (two
runs of the same input differ by 1e-11), so the mixed form to its tolerance."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from cases import rel_err
from openvort_b200 import geometry as G
from openvort_b200._lib import Vec3d
from openvort_b200.tangle import Flow, Params

pytestmark = pytest.mark.gpu

VALUES = [np.nan, -np.nan, np.inf, 1e300]
IDS = ["nan", "-nan", "inf", "1e300"]
D, DT, TOL_MIXED = 0.1, 1e-6, 1e-5
PARAMS = dict(kappa=9.97e-4, core_a=1e-8, alpha=0.098, alpha_p=0.016, use_mf=1, dl_max=1e-3, bh_theta=0.5,
              vn=Flow("simple", {"external_v": (0.5, 0, 0)}))


@pytest.fixture(scope="module")
def ov():
    import openvort_b200 as ov
    lib = ov.load()
    assert lib.ov_init(0) == 0, lib.ov_last_error_message()
    yield ov
    ov.configure(Params(**PARAMS), ov.OV_PREC_FP64)


def same(a, b, precision):
    if not np.all(np.isfinite(a)):
        return False
    return np.array_equal(a, b) if precision == 0 else rel_err(b, a) < TOL_MIXED


def holed(t, value):
    """t with `value` at its EMPTY slots"""
    out = t.copy()
    out.pos[~t.active] = value
    assert (~t.active).sum() >= 7
    return out


# around the block of 128 slots whose small sums take the geometry along; more
# than the interactions of such a sum; Barnes-Hut
@pytest.mark.parametrize("value", VALUES, ids=IDS)
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("boundary,rings,use_bh", [("open", 2, 0), ("periodic-26", 4, 0), ("periodic-26", 40, 0),
                                                   ("periodic-26", 12, 1)])
def test_updates_runs_and_points(ov, boundary, rings, use_bh, precision, value):
    t = G.random_ring_tangle(5 + rings, rings, D, boundary=boundary, empty_slots=7)
    p = Params(use_bh=use_bh, **PARAMS)
    pts = np.random.default_rng(1).uniform(0, D, size=(40, 3))
    got = []
    for hole in (D / 2, value):
        ov.configure(p, precision)
        h = holed(t, hole)
        ov.update_tangle(h, 0.0)
        res = [h.vels[t.active], h.vs[t.active], h.tangents[t.active], h.normals[t.active]]
        ov.rk4_step(h, 0.0, DT)
        res.append(h.pos[t.active])
        st = ov.DeviceState(holed(t, hole))
        st.run(0.0, DT, 2)
        st.download()
        res += [st.t.pos[t.active], st.t.vels[t.active], st.eval_points(pts, method=0), st.eval_points(pts, method=1)]
        st.close()
        lib = ov.load()
        h = holed(t, hole)
        v = lib.calculate_vs(h.ptr(), Vec3d((C.c_double * 3)(*pts[0])), -1)
        res.append(np.array(v.p[:]))
        k = int(np.nonzero(t.active)[0][3])
        ov.update_tangle(h, 0.0)
        lib.update_velocity(h.ptr(), k, 0.0, None)
        ov.check(lib)
        res.append(h.vels[k])
        got.append(res)
    for i, (a, b) in enumerate(zip(*got)):
        assert same(a, b, precision), i


@pytest.mark.parametrize("value", VALUES, ids=IDS)
@pytest.mark.parametrize("systems", [3, 400])
def test_fp64_ensembles(ov, systems, value):
    """Few systems (their sources summed in shares) and many."""
    t, off = holed_ensemble(systems)
    assert_same_ensemble(ov, t, off, value, ov.OV_PREC_FP64, [(128, 128), (64, 0)])


@pytest.mark.parametrize("value", VALUES, ids=IDS)
@pytest.mark.parametrize("systems", [3, 400])
def test_mixed_ensembles(ov, systems, value):
    """Every kind of mixed kernel: offsets from the first target, from the
    middle one, and in chain order."""
    t, off = holed_ensemble(systems)
    assert_same_ensemble(ov, t, off, value, ov.OV_PREC_MIXED, [(128, 128), (256, 64), (64, 64), (64, 256), (128, 0)])


def holed_ensemble(systems):
    """ring pairs of 5 .. 140 nodes a ring, with EMPTY slots at the front, in
    the middle and at the end of each system"""
    rng = np.random.default_rng(systems)
    parts, off = [], [0]
    for _ in range(systems):
        rings = [G.ring_points(rng.uniform(-0.02, 0.02, 3), rng.normal(size=3), rng.uniform(5e-3, 1e-2),
                               int(rng.integers(5, 140))) for _ in range(2)]
        parts.append(rings)
    pos, fwd, rev, status = [], [], [], []
    for rings in parts:
        n0 = off[-1]
        at = n0 + 2
        for r in rings:
            n, i = len(r), np.arange(len(r))
            pos += [np.zeros((2, 3)), r]
            fwd += [[-1, -1], at + (i + 1) % n]
            rev += [[-1, -1], at + (i - 1) % n]
            status += [[-1, -1], np.zeros(n, int)]
            at += n + 2
        pos.append(np.zeros((1, 3)))
        fwd.append([-1])
        rev.append([-1])
        status.append([-1])
        off.append(at - 1)
    from openvort_b200.tangle import HostTangle
    cat = lambda x: np.concatenate(x).astype(np.int32)
    t = HostTangle(np.concatenate(pos), cat(fwd), cat(rev), cat(status), None, (-0.05,) * 3, (0.05,) * 3, "open")
    return t, off


def assert_same_ensemble(ov, t, off, value, precision, shapes):
    act = t.active
    for shape in shapes:
        got = []
        for hole in (0.0, value):
            ov.configure(Params(**PARAMS), precision)
            b = ov.DeviceBatch(holed(t, hole), off)
            b.set_tuning(*shape)
            b.update(0.0)
            b.download()
            res = [b.t.vels[act].copy()]
            b.run(0.0, DT, 2)
            b.download()
            got.append(res + [b.t.pos[act].copy()])
            b.close()
        for x, y in zip(*got):
            assert same(x, y, precision), shape


@pytest.mark.parametrize("value", VALUES, ids=IDS)
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("boundary", ["open", "periodic-26"])
def test_reconnection(ov, boundary, precision, value):
    side = 0.05
    t = G.random_ring_tangle(17, 40, side, dl=side / 100, boundary=boundary, empty_slots=9)
    p = Params(**PARAMS)
    lib = ov.load()
    got = []
    for hole in (side / 2, value):
        ov.configure(p, precision)
        h = holed(t, hole)
        ov.update_tangle(h, 0.0)
        h.recalc[:] = 0
        n = lib.ov_reconnect_vortices(h.ptr(), 0.0, 2.5 * side / 100, 0.087)
        ov.check(lib)
        assert n > 3
        got.append(h)
    a, b = got
    assert np.array_equal(a.links, b.links) and np.array_equal(a.recalc, b.recalc)
    assert same(a.vels[t.active], b.vels[t.active], precision)


@pytest.mark.parametrize("value", VALUES, ids=IDS)
@pytest.mark.parametrize("nodes", [30, 127, 301])
def test_adjoint(ov, nodes, value):
    """Velocity, its vector-Jacobian product and the gradient through four
    steps, two from a checkpoint.  The pair passes add with atomics, in no fixed
    order: some hundred roundings of partial sums up to a few ten times the
    result, so 1e-12 of the largest entry."""
    from openvort_b200.adjoint import Adjoint
    rng = np.random.default_rng(nodes)
    rings = [G.ring_points(c, rng.normal(size=3), 1e-2, n)
             for c, n in (((0, 0, 0), nodes // 3), ((5e-3, 0, 0), nodes - nodes // 3))]
    t = G.rings_to_tangle(rings, (-0.05,) * 3, (0.05,) * 3, "open", empty_slots=9)
    act = t.active
    g = np.where(act[:, None], rng.normal(size=(t.n, 3)), 0.0)
    vn = np.array([0.2, 0.0, 0.1])
    got = []
    for hole in (0.0, value):
        ov.configure(Params(**PARAMS), ov.OV_PREC_FP64)
        h = holed(t, hole)
        a = Adjoint(h)
        x_bar, vn_bar = a.velocity_vjp(h.pos, g, vn)
        res = [a.velocity(h.pos, vn)[act], x_bar[act], vn_bar]
        res.append(a.forward(h.pos, vn, 0.0, DT, 4, every=2)[act])
        x_bar, vn_bar = a.backward(g)
        got.append(res + [x_bar[act], vn_bar])
        a.close()
    for i, (a, b) in enumerate(zip(*got)):
        assert np.all(np.isfinite(b)) and np.abs(a - b).max() <= 1e-12 * np.abs(a).max(), i


@pytest.mark.parametrize("precision", [0, 1])
def test_adjoint_without_nodes(ov, precision):
    """Slots that are all EMPTY: nothing moves, and the gradient passes through."""
    from openvort_b200.adjoint import Adjoint
    from openvort_b200.tangle import HostTangle
    n = 6
    none = -np.ones(n, np.int32)
    t = HostTangle(np.ones((n, 3)), none, none, none, none, (-0.05,) * 3, (0.05,) * 3, "open")
    ov.configure(Params(**PARAMS), precision)
    a = Adjoint(t)
    g = np.random.default_rng(2).normal(size=(n, 3))
    assert np.array_equal(a.forward(t.pos, np.zeros(3), 0.0, DT, 3, every=2), t.pos)
    x_bar, vn_bar = a.backward(g)
    assert np.array_equal(x_bar, g) and np.all(vn_bar == 0)
    x_bar, vn_bar = a.velocity_vjp(t.pos, g, np.zeros(3))
    assert np.all(x_bar == 0) and np.all(vn_bar == 0)
    a.close()


@pytest.mark.parametrize("value", VALUES, ids=IDS)
def test_walls_pinned_nodes_and_remesh(ov, value):
    """Mirror images with pinned nodes (the second geometry pass, the walk per
    image), and the passes that change a tangle: remeshing takes EMPTY slots for
    new nodes, boundary enforcement and small-loop removal visit all slots."""
    from cases import load
    lib = ov.load()
    wall, pw, _, _ = load("wall_half_ring")
    got = []
    for hole in (D / 2, value):
        res = []
        for use_bh in (0, 1):
            ov.configure(dataclasses.replace(pw, use_bh=use_bh, bh_theta=0.5), 0)
            h = with_holes(wall, hole)
            ov.update_tangle(h, 0.0)
            res.append(h.vels[h.active].copy())
            ov.rk4_step(h, 0.0, 1e-7)
            res.append(h.pos[h.active].copy())
        ov.configure(Params(**PARAMS), 0)
        h = holed(G.random_ring_tangle(8, 6, D, boundary="periodic-26", empty_slots=40), hole)
        ov.update_tangle(h, 0.0)
        live = np.nonzero(h.active)[0]
        h.pos[live[::9]] = 0.5 * (h.pos[live[::9]] + h.pos[h.links[live[::9], 0]])
        ov.update_tangle(h, 0.0)
        seg = np.median(h.dxi[h.active])
        changes = lib.ov_remesh(h.ptr(), 0.6 * seg, 1.4 * seg, None)
        ov.check(lib)
        assert changes > 3
        lib.ov_enforce_boundaries(h.ptr())
        lib.ov_eliminate_small_loops(h.ptr(), 5)
        ov.check(lib)
        ov.update_tangle(h, 0.0)
        got.append(res + [h.stat[:, 0].copy(), h.links[h.active].copy(), h.pos[h.active].copy(), h.vels[h.active].copy()])
    for i, (a, b) in enumerate(zip(*got)):
        assert np.all(np.isfinite(b)) and np.array_equal(a, b), i


def with_holes(t, value):
    """t with three EMPTY slots behind its nodes"""
    from openvort_b200.tangle import HostTangle
    none = np.full(3, -1, np.int32)
    return HostTangle(np.concatenate([t.pos, np.full((3, 3), value)]), np.concatenate([t.links[:, 0], none]),
                      np.concatenate([t.links[:, 1], none]), np.concatenate([t.stat[:, 0], none]),
                      np.concatenate([t.stat[:, 1], none]), t.box_lo, t.box_hi, t.boundary)
