"""GPU: ov_get_last_stats tells of the last velocity evaluation on the thread,
its counters and its times alike."""
import dataclasses
import time

import numpy as np
import pytest

from openvort_b200 import geometry as G
from openvort_b200.tangle import Params

pytestmark = pytest.mark.gpu

P = Params(core_a=1e-8, dl_max=1e-3, use_bh=1, bh_theta=0.5)


@pytest.fixture(scope="module")
def ov():
    import openvort_b200 as ov
    lib = ov.load()
    assert lib.ov_init(0) == 0, lib.ov_last_error_message()
    yield ov
    ov.configure(P, ov.OV_PREC_FP64)


def fields(s):
    return s.interactions, s.cell_interactions, s.cells, s.eval_ms, s.build_ms, s.total_ms


def test_times_follow_the_evaluation(ov):
    t = G.random_ring_tangle(31, 40, 0.1, boundary="periodic-26")
    ov.configure(P, 0)
    st = ov.DeviceState(t)
    st.reset_stats()
    st.run(0.0, 1e-7, 3)
    s = ov.stats()
    assert s.cell_interactions > 0 and s.cells > 0 and s.eval_ms > 0 and s.build_ms > 0
    assert s.total_ms == pytest.approx(s.eval_ms + s.build_ms)
    # twelve evaluations of a few hundred microseconds each
    assert s.eval_ms < st.stats().bs_kernel_ms / 3
    # a point query is no evaluation: the times stay, however long ago it was
    before = ov.stats()
    time.sleep(0.2)
    st.eval_points(np.full((40, 3), 0.05), method=1)
    after = ov.stats()
    assert (after.eval_ms, after.build_ms) == (before.eval_ms, before.build_ms)
    st.close()
    # an evaluation without a sum has no times
    ov.configure(dataclasses.replace(P, lia_only=1), 0)
    st = ov.DeviceState(t)
    st.update_tangle(0.0)
    assert fields(ov.stats()) == (0, 0, 0, 0, 0, 0)
    st.close()


def test_no_times_of_the_walk_after_it(ov):
    """Local induction alone on a state that has walked before."""
    t = G.random_ring_tangle(32, 10, 0.1, boundary="periodic-26")
    ov.configure(P, 0)
    h = t.copy()
    ov.update_tangle(h, 0.0)
    assert ov.stats().eval_ms > 0
    ov.configure(dataclasses.replace(P, lia_only=1), 0)
    ov.update_tangle(h, 0.0)
    assert fields(ov.stats()) == (0, 0, 0, 0, 0, 0)
