"""Sweeps with the DWR indicator in turn with plain ones, from several iterations and over fewer and more
steps, against the same sweep on a context that does nothing else."""
import numpy as np
import pytest

from discrete_adjoint_b200 import GeoflowContext, TimeProps, _ffi, adjoint_run, inputs
from discrete_adjoint_b200.dwr import Indicator, error_grid

pytestmark = pytest.mark.gpu


def same(a, b):
    for k in ("J", "dJ_dintfrict", "forward_steps"):
        assert getattr(a, k) == getattr(b, k), k
    for k in ("dJ_dbedfrict", "dJ_dpile", "lambda0", "dwr_cell", "dwr_steps"):
        x, y = getattr(a, k, None), getattr(b, k, None)
        assert (x is None) == (y is None) and (x is None or np.array_equal(x, y)), k


@pytest.mark.parametrize("precision", [_ffi.DA_PREC_FP64, _ffi.DA_PREC_FP32_SPLIT])
def test_indicator_sweeps_in_turn_with_plain_ones(precision):
    w = inputs.test_case(seed=3)
    m = w.mesh
    g = error_grid(w)
    box = (m.x.min(), m.x.max(), m.y.min(), m.y.max())

    def start(c, iter0):
        c.set_state(m.h0, m.hu0, m.hv0)
        c.set_time(0.0, iter0)

    def sweep(c, steps, snaps, dwr):
        return adjoint_run(c, box, steps, snaps, m.dh0_dpile, want_lambda0=True, dwr=dwr)

    # (first iteration, steps, checkpoints, indicator): across the friction threshold's change at 50, with
    # repeats and with fewer steps after more
    calls = [(0, 9, 2, True), (0, 9, 2, False), (47, 9, 2, True), (47, 9, 2, False), (60, 9, 2, True), (60, 4, 2, True),
             (0, 9, 2, True), (0, 12, 3, True), (0, 9, 2, False)]
    with GeoflowContext(w.mat, TimeProps(), precision=precision) as c:
        c.upload_mesh(m)
        ind = Indicator(c, g)
        for iter0, steps, snaps, dwr in calls:
            start(c, iter0)
            got = sweep(c, steps, snaps, dwr)
            with GeoflowContext(w.mat, TimeProps(), precision=precision) as d:
                d.upload_mesh(m)
                Indicator(d, g)
                start(d, iter0)
                same(got, sweep(d, steps, snaps, dwr))
        # a single step between them, and a new error grid: the sweeps on it are captured anew
        start(c, 0)
        ind.step(np.ones((3, m.n)))
        Indicator(c, g)
        a = sweep(c, 9, 2, True)
        start(c, 0)
        same(a, sweep(c, 9, 2, True))
