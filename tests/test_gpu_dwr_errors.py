"""An error of the error grid's step reaches the caller, once: the next indicator starts without it."""
import numpy as np
import pytest

from discrete_adjoint_b200 import GeoflowContext, TimeProps, _ffi, adjoint_run, inputs
from discrete_adjoint_b200.dwr import Indicator, error_grid

pytestmark = pytest.mark.gpu


def test_error_of_the_error_grid_is_reported_and_does_not_last():
    w = inputs.test_case(seed=1)
    m = w.mesh
    wet = m.h0 > 1.0
    box = (m.x.min(), m.x.max(), m.y.min(), m.y.max())
    # gravity on the error grid alone that makes the wave speed exceed its bound where the pile stands
    # and nowhere else
    bad, good = error_grid(w), error_grid(w)
    n, nf = m.n, bad.fine.n
    g = bad.fine.gravity.reshape(3, nf)
    g[2, wet[bad.parent]] = 1e30
    bad.fine._soa = None
    # a state that is dry there
    far = np.abs(m.x - m.x[wet].mean()) > 0.25 * (m.x.max() - m.x.min())
    off = np.where(far & (m.h0 == 0), 2.0, 0.0)
    lam = np.ones((3, n))
    with GeoflowContext(w.mat, TimeProps()) as c:
        c.upload_mesh(m)
        ind = Indicator(c, good)
        c.set_state(off, 0 * off, 0 * off)
        ref = ind.step(lam)
        ref_run = adjoint_run(c, box, 3, 1, dwr=True)
    with GeoflowContext(w.mat, TimeProps()) as c:
        c.upload_mesh(m)
        ind = Indicator(c, bad)
        for _ in range(2):
            c.set_state(m.h0, m.hu0, m.hv0)
            c.set_time(0.0, 0)
            with pytest.raises(_ffi.DAError) as e:
                ind.step(lam)
            assert e.value.code == _ffi.DA_ERR_EIGEN
            with pytest.raises(_ffi.DAError) as e:
                adjoint_run(c, box, 3, 1, dwr=True)
            assert e.value.code == _ffi.DA_ERR_EIGEN
            # the coarse context is where it was and has no error of its own
            assert all(np.array_equal(a, b) for a, b in zip(c.get_state(), (m.h0, m.hu0, m.hv0)))
            assert c.step().iter == 1
            c.set_state(off, 0 * off, 0 * off)
            c.set_time(0.0, 0)
            got = ind.step(lam)
            run = adjoint_run(c, box, 3, 1, dwr=True)
            for a, b in zip(got, ref):
                assert np.array_equal(a, b)
            assert np.array_equal(run.dwr_cell, ref_run.dwr_cell) and np.array_equal(run.dwr_steps, ref_run.dwr_steps)


def test_failed_setups_leave_nothing_behind():
    # the error grid's context, its stream included, goes with a setup that fails in the mesh's checks: a
    # stream left behind takes half a megabyte of device memory
    import torch
    w = inputs.test_case(seed=1)
    g = error_grid(w)
    g.fine.material[0] = 99
    g.fine._soa = None
    with GeoflowContext(w.mat, TimeProps()) as c:
        c.upload_mesh(w.mesh)
        free = []
        for k in range(102):
            with pytest.raises(_ffi.DAError):
                Indicator(c, g)
            free.append(torch.cuda.mem_get_info()[0])
        assert free[1] - free[-1] < 8 << 20
