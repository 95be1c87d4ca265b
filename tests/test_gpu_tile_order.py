"""Adjoint sweeps whose tiles are taken in another order than plain: results do not depend on it."""
import numpy as np
import pytest

from discrete_adjoint_b200 import (Ensemble, GeoflowContext, MatProps, Member, TimeProps, _ffi, adjoint_run, inputs)

pytestmark = pytest.mark.gpu

TILE = 256
PLAIN = 296 * TILE  # cells up to which the tiles stay in plain order on 148 SMs


def box_of(m):
    wet = m.h0 > 1.0
    return m.x[wet].min(), m.x[wet].max() + 100.0, m.y[wet].min(), m.y[wet].max()


def test_ordered_ensemble_equals_single_runs():
    # members alike in their tiles, so that their flows fall on the same blocks in plain order; enough
    # steps for a second order inside the sweep
    mbs = []
    for seed in (1, 2, 3, 4, 5, 6):
        m = inputs.test_case(seed=seed, nx0=60, ny0=48).mesh
        mbs.append(Member(m, MatProps(intfrict_deg=30.0 + seed, bedfrict_deg=[20.0, 16.0]), box_of(m)))
    assert sum(mb.mesh.n for mb in mbs) > PLAIN
    with Ensemble(mbs) as ens:
        runs = [ens.adjoint(40, 4)[0] for _ in range(2)]  # the second sweep starts in the first one's last order
        for k, mb in enumerate(mbs):
            with GeoflowContext(mb.mat, TimeProps()) as c:
                c.upload_mesh(mb.mesh)
                c.set_state(mb.mesh.h0, mb.mesh.hu0, mb.mesh.hv0)
                g = adjoint_run(c, mb.box, 40, 4, mb.mesh.dh0_dpile[0])
            for e in (runs[0][k], runs[1][k]):
                assert e.J == runs[0][k].J and e.dJ_dintfrict == runs[0][k].dJ_dintfrict
                for x, y in [(e.J, g.J), (e.dJ_dintfrict, g.dJ_dintfrict), (e.dJ_dpile[0], g.dJ_dpile[0])] + \
                        list(zip(e.dJ_dbedfrict, g.dJ_dbedfrict)):
                    assert abs(x - y) <= 1e-12 * max(abs(y), 1e-30), (k, x, y)


@pytest.mark.parametrize("staging", [1, 2, 3])
def test_ordered_fp32_adjoint_equals_plain(staging):
    # against the unstaged phases, which keep plain order; gathers by tiles and by quarter tiles
    w = inputs.test_case(seed=2, nx0=160, ny0=120)
    m = w.mesh
    assert m.n > PLAIN
    out = []
    for st in (0, staging):
        with GeoflowContext(w.mat, TimeProps(), precision=_ffi.DA_PREC_FP32_SPLIT, tile_staging=st) as c:
            c.upload_mesh(m)
            c.set_state(m.h0, m.hu0, m.hv0)
            out.append([adjoint_run(c, box_of(m), 40, 4, m.dh0_dpile, want_lambda0=True) for _ in range(2)])
    for a, b in zip(*out):
        assert np.array_equal(a.lambda0, b.lambda0)
        assert a.J == b.J and a.dJ_dintfrict == b.dJ_dintfrict
        assert np.array_equal(a.dJ_dbedfrict, b.dJ_dbedfrict) and np.array_equal(a.dJ_dpile, b.dJ_dpile)
