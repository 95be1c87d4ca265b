"""The ranges that the branch-free FP64 quotients (csrc/quot.cuh) ask of materials, gravity, states, time steps
and an ensemble's members, inside and outside, in forward steps and in the reverse step's gather: the same
bits as the global-memory phases, which divide with the operator throughout."""
import math

import numpy as np
import pytest

from discrete_adjoint_b200 import (Ensemble, GeoflowContext, MatProps, Member, TimeProps, _ffi, adjoint_run, inputs,
                                   set_dt_replay)
from discrete_adjoint_b200.solver import PI_REF

pytestmark = pytest.mark.gpu

TINY = 1.0e-4


def scaled(m, **factors):
    for k, f in factors.items():
        setattr(m, k, np.ascontiguousarray(getattr(m, k) * f))
    m._soa = None
    return m


def box_of(m):
    return m.x.min(), m.x.max(), m.y.min(), m.y.max()


def forward(mat, m, state, staging, steps):
    """State, dt, time and status of some steps (a wave speed above its bound raises but is computed)."""
    with GeoflowContext(mat, TimeProps(), tile_staging=staging) as c:
        c.upload_mesh(m)
        c.set_state(*state)
        code, s = 0, None
        try:
            s = c.run(steps)
        except _ffi.DAError as e:
            code = e.code
        return [*c.get_state(), np.array([s.dt, s.time] if s else [0.0, 0.0]), np.array([code])]


def backward(mat, m, state, staging, steps=10, snaps=3, dt=None):
    with GeoflowContext(mat, TimeProps(), tile_staging=staging) as c:
        c.upload_mesh(m)
        c.set_state(*state)
        if dt is not None:
            set_dt_replay(c, [dt] * (steps + 1), 0)
        g = adjoint_run(c, box_of(m), steps, snaps, m.dh0_dpile, want_lambda0=True)
        return [g.lambda0, np.array([g.J, g.dJ_dintfrict]), np.asarray(g.dJ_dbedfrict), np.asarray(g.dJ_dpile),
                *c.get_state()]


def same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(np.asarray(x).view(np.uint64), np.asarray(y).view(np.uint64))


def all_stagings(fn, *args, **kw):
    ref = fn(*args, 0, **kw)
    for staging in (1, 2, 3):
        same(fn(*args, staging, **kw), ref)
    return ref


def moving(m, scale=1.0, vx=0.3, vy=-0.1):
    h = m.h0 * scale
    return h, vx * h, vy * h


# k act/pass [2^-60, 2^60] by its factor epsilon: below, in, at the upper edge and above (depths that keep
# the wave speed in its bound)
@pytest.mark.parametrize("eps,depth", [(2.0 ** -64, 1.0), (2.0 ** -58, 1.0), (2.0 ** 58, 0.005), (2.0 ** 61, 0.002)])
def test_materials_by_their_factor(eps, depth):
    w = inputs.test_case(seed=3)
    mat = MatProps(w.mat.intfrict_deg, list(w.mat.bedfrict_deg), epsilon=eps)
    m = w.mesh
    s = moving(m, depth / m.h0.max() * 5)
    assert forward(mat, m, s, 1, 8)[4][0] == 0
    all_stagings(lambda st: forward(mat, m, s, st, 8))
    all_stagings(lambda st: backward(mat, m, s, st))


# friction angles with k = 0 (the flux's speeds are then the velocities), and with k above 2^60
@pytest.mark.parametrize("intfrict,bedfrict,depth", [
    (10.0, 60.0, 1.0), ((math.pi / 2 - 1.0e-9) * 180.0 / PI_REF, 20.0, 0.002)])
def test_materials_by_their_angles(intfrict, bedfrict, depth):
    w = inputs.test_case(seed=4)
    mat = MatProps(intfrict, [bedfrict] * len(w.mat.bedfrict_deg))
    m = w.mesh
    s = moving(m, depth / m.h0.max() * 5)
    all_stagings(lambda st: forward(mat, m, s, st, 8))
    all_stagings(lambda st: backward(mat, m, s, st))


# g_z [2^-40, 2^40], about 10 here
@pytest.mark.parametrize("scale", [2.0 ** -46, 2.0 ** -42, 2.0 ** 35, 2.0 ** 40])
def test_gravity(scale):
    w = inputs.test_case(seed=5)
    m = w.mesh
    m.gravity = np.ascontiguousarray(m.gravity.reshape(3, m.n) * np.array([[1.0], [1.0], [scale]]))
    m._soa = None
    s = moving(m)
    all_stagings(lambda st: forward(w.mat, m, s, st, 8))
    all_stagings(lambda st: backward(w.mat, m, s, st))


# states on both sides of 2^100, one step (the wave speed's bound is passed, the step is computed all the same)
@pytest.mark.parametrize("h,mom", [(1.0, 2.0 ** 99), (1.0, 2.0 ** 101), (2.0 ** 99, 1.0), (2.0 ** 101, 2.0 ** 40)])
def test_large_states(h, mom):
    w = inputs.test_case(seed=6)
    m = w.mesh
    pick = np.random.default_rng(3).random(m.n) < 0.05
    s = (np.where(pick, h, m.h0), np.where(pick, mom, 0.2 * m.h0), np.where(pick, -mom, 0.1 * m.h0))
    ref = all_stagings(lambda st: forward(w.mat, m, s, st, 1))
    assert ref[4][0] in (0, _ffi.DA_ERR_EIGEN)


# the reverse step: momenta next to 2^-150 and denormal, depths at the wet threshold
@pytest.mark.parametrize("tiny", [0.0, 2.0 ** -149, 2.0 ** -151, 5e-324])
def test_adjoint_with_small_momenta_and_threshold_depths(tiny):
    w = inputs.test_case(seed=3)
    m = w.mesh
    rng = np.random.default_rng(7)
    h = np.where(rng.random(m.n) < 0.2, TINY, m.h0)
    s = (h, np.where(rng.random(m.n) < 0.1, tiny, 0.3) * h, np.where(rng.random(m.n) < 0.1, -tiny, -0.1) * h)
    all_stagings(lambda st: backward(w.mat, m, s, st))


# cell sizes at the edges of [2^-40, 2^40] in the reverse step: the whole geometry scaled
@pytest.mark.parametrize("scale", [2.0 ** -43, 2.0 ** -60, 2.0 ** 33, 2.0 ** 60])
def test_adjoint_on_scaled_meshes(scale):
    w = inputs.test_case(seed=4)
    m = scaled(w.mesh, x=scale, y=scale, dx=scale, dy=scale)
    s = moving(m)
    all_stagings(lambda st: backward(w.mat, m, s, st))


# the gather divides dt by the cell sizes: replayed steps next to 2^-150
@pytest.mark.parametrize("dt", [2.0 ** -20, 2.0 ** -149, 2.0 ** -151, 2.0 ** -400])
def test_adjoint_with_small_time_steps(dt):
    w = inputs.test_case(seed=5)
    m = w.mesh
    s = moving(m)
    all_stagings(lambda st: backward(w.mat, m, s, st, dt=dt))


# one member's material outside the range takes all of them to the operator
@pytest.mark.parametrize("odd", [None, 1])
def test_ensemble_with_a_member_outside_the_range(odd):
    mbs = []
    for k, seed in enumerate((1, 2, 5)):
        m = inputs.test_case(seed=seed, nx0=14, ny0=12).mesh
        m.h0, m.hu0, m.hv0 = moving(m, 0.01 / m.h0.max())
        phi = (math.pi / 2 - 1.0e-9) * 180.0 / PI_REF if k == odd else 30.0 + k
        mbs.append(Member(m, MatProps(phi, [20.0, 16.0]), box_of(m)))
    with Ensemble(mbs) as ens:
        ens.forward(10)
        got = [ens.get_state(k) for k in range(3)]
        grads, _ = ens.adjoint(6, 2)
    for mb, u, e in zip(mbs, got, grads):
        with GeoflowContext(mb.mat, TimeProps(), tile_staging=0) as c:
            c.upload_mesh(mb.mesh)
            c.set_state(mb.mesh.h0, mb.mesh.hu0, mb.mesh.hv0)
            c.run(10)
            same(u, c.get_state())
            g = adjoint_run(c, mb.box, 6, 2, mb.mesh.dh0_dpile[0])
        # the members' sums run in another order
        for x, y in [(e.J, g.J), (e.dJ_dintfrict, g.dJ_dintfrict), (e.dJ_dpile[0], g.dJ_dpile[0])] + \
                list(zip(e.dJ_dbedfrict, g.dJ_dbedfrict)):
            assert abs(x - y) <= 1e-12 * max(abs(y), 1e-30), (x, y)


# the reduction of an ensemble's gradients with different numbers of materials per member
def test_ensemble_gradients_with_several_materials():
    mbs = []
    for k, (seed, n_mat) in enumerate([(1, 1), (2, 5), (3, 3), (4, 16)]):
        m = inputs.test_case(seed=seed, nx0=14, ny0=12).mesh
        m.material = np.ascontiguousarray(np.random.default_rng(k).integers(0, n_mat, m.n), dtype=np.int32)
        m._soa = None
        mbs.append(Member(m, MatProps(30.0 + k, [14.0 + 0.5 * q for q in range(n_mat)]), box_of(m)))
    with Ensemble(mbs) as ens:
        grads, _ = ens.adjoint(20, 4)
    for mb, e in zip(mbs, grads):
        with GeoflowContext(mb.mat, TimeProps()) as c:
            c.upload_mesh(mb.mesh)
            c.set_state(mb.mesh.h0, mb.mesh.hu0, mb.mesh.hv0)
            g = adjoint_run(c, mb.box, 20, 4, mb.mesh.dh0_dpile[0])
        assert len(e.dJ_dbedfrict) == len(g.dJ_dbedfrict) == len(mb.mat.bedfrict_deg)
        big = np.abs(g.dJ_dbedfrict).max()
        assert np.abs(np.subtract(e.dJ_dbedfrict, g.dJ_dbedfrict)).max() <= 1e-12 * big
        assert abs(e.dJ_dintfrict - g.dJ_dintfrict) <= 1e-12 * abs(g.dJ_dintfrict)
