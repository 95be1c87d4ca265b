"""The staged FP64 phases where their branch-free quotients (csrc/quot.cuh) hand over to the division
operator: states, meshes and materials on both sides of the declared ranges must give the same
bits as the global-memory phases, which divide with the operator throughout."""
import numpy as np
import pytest

from discrete_adjoint_b200 import GeoflowContext, TimeProps, inputs

pytestmark = pytest.mark.gpu


def _run(w, h, hu, hv, staging, steps, **mesh):
    with GeoflowContext(w.mat, TimeProps(), tile_staging=staging) as c:
        c.upload_mesh(w.mesh)
        c.set_state(h, hu, hv)
        s = c.run(steps)
        return (*c.get_state(), s.dt, s.time)


# momenta at the edges of the range [2^-150, 2^100] (and denormal), on some cells of some tiles
@pytest.mark.parametrize("tiny", [0.0, 2.0 ** -149, 2.0 ** -150, 2.0 ** -151, 2.0 ** -400, 5e-324])
def test_small_momenta_take_either_path(tiny):
    w = inputs.test_case(seed=3)
    m = w.mesh
    rng = np.random.default_rng(7)
    h = m.h0 + np.where(rng.random(m.n) < 0.2, 0.5, 0.0)
    hu = np.where(rng.random(m.n) < 0.1, tiny, 0.3) * h
    hv = np.where(rng.random(m.n) < 0.1, -tiny, -0.1) * h
    a, b = _run(w, h, hu, hv, 1, 12), _run(w, h, hu, hv, 0, 12)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


# cell sizes at the edges of the mesh's range [2^-40, 2^40]: the whole geometry scaled
@pytest.mark.parametrize("scale", [2.0 ** -43, 2.0 ** -60, 1.0, 2.0 ** 33, 2.0 ** 60])
def test_mesh_scales_take_either_path(scale):
    w = inputs.test_case(seed=4)
    m = w.mesh
    for k in ("x", "y", "dx", "dy"):
        setattr(m, k, np.ascontiguousarray(getattr(m, k) * scale))
    m._soa = None
    a, b = _run(w, m.h0, m.hu0, m.hv0, 1, 10), _run(w, m.h0, m.hu0, m.hv0, 0, 10)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))


# depths exactly at the wet threshold: dry for the coefficients, wet for the fluxes
def test_depths_at_the_wet_threshold():
    w = inputs.test_case(seed=5)
    m = w.mesh
    rng = np.random.default_rng(1)
    h = np.where(rng.random(m.n) < 0.3, 1.0e-4, m.h0)
    hu, hv = 0.2 * h, -0.3 * h
    a, b = _run(w, h, hu, hv, 1, 15), _run(w, h, hu, hv, 0, 15)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
