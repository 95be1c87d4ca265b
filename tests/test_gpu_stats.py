"""Flow statistics (da_compute_stats) at the sizes where its partition can go wrong: fewer cells
than blocks, ragged ranges, more than one cell per thread, a dry map, both precisions, no and several
planes.  Against the sums in numpy; FP64 sums of n terms in any order agree within n 2^-53 of the
sum of magnitudes, and the statistics are quotients of such sums (1e-12 for n < 1e4 cells)."""
import numpy as np
import pytest

from discrete_adjoint_b200 import GeoflowContext, Mesh, MeshSpec, TimeProps, _ffi, inputs

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, level):
    dem = inputs.inclined_plane(400.0, 400.0, 10.0, 25.0, 300.0)
    spec = MeshSpec(xmin=0.0, ymin=0.0, dx0=400.0 / nx, dy0=400.0 / ny, nx0=nx, ny0=ny, max_level=level, uniform=True)
    return Mesh.build(spec, dem, [])


@pytest.mark.parametrize("nx,ny,level", [(1, 1, 0), (3, 5, 1), (7, 9, 1), (8, 8, 1), (17, 15, 0), (16, 16, 2), (33, 31, 1)])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("wet", [0.0, 0.4, 1.0])
def test_statistics_of_any_size(nx, ny, level, fp32, wet):
    m = _mesh(nx, ny, level)
    rng = np.random.default_rng(nx * 100 + ny)
    h = np.where(rng.random(m.n) < wet, rng.uniform(0.01, 3.0, m.n), 0.0)
    hu, hv = h * rng.uniform(0.5, 2.0, m.n), h * rng.uniform(0.5, 2.0, m.n)
    if fp32:
        h, hu, hv = (a.astype(np.float32).astype(np.float64) for a in (h, hu, hv))
    dx, dy = (a.astype(np.float32).astype(np.float64) if fp32 else a for a in (m.dx, m.dy))
    planes = [(0.0, 400.0, 201.0, 199.0), (150.0, 150.5, 0.0, 400.0), (10.0, 390.0, 20.0, 380.0)][:nx % 4]
    dis = np.zeros(len(planes))
    w = inputs.test_case(seed=1)
    with GeoflowContext(w.mat, TimeProps(), precision=_ffi.DA_PREC_FP32_SPLIT if fp32 else _ffi.DA_PREC_FP64) as c:
        c.upload_mesh(m)
        c.set_state(h, hu, hv)
        first = c.stats(0.5, (0.5, 200.0, 200.0), 0.0, planes, dis if planes else None)
        again = c.stats(0.5, (0.5, 200.0, 200.0), 0.0, planes, dis.copy() if planes else None)
    assert all(again[k] == v or (np.isnan(v) and np.isnan(again[k])) for k, v in first.items())
    on = h > 1.0e-4
    if not on.any():
        assert first["area"] == 0.0 and first["statvolume"] == 0.0 and first["hmax"] == 0.0
        assert np.all(dis == 0.0)
        return
    A = (dx * dy)[on]
    V = h[on] * A
    x, y = m.x[on], m.y[on]
    near = lambda a, b: abs(a - b) <= 1e-12 * max(abs(b), 1e-300)  # noqa: E731
    assert near(first["area"], A.sum()) and near(first["statvolume"], V.sum())
    assert near(first["xcen"], (x * V).sum() / V.sum()) and near(first["ycen"], (y * V).sum() / V.sum())
    assert near(first["vxmean"], (hu[on] * A).sum() / V.sum()) and near(first["vymean"], (hv[on] * A).sum() / V.sum())
    assert near(first["vmean"], (np.hypot(hu, hv)[on] * A).sum() / V.sum())
    assert first["hmax"] == h.max()
    deep = h >= 1.0e-3
    assert (first["xmin"], first["xmax"]) == (m.x[deep].min(), m.x[deep].max())
    assert (first["ymin"], first["ymax"]) == (m.y[deep].min(), m.y[deep].max())
    d2 = np.where(on, (m.x - 200.0) ** 2 + (m.y - 200.0) ** 2, np.inf)
    assert first["testpoint_reach"] == int(np.any(h[d2 == d2.min()] >= 0.5))
    if planes and wet == 1.0 and m.n > 1:
        assert np.all(dis != 0.0)
