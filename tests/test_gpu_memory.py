"""Device memory of a context: a forward run keeps nothing that only an adjoint needs."""
import numpy as np
import pytest

from discrete_adjoint_b200 import Ensemble, GeoflowContext, MatProps, Member, TimeProps, adjoint_run, inputs
from discrete_adjoint_b200.mesh import Mesh, MeshSpec

pytestmark = pytest.mark.gpu


# mesh: 8 neighbours of 4 B and of 2 B, flag, material, x, y, dx, dy, 3 + 2 + 2 geometry doubles; two
# states of 3 doubles; k act/pass, 5 kept doubles and the friction signs
FORWARD = 32 + 16 + 2 + 8 * (4 + 7) + 8 * 6 + 8 + 8 * 5 + 1


def uniform(nx, ny):
    # arrays of 8 n bytes fill whole 2 MB blocks, so the difference of the free memory is what they take
    dem = inputs.analytic_dem(lambda X, Y: 1000.0 - 0.2 * X, 0.0, 0.0, 10.0 * nx, 10.0 * ny, 40.0)
    spec = MeshSpec(xmin=0.0, ymin=0.0, dx0=10.0, dy0=10.0, nx0=nx, ny0=ny, max_level=0, random_frac=0.0, seed=1)
    m = Mesh.build(spec, dem, [])
    assert m.n == nx * ny
    m.h0[:200] = 1.0
    return m


def test_bytes_per_cell():
    import torch
    m = uniform(1024, 512)
    n = m.n
    warm = inputs.test_case(seed=1)
    with GeoflowContext(warm.mat, TimeProps()) as c:  # the kernels' own memory
        c.upload_mesh(warm.mesh)
        c.set_state(warm.mesh.h0, warm.mesh.hu0, warm.mesh.hv0)
        c.run(2)
        adjoint_run(c, (0.0, 1.0, 0.0, 1.0), 4, 1)
    free0 = torch.cuda.mem_get_info()[0]
    with GeoflowContext(MatProps(), TimeProps()) as c:
        c.upload_mesh(m)
        c.set_state(m.h0, m.hu0, m.hv0)
        c.run(2)
        used = free0 - torch.cuda.mem_get_info()[0]
        cell = FORWARD
        # halos (about 68 cells of 4 B a 256-cell tile), segment and tile arrays: below 4 B a cell; and
        # 2 MB for what is rounded up
        assert used <= (cell + 4) * n + (6 << 20), used / n
        adjoint_run(c, (0.0, 1.0, 0.0, 1.0), 4, 1)
        used = free0 - torch.cuda.mem_get_info()[0]
        # branch bytes, two lambdas, A, B, two running sensitivities, the base and one checkpoint
        cell += 1 + 8 * 6 + 8 * 7 + 8 * 2 + 2 * 24
        assert used <= (cell + 8) * n + (12 << 20), used / n


@pytest.mark.parametrize("moving", [False, True])
def test_ensemble_bytes_per_cell_and_restart(moving):
    # members that start at rest keep their initial depths on the device for a restart, others their momenta too
    import torch
    m = uniform(512, 256)
    small = uniform(32, 16)
    for k in (m, small):
        k.hu0[:] = -0.0 if moving else 0.0  # a zero whose sign a restart has to keep
        k.hv0[:] = 0.5 * k.h0 if moving else 0.0
    with Ensemble([Member(small, MatProps(), (0.0, 1.0, 0.0, 1.0), pile=-1)]) as e:
        e.forward(2)
        e.restart()
    free0 = torch.cuda.mem_get_info()[0]
    with Ensemble([Member(m, MatProps(), (0.0, 1.0, 0.0, 1.0), pile=-1) for _ in range(4)]) as e:
        n = 4 * m.n
        used = free0 - torch.cuda.mem_get_info()[0]
        assert used <= (FORWARD + 4 + (24 if moving else 8)) * n + (6 << 20), used / n
        for _ in range(2):
            e.forward(3)
            e.restart()
            for k in (0, 3):
                for a, b in zip(e.get_state(k), (m.h0, m.hu0, m.hv0)):
                    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
