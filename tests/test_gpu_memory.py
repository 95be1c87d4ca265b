"""Device memory of a context: a forward run keeps nothing that only an adjoint needs."""
import pytest

from discrete_adjoint_b200 import GeoflowContext, MatProps, TimeProps, adjoint_run, inputs
from discrete_adjoint_b200.mesh import Mesh, MeshSpec

pytestmark = pytest.mark.gpu


def test_bytes_per_cell():
    import torch
    # arrays of 8 n bytes fill whole 2 MB blocks, so the difference of the free memory is what they take
    nx, ny = 1024, 512
    n = nx * ny
    dem = inputs.analytic_dem(lambda X, Y: 1000.0 - 0.2 * X, 0.0, 0.0, 10.0 * nx, 10.0 * ny, 40.0)
    spec = MeshSpec(xmin=0.0, ymin=0.0, dx0=10.0, dy0=10.0, nx0=nx, ny0=ny, max_level=0, random_frac=0.0, seed=1)
    m = Mesh.build(spec, dem, [])
    assert m.n == n
    m.h0[:200] = 1.0
    warm = inputs.test_case(seed=1)
    with GeoflowContext(warm.mat, TimeProps()) as c:  # the kernels' own memory
        c.upload_mesh(warm.mesh)
        c.set_state(warm.mesh.h0, warm.mesh.hu0, warm.mesh.hv0)
        adjoint_run(c, (0.0, 1.0, 0.0, 1.0), 4, 1)
    free0 = torch.cuda.mem_get_info()[0]
    with GeoflowContext(MatProps(), TimeProps()) as c:
        c.upload_mesh(m)
        c.set_state(m.h0, m.hu0, m.hv0)
        c.run(2)
        used = free0 - torch.cuda.mem_get_info()[0]
        # mesh: 8 neighbours of 4 B and of 2 B, flag, material, x, y, dx, dy, 3 + 2 + 2 geometry doubles; two
        # states of 3 doubles; k act/pass, 5 kept doubles and the friction signs
        cell = 32 + 16 + 2 + 8 * (4 + 7) + 8 * 6 + 8 + 8 * 5 + 1
        # halos (about 68 cells of 4 B a 256-cell tile), segment and tile arrays: below 4 B a cell; and
        # 2 MB for what is rounded up
        assert used <= (cell + 4) * n + (6 << 20), used / n
        adjoint_run(c, (0.0, 1.0, 0.0, 1.0), 4, 1)
        used = free0 - torch.cuda.mem_get_info()[0]
        # branch bytes, two lambdas, A, B, two running sensitivities, the base and one checkpoint
        cell += 1 + 8 * 6 + 8 * 7 + 8 * 2 + 2 * 24
        assert used <= (cell + 8) * n + (12 << 20), used / n
