"""Parameters set on a live ensemble context: the gradients stay the members' own."""
import ctypes as C

import numpy as np
import pytest

from discrete_adjoint_b200 import Ensemble, MatProps, Member, _ffi, inputs

pytestmark = pytest.mark.gpu


# the partial sums' buffer is allocated by the first adjoint; the second writes more outputs per member
@pytest.mark.parametrize("n_members,n_materials", [(17, 4), (24, _ffi.DA_MAX_MATERIALS)])
def test_more_materials_after_the_first_adjoint(n_members, n_materials):
    mbs = []
    for k in range(n_members):
        m = inputs.test_case(seed=1 + k % 5, nx0=12, ny0=10).mesh
        m.material[:] = 0
        m._soa = None
        mbs.append(Member(m, MatProps(intfrict_deg=30.0, bedfrict_deg=[15.0 + 0.2 * k]),
                          (m.x.min(), m.x.max(), m.y.min(), m.y.max())))
    with Ensemble(mbs) as ens:
        a, _ = ens.adjoint(8, 2)
        p = _ffi.da_params()
        C.memmove(C.byref(p), C.byref(ens.params), C.sizeof(p))
        p.n_materials = n_materials
        for q in range(n_materials):
            p.bedfrict[q] = ens.params.bedfrict[0]
        ens._check(ens.lib.da_set_params(ens.ctx, C.byref(p)), "da_set_params")
        b, _ = ens.adjoint(8, 2)
    same(a, b)


# fewer materials than a member has: its gradients are still all of its own
def test_fewer_materials_after_the_upload():
    mbs = []
    for k, n_mat in enumerate((3, 1, 6)):
        m = inputs.test_case(seed=1 + k, nx0=12, ny0=10).mesh
        m.material = np.ascontiguousarray(np.random.default_rng(k).integers(0, n_mat, m.n), dtype=np.int32)
        m._soa = None
        mbs.append(Member(m, MatProps(intfrict_deg=30.0, bedfrict_deg=[15.0 + q for q in range(n_mat)]),
                          (m.x.min(), m.x.max(), m.y.min(), m.y.max())))
    with Ensemble(mbs) as ens:
        a, _ = ens.adjoint(8, 2)
        p = _ffi.da_params()
        C.memmove(C.byref(p), C.byref(ens.params), C.sizeof(p))
        p.n_materials = 1
        ens._check(ens.lib.da_set_params(ens.ctx, C.byref(p)), "da_set_params")
        b, _ = ens.adjoint(8, 2)
    same(a, b)


def same(a, b):
    for x, y in zip(a, b):
        assert x.J == y.J and x.dJ_dintfrict == y.dJ_dintfrict
        assert np.array_equal(x.dJ_dbedfrict, y.dJ_dbedfrict) and np.array_equal(x.dJ_dpile, y.dJ_dpile)
