"""A wait inside the one-launch solve that runs out: one CTA of the cluster never sends its part of a sum, so no CTA's
wait for it can end.  Each gives up after the limit that the test sets, the whole cluster leaves the kernel together, every CTA
reports AMR_ETIMEOUT, and the handle solves as before."""
import ctypes as C

import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu
ETIMEOUT = -8


def _wait(model, exact, rank, limit_ms):
    f = L.lib().amr_test_resident_wait
    f.argtypes = [C.c_void_p, C.c_int32, C.c_int32, C.c_double, C.c_void_p, C.c_void_p]
    status, ctas = np.zeros(16, np.int32), C.c_int32(0)
    rc = f(model.dev.h, exact, rank, limit_ms, L.ptr(status), C.addressof(ctas))
    return rc, status[:ctas.value]


@pytest.mark.parametrize("exact", [1, 0])
@pytest.mark.parametrize("cell,n", [(A.HEX8, (24, 5, 2)), (A.HEX8, (3, 2, 2)), (A.QUAD8, (40, 20))])
def test_every_cta_reports_the_wait_that_gave_up(cell, n, exact):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 1.0]]
    model = A.FEModel(A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n)))),
                      [("all", A.LinearElastic(E=1e3, nu=0.3))])
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(tx=1.0))])
    model.dev.assemble_K()
    U0, F0 = model.get_bc_vals(setup)
    before = model.dev.solve(U0, F0, L.default_solve_opts(rtol=1e-9))
    rc, status = _wait(model, exact, 0, 20.0)
    assert rc == 0 and len(status) >= 1 and (status == ETIMEOUT).all()
    if len(status) > 1:
        rc, status = _wait(model, exact, len(status) - 1, 20.0)
        assert rc == 0 and (status == ETIMEOUT).all()
    after = model.dev.solve(U0, F0, L.default_solve_opts(rtol=1e-9))
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])


def test_refuses_a_rank_that_is_not_there():
    model = A.FEModel(A.Mesh(A.Block([[0, 0], [1.0, 1.0]], nx=2, ny=2, cellshape=A.QUAD4)),
                      [("all", A.LinearElastic(E=1e3, nu=0.3))])
    model.configure_dofs([("x==0", A.SurfaceBC(ux=0, uy=0))])
    model.dev.assemble_K()
    assert _wait(model, 1, 16, 20.0)[0] == -1
