"""The multigrid's Galerkin product on levels on both sides of the number of coarse blocks from which it takes four lanes per
block: a wrong operator costs the coarse correction, so iterations grow to block-Jacobi's several hundred.  The solution is
compared with block-Jacobi's, both to 1e-10 of the residual, amplified by at most cond(K), below 1e5 here."""
import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,n", [(A.HEX8, (80, 40, 40)), (A.HEX8, (60, 30, 30)), (A.QUAD8, (180, 180)), (A.QUAD8, (140, 140))])
def test_both_sides_of_the_rule(cell, n):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 2.0]]
    model = A.FEModel(A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n)))),
                      [("all", A.LinearElastic(E=1e3, nu=0.3))])
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(tx=1.0, ty=0.1))])
    model.dev.assemble_K()
    U0, F0 = model.get_bc_vals(setup)
    ref, _, _ = model.dev.solve(U0, F0, L.default_solve_opts(method=L.SOLVER_FP64, rtol=1e-10, max_iters=100000))
    for method in (L.SOLVER_AMG, L.SOLVER_AMG_FP64):
        U, _, st = model.dev.solve(U0, F0, L.default_solve_opts(method=method, rtol=1e-10))
        assert st.iterations <= 100
        assert np.abs(U - ref).max() <= 2e-5 * np.abs(ref).max()
