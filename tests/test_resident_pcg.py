"""The mixed solver's one-launch form for small models (a cluster of CTAs, the matrix in shared memory): one CTA and
several, one, two and four threads per row, slices around the edges of a warp of rows, both dimensions, long rows,
and models just past the size that fits, which take a launch per step.

Two solves of the same system to a relative residual of 1e-10 differ by at most cond(K) (here up to about 1e4) times
2e-10 of the solution, so 1e-5 bounds the difference; the residual itself is checked on K64 by the solver."""
import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


def _model(cell, n, extra=0):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 1.0]]
    mesh = A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n))))
    E = 1e3 * np.exp(np.random.default_rng(7).normal(0.0, 0.3, len(mesh.shape)))
    if extra:
        mesh.coords = np.vstack([mesh.coords, np.full((extra, 3), 9.0)])
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.3))], E=E)
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(ux=1e-3)),
                                  ("y==1", A.SurfaceBC(ty=-1.0))])
    model.dev.assemble_K()
    return model, model.get_bc_vals(setup)


SIZES = [(A.HEX8, (1, 1, 1)), (A.HEX8, (3, 3, 1)), (A.HEX8, (7, 4, 3)), (A.HEX8, (15, 7, 3)), (A.HEX8, (33, 9, 6)),
         (A.HEX8, (36, 9, 9)), (A.HEX8, (40, 16, 16)), (A.TET4, (6, 5, 4)), (A.HEX20, (4, 3, 3)), (A.TET10, (4, 3, 3)),
         (A.QUAD4, (5, 5)), (A.QUAD4, (63, 33)), (A.QUAD8, (3, 3)), (A.QUAD8, (21, 21)), (A.QUAD8, (60, 60)),
         (A.QUAD8, (75, 75)), (A.TRI3, (40, 40)), (A.QUAD9, (12, 9))]


@pytest.mark.parametrize("cell,n", SIZES)
def test_solution_and_reactions(cell, n):
    model, (U0, F0) = _model(cell, n)
    Um, Fm, sm = model.dev.solve(U0, F0, L.default_solve_opts(method=L.SOLVER_MIXED, rtol=1e-10))
    Ud, Fd, sd = model.dev.solve(U0, F0, L.default_solve_opts(method=L.SOLVER_FP64, rtol=1e-10))
    assert sm.rel_residual <= 1e-10
    assert np.abs(Um - Ud).max() <= 1e-5 * np.abs(Ud).max()
    assert np.abs(Fm - Fd).max() <= 1e-5 * np.abs(Fd).max()
    U2, F2, s2 = model.dev.solve(U0, F0, L.default_solve_opts(method=L.SOLVER_MIXED, rtol=1e-10))
    assert np.array_equal(Um, U2) and np.array_equal(Fm, F2) and s2.iterations == sm.iterations


@pytest.mark.parametrize("extra", [1, 40])
def test_unused_nodes_change_nothing(extra):
    a, (U0, F0) = _model(A.HEX8, (9, 4, 4))
    b, (U1, F1) = _model(A.HEX8, (9, 4, 4), extra)
    o = L.default_solve_opts(rtol=1e-9)
    assert np.array_equal(a.dev.solve(U0, F0, o)[0], b.dev.solve(U1, F1, o)[0])


def test_limits_and_empty_loads():
    model, (U0, F0) = _model(A.QUAD8, (20, 9))
    with pytest.raises(A.AmrError):
        model.dev.solve(U0, F0, L.default_solve_opts(rtol=1e-10, max_iters=5))
    z, _, st = model.dev.solve(np.zeros_like(U0), np.zeros_like(F0), L.default_solve_opts(rtol=1e-10))
    assert st.iterations == 0 and not z.any()
    st = model.dev.solve(U0, F0, L.default_solve_opts(rtol=1e-10, refine_every=1))[2]  # a refresh every 16 iterations
    assert st.rel_residual <= 1e-10 and st.refinements >= st.iterations // 16
