"""The multigrid's dense coarsest level, inverted by a blocked sweep in tiles of 32 rows: coarse levels of one partial
tile, of a few rows past a tile edge, of several tiles, and a batch's block-diagonal level.

A wrong inverse leaves the coarse error uncorrected: the Krylov count then grows to block-Jacobi's (several hundred on
these blocks) or the solve fails.  The solution is compared with the all-FP64 block-Jacobi solve to the tolerance
both are solved to: 1e-10 on the residual, amplified by at most cond(K) ~ 1e3 on these blocks."""
import numpy as np
import pytest

import amaru_gpu as A

pytestmark = pytest.mark.gpu


def _model(cell, n):
    box = [[0, 0, 0], [1.0, 0.5, 0.5]] if len(n) == 3 else [[0, 0], [1.0, 0.5]]
    div = dict(zip(("nx", "ny", "nz"), n))
    mesh = A.Mesh(A.Block(box, cellshape=cell, **div))
    E = 1e3 * np.exp(np.random.default_rng(3).normal(0.0, 0.2, len(mesh.shape)))
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.3))], E=E)
    fix = dict(ux=0, uy=0, uz=0) if len(n) == 3 else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==1", A.SurfaceBC(ty=-1.0))])
    return model, model.get_bc_vals(setup)


@pytest.mark.parametrize("cell,n", [(A.HEX8, (2, 1, 1)), (A.HEX8, (6, 3, 3)), (A.HEX8, (13, 5, 4)), (A.TET10, (5, 3, 2)),
                                    (A.HEX20, (9, 4, 4)), (A.HEX8, (31, 15, 14)), (A.QUAD8, (7, 5)), (A.QUAD4, (64, 33))])
def test_dense_level_corrects_the_coarse_error(cell, n):
    model, (U0, F0) = _model(cell, n)
    model.dev.assemble_K()
    sols = {}
    for name, method in (("amg", A._lib.SOLVER_AMG), ("amg_fp64", A._lib.SOLVER_AMG_FP64), ("fp64", A._lib.SOLVER_FP64)):
        U, _, st = model.dev.solve(U0, F0, A._lib.default_solve_opts(method=method, rtol=1e-10))
        sols[name] = (U, st.iterations)
    ref = np.abs(sols["fp64"][0]).max()
    for name in ("amg", "amg_fp64"):
        assert np.abs(sols[name][0] - sols["fp64"][0]).max() <= 1e-7 * ref
        assert sols[name][1] <= 100


def test_dense_level_of_a_batch_is_block_diagonal():
    """Parts of different sizes joined: each part's solution is the one it has alone."""
    rng = np.random.default_rng(5)
    bcs = [("x==0", A.SurfaceBC(ux=0, uy=0)), ("x==2", A.SurfaceBC(tx=1.0))]

    def models(device):
        return [A.FEModel(A.Mesh(A.Block([[0, 0], [2.0, 1.0]], nx=int(k), ny=int(k), cellshape=A.QUAD8)),
                          [("all", A.LinearElastic(E=float(e), nu=0.3))], A.MechContext(stressmodel="planestrain"),
                          device=device) for k, e in zip((1, 3, 9, 17, 4, 12), 1e3 * np.exp(rng.normal(size=6)))]
    state = rng.bit_generator.state
    ba = A.BatchAnalysis(models(False))
    ba.addstage(bcs)
    assert all(ok for ok, _ in ba.solve(solver="amg", linear_rtol=1e-10))
    rng.bit_generator.state = state
    for part, m in zip(ba.models, models(True)):
        ana = A.MechAnalysis(m)
        ana.addstage(bcs)
        assert ana.solve(solver="amg", linear_rtol=1e-10)[0]
        np.testing.assert_allclose(part.U, m.U, rtol=0, atol=1e-7 * np.abs(m.U).max())


@pytest.mark.parametrize("scale", [1e-6, 1e6, 1e22])
def test_dense_level_at_any_scale(scale):
    """The inverse's digits and reciprocals follow the matrix's exponents: with all moduli scaled (upwards far; far below
    1 element entries fall under the assembly's eps and are dropped), the same iterations
    (one more or less, where the residual passes the tolerance) and the scaled solution (both solved to 1e-10, as
    above)."""
    out = []
    for f in (1.0, scale):
        model, (U0, F0) = _model(A.HEX8, (13, 5, 4))
        model.dev.set_youngs(f * model.mat_params[:, 0])
        model.dev.assemble_K()
        U, _, st = model.dev.solve(U0, F0 * f, A._lib.default_solve_opts(method=A._lib.SOLVER_AMG, rtol=1e-10))
        out.append((U, st.iterations))
    assert abs(out[0][1] - out[1][1]) <= 1
    assert np.abs(out[1][0] - out[0][0]).max() <= 1e-7 * np.abs(out[0][0]).max()
