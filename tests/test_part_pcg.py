"""Parts of a batch whose matrices do not fit a cluster's shared memory: the solve that streams them (a cluster of CTAs per
part of 2 048 nodes or more, a CTA per smaller one), alone and beside parts that do fit, on the same launch of a batch.

Every part is solved to its relative residual and compared with the same model alone under the all-FP64 solver, to
1e-5 of the solution: two solutions to 1e-9 of the residual differ by at most cond(K), here below 1e4 each way."""
import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


def _part(cell, n, E, device):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 1.0]]
    mesh = A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n))))
    ctx = [] if three else [A.MechContext(stressmodel="planestrain")]
    return A.FEModel(mesh, [("all", A.LinearElastic(E=E, nu=0.3))], *ctx, device=device)


def _bcs(three, t=1.0):
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    return [("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(tx=t))]


MIXES = [  # (cell, sizes): beyond the shared memory first
    (A.QUAD8, [(64, 64)]),                                   # one that streams, nothing beside it
    (A.QUAD8, [(70, 70), (6, 5), (20, 20), (40, 40)]),        # with resident groups of several cluster sizes
    (A.HEX20, [(12, 8, 8), (10, 6, 6), (5, 4, 4), (2, 2, 2), (9, 5, 5)]),  # (10, 6, 6): 1 953 nodes, a CTA
    (A.HEX8, [(33, 12, 12), (3, 3, 3), (14, 10, 10)]),
]


@pytest.mark.parametrize("cell,sizes", MIXES)
def test_parts_that_stream_beside_parts_that_fit(cell, sizes):
    three = len(sizes[0]) == 3
    E = [1e3 * (1 + 0.3 * i) for i in range(len(sizes))]
    ba = A.BatchAnalysis([_part(cell, n, e, False) for n, e in zip(sizes, E)])
    U, F = ba.configure([_bcs(three)] * len(sizes))
    J = ba.joined
    J.dev.assemble_K()
    o = L.default_solve_opts(rtol=1e-9, max_iters=20000)
    U1, F1, st = J.dev.solve(U, F, o)
    U2, F2, _ = J.dev.solve(U, F, o)
    assert st.rel_residual <= 1e-9 and np.array_equal(U1, U2) and np.array_equal(F1, F2)
    for k, (n, e) in enumerate(zip(sizes, E)):
        m = _part(cell, n, e, True)
        setup = m.configure_dofs(_bcs(three))
        U0, F0 = m.get_bc_vals(setup)
        m.dev.assemble_K()
        Ud, Fd, _ = m.dev.solve(U0, F0, L.default_solve_opts(method=L.SOLVER_FP64, rtol=1e-9, max_iters=20000))
        want = np.zeros((len(m.mesh.coords), 3 if three else 2))
        want[m.dof_node, m.dof_comp] = Ud
        assert np.abs(ba.split(U1)[k] - want).max() <= 1e-5 * np.abs(want).max()
        alone = A.BatchAnalysis([_part(cell, n, e, False)])
        Ua, Fa = alone.configure([_bcs(three)])
        alone.joined.dev.assemble_K()
        Ua, _, _ = alone.joined.dev.solve(Ua, Fa, o)
        assert np.array_equal(alone.split(Ua)[0], ba.split(U1)[k])


def test_elastoplastic_stage_of_streaming_and_resident_parts():
    sizes = [(66, 64), (8, 6), (30, 25)]
    def parts(device):
        out = []
        for n in sizes:
            mesh = A.Mesh(A.Block([[0, 0], [2.0, 1.0]], nx=n[0], ny=n[1], cellshape=A.QUAD8))
            out.append(A.FEModel(mesh, [("all", A.VonMises(E=200e3, nu=0.3, fy=0.9, H=1e3))],
                                 A.MechContext(stressmodel="planestrain"), device=device))
        return out
    ba = A.BatchAnalysis(parts(False))
    ba.addstage(_bcs(False), nincs=2)
    assert all(ok for ok, _ in ba.solve(tol=1e-6))
    for k, m in enumerate(parts(True)):
        ana = A.MechAnalysis(m)
        ana.addstage(_bcs(False), nincs=2)
        assert ana.solve(tol=1e-6)[0]
        assert ba.part_stats[0][k].iterations == ana.stats[0].iterations
        assert np.abs(ba.models[k].U - m.U).max() <= 1e-5 * np.abs(m.U).max()
        assert m.state()[:, 12].max() > 0


@pytest.mark.parametrize("cell,n", [(A.QUAD8, (64, 64)), (A.HEX20, (12, 8, 8))])
def test_limits_of_the_streaming_solve(cell, n):
    three = len(n) == 3
    ba = A.BatchAnalysis([_part(cell, n, 1e3, False)])
    U, F = ba.configure([_bcs(three)])
    ba.joined.dev.assemble_K()
    with pytest.raises(A.AmrError):
        ba.joined.dev.solve(U, F, L.default_solve_opts(rtol=1e-9, max_iters=5))
    z, _, st = ba.joined.dev.solve(np.zeros_like(U), np.zeros_like(F), L.default_solve_opts(rtol=1e-9))
    assert st.iterations == 0 and not z.any()
