"""K in the reference's order of operations and its export as CSC.

Element kernel: every quadrature the shapes take (points handled in chunks of 8: fewer, exactly, more), on distorted
meshes, where no entry of a Jacobian or of B is zero by chance; values and pattern bitwise equal to the oracle's.
Export: equation numbers in any order (rows are ranked in each column), and more entries than one chunk of the
read-back; the same matrix bitwise, permuted."""
import numpy as np
import pytest

import oracle as O
import amaru_gpu as A

pytestmark = pytest.mark.gpu


def _pair(cell, n, nips, stressmodel, mat):
    dim = len(n)
    box = [[0.5, 0, 0], [1.5, 0.6, 0.7]] if dim == 3 else [[0.5, 0], [1.5, 0.6]]
    div = dict(zip(("nx", "ny", "nz"), n))
    mo, mg = O.Mesh(O.Block(box, cellshape=cell, **div)), A.Mesh(A.Block(box, cellshape=cell, **div))
    shift = np.random.default_rng(7).uniform(-0.01, 0.01, mo.coords[:, :dim].shape)
    mo.coords[:, :dim] += shift
    mg.coords = np.ascontiguousarray(mo.coords)
    om = O.FEModel(mo, [("all", O.LinearElastic(**mat))], stressmodel=stressmodel, thickness=0.3, nips=nips)
    gm = A.FEModel(mg, [("all", A.LinearElastic(**mat))], A.MechContext(stressmodel=stressmodel), thickness=0.3, nips=nips)
    fix = dict(ux=0, uy=0, uz=0) if dim == 3 else dict(ux=0, uy=0)
    dofs, _, _ = O.configure_dofs(om, [("x<=0.52", O.NodeBC(**fix))])
    gm.configure_dofs([("x<=0.52", A.NodeBC(**fix))])
    assert (gm.eq_id == om.eq_id).all()
    return om, gm, len(dofs)


CASES = [(A.HEX8, (3, 2, 2), 8, "d3"), (A.HEX8, (2, 2, 1), 27, "d3"), (A.HEX20, (2, 1, 1), 8, "d3"),
         (A.HEX20, (2, 1, 2), 27, "d3"), (A.TET4, (2, 1, 1), 1, "d3"), (A.TET10, (2, 1, 1), 4, "d3"),
         (A.QUAD4, (3, 2), 4, "planestress"), (A.QUAD8, (2, 2), 4, "planestrain"), (A.QUAD8, (3, 2), 9, "axisymmetric"),
         (A.QUAD9, (2, 2), 16, "planestress"), (A.TRI3, (3, 2), 1, "axisymmetric"), (A.TRI6, (2, 2), 3, "planestrain")]


@pytest.mark.parametrize("cell,n,nips,stressmodel", CASES)
def test_reference_order_on_distorted_meshes(cell, n, nips, stressmodel):
    om, gm, nd = _pair(cell, n, nips, stressmodel, dict(E=3e4, nu=0.27))
    Ko, Kg = O.mount_K(om, nd).tocsc(), gm.mount_K()
    assert (Kg.indptr == Ko.indptr).all() and (Kg.indices == Ko.indices).all()
    assert np.array_equal(Kg.data, Ko.data)


@pytest.mark.parametrize("cell,n", [(A.HEX8, (3, 2, 2)), (A.QUAD8, (5, 3)), (A.HEX20, (17, 9, 9))])
def test_export_under_any_numbering(cell, n):
    box = [[0, 0, 0], [1.0, 0.6, 0.7]] if len(n) == 3 else [[0, 0], [1.0, 0.6]]
    mesh = A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n))))
    gm = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.3))], A.MechContext(
        stressmodel="d3" if len(n) == 3 else "planestrain"))
    gm.configure_dofs([("x==0", A.NodeBC(ux=0))])
    K = gm.mount_K()
    assert K.has_sorted_indices and abs(K @ np.ones(K.shape[0])).max() <= 1e-10 * abs(K.data).max()
    if cell == A.HEX20:
        assert K.nnz > 1 << 21  # more than one chunk
    nd = K.shape[0]
    p = np.random.default_rng(2).permutation(nd)
    eq = np.where(gm.eq_id >= 0, p[gm.eq_id], -1)
    gm.dev.set_dofs(eq, nd, gm.nu)
    Kp = gm.mount_K()
    assert all(np.all(np.diff(Kp.indices[a:b]) > 0) for a, b in zip(Kp.indptr[:200], Kp.indptr[1:201]))
    back = Kp[p][:, p].tocsc()
    back.sort_indices()
    assert (back.indptr == K.indptr).all() and (back.indices == K.indices).all() and np.array_equal(back.data, K.data)
