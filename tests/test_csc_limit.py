"""K as CSC on both sides of the number of entries up to which the host makes its columns: pattern and values bitwise the
oracle's, in the analysis' numbering and in any other."""
import numpy as np
import pytest

import oracle as O
import amaru_gpu as A

pytestmark = pytest.mark.gpu

CASES = [(A.HEX8, (1, 1, 1), "d3"), (A.HEX8, (4, 3, 3), "d3"), (A.HEX8, (4, 4, 3), "d3"), (A.HEX8, (7, 5, 4), "d3"),
         (A.TET10, (2, 2, 1), "d3"), (A.TET10, (3, 3, 2), "d3"), (A.HEX20, (2, 1, 1), "d3"), (A.HEX20, (3, 2, 2), "d3"),
         (A.QUAD8, (7, 7), "planestrain"), (A.QUAD8, (9, 9), "axisymmetric"), (A.QUAD4, (14, 13), "planestress"),
         (A.QUAD4, (20, 20), "planestrain"), (A.TRI6, (6, 5), "planestress")]


@pytest.mark.parametrize("cell,n,stressmodel", CASES)
def test_both_sides_of_the_limit(cell, n, stressmodel):
    dim = len(n)
    box = [[0.5, 0, 0], [1.5, 0.6, 0.7]] if dim == 3 else [[0.5, 0], [1.5, 0.6]]
    div = dict(zip(("nx", "ny", "nz"), n))
    mo, mg = O.Mesh(O.Block(box, cellshape=cell, **div)), A.Mesh(A.Block(box, cellshape=cell, **div))
    assert np.allclose(mo.coords, mg.coords, rtol=0, atol=1e-15)
    mg.coords = np.ascontiguousarray(mo.coords)  # entries near eps() follow the coordinates' last bits
    om = O.FEModel(mo, [("all", O.LinearElastic(E=3e4, nu=0.27))], stressmodel=stressmodel)
    gm = A.FEModel(mg, [("all", A.LinearElastic(E=3e4, nu=0.27))], A.MechContext(stressmodel=stressmodel))
    fix = dict(ux=0, uy=0, uz=0) if dim == 3 else dict(ux=0, uy=0)
    dofs, _, _ = O.configure_dofs(om, [("x<=0.52", O.NodeBC(**fix))])
    gm.configure_dofs([("x<=0.52", A.NodeBC(**fix))])
    Ko, Kg = O.mount_K(om, len(dofs)).tocsc(), gm.mount_K()
    assert (Kg.indptr == Ko.indptr).all() and (Kg.indices == Ko.indices).all() and np.array_equal(Kg.data, Ko.data)
    p = np.random.default_rng(2).permutation(len(dofs))
    gm.dev.set_dofs(np.where(gm.eq_id >= 0, p[gm.eq_id], -1), len(dofs), gm.nu)
    Kp = gm.mount_K()
    assert all(np.all(np.diff(Kp.indices[a:b]) > 0) for a, b in zip(Kp.indptr[:-1], Kp.indptr[1:]))
    back = Kp[p][:, p].tocsc()
    back.sort_indices()
    assert (back.indices == Ko.indices).all() and np.array_equal(back.data, Ko.data)
