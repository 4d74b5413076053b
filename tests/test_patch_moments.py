"""Patch recovery from the elements' moments: every width of lanes per element (up to 4, 8, 27 points), fields that
fill half a warp and more, field sets of several materials, patches on the pseudo-inverse path beside them, and meshes
far from the origin.  Against the oracle's least-squares fit in global coordinates.

Tolerance: both solve for 7 terms (6 in 2-D) from sums of m <= 216 points.  The oracle's own conditioning rules: its
regression columns reach L^2 at distance L from the origin of a patch of size h, so its fit carries
eps * (L/h)^2 * m ~ 2e-16 * 30^2 * 216 = 4e-11 of the field's scale; 1e-9 leaves 25 times that."""
import numpy as np
import pytest

import amaru_gpu as A
import oracle as O

pytestmark = pytest.mark.gpu

CASES = [(A.HEX8, (4, 3, 3), 8, "elastic"), (A.HEX8, (3, 3, 2), 27, "vonmises"), (A.HEX20, (3, 2, 3), 27, "mixed"),
         (A.HEX20, (2, 3, 2), 8, "elastic"), (A.TET4, (3, 3, 3), 1, "elastic"), (A.TET10, (2, 2, 2), 4, "mixed"),
         (A.QUAD4, (5, 4), 4, "vonmises"), (A.QUAD8, (4, 5), 9, "mixed"), (A.QUAD9, (3, 3), 16, "elastic"),
         (A.TRI6, (4, 3), 3, "mixed"), (A.HEX8, (4, 1, 2), 8, "elastic")]


@pytest.mark.parametrize("shift", [0.0, 20.0])
@pytest.mark.parametrize("cell,n,nips,mat", CASES)
def test_recovery_from_moments(cell, n, nips, mat, shift):
    dim = len(n)
    box = [[shift] * dim, [shift + 1.5, shift + 1.0, shift + 0.8][:1] + [shift + 1.0, shift + 0.8][:dim - 1]]
    div = dict(zip(("nx", "ny", "nz"), n))
    ctx = "d3" if dim == 3 else "planestrain"
    mo, mg = O.Mesh(O.Block(box, cellshape=cell, **div)), A.Mesh(A.Block(box, cellshape=cell, **div))
    rng = np.random.default_rng(4)
    mo.coords[:, :dim] += rng.uniform(-0.02, 0.02, mo.coords[:, :dim].shape)
    mg.coords = np.ascontiguousarray(mo.coords)
    x0 = shift + 0.75

    def mats(M):
        e, v = M.LinearElastic(E=1e4, nu=0.25), M.VonMises(E=1e4, nu=0.25, fy=8.0, H=100.0)
        return [("all", v if mat == "vonmises" else e)] + ([("x<=%g" % x0, v)] if mat == "mixed" else [])
    om = O.FEModel(mo, mats(O), stressmodel=ctx, nips=nips)
    gm = A.FEModel(mg, mats(A), A.MechContext(stressmodel=ctx), nips=nips)
    st = gm.state()
    st[:, :13] = rng.normal(size=(len(st), 13))
    gm.set_state(st)
    om.state[:] = gm.state()
    Vo, no = O.nodal_patch_recovery(om)
    Vg, ng = gm.nodal_patch_recovery()
    assert ng == no
    for j, k in enumerate(no):
        assert np.abs(Vg[:, j] - Vo[:, j]).max() <= 1e-9 * np.abs(Vo[:, j]).max(), k
