"""IP states on both sides of the number of points up to which the host transposes them: rows in the caller's order of
elements of two kinds, got as they were set, and the points' own stresses after an update."""
import numpy as np
import pytest

import amaru_gpu as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [1, 15, 16, 60])
def test_both_sides_of_the_limit(ny):
    shapes = [A.TET4, A.HEX8, A.TET4, A.HEX8]
    mesh = A.Mesh(*[A.Block([[k, 0, 0], [k + 1.0, 1.0, 1.0]], nx=1, ny=ny, nz=3, cellshape=s) for k, s in enumerate(shapes)])
    E = 1e3 * (1.0 + np.arange(len(mesh.shape)) % 7)
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.25))], E=E)
    model.configure_dofs([("x==0", A.NodeBC(ux=0))])
    rng = np.random.default_rng(ny)
    st = model.state()
    nips = model.dev.elem_nips()
    assert st.shape == (nips.sum(), 16) and len(set(nips)) > 1
    new = rng.normal(size=st.shape)
    model.set_state(new)
    got = model.state()
    assert np.array_equal(got[:, :14], new[:, :14]) and (got[:, 14:] == 0).all()
    model.set_state(np.zeros_like(st))
    model.update_state(np.where(model.dof_comp == 0, 1e-3 * mesh.coords[model.dof_node, 0], 0.0))
    st = model.state()
    elem = np.repeat(np.arange(len(E)), nips)
    np.testing.assert_allclose(st[:, 0], E[elem] * 1e-3 * 0.75 / (1.25 * 0.5), rtol=1e-11)


def test_the_sizes_lie_on_both_sides():
    rows = []
    for ny in (15, 16):
        mesh = A.Mesh(*[A.Block([[k, 0, 0], [k + 1.0, 1.0, 1.0]], nx=1, ny=ny, nz=3, cellshape=s)
                        for k, s in enumerate([A.TET4, A.HEX8, A.TET4, A.HEX8])])
        model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.25))])
        rows.append(int(model.dev.elem_nips().sum()))
    assert rows[0] <= 3000 < rows[1]
