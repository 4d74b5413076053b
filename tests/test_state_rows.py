"""IP states to and from the caller's order: rows follow the caller's elements where the device sorts them by shape, and
more rows than one chunk of 32 MB takes.  Values are copied, so they are equal; the planted strain is uniform, so each
element's stress is its own modulus times a constant, to rounding of the shape functions' sums (20 terms: 1e-12)."""
import numpy as np
import pytest

import amaru_gpu as A

pytestmark = pytest.mark.gpu


def test_rows_follow_the_callers_elements():
    shapes = [A.TET4, A.HEX8, A.TET4, A.TET4, A.HEX8, A.HEX8]
    mesh = A.Mesh(*[A.Block([[k, 0, 0], [k + 1.0, 1.0, 1.0]], nx=2, ny=1, nz=2, cellshape=s) for k, s in enumerate(shapes)])
    E = 1e3 * (1.0 + np.arange(len(mesh.shape)))
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.25))], E=E)
    model.configure_dofs([("x==0", A.NodeBC(ux=0))])
    dU = np.where(model.dof_comp == 0, 1e-3 * mesh.coords[model.dof_node, 0], 0.0)
    model.update_state(dU)
    st = model.state()
    elem = np.repeat(np.arange(len(E)), model.dev.elem_nips())
    assert len(set(model.dev.elem_nips())) > 1
    np.testing.assert_allclose(st[:, 6], 1e-3, rtol=1e-11)
    np.testing.assert_allclose(st[:, 0], E[elem] * 1e-3 * 0.75 / (1.25 * 0.5), rtol=1e-11)
    assert (st[:, 14:] == 0).all()
    new = np.random.default_rng(1).normal(size=st.shape)
    model.set_state(new)
    got = model.state()
    assert np.array_equal(got[:, :14], new[:, :14]) and (got[:, 14:] == 0).all()


@pytest.mark.parametrize("n", [(1, 1, 1), (22, 22, 23)])
def test_rows_of_one_point_count_and_of_several_chunks(n):
    mesh = A.Mesh(A.Block([[0, 0, 0], [1, 1, 1]], nx=n[0], ny=n[1], nz=n[2], cellshape=A.HEX8))
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.25))], nips=27)
    rows = 27 * len(mesh.shape)
    assert n == (1, 1, 1) or rows * 128 > 1 << 25
    new = np.random.default_rng(2).normal(size=(rows, 16))
    model.set_state(new)
    assert np.array_equal(model.state()[:, :14], new[:, :14])
