"""The one-launch solve of a small model and the launch-per-step solve that larger ones take: the same operations in the same
order, so the same bits, iterations and refreshes, whatever the model's size (one to sixteen CTAs, one, two and four
threads per row, long rows, rows without blocks) and however small or large its loads.

alpha and beta are the nearest FP32 numbers to the quotients of the exact sums on one side and of FP64 sums on the other: a
quotient within about 2^-52 of the middle between two FP32 numbers would differ, some 2^-27 of them.  The cases here take
fewer than 2^15 iterations in all, so that one of them differs by that has a probability below 2^-11; the inputs are fixed, so
a difference is an error in the order."""
import ctypes as C

import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


def _fail(after):
    f = L.lib().amr_test_fail_alloc
    f.argtypes, f.restype = [C.c_int64], None
    f(after)


def _model(cell, n, extra=0):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 1.0]]
    mesh = A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n))))
    E = 1e3 * np.exp(np.random.default_rng(11).normal(0.0, 0.3, len(mesh.shape)))
    if extra:
        mesh.coords = np.vstack([mesh.coords, np.full((extra, 3), 9.0)])
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1e3, nu=0.3))], E=E)
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(ux=1e-3)),
                                  ("y==1", A.SurfaceBC(ty=-1.0))])
    model.dev.assemble_K()
    return model, model.get_bc_vals(setup)


def _launches(model, U, F, opts):
    before = model.dev.launch_count()
    U, F, st = model.dev.solve(U, F, opts)
    return U, F, st, model.dev.launch_count() - before


def _both(model, U0, F0, opts):
    """The solve without memory for the one-launch form's arrays, and with it."""
    model.dev.solve(np.zeros_like(U0), np.zeros_like(F0), L.default_solve_opts(method=L.SOLVER_FP64))  # the work arrays
    for after in range(32):
        _fail(after)
        try:
            steps = _launches(model, U0, F0, opts)
        except A.AmrError:
            continue
        finally:
            _fail(-1)
        return steps, _launches(model, U0, F0, opts)
    raise AssertionError("no allocation of the one-launch form was met")


ONE = [(A.HEX8, (1, 1, 1)), (A.HEX8, (7, 4, 3)), (A.HEX8, (24, 5, 2)), (A.HEX8, (20, 7, 6)), (A.TET4, (9, 6, 5)),
       (A.TET10, (4, 3, 3)), (A.HEX20, (4, 2, 2)), (A.QUAD4, (40, 33)), (A.QUAD8, (3, 3)), (A.QUAD8, (61, 7)),
       (A.QUAD8, (33, 31)), (A.TRI6, (14, 9))]


def _same(steps, one):
    assert steps[2].iterations == one[2].iterations and steps[2].refinements == one[2].refinements
    assert np.array_equal(steps[0], one[0]) and np.array_equal(steps[1], one[1])
    assert steps[2].rel_residual == one[2].rel_residual
    assert steps[3] >= 3 * steps[2].iterations > 0 and one[3] < 20


@pytest.mark.parametrize("cell,n", ONE)
def test_same_bits_and_the_form_that_ran(cell, n):
    model, (U0, F0) = _model(cell, n)
    _same(*_both(model, U0, F0, L.default_solve_opts(rtol=1e-9)))


@pytest.mark.parametrize("scale", [2.0 ** -37, 2.0 ** -33, 2.0 ** -28, 2.0 ** 30])
@pytest.mark.parametrize("cell,n", [(A.HEX8, (7, 4, 3)), (A.QUAD8, (33, 31))])
def test_same_bits_at_any_load(cell, n, scale):
    """Down to loads whose r.z is near the least normal FP32 number, where the halves of a sum of FP32 pairs no longer are."""
    model, (U0, F0) = _model(cell, n)
    _same(*_both(model, U0 * scale, F0 * scale, L.default_solve_opts(rtol=1e-6)))


def test_same_bits_with_nodes_that_no_element_uses():
    model, (U0, F0) = _model(A.HEX8, (9, 4, 4), extra=70)
    _same(*_both(model, U0, F0, L.default_solve_opts(rtol=1e-9, refine_every=2)))


@pytest.mark.parametrize("cell,fits,beyond", [(A.HEX8, (20, 7, 6), (24, 9, 9)), (A.QUAD8, (50, 50), (54, 54))])
def test_the_size_that_fits_takes_one_launch(cell, fits, beyond):
    for n, one in ((fits, True), (beyond, False)):
        model, (U0, F0) = _model(cell, n)
        _, _, st, launches = _launches(model, U0, F0, L.default_solve_opts(rtol=1e-6))
        assert launches < 20 if one else launches >= 3 * st.iterations
