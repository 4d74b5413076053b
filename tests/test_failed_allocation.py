"""Solves whose device allocations fail, one after the other: the call raises or does without, and the next solve on the
same handle, with memory there, gives what a handle gives that never met a failure.  The failure is made on the host: the
library's allocator reports one as it would when the device is full."""
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


def _model(cell, n):
    three = len(n) == 3
    box = [[0, 0, 0], [2.0, 1.0, 1.0]] if three else [[0, 0], [2.0, 1.0]]
    model = A.FEModel(A.Mesh(A.Block(box, cellshape=cell, **dict(zip(("nx", "ny", "nz"), n)))),
                      [("all", A.LinearElastic(E=1e3, nu=0.3))])
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    setup = model.configure_dofs([("x==0", A.SurfaceBC(**fix)), ("x==2", A.SurfaceBC(tx=1.0))])
    model.dev.assemble_K()
    return model, model.get_bc_vals(setup)


def _each_failure(cell, n, method):
    """The solve with each of its allocations failing in turn; returns their number."""
    model, (U0, F0) = _model(cell, n)
    opts = L.default_solve_opts(method=method, rtol=1e-9)
    U, F, _ = model.dev.solve(U0, F0, opts)
    failures = 0
    for after in range(400):
        model, (U0, F0) = _model(cell, n)
        before = model.dev.alloc_count()
        _fail(after)
        try:
            got = model.dev.solve(U0, F0, opts)
        except A.AmrError as e:
            assert "device allocation" in str(e)
            got = None
        finally:
            _fail(-1)
        asked = model.dev.alloc_count() - before
        for u, f in ([got[:2]] if got else []) + [model.dev.solve(U0, F0, opts)[:2] for _ in range(2)]:
            assert np.array_equal(u, U) and np.array_equal(f, F)
        if got is not None and asked <= after:
            return failures
        failures += 1
    raise AssertionError("the solve went on allocating")


@pytest.mark.parametrize("cell,n,method,least", [
    (A.HEX8, (40, 18, 18), L.SOLVER_MIXED, 9), (A.HEX8, (5, 3, 2), L.SOLVER_FP64, 13),
    (A.QUAD8, (9, 7), L.SOLVER_FP64, 13), (A.HEX8, (6, 4, 3), L.SOLVER_AMG, 9), (A.HEX8, (6, 4, 3), L.SOLVER_AMG_FP64, 13)])
def test_work_arrays_without_memory(cell, n, method, least):
    assert _each_failure(cell, n, method) >= least


@pytest.mark.parametrize("cell,n", [(A.HEX8, (5, 3, 2)), (A.QUAD8, (9, 7))])
def test_one_launch_solve_without_memory(cell, n):
    """Without its own arrays the solve takes a launch per step, and gives the same."""
    assert _each_failure(cell, n, L.SOLVER_MIXED) >= 13
