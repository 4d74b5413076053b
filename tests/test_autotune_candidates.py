"""What the tuner times for the internal-force kernel: the elements per CTA that the kernel takes untuned among them, all
within the kernel's shared memory; and tuning a 3-D model before its first assembly changes no result."""
import ctypes as C

import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L


def _candidates(dim, nen, nip, cached):
    f = L.lib().amr_test_internal_candidates
    f.argtypes = [C.c_int32] * 4 + [C.c_void_p, C.c_void_p]
    epb, smem = np.zeros(8, np.int32), np.zeros(8, np.int64)
    n = f(dim, nen, nip, cached, L.ptr(epb), L.ptr(smem))
    return epb[:n].tolist(), smem[:n].tolist()


@pytest.mark.parametrize("nen,nip", [(4, 1), (4, 4), (10, 4), (8, 8), (8, 1), (20, 8), (20, 27)])
def test_cached_kernel(nen, nip):
    epb, smem = _candidates(3, nen, nip, 1)
    assert epb[0] == max(1, 64 // nip) and len(set(epb)) == len(epb)
    assert smem == [8 * e * (3 * nen + 7 * nip) for e in epb] and max(smem) <= 48 * 1024
    assert {1, 2, 4, 8, 16} <= set(epb)


@pytest.mark.parametrize("dim,nen,nip", [(2, 3, 1), (2, 8, 9), (2, 4, 4), (3, 20, 27), (3, 8, 8)])
def test_kernel_without_the_cache(dim, nen, nip):
    epb, smem = _candidates(dim, nen, nip, 0)
    assert epb[0] == (4 if nip >= 16 else 16) and max(smem) <= 200 * 1024


@pytest.mark.gpu
@pytest.mark.parametrize("cells", [(A.HEX8, A.HEX8, A.TET4), (A.HEX20, A.TET10, A.HEX20)])
def test_tuning_a_fresh_model_changes_no_result(cells):
    def parts():
        out = []
        for i, cell in enumerate(cells):
            mesh = A.Mesh(A.Block([[0, 0, 0], [2.0, 1.0, 1.0]], nx=3 + i, ny=2, nz=2, cellshape=cell))
            out.append(A.FEModel(mesh, [("all", A.LinearElastic(E=200e3, nu=0.3))], device=False))
        return out
    runs = []
    for tune in (False, True):
        ba = A.BatchAnalysis(parts())
        ba.addstage([("x==0", A.SurfaceBC(ux=0, uy=0, uz=0)), ("x==2", A.SurfaceBC(tx=1.0))], nincs=2)
        if tune:
            ba.configure(ba.stages[0].bcs)
            t = ba.joined.dev.autotune()  # before any assembly
            assert min(t.internal_epb[:t.ngroups]) >= 1
        assert all(ok for ok, _ in ba.solve(tol=1e-6))
        runs.append(ba)
    for a, b in zip(runs[0].models, runs[1].models):
        assert np.array_equal(a.U, b.U) and np.array_equal(a.F, b.F)
