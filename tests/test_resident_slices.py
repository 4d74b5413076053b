"""How a model is cut for the one-launch solve: every CTA of the cluster has rows.

A sum over the cluster ends, in a CTA, when the sums of all rows have arrived there.  A CTA without rows sends nothing, so
the others never wait for it and may write the next sum into its shared memory while it reads the last one; the layout
must not have such a CTA.  Slices are whole groups of 64 rows, cover the rows once and stay within the shared memory."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import amaru_gpu as A
from amaru_gpu import _lib as L

CELLS = [(A.HEX8, 3), (A.TET4, 3), (A.TET10, 3), (A.HEX20, 3), (A.QUAD4, 2), (A.QUAD8, 2), (A.TRI3, 2), (A.TRI6, 2)]


def _pattern(mesh):
    rows, cols = [], []
    for q in range(len(mesh.shape)):
        e = np.asarray(mesh.conn[mesh.conn_ptr[q]:mesh.conn_ptr[q + 1]])
        rows.append(np.repeat(e, len(e)))
        cols.append(np.tile(e, len(e)))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    m = sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(len(mesh.coords),) * 2)
    m.sum_duplicates()
    m.sort_indices()
    return m.indptr.astype(np.int64), m.indices.astype(np.int32)


def _shape(ndim, rp, cj, prefer, exact, most=16):
    bounds, nbytes = np.zeros(most + 1, np.int64), C.c_int64()
    f = L.lib().amr_test_resident_shape
    f.argtypes = [C.c_int32, C.c_int64, C.c_void_p, C.c_void_p, C.c_int64, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p]
    ctas = f(ndim, len(rp) - 1, L.ptr(rp), L.ptr(cj), prefer, exact, most, L.ptr(bounds), C.addressof(nbytes))
    return ctas, bounds[:ctas + 1], nbytes.value


@pytest.mark.parametrize("cell,ndim", CELLS)
def test_every_cta_has_rows(cell, ndim):
    sizes = [(k, a, b) for k in (1, 2, 5, 13, 24, 29) for a in (1, 3, 5) for b in (1, 2, 5)] if ndim == 3 else \
        [(k, a) for k in (1, 4, 9, 25, 39) for a in (1, 6, 17, 38)]
    cut = 0
    for n in sizes:
        mesh = A.Mesh(A.Block([[0.0] * ndim, [1.0] * ndim], cellshape=cell, **dict(zip(("nx", "ny", "nz"), n))))
        rp, cj = _pattern(mesh)
        for prefer in (24 << 10, 48 << 10, 100 << 10, 206 << 10):
            ctas, bounds, nbytes = _shape(ndim, rp, cj, prefer, 1)
            if ctas == 0:
                continue
            cut += ctas > 1
            assert bounds[0] == 0 and bounds[-1] == len(mesh.coords) and nbytes <= 206 << 10
            assert (np.diff(bounds) > 0).all() and (np.diff(bounds) <= 1024).all()
            assert (bounds[:-1] % 64 == 0).all()
    assert cut > 0


def test_rows_of_very_different_length():
    """A few nodes with very long rows: equal shares of the blocks would leave CTAs without a group of rows."""
    n, hubs = 500, 4
    m = sp.lil_matrix((n, n))
    m.setdiag(1)
    m[:hubs, :] = 1
    m[:, :hubs] = 1
    m = m.tocsr()
    m.sort_indices()
    ctas, bounds, nbytes = _shape(2, m.indptr.astype(np.int64), m.indices.astype(np.int32), 24 << 10, 1)
    assert ctas > 1 and (np.diff(bounds) > 0).all()
