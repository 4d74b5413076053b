"""The inverse that the dense coarsest level of the multigrid takes, against one in extended precision, for matrices whose
rows mix magnitudes: rotations beside translations, stiff materials beside soft ones.

A = S B S with S diagonal is inverted by an elimination in FP64 as B is: the error of S X S is at most about
n 2^-52 cond(B) of its largest entry, whatever S.  An elimination by tiles with the tiles' explicit inverses, or products
formed from slices relative to a row's largest entry, hold that only if the factors of a product are of one magnitude and
do not grow with a tile's condition number."""
import ctypes as C

import numpy as np
import pytest

import amaru_gpu as A
from amaru_gpu import _lib as L

pytestmark = pytest.mark.gpu


def _inverse(K):
    f = L.lib().amr_test_dense_inverse
    f.argtypes = [C.c_int32, C.c_void_p, C.c_void_p]
    K = np.ascontiguousarray(K, np.float64)
    X = np.zeros_like(K)
    assert f(len(K), L.ptr(K), L.ptr(X)) == 0
    return X


def _exact(K):
    """Elimination in extended precision (64 bits on x86, 113 on Arm)."""
    n = len(K)
    W = np.concatenate([K.astype(np.longdouble), np.eye(n, dtype=np.longdouble)], axis=1)
    for p in range(n):
        W[p] /= W[p, p]
        f = W[:, p].copy()
        f[p] = 0
        W -= np.outer(f, W[p])
    return W[:, n:]


def _check(K):
    s = 1 / np.sqrt(np.diag(K))
    B = K * s[:, None] * s[None, :]
    cond = np.linalg.cond(B)
    X, Xe = _inverse(K), _exact(K)
    scale = (1 / s)[:, None] * (1 / s)[None, :]
    err = np.abs((X - Xe) * scale).max() / np.abs(Xe * scale).max()
    assert err <= len(K) * 2.0 ** -52 * cond, (err, cond)
    return float(err), float(cond)


def _spd(rng, n, cond):
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    return (Q * np.logspace(0, np.log10(cond), n)) @ Q.T


@pytest.mark.parametrize("n", [1, 20, 32, 33, 64, 95, 130, 201])
@pytest.mark.parametrize("spread", [0, 4, 10, 20, 30])
def test_rows_of_mixed_magnitudes(n, spread):
    rng = np.random.default_rng(100 * n + spread)
    B = _spd(rng, n, 1e3)
    S = 2.0 ** rng.uniform(-spread, spread, n)
    _check((B + B.T) / 2 * S[:, None] * S[None, :])


@pytest.mark.parametrize("n,cond", [(33, 1e6), (33, 1e10), (70, 1e8), (201, 1e10)])
def test_ill_conditioned_tiles(n, cond):
    B = _spd(np.random.default_rng(n), n, cond)
    _check((B + B.T) / 2)


@pytest.mark.parametrize("contrast", [1.0, 1e4, 1e6, 1e8])
@pytest.mark.parametrize("cell,n", [(A.HEX8, (4, 3, 2)), (A.QUAD8, (6, 4))])
def test_two_interleaved_materials(cell, n, contrast):
    three = len(n) == 3
    mesh = A.Mesh(A.Block([[0, 0, 0], [1.0, 0.5, 0.5]] if three else [[0, 0], [1.0, 0.5]], cellshape=cell,
                          **dict(zip(("nx", "ny", "nz"), n))))
    E = np.where(np.arange(len(mesh.shape)) % 2 == 0, 1.0, contrast)
    model = A.FEModel(mesh, [("all", A.LinearElastic(E=1.0, nu=0.3))], E=E)
    fix = dict(ux=0, uy=0, uz=0) if three else dict(ux=0, uy=0)
    model.configure_dofs([("x==0", A.SurfaceBC(**fix))])
    K = model.mount_K().toarray()[:model.nu, :model.nu]
    _check((K + K.T) / 2)
