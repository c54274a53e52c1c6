"""Block QR and RQ over real and complex entries at the sizes where the kernel changes (one column, odd numbers
of columns, more column pairs than warps, blocks beyond shared memory), for rank-deficient blocks and for
scales near the ends of the number range, against numpy.

Householder QR is backward stable: |A - Q R| and the defect of Q's orthonormality are at most a small multiple
of max(m, n) eps (relative to the largest entry's scale); the multiple here is 8."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


def _matrix(rng, m, n, cplx, kind):
    a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
    if kind == "rank":                         # every third row and column zero, the rest of rank three
        a = a[:, :3] @ a[:3, :] if min(m, n) >= 3 else a
        a[::3] = 0
        a[:, 1::3] = 0
    return a * {"tiny": 2.0**-700, "huge": 2.0**900}.get(kind, 1.0)


@pytest.mark.parametrize("kind", ["random", "rank", "tiny", "huge"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 5), (5, 1), (2, 2), (7, 3), (3, 7), (32, 33), (64, 21), (21, 64), (130, 150), (190, 150)])
def test_qr_and_rq(gpu, m, n, cplx, kind):
    rng = np.random.default_rng(m * 100 + n)
    t = cs.BlockSparse((m, n), (1, -1), [np.zeros(m, np.int32), np.zeros(n, np.int32)],
                       dtype=cs.CT_DOUBLE_COMPLEX if cplx else cs.CT_DOUBLE_REAL)
    a = _matrix(rng, m, n, cplx, kind)
    t.blocks[t.allowed[0]] = a
    ca = c_bst(t)
    k, tol = min(m, n), 8 * max(m, n) * np.finfo(np.float64).eps
    scale = max(np.abs(a).max(), 1e-300)
    q, r = cs.BlockSparseTensor(), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_qr(C.byref(ca), 0, C.byref(q), C.byref(r)) == 0
    Q, R = cs.read_bst(q).to_dense(), cs.read_bst(r).to_dense()
    assert np.abs(Q @ (R / scale) - a / scale).max() <= tol * np.sqrt(k)
    np.testing.assert_allclose(Q.conj().T @ Q, np.eye(k), rtol=0, atol=tol)
    assert np.all(np.tril(R, -1) == 0) and np.all(np.diag(R).imag == 0)
    r2, q2 = cs.BlockSparseTensor(), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_rq(C.byref(ca), 0, C.byref(r2), C.byref(q2)) == 0
    Q2, R2 = cs.read_bst(q2).to_dense(), cs.read_bst(r2).to_dense()
    assert np.abs((R2 / scale) @ Q2 - a / scale).max() <= tol * np.sqrt(k)
    np.testing.assert_allclose(Q2 @ Q2.conj().T, np.eye(k), rtol=0, atol=tol)
    if kind == "random":
        # LAPACK's signs: R of QR directly, R of RQ from the QR of the reversed conjugate transpose
        ref = np.linalg.qr(a)[1]
        np.testing.assert_array_equal(np.sign(np.diag(R).real), np.sign(np.diag(ref).real))
        ref = np.linalg.qr(a.conj().T[::-1, ::-1])[1]
        np.testing.assert_array_equal(np.sign(np.diag(R2[::-1, ::-1]).real)[:k], np.sign(np.diag(ref).real))
    for x in (q, r, r2, q2, ca):
        cs.free_bst(x)
