"""Block QR and RQ of blocks that are not finite and of columns far below the others.

A reflector whose vector holds NaN or an infinity has no finite norm: R's diagonal entry there is not finite
(LAPACK's dgeqrf and dgerqf give NaN), and a finite part in front of it stays what it is."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


def _factors(lib, a, name):
    m, n = a.shape
    t = cs.BlockSparse((m, n), (1, -1), [np.zeros(m, np.int32), np.zeros(n, np.int32)],
                       dtype=cs.CT_DOUBLE_COMPLEX if np.iscomplexobj(a) else cs.CT_DOUBLE_REAL)
    t.blocks[t.allowed[0]] = a
    ca, x, y = c_bst(t), cs.BlockSparseTensor(), cs.BlockSparseTensor()
    assert getattr(lib, "ctgpu_block_sparse_tensor_" + name)(C.byref(ca), 0, C.byref(x), C.byref(y)) == 0
    out = cs.read_bst(x).to_dense(), cs.read_bst(y).to_dense()
    for z in (ca, x, y):
        cs.free_bst(z)
    return out


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("m,n", [(5, 1), (1, 5), (7, 4), (40, 33), (190, 150)])
def test_not_finite(gpu, m, n, value, cplx):
    rng = np.random.default_rng(m + n)
    a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
    c = min(m, n) // 2
    a[m // 2, c] = value
    q, r = _factors(gpu, a, "qr")
    # columns in front of the bad one are untouched by it; it and those behind it have no finite R entry
    ref = np.linalg.qr(np.where(np.isfinite(a), a, 0))[1]
    np.testing.assert_allclose(np.abs(r[:c, :c]), np.abs(ref[:c, :c]), rtol=0, atol=8 * max(m, n) * 2.3e-16 * np.abs(ref).max())
    assert not np.any(np.isfinite(np.diag(r)[c:])), np.diag(r)
    assert m == 1 or not np.all(np.isfinite(q))          # one row: nothing to eliminate, Q is 1
    r2, q2 = _factors(gpu, a.conj().T[::-1, ::-1].copy(), "rq")
    assert not np.any(np.isfinite(np.diag(r2[::-1, ::-1])[c:])), np.diag(r2)
    assert m == 1 or not np.all(np.isfinite(q2))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("small", [1e-140, 1e-146, 1e-150])
def test_small_columns(gpu, small, cplx):
    """Columns far below the others, down to squared norms of 1e-300, still get their own reflector: every
    column of R has that column's norm."""
    rng = np.random.default_rng(1)
    a = rng.standard_normal((20, 6)) + (1j * rng.standard_normal((20, 6)) if cplx else 0)
    a[:, 2] = 0                                # so that the small columns meet no larger ones in their rows
    a[:10, 3:] = 0
    a[10:, :2] = 0
    a[:, 3:] *= small
    q, r = _factors(gpu, a, "qr")
    np.testing.assert_allclose(np.linalg.norm(r[:, 3:] / small, axis=0), np.linalg.norm(a[:, 3:] / small, axis=0), rtol=1e-13)
    np.testing.assert_allclose(q.conj().T @ q, np.eye(6), rtol=0, atol=8 * 20 * 2.3e-16)
    np.testing.assert_allclose((q @ (r / small))[:, 3:], a[:, 3:] / small, rtol=0, atol=1e-13)
