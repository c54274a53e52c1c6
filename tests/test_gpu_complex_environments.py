"""Environment updates over complex128 tensors, whose bra is read conjugated in the products (no copy): narrow, wide and
square blocks, contractions that are split into shares, against numpy.

The bound is componentwise: three products in a row with k1, k2 and k3 terms, each off by at most 4 (k + 2) eps of its
magnitudes; numpy's own take half of that."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


def _tensor(rng, dims, dirs):
    t = cs.BlockSparse(dims, dirs, [np.zeros(n, np.int32) for n in dims], dtype=cs.CT_DOUBLE_COMPLEX)
    t.blocks[(0,) * len(dims)] = rng.standard_normal(dims) + 1j * rng.standard_normal(dims)
    return t


def _call(fn, *ts):
    c, out = [c_bst(t) for t in ts], cs.BlockSparseTensor()
    assert fn(*[C.byref(x) for x in c], C.byref(out)) == 0
    r = cs.read_bst(out).to_dense()
    for x in (*c, out):
        cs.free_bst(x)
    return r


@pytest.mark.parametrize("d0,d,d1,w0,w1", [
    (1, 1, 1, 1, 1), (3, 2, 130, 5, 4), (130, 3, 7, 1, 6), (65, 2, 67, 3, 3), (33, 4, 31, 6, 5), (900, 1, 16, 2, 1), (16, 1, 900, 1, 2),
])
def test_steps_with_a_conjugated_bra(gpu, d0, d, d1, w0, w1):
    rng = np.random.default_rng(d0 + d1)
    a = _tensor(rng, (d0, d, d1), (1, 1, -1))
    w = _tensor(rng, (w0, d, d, w1), (1, 1, -1, -1))
    A, W = a.to_dense(), w.to_dense()
    eps = np.finfo(np.float64).eps
    # l[1, alpha, wl, alpha'], r[beta, wr, beta', 1]; the bra has the primed indices
    left = "xpwq,qtv,wtsz,psu->xuzv"
    env = _tensor(rng, (1, d0, w0, d0), (1, -1, -1, 1))
    L = env.to_dense()
    ref = np.einsum(left, L, A.conj(), W, A, optimize=True)
    mag = np.einsum(left, *[np.abs(x) for x in (L, A, W, A)], optimize=True)
    got = _call(gpu.ctgpu_contraction_operator_step_left, a, w, env)
    assert np.all(np.abs(got - ref) <= 1.5 * 4 * (d0 + w0 * d + d0 * d + 6) * eps * mag)
    right = "psu,uzvx,wtsz,qtv->pwqx"
    env = _tensor(rng, (d1, w1, d1, 1), (1, 1, -1, 1))
    R = env.to_dense()
    ref = np.einsum(right, A, R, W, A.conj(), optimize=True)
    mag = np.einsum(right, *[np.abs(x) for x in (A, R, W, A)], optimize=True)
    got = _call(gpu.ctgpu_contraction_operator_step_right, a, w, env)
    assert np.all(np.abs(got - ref) <= 1.5 * 4 * (d1 + w1 * d + d1 * d + 6) * eps * mag)
