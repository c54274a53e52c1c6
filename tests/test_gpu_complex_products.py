"""complex128 block products over the tile classes of the work lists (narrow, wide, square, long
contractions that are split into shares, contractions short enough to skip the staging) against numpy.

The bound is componentwise: a sum of k complex products in FP64, in any order, is off by at most
4 (k + 2) eps (|A| |B|); numpy's own sum takes half of that."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


def _tensor(rng, dims, dirs, nq):
    t = cs.BlockSparse(dims, dirs, [(np.arange(d) % nq).astype(np.int32) for d in dims], dtype=cs.CT_DOUBLE_COMPLEX)
    for idx in t.allowed:
        shp = t.block_shape(idx)
        t.blocks[idx] = rng.standard_normal(shp) + 1j * rng.standard_normal(shp)
    return t


@pytest.mark.parametrize("m,k,n,nq", [
    (1, 1, 1, 1), (3, 200, 70, 1), (70, 200, 3, 1), (7, 33, 130, 1), (130, 33, 7, 1), (16, 900, 16, 1), (17, 16, 65, 1),
    (65, 17, 16, 1), (129, 65, 67, 1), (40, 4, 40, 1), (41, 5, 39, 1), (90, 120, 100, 3),
])
def test_complex_product(gpu, m, k, n, nq):
    rng = np.random.default_rng(m * 7 + k * 11 + n)
    a, b = _tensor(rng, (m, k), (1, -1), nq), _tensor(rng, (k, n), (1, -1), nq)
    ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
    got = cs.read_bst(out).to_dense()
    A, B = a.to_dense(), b.to_dense()
    bound = 4 * (k + 2) * np.finfo(np.float64).eps * (np.abs(A) @ np.abs(B))
    assert np.all(np.abs(got - A @ B) <= bound)
    for x in (out, ca, cb):
        cs.free_bst(x)
