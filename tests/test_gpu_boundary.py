"""Tensors across the C boundary, exactly: sizes below and above what the host threads share, one large block
and many small ones, more than the pinned staging area holds, empty and complex tensors."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n,nq", [(3, 2, 1), (0, 0, 2), (255, 257, 1), (257, 257, 1), (700, 900, 40), (1500, 333, 3), (3001, 2999, 1)])
def test_round_trip(gpu, m, n, nq, cplx):
    rng = np.random.default_rng(m + n)
    dtype = cs.CT_DOUBLE_COMPLEX if cplx else cs.CT_DOUBLE_REAL
    if m == 0:                                 # no allowed block
        t = cs.BlockSparse((2, 3), (1, -1), [np.zeros(2, np.int32), np.ones(3, np.int32)], dtype=dtype)
    else:
        t = cs.BlockSparse((m, n), (1, -1), [np.sort(rng.integers(0, nq, d)).astype(np.int32) for d in (m, n)], dtype=dtype)
    for idx in t.allowed:
        t.blocks[idx] = rng.standard_normal(t.block_shape(idx)) + (1j * rng.standard_normal(t.block_shape(idx)) if cplx else 0)
    ct, once, twice = c_bst(t), cs.BlockSparseTensor(), cs.BlockSparseTensor()
    perm = (C.c_int * 2)(1, 0)
    assert gpu.ctgpu_block_sparse_tensor_transpose(perm, C.byref(ct), C.byref(once)) == 0
    assert gpu.ctgpu_block_sparse_tensor_transpose(perm, C.byref(once), C.byref(twice)) == 0
    a, b = cs.read_bst(once), cs.read_bst(twice)
    assert b.allowed == t.allowed
    for idx in t.allowed:
        np.testing.assert_array_equal(a.blocks[idx[::-1]], t.blocks[idx].T)
        np.testing.assert_array_equal(b.blocks[idx], t.blocks[idx])
    for x in (ct, once, twice):
        cs.free_bst(x)
