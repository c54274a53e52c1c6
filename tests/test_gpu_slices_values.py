"""Digit-slice products (large FP64 products) where one operand block is all zeros and the other holds a
number that is not finite: NaN where BLAS has NaN, in tiles of one CTA and in tiles whose sum is split."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu

# (m, n, k) of the sectors: 20000 terms are split into shares; the last sector makes the product large
# enough for the slices
SECTORS = [(40, 50, 64), (40, 50, 64), (9, 70, 20000), (70, 9, 20000), (600, 513, 500)]


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("zero", [0, 1])
def test_zeros_times_not_finite(gpu, value, zero):
    rng = np.random.default_rng(3)
    qm, qn, qk = (np.repeat(np.arange(len(SECTORS)), [s[i] for s in SECTORS]).astype(np.int32) for i in range(3))
    ops = [cs.BlockSparse((len(qm), len(qk)), (1, -1), [qm, qk]), cs.BlockSparse((len(qk), len(qn)), (1, -1), [qk, qn])]
    for t in ops:
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
    for i, idx in enumerate(ops[0].allowed[:-1]):
        ops[zero].blocks[idx][...] = 0.0
        ops[1 - zero].blocks[idx][3, 5] = value
    ca, cb, out = c_bst(ops[0]), c_bst(ops[1]), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
    got = cs.read_bst(out)
    for x in (out, ca, cb):
        cs.free_bst(x)
    for idx in got.allowed[:-1]:
        with np.errstate(invalid="ignore"):
            ref = ops[0].blocks[idx] @ ops[1].blocks[idx]
        assert np.isnan(ref).any()
        np.testing.assert_array_equal(got.blocks[idx], ref)
    assert np.all(np.isfinite(got.blocks[got.allowed[-1]]))
