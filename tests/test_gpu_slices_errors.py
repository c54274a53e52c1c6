"""A large FP64 product (digit slices) whose bounded waits run out: the limit is lowered to one poll, so the kernel takes
its own error exit (it records a flag, lets its copies and matrix products end, frees its tensor memory and
returns) and the call reports it. The next call of the same product, whose plan counts the shares of split sums,
gives the right result."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs, native
from helpers import c_bst

pytestmark = pytest.mark.gpu


def test_product_after_a_wait_that_ran_out(gpu):
    rng = np.random.default_rng(2)
    dims = [(90, 70, 20000), (600, 513, 500)]
    qm, qn, qk = (np.repeat([0, 1], [d[i] for d in dims]).astype(np.int32) for i in range(3))
    a = cs.BlockSparse((len(qm), len(qk)), (1, -1), [qm, qk])
    b = cs.BlockSparse((len(qk), len(qn)), (1, -1), [qk, qn])
    for t in (a, b):
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
    ca, cb = c_bst(a), c_bst(b)

    def run():
        out = cs.BlockSparseTensor()
        ret = gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out))
        r = cs.read_bst(out) if ret == 0 else None
        if ret == 0:
            cs.free_bst(out)
        return ret, r

    ret, first = run()
    assert ret == 0
    try:
        gpu.ctgpu_set_tc_wait_limit(1)
        ret, _ = run()
        msg = native.last_error()
    finally:
        gpu.ctgpu_set_tc_wait_limit(0)
    assert ret == -5 and "timed out" in msg, (ret, msg)
    for _ in range(2):
        ret, again = run()
        assert ret == 0
        for idx in first.allowed:
            np.testing.assert_array_equal(again.blocks[idx], first.blocks[idx])
    for t in (ca, cb):
        cs.free_bst(t)
