"""Large FP64 block products (digit slices) keep the accuracy of every row and column: operands whose rows and
columns differ in scale by up to 1e20, and contracted sectors of different scale, against numpy.

The bound is componentwise, as for the products on the FP64 pipe: a sum of k products in FP64, in any order,
is off by at most (k + 2) eps (|A| |B|); numpy's own sum takes as much again."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu

# rows, columns, terms; the last makes the product large enough for the slices
SECTORS = [(33, 31, 17), (129, 65, 128), (65, 129, 256), (8, 9, 129), (200, 190, 15), (70, 9, 20000), (600, 513, 500)]


def _check(gpu, a, axs, b, axt, nmult=1):
    ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), axs, C.byref(cb), axt, nmult, C.byref(out)) == 0
    got = cs.read_bst(out)
    for x in (out, ca, cb):
        cs.free_bst(x)
    return got


def _bounded(got, x, y):
    k = x.shape[1]
    bound = 2 * (k + 2) * np.finfo(np.float64).eps * (np.abs(x) @ np.abs(y))
    assert np.all(np.abs(got - x @ y) <= bound), float(np.max(np.abs(got - x @ y) / np.maximum(bound, 5e-324)))


@pytest.mark.parametrize("axs,axt", [(1, 0), (0, 1)])
@pytest.mark.parametrize("scale", [1e-6, 1e-10, 1e-14, 1e-20])
def test_scaled_rows_and_columns(gpu, scale, axs, axt):
    rng = np.random.default_rng(int(-np.log10(scale)))
    qm, qn, qk = (np.repeat(np.arange(len(SECTORS)), [s[i] for s in SECTORS]).astype(np.int32) for i in range(3))
    a = cs.BlockSparse((len(qm), len(qk)), (1, -1), [qm, qk]) if axs else cs.BlockSparse((len(qk), len(qm)), (-1, 1), [qk, qm])
    b = cs.BlockSparse((len(qn), len(qk)), (-1, 1), [qn, qk]) if axt else cs.BlockSparse((len(qk), len(qn)), (1, -1), [qk, qn])
    for t, lead in ((a, axs == 1), (b, axt == 1)):
        for idx in t.allowed:
            x = rng.standard_normal(t.block_shape(idx))
            s = scale ** rng.uniform(0, 1, x.shape[0 if lead else 1])
            s[0] = scale
            t.blocks[idx] = x * (s[:, None] if lead else s[None, :])
    got = _check(gpu, a, axs, b, axt)
    for idx in got.allowed:
        _bounded(got.blocks[idx], a.blocks[idx] if axs else a.blocks[idx].T, b.blocks[idx].T if axt else b.blocks[idx])
