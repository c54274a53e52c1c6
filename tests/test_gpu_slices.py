"""FP64 block products by digit slices on the tensor cores (large products) against extended precision."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu

# block sizes (m, n, k) of the sectors: edges of the 128 x 64 tiles, of their halves of 32, of 8 rows, of the
# 16 terms of a stage and the 128 of a flush; the last makes the product large enough for the slices
SECTORS = [(1, 300, 500), (300, 1, 333), (33, 31, 17), (128, 64, 16), (129, 65, 128), (64, 128, 640), (8, 9, 129),
           (200, 190, 15), (31, 97, 1), (600, 513, 500)]


def _operands(rng, axs, axt, grade):
    """A of shape (m, k) or (k, m), B of (k, n) or (n, k); one block per sector."""
    rows = [np.repeat(np.arange(len(SECTORS)), [s[i] for s in SECTORS]).astype(np.int32) for i in range(3)]
    qm, qn, qk = rows
    if axs == 1:
        a = cs.BlockSparse((len(qm), len(qk)), (1, -1), [qm, qk])
    else:
        a = cs.BlockSparse((len(qk), len(qm)), (-1, 1), [qk, qm])
    if axt == 0:
        b = cs.BlockSparse((len(qk), len(qn)), (1, -1), [qk, qn])
    else:
        b = cs.BlockSparse((len(qn), len(qk)), (-1, 1), [qn, qk])
    for t in (a, b):
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx)) * 2.0 ** int(rng.integers(-40, 40))
            if grade:
                t.blocks[idx] *= 10.0 ** rng.uniform(-8, 0, size=t.block_shape(idx))
    return a, b


def _dot(gpu, a, axs, b, axt):
    ca, cb = c_bst(a), c_bst(b)
    out = cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), axs, C.byref(cb), axt, 1, C.byref(out)) == 0
    r = cs.read_bst(out)
    for t in (out, ca, cb):
        cs.free_bst(t)
    return r


def _dropped(x, y):
    """The digit products that the slices drop: seven per term, of 2^-76 of the blocks' powers of two times two
    digits of 74 rms (2^-62.2 together), eight standard deviations of their sum."""
    top = 2.0 ** (np.floor(np.log2(float(np.abs(x).max()))) + 1 + np.floor(np.log2(float(np.abs(y).max()))) + 1)
    return 8 * np.sqrt(x.shape[1]) * 2.0**-62 * top


@pytest.mark.parametrize("axs,axt,grade", [(1, 0, False), (0, 0, False), (1, 1, True), (0, 1, True)])
def test_large_products_round_once(gpu, axs, axt, grade):
    rng = np.random.default_rng(10 * axs + axt)
    a, b = _operands(rng, axs, axt, grade)
    r = _dot(gpu, a, axs, b, axt)
    assert len(r.allowed) == len(SECTORS)
    for idx in r.allowed:
        x = a.blocks[idx] if axs == 1 else a.blocks[idx].T
        y = b.blocks[idx] if axt == 0 else b.blocks[idx].T
        k = x.shape[1]
        # every entry of the small blocks, some of the large ones, in extended precision
        n = x.shape[0] * y.shape[1]
        at = np.arange(n) if n <= 5000 else np.sort(rng.choice(n, 5000, replace=False))
        i, j = at // y.shape[1], at % y.shape[1]
        ref = np.array([np.dot(x[p].astype(np.longdouble), y[:, q].astype(np.longdouble)) for p, q in zip(i, j)])
        tol = np.abs(ref) * 2.0**-53 * 1.001 + _dropped(x, y)
        assert np.all(np.abs(r.blocks[idx][i, j] - ref) <= tol), idx


def test_values_out_of_the_slices_range(gpu):
    """Blocks with infinities, NaN, denormal or huge entries take FP64 sums; zero blocks give zeros."""
    rng = np.random.default_rng(5)
    a, b = _operands(rng, 1, 0, False)
    for i, idx in enumerate(a.allowed):
        x, y = a.blocks[idx], b.blocks[idx]
        if i == 0: x[0, 0] = np.inf
        if i == 2: y[0, -1] = np.nan
        if i == 3: x[...] = 5e-310
        if i == 4: y[...] = 0.0
        if i == 5: x *= 1e300 / np.abs(x).max()
        if i == 6:
            x *= 1e200 / np.abs(x).max()
            y *= 1e200 / np.abs(y).max()
        if i == 7:
            x *= 1e-200 / np.abs(x).max()
            y *= 1e-130 / np.abs(y).max()
    r = _dot(gpu, a, 1, b, 0)
    for i, idx in enumerate(r.allowed):
        with np.errstate(all="ignore"):
            ref = a.blocks[idx] @ b.blocks[idx]
            mag = np.abs(a.blocks[idx]) @ np.abs(b.blocks[idx])
        got = r.blocks[idx]
        assert np.array_equal(np.isnan(got), np.isnan(ref)), i
        # a sum that overflows may do so in another order of its terms: only its not being finite is common
        fin = np.isfinite(ref) & np.isfinite(mag)
        assert np.all(np.isfinite(got[fin])), i
        if i != 6:
            assert np.array_equal(np.isinf(got), np.isinf(ref)), i
        # FP64 sums on both sides, or one on the slices
        n = a.blocks[idx].shape[1]
        tol = 2 * n * 2.0**-53 * mag[fin] + 5e-324 * n
        if i in (1, 8, 9):
            tol = tol + _dropped(a.blocks[idx], b.blocks[idx])
        assert np.all(np.abs(got[fin] - ref[fin]) <= tol), i
