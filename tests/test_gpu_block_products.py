"""FP64 block products over the forms of a tile's list of terms: one contribution and many, more than the 64
terms and more than the 64 contributions that are tabulated at a time, stages of 16 terms that end inside a
contribution, shares of a split sum, blocks without contributions; against numpy.

The bound is componentwise: a sum of k products in FP64, in any order, is off by at most (k + 2) eps (|A| |B|);
numpy's own sum takes as much again."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu

# multiplicities of the sectors of the two contracted axes: contribution i has p[i] q[i] terms
SECTORS = {"one": ([1], [1]), "k16": ([4], [4]), "k17": ([17], [1]), "k64": ([8], [8]), "k65": ([13], [5]),
           "long": ([30], [30]), "mixed": ([3, 1, 5, 2, 7, 1], [2, 1, 3, 8, 9, 1]), "many": ([1] * 70, [1] * 70),
           "even": ([2] * 40, [2] * 40), "tail": ([1] * 60 + [11], [1] * 60 + [17])}


def _axis(mult):
    return np.repeat(np.arange(len(mult)), mult).astype(np.int32)


@pytest.mark.parametrize("lead", [False, True])
@pytest.mark.parametrize("kind", list(SECTORS))
@pytest.mark.parametrize("m,n", [(1, 1), (17, 16), (3, 130), (70, 5), (40, 33), (200, 150)])
def test_block_product(gpu, m, n, kind, lead):
    p, q = SECTORS[kind]
    rng = np.random.default_rng(m + n)
    # free axes: sector 0, and two entries of a sector that no contracted pair reaches
    qm, qn = (np.r_[np.zeros(d), [100, 100]].astype(np.int32) for d in (m, n))
    qp, qq = _axis(p), _axis(q)
    if lead:                                   # both operands contracted over their leading axes
        a = cs.BlockSparse((len(qp), len(qq), m + 2), (-1, 1, 1), [qp, qq, qm])
    else:
        a = cs.BlockSparse((m + 2, len(qp), len(qq)), (1, -1, 1), [qm, qp, qq])
    b = cs.BlockSparse((len(qp), len(qq), n + 2), (1, -1, -1), [qp, qq, qn])
    for t in (a, b):
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
    ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), 0 if lead else 1, C.byref(cb), 0, 2, C.byref(out)) == 0
    got = cs.read_bst(out).to_dense()
    A, B = a.to_dense(), b.to_dense()
    axes = ((0, 1) if lead else (1, 2), (0, 1))
    k = int(np.dot(p, q))
    bound = 2 * (k + 2) * np.finfo(np.float64).eps * np.tensordot(np.abs(A), np.abs(B), axes)
    assert np.all(np.abs(got - np.tensordot(A, B, axes)) <= bound)
    for x in (out, ca, cb):
        cs.free_bst(x)


_EMPTY_LARGE = """
import ctypes as C
import numpy as np
from chemtensor_gb300 import ctstructs as cs, native
from helpers import c_bst
lib = native.lib()
rng = np.random.default_rng(3)
k = 60000
q = lambda *n: np.concatenate([np.full(c, i) for i, c in enumerate(n)]).astype(np.int32)
a = cs.BlockSparse((140, k), (1, -1), [q(40, 100), np.zeros(k, np.int32)])
b = cs.BlockSparse((k, 140), (1, -1), [np.zeros(k, np.int32), q(40, 100)])
for t in (a, b):
    for idx in t.allowed:
        t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
A, B = a.to_dense(), b.to_dense()
for _ in range(2):                             # dirty the allocator's memory, then use it
    ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
    assert lib.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
    got = cs.read_bst(out).to_dense()
    bound = 2 * (k + 2) * np.finfo(np.float64).eps * (np.abs(A) @ np.abs(B))
    assert np.all(np.abs(got - A @ B) <= bound)
"""


def test_large_block_without_terms(gpu):
    """A product large enough for the largest tiles whose only block of that size has no terms: the block is
    zeros. (On the FP64 tiles: the digit slices, which such products normally take, are off.)"""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, CTGPU_SLICE_GEMM="0", PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", _EMPTY_LARGE], cwd=root, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
