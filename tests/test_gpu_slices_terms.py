"""Large FP64 block products (digit slices) keep the accuracy of every entry: sectors and terms of different scale along
the contraction, graded operands times an identity, terms that cancel, in unsplit and split sums, against numpy.

The bound is componentwise, as for the products on the FP64 pipe: a sum of k products in FP64, in any order,
is off by at most (k + 2) eps (|A| |B|); numpy's own sum takes as much again."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


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


def _sectors(rng, scale, kind, m=300, n=260):
    """Contraction over two axes of four sectors each; free axes of one sector."""
    p, q = [30, 7, 50, 1], [40, 3, 20, 9]
    qp, qq = (np.repeat(np.arange(len(x)), x).astype(np.int32) for x in (p, q))
    a = cs.BlockSparse((m, len(qp), len(qq)), (1, -1, 1), [np.zeros(m, np.int32), qp, qq])
    b = cs.BlockSparse((len(qp), len(qq), n), (1, -1, -1), [qp, qq, np.zeros(n, np.int32)])
    for i, (ia, ib) in enumerate(zip(a.allowed, b.allowed)):
        x, y = rng.standard_normal(a.block_shape(ia)), rng.standard_normal(b.block_shape(ib))
        if kind == "blocks":                   # A = U S, B = S^-1 V, S constant in a sector
            s = scale ** (i / 3.0)
            x, y = x * s, y / s
        elif kind == "terms":                  # the same with S graded inside the sectors
            s = scale ** rng.uniform(0, 1, x.shape[1:])
            x, y = x * s, y / s[:, :, None]
        elif kind == "identity" and i == 0:    # a graded operand times an identity (and zeros elsewhere)
            x = x * scale ** rng.uniform(0, 1, x.shape[1:])
            y = np.eye(y[..., 0].size, n).reshape(y.shape)
        elif kind == "identity":
            y = np.zeros_like(y)
        a.blocks[ia], b.blocks[ib] = x, y
    return a, b


@pytest.mark.parametrize("kind", ["blocks", "terms", "identity"])
@pytest.mark.parametrize("scale", [1e-3, 1e-6, 1e-12])
def test_scales_along_the_contraction(gpu, scale, kind):
    """Terms whose factors lie far from the largest ones of their row and column: the result is as accurate as
    the FP64 pipe's."""
    a, b = _sectors(np.random.default_rng(7), scale, kind)
    A, B = a.to_dense(), b.to_dense()
    got = _check(gpu, a, 1, b, 0, 2).to_dense()
    _bounded(got, A.reshape(A.shape[0], -1), B.reshape(-1, B.shape[2]))


@pytest.mark.parametrize("m,n", [(70, 9), (9, 70), (150, 140)])
@pytest.mark.parametrize("kind", ["cancel", "disjoint", "graded"])
def test_small_results_of_long_sums(gpu, m, n, kind):
    """20000 terms (split into shares) beside a block that makes the product large: pairs of terms that cancel,
    rows and columns that are large where the other is zero, rows graded against the columns."""
    rng = np.random.default_rng(m)
    k = 20000
    dims = [(m, n, k), (600, 513, 500)]
    qm, qn, qk = (np.repeat([0, 1], [d[i] for d in dims]).astype(np.int32) for i in range(3))
    a = cs.BlockSparse((len(qm), len(qk)), (1, -1), [qm, qk])
    b = cs.BlockSparse((len(qk), len(qn)), (1, -1), [qk, qn])
    for t in (a, b):
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
    x, y = a.blocks[a.allowed[0]], b.blocks[b.allowed[0]]
    if kind == "cancel":
        x[:, 1::2], y[1::2] = -x[:, ::2], y[::2]
        x[:, 0] *= 1 + 1e-12
    elif kind == "disjoint":
        x[:, k // 2:] *= 1e-11
        y[:k // 2] = 0
    else:
        g = 10.0 ** rng.uniform(-9, 0, k)
        x *= g
        y *= g.min() / g[:, None]
    got = _check(gpu, a, 1, b, 0)
    _bounded(got.blocks[got.allowed[0]], x, y)


def test_small_products_on_the_slices(gpu):
    """The tests of block products, of single operations and of searches with every FP64 product on the slices: groups of
    several blocks, transposed results, blocks without terms."""
    here = os.path.dirname(os.path.abspath(__file__))
    files = [os.path.join(here, f"test_gpu_{f}.py") for f in ("block_products", "ops", "dmrg", "inner")]
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", *files], cwd=os.path.dirname(here),
                       env=dict(os.environ, CTGPU_SLICE_GEMM="1"), capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:]
