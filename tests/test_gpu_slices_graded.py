"""Large FP64 block products (digit slices) of which most results are small beside their rows' largest entries (rows graded
against the other operand's columns): at the edges of a tile, with several blocks along the contraction, with some of the
results only, and beside rows that are not finite, tiny or huge, against numpy; and they take no longer than on the
FP64 pipe.

The bound is componentwise: a sum of k products in FP64, in any order, is off by at most (k + 2) eps (|A| |B|); numpy's
own sum takes as much again."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from helpers import c_bst

pytestmark = pytest.mark.gpu


def _operands(rng, m, n, k):
    """Charge 0: m x n results of k + 65 terms in three blocks; charge 5: a block that makes the product large."""
    q = lambda charges, sizes: np.repeat(charges, sizes).astype(np.int32)
    qm, qn = q([0, 5], [m, 600]), q([0, 5], [n, 513])
    qp, qq = q([0, 1, 2, 5], [k, 5, 1, 500]), q([0, 1, 2], [1, 7, 30])
    a = cs.BlockSparse((len(qm), len(qp), len(qq)), (1, -1, 1), [qm, qp, qq])
    b = cs.BlockSparse((len(qp), len(qq), len(qn)), (1, -1, -1), [qp, qq, qn])
    for t in (a, b):
        for idx in t.allowed:
            t.blocks[idx] = rng.standard_normal(t.block_shape(idx))
    return a, b, [(0, 0, 0), (0, 1, 1), (0, 2, 2)], [(0, 0, 0), (1, 1, 0), (2, 2, 0)]


def _product(gpu, a, b):
    ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
    assert gpu.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 2, C.byref(out)) == 0
    got = cs.read_bst(out)
    for t in (out, ca, cb):
        cs.free_bst(t)
    return got.blocks[(0, 0)]


@pytest.mark.parametrize("kind", ["all", "half", "rows"])
@pytest.mark.parametrize("m,n,k", [(128, 64, 31), (129, 65, 700), (97, 8, 2100), (9, 130, 33), (300, 200, 600), (520, 333, 131), (333, 1000, 64)])
def test_graded_rows_against_columns(gpu, m, n, k, kind):
    rng = np.random.default_rng(m + n)
    a, b, ia, ib = _operands(rng, m, n, k)
    for i, j in zip(ia, ib):
        x, y = a.blocks[i], b.blocks[j]
        s = 10.0 ** rng.uniform(-9, 0, x.shape[1:])
        x[: m if kind != "half" else m // 2] *= s
        y /= s[:, :, None]
        if kind == "rows":
            x[m // 3] *= 1e-290
            x[m // 2] *= 1e290
            y[..., n // 2] *= 1e-3
    if kind == "rows":
        a.blocks[ia[0]][1, 3] = np.inf
        a.blocks[ia[1]][2, 0, 0] = np.nan
        b.blocks[ib[0]][7, 0, 0] = -np.inf
    flat = lambda t, idx, axis: np.concatenate([t.blocks[i].reshape(t.blocks[i].shape[0], -1) if axis else
                                                t.blocks[i].reshape(-1, t.blocks[i].shape[2]) for i in idx], axis)
    x, y = flat(a, ia, 1), flat(b, ib, 0)
    got = _product(gpu, a, b)
    with np.errstate(all="ignore"):
        want, size = x @ y, np.abs(x) @ np.abs(y)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    np.testing.assert_array_equal(got[inf], want[inf])
    ok = np.isfinite(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= 2 * (x.shape[1] + 2) * np.finfo(np.float64).eps * size[ok])


_TIME = """
import ctypes as C
import time
import numpy as np
from chemtensor_gb300 import ctstructs as cs, native
from helpers import c_bst
lib = native.lib()
rng = np.random.default_rng(0)
n, k = 1024, 8192
s = 10.0 ** rng.uniform(-8, 0, k)
z = lambda n: np.zeros(n, np.int32)
a, b = cs.BlockSparse((n, k), (1, -1), [z(n), z(k)]), cs.BlockSparse((k, n), (1, -1), [z(k), z(n)])
a.blocks[(0, 0)], b.blocks[(0, 0)] = rng.standard_normal((n, k)) * s, rng.standard_normal((k, n)) / s[:, None]
ca, cb = c_bst(a), c_bst(b)
best = 1e30
for _ in range(5):
    out = cs.BlockSparseTensor()
    t = time.perf_counter()
    assert lib.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
    best = min(best, time.perf_counter() - t)
    cs.free_bst(out)
print(1e3 * best)
"""


def test_time_beside_the_pipe(gpu):
    """All results suspect: the slices are then of no use, and may cost a fifth of the pipe's time on top of it."""
    def run(**env):
        root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
        env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]), **env)
        r = subprocess.run([sys.executable, "-c", _TIME], cwd=root, env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        return float(r.stdout)
    slices, pipe = run(), run(CTGPU_SLICE_GEMM="0")
    print(slices, pipe)
    assert slices <= 1.2 * pipe
