"""Digit-slice products with more than 55800 terms in one share (437 flushes of the tensor-core sums, where the offsets of
the sums pass 63 bits) and, on the FP64 pipe, with more terms than the slices' integers hold."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_RUN = """
import ctypes as C
import sys
import numpy as np
from chemtensor_gb300 import ctstructs as cs, native
from helpers import c_bst
lib = native.lib()
nsec, k = int(sys.argv[1]), int(sys.argv[2])
rng = np.random.default_rng(1)
q, qk = np.arange(nsec, dtype=np.int32), np.repeat(np.arange(nsec), k).astype(np.int32)
a, b = cs.BlockSparse((nsec, nsec * k), (1, -1), [q, qk]), cs.BlockSparse((nsec * k, nsec), (1, -1), [qk, q])
for t in (a, b):
    for idx in t.allowed:
        t.blocks[idx] = np.abs(rng.standard_normal(t.block_shape(idx)))
ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
assert lib.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
got = cs.read_bst(out)
for i, idx in enumerate(got.allowed):
    x, y = a.blocks[a.allowed[i]].ravel(), b.blocks[b.allowed[i]].ravel()
    ref = np.dot(x.astype(np.longdouble), y.astype(np.longdouble))
    # the slices: one rounding and the digits cut off (8 standard deviations); the FP64 pipe: its sum
    tol = ref * 2.0**-53 * 1.001 + 8 * np.sqrt(k) * 2.0**-62 * 64 if k < 1 << 21 else (k + 2) * 2.0**-52 * ref
    assert abs(got.blocks[idx][0, 0] - ref) <= tol, (i, got.blocks[idx][0, 0], ref)
"""


@pytest.mark.parametrize("nsec,k", [(160, 56000), (1, (1 << 21) + 3)])
def test_long_sums(gpu, nsec, k):
    """160 sums of 56000 terms are a share each on 152 SMs."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, CTGPU_SLICE_GEMM="1", PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", _RUN, str(nsec), str(k)], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
