"""The tile choices of reduced-precision products that are kept in a file: they are read back by later processes, and
a line that was timed against other kernels (a key without the form of the FP64 product and the version) is not."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_RUN = """
import ctypes as C
import numpy as np
from chemtensor_gb300 import ctstructs as cs, native
from helpers import c_bst
lib = native.lib()
z = lambda n: np.zeros(n, np.int32)
s, t = cs.BlockSparse((200, 150), (1, 1), [z(200), z(150)]), cs.BlockSparse((150, 250), (-1, 1), [z(150), z(250)])
for x in (s, t):
    x.blocks[(0, 0)] = np.ones(x.block_shape((0, 0)))
native.set_precision(native.PRECISION_BF16X3)
ca, cb, out = c_bst(s), c_bst(t), cs.BlockSparseTensor()
assert lib.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
for e in native.tile_tuning():
    print("ENTRY", e["key"], e["bn"], e["source"])
"""


def _run(path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, CTGPU_TUNE_FILE=str(path), PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", _RUN], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [ln.split()[1:] for ln in r.stdout.splitlines() if ln.startswith("ENTRY")]


def test_lines_of_other_kernels_are_not_used(gpu, tmp_path):
    path = tmp_path / "tuning.txt"
    (key, bn, source), = _run(path)
    assert source == "timed"
    assert _run(path) == [[key, bn, "file"]]
    # the same product's line as it was written before the key named the timed kernels
    path.write_text(key.split("_s")[0] + " 128 1.0 0.5 1.0 1.0\n")
    entries = _run(path)
    assert [key, "timed"] in [[e[0], e[2]] for e in entries], entries
