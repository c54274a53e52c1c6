"""A local-Hamiltonian application whose MPO tensor is larger than the intermediate that it meets, as on the bonds of a
wide MPO where the state has become small, with rows and terms of very different scale: every entry is as
accurate as the FP64 pipe's, and the application takes no longer than there.

The bound is componentwise: two FP64 evaluations of the three products differ by at most
2 (k1 + k2 + k3 + 6) eps times the same application to the operands' magnitudes."""

import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_RUN = """
import ctypes as C
import sys
import numpy as np
from chemtensor_gb300 import ctstructs as cs, native, workloads as wl
from helpers import c_bst
lib = native.lib()
D, Dw = 96, 480
a, w, l, r = wl.local_h_microbench(D=D, nsec=7, sigma=2.0, Dw=Dw, seed=3)
rng = np.random.default_rng(5)
w_scale, r_scale = 10.0 ** rng.uniform(-6, 0, Dw), 10.0 ** rng.uniform(-6, 0, Dw)
sectors = [np.flatnonzero(w.qnums_logical[3] == q) for q in w.qnums_blocks[3]]
for i, b in w.blocks.items():                  # a few nonzero terms in a row
    w.blocks[i] = b * (rng.uniform(0, 1, b.shape) < 0.02) * w_scale[sectors[i[3]]]
for i, b in r.blocks.items():
    r.blocks[i] = b * r_scale[sectors[i[1]]][None, :, None, None]
if sys.argv[1] == "magnitudes":
    for t in (a, w, l, r):
        for i in t.blocks:
            t.blocks[i] = np.abs(t.blocks[i])
ops = [c_bst(t) for t in (a, w, l, r)]
out = cs.BlockSparseTensor()
assert lib.ctgpu_apply_local_hamiltonian(*[C.byref(t) for t in ops], C.byref(out)) == 0
cs.read_bst(out).to_dense().tofile(sys.argv[2])
ms, flops = C.c_double(), C.c_double()
best = 1e30
for _ in range(4):
    assert lib.ctgpu_time_local_hamiltonian(*[C.byref(t) for t in ops], 4, C.byref(ms), C.byref(flops)) == 0
    best = min(best, ms.value / 4)
print(best, flops.value)
"""


def _run(path, what, **env):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]), **env)
    r = subprocess.run([sys.executable, "-c", _RUN, what, str(path)], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    print(what, env.get("CTGPU_SLICE_GEMM"), r.stdout.strip())
    return np.fromfile(path), float(r.stdout.split()[0])


def test_mpo_larger_than_the_intermediate(gpu, tmp_path):
    got, ms = _run(tmp_path / "a", "values")
    want, ms_pipe = _run(tmp_path / "b", "values", CTGPU_SLICE_GEMM="0")
    size, _ = _run(tmp_path / "c", "magnitudes", CTGPU_SLICE_GEMM="0")
    k = 96 + 16 * 480 + 96 * 480
    assert np.any(got != want)                 # the digit slices did take part
    assert np.all(np.abs(got - want) <= 2 * (k + 6) * np.finfo(np.float64).eps * size)
    assert ms <= ms_pipe
