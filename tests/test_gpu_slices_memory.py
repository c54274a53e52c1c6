"""Large FP64 products where the digits of their operands may not be held (a limit of one byte, which stands for a device
without room for them): they run on the FP64 pipe, with its results to the last bit, in single products, in a
local-Hamiltonian application and in a search."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_RUN = """
import ctypes as C
import hashlib
import numpy as np
from chemtensor_gb300 import ctstructs as cs, hamiltonians as hm, native, workloads as wl
from helpers import c_bst, run_gpu_dmrg
lib = native.lib()
rng = np.random.default_rng(0)
z = lambda n: np.zeros(n, np.int32)
a, b = cs.BlockSparse((600, 500), (1, -1), [z(600), z(500)]), cs.BlockSparse((500, 513), (1, -1), [z(500), z(513)])
for t in (a, b):
    t.blocks[(0, 0)] = rng.standard_normal(t.block_shape((0, 0)))
ca, cb, out = c_bst(a), c_bst(b), cs.BlockSparseTensor()
assert lib.ctgpu_block_sparse_tensor_dot(C.byref(ca), 1, C.byref(cb), 0, 1, C.byref(out)) == 0
print(hashlib.sha1(cs.read_bst(out).serialize().tobytes()).hexdigest())
ops = [c_bst(t) for t in wl.local_h_microbench(D=300, nsec=7, sigma=3.0, Dw=12, seed=1)]
out = cs.BlockSparseTensor()
assert lib.ctgpu_apply_local_hamiltonian(*[C.byref(t) for t in ops], C.byref(out)) == 0
print(hashlib.sha1(cs.read_bst(out).serialize().tobytes()).hexdigest())
tkin, vint = wl.molecular_integrals(6, 3)
psi = native.random_mps(6, 4, hm.HUBBARD_QSITE, hm.encode_quantum_number_pair(6, 0), 64, 5)
ret, en, *_ = run_gpu_dmrg(lib, hm.spin_molecular(tkin, vint), cs.read_mps(psi), 1, 5, 1e-10, 64)
assert ret == 0
print(en.tobytes().hex())
"""


def _run(**env):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]), **env)
    r = subprocess.run([sys.executable, "-c", _RUN], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split()


def test_no_room_for_the_digits(gpu):
    tiles = _run(CTGPU_SLICE_GEMM="0")
    assert _run(CTGPU_SLICE_BYTES="1") == tiles
    assert _run(CTGPU_SLICE_BYTES="1", CTGPU_SLICE_GEMM="1") == tiles
    slices = _run()
    assert slices[0] != tiles[0] and slices[1] != tiles[1]
