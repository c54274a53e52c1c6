"""Block SVD as a truncating caller runs it (the split of a two-site tensor): FP32 sweeps from rank 16 on, on a sub-cluster
of one, two, four or eight CTAs by rank, twelve warps from 129 columns on; and the factors of the complex SVD at every
cluster size and beyond its shared memory. Reconstruction, orthonormal factors and singular values against
LAPACK (numpy); the number of FP32 sweeps from the library's phase counters.

The bounds follow from backward stability: |A - U S V^H| and the errors of the singular values are at most a small
multiple of max(m, n) eps sigma_max, the factors' orthogonality a small multiple of max(m, n) eps; the multiple
here is 8. The weight that may be discarded, 1e-60, is below all of the values."""

import os
import re
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
from test_zz_svd_small_ranks import _matrix
lib = native.lib()
cplx, discard = int(sys.argv[1]), float(sys.argv[2])
for size in sys.argv[3:]:
    m, n = map(int, size.split("x"))
    k = min(m, n)
    for kind in ("random", "scaled", "level"):
        rng = np.random.default_rng(m * 1000 + n)
        a = _matrix(rng, m, n, kind)
        if cplx:
            p = np.exp(2j * np.pi * rng.uniform(size=(m, m)))
            a = np.linalg.qr(p)[0] @ a @ np.linalg.qr(np.exp(2j * np.pi * rng.uniform(size=(n, n))))[0]
        t = cs.BlockSparse((m, n), (1, -1), [np.zeros(m, np.int32), np.zeros(n, np.int32)],
                           dtype=cs.CT_DOUBLE_COMPLEX if cplx else cs.CT_DOUBLE_REAL)
        t.blocks[(0, 0)] = a
        ca, cu, cv, s, ns = c_bst(t), cs.BlockSparseTensor(), cs.BlockSparseTensor(), np.zeros(k), C.c_int64()
        print("CALL", m, n, kind, file=sys.stderr, flush=True)
        assert lib.ctgpu_block_sparse_tensor_svd(C.byref(ca), discard, C.byref(cu), s.ctypes.data, C.byref(ns), C.byref(cv)) == 0
        u, vh = cs.read_bst(cu).to_dense(), cs.read_bst(cv).to_dense()
        for x in (ca, cu, cv):
            cs.free_bst(x)
        ref = np.linalg.svd(a, compute_uv=False)
        tol = 8 * max(m, n) * np.finfo(np.float64).eps
        for name, got, want, scale in (("values", s, ref, ref[0]), ("product", (u * s) @ vh, a, ref[0]),
                                       ("u", u.conj().T @ u, np.eye(k), 1), ("vh", vh @ vh.conj().T, np.eye(k), 1)):
            assert np.abs(got - want).max() <= tol * scale, (size, kind, name, np.abs(got - want).max() / scale, tol)
"""


def _run(cplx, discard, sizes):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, CTGPU_SVD_PHASES="2", PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", _RUN, str(cplx), str(discard), *[f"{m}x{n}" for m, n in sizes]], cwd=root, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return re.findall(r"CALL (\d+) (\d+) \w+\n.*?FP32 sweeps (\d+)", r.stderr)


SIZES = [(15, 15), (16, 16), (17, 17), (16, 40), (31, 31), (32, 32), (33, 33), (40, 33), (64, 64), (65, 65), (128, 128), (129, 129),
         (190, 150)]


@pytest.mark.parametrize("discard,smallest", [(1e-60, 16), (0.0, 32)])
def test_factors(gpu, discard, smallest):
    calls = _run(0, discard, SIZES)
    assert len(calls) == 3 * len(SIZES)
    for m, n, sweeps in calls:
        assert (int(sweeps) > 0) == (min(int(m), int(n)) >= smallest), (m, n, sweeps)


@pytest.mark.parametrize("discard", [1e-60, 0.0])
def test_complex_factors(gpu, discard):
    _run(1, discard, [(8, 8), (9, 15), (16, 16), (33, 32), (64, 65), (100, 129), (224, 224), (232, 240)])
