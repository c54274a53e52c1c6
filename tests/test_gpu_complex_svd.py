"""complex128 block SVD at the sizes where its forms change: one CTA to sixteen per block, groups of one to
several columns, the smallest block whose sweeps start in FP32 (16), wide and tall blocks, blocks beyond
the shared memory of a cluster (more than 224 columns at square shape), many blocks of different sizes in
one call; and spectra that are graded, degenerate, nearly level or of extreme scale.

Backward stability bounds the error of every singular value by a small multiple of max(m, n) eps times the
largest one; the multiple here is 8. A two-site search checks the factors: the rows of a
returned state whose blocks reach the FP32 sweeps, and its energy against the search with real entries."""

import ctypes as C

import numpy as np
import pytest

from chemtensor_gb300 import ctstructs as cs
from chemtensor_gb300 import hamiltonians as hm
from chemtensor_gb300 import native
from chemtensor_gb300 import workloads as wl
from helpers import c_bst, run_gpu_dmrg

pytestmark = pytest.mark.gpu


def _matrix(rng, m, n, kind):
    k = min(m, n)
    if kind == "random":
        return rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))
    s = {"graded": np.logspace(0, -12, k), "equal": np.repeat(np.logspace(0, -6, (k + 3) // 4), 4)[:k],
         "level": 1 + 1e-3 * rng.uniform(-1, 1, k), "tiny": np.logspace(-150, -156, k), "rank": np.r_[np.ones((k + 1) // 2), np.zeros(k // 2)]}
    u = np.linalg.qr(rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k)))[0]
    v = np.linalg.qr(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))[0]
    return (u * s[kind]) @ v.conj().T


def _values(gpu, t):
    ct = c_bst(t)
    k = min(t.dim_logical)
    sig, ns = np.zeros(k), C.c_int64()
    assert gpu.ctgpu_block_sparse_tensor_svd_values(C.byref(ct), sig.ctypes.data, C.byref(ns)) == 0
    cs.free_bst(ct)
    return np.sort(sig[:ns.value])[::-1]


@pytest.mark.parametrize("kind", ["random", "graded", "equal", "level", "tiny", "rank"])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 3), (8, 9), (15, 15), (16, 16), (17, 40), (33, 32), (65, 64), (40, 130), (129, 128)])
def test_singular_values(gpu, m, n, kind):
    rng = np.random.default_rng(m * 1000 + n)
    t = cs.BlockSparse((m, n), (1, -1), [np.zeros(m, np.int32), np.zeros(n, np.int32)], dtype=cs.CT_DOUBLE_COMPLEX)
    a = _matrix(rng, m, n, kind)
    t.blocks[t.allowed[0]] = a
    ref = np.linalg.svd(a, compute_uv=False)
    np.testing.assert_allclose(_values(gpu, t), ref, rtol=0, atol=8 * max(m, n) * np.finfo(np.float64).eps * ref[0])


@pytest.mark.parametrize("big", [30, 224, 232])
def test_blocks_of_many_sizes(gpu, big):
    rng = np.random.default_rng(big)
    rows, cols = [3, 40, 1, 17, 26, 9, big], [5, 38, 4, 1, 30, 9, big]
    q = [np.repeat(np.arange(len(x)), x).astype(np.int32) for x in (rows, cols)]
    t = cs.BlockSparse((sum(rows), sum(cols)), (1, -1), q, dtype=cs.CT_DOUBLE_COMPLEX)
    ref = []
    for idx in t.allowed:
        a = _matrix(rng, *t.block_shape(idx), "random")
        t.blocks[idx] = a
        ref.append(np.linalg.svd(a, compute_uv=False))
    ref = np.sort(np.concatenate(ref))[::-1]
    np.testing.assert_allclose(_values(gpu, t), ref, rtol=0, atol=8 * max(big, 40) * np.finfo(np.float64).eps * ref[0])


def test_factors_in_a_search(gpu):
    """A two-site search at bond dimension 96 (blocks of up to 30 columns): the returned tensors right of the
    first one have orthonormal rows to the SVD's own accuracy, the energy is that of the search over real
    entries, of which the complex Hamiltonian and state are a gauge transform."""
    L, D = 8, 96
    H = hm.fermi_hubbard_1d(L, 1.0, 4.0, 0.0)
    sector = hm.encode_quantum_number_pair(L, 0)
    m = native.random_mps(L, 4, hm.HUBBARD_QSITE, sector, D, 7)
    psi = cs.read_mps(m)
    en = {}
    for z in (False, True):
        ret, e, _, out = run_gpu_dmrg(gpu, wl.complex_gauge(H, 3) if z else H, wl.complex_gauge(psi, 4) if z else psi, 2, 10, 1e-10, D)
        assert ret == 0
        en[z] = e[-1]
    np.testing.assert_allclose(en[True], en[False], rtol=1e-10)
    for t in out.tensors[1:]:
        a = t.to_dense()
        a = a.reshape(a.shape[0], -1)
        np.testing.assert_allclose(a @ a.conj().T, np.eye(len(a)), rtol=0, atol=8 * a.shape[1] * np.finfo(np.float64).eps)
