"""Block SVD factors around the smallest ranks whose Jacobi sweeps start from an FP32-preconditioned
basis (16), and on spectra that keep the FP32 sweeps turning wide angles, so that they go on after
the usual number of sweeps: reconstruction, orthonormal factors and singular values against LAPACK
(numpy).

The bounds follow from backward stability: |A - U S V^H| and the errors of the singular values are at
most a small multiple of max(m, n) eps sigma_max, the factors' orthogonality a small multiple of
max(m, n) eps (the sweeps stop at cosines of n eps); the multiple here is 8.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(rng, m, n, kind):
    if kind == "random":
        return rng.standard_normal((m, n))
    if kind == "scaled":                       # column norms over four decades in random order
        return rng.standard_normal((m, n)) * 10.0 ** rng.uniform(-4, 0, n)
    k = min(m, n)                              # nearly equal singular values: angles stay wide
    u, _ = np.linalg.qr(rng.standard_normal((m, k)))
    v, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return (u * (1.0 + 1e-3 * rng.uniform(-1, 1, k))) @ v.T


@pytest.mark.parametrize("kind", ["random", "scaled", "level"])
@pytest.mark.parametrize("m,n", [(15, 15), (16, 16), (17, 16), (16, 40), (31, 33), (90, 33), (97, 150), (190, 180)])
def test_svd_factors_small_and_slow(gpu, m, n, kind):
    torch = pytest.importorskip("torch")
    fn = gpu.ctgpu_dense_svd_noalloc
    fn.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    dev = torch.device("cuda:0")
    a = _matrix(np.random.default_rng(m * 1000 + n), m, n, kind)
    k = min(m, n)
    d_a = torch.from_numpy(a).to(dev)
    d_u = torch.zeros((m * k,), dtype=torch.float64, device=dev)
    d_s = torch.zeros((k,), dtype=torch.float64, device=dev)
    d_vh = torch.zeros((k * n,), dtype=torch.float64, device=dev)
    d_info = torch.full((1,), 7, dtype=torch.int32, device=dev)
    assert fn(d_a.data_ptr(), m, n, d_u.data_ptr(), d_s.data_ptr(), d_vh.data_ptr(), d_info.data_ptr(),
              torch.cuda.current_stream(dev).cuda_stream) == 0
    torch.cuda.synchronize(dev)
    assert int(d_info.item()) == 0
    u, s, vh = d_u.cpu().numpy().reshape(m, k), d_s.cpu().numpy(), d_vh.cpu().numpy().reshape(k, n)
    ref = np.linalg.svd(a, compute_uv=False)
    tol = 8 * max(m, n) * np.finfo(np.float64).eps
    np.testing.assert_allclose(s, ref, rtol=0, atol=tol * ref[0])
    np.testing.assert_allclose((u * s) @ vh, a, rtol=0, atol=tol * ref[0])
    np.testing.assert_allclose(u.T @ u, np.eye(k), rtol=0, atol=tol)
    np.testing.assert_allclose(vh @ vh.T, np.eye(k), rtol=0, atol=tol)
