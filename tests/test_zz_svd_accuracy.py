"""Dense block SVD of blocks with a flat spectrum, whose FP64 finish turns columns by the widest angles: reconstruction,
singular values and factors as accurate as LAPACK's, not only to the bound of backward stability.

The bounds: a Householder QR, the rotations and a product each leave a few eps in the residual (Frobenius norm relative
to A's) and in the singular values (relative to the largest), and a few eps in every entry of the factors' Gram
matrices: 16 eps each."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(64, 60), (100, 90), (128, 128), (190, 150), (150, 200)])
def test_flat_spectrum(gpu, m, n):
    torch = pytest.importorskip("torch")
    fn = gpu.ctgpu_dense_svd_noalloc
    fn.argtypes = [C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 5
    fn.restype = C.c_int
    eps, k = np.finfo(np.float64).eps, min(m, n)
    for seed in range(3):
        a = np.random.default_rng(seed).standard_normal((m, n))
        d = torch.from_numpy(a).cuda()
        u, s, vh = (torch.zeros(x, dtype=torch.float64, device="cuda") for x in ((m, k), (k,), (k, n)))
        info = torch.full((1,), 7, dtype=torch.int32, device="cuda")
        assert fn(d.data_ptr(), m, n, u.data_ptr(), s.data_ptr(), vh.data_ptr(), info.data_ptr(),
                  torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert int(info.item()) == 0
        u, s, vh = u.cpu().numpy(), s.cpu().numpy(), vh.cpu().numpy()
        ref = np.linalg.svd(a, compute_uv=False)
        assert np.linalg.norm((u * s) @ vh - a) <= 16 * eps * np.linalg.norm(a)
        assert np.abs(s - ref).max() <= 16 * eps * ref[0]
        for q in (u.T @ u, vh @ vh.T):
            assert np.linalg.norm(q - np.eye(k)) <= 16 * eps * k
