"""Block QR of blocks whose entries fill just under 48 KB of shared memory, the limit for static and dynamic
shared memory together that holds until a kernel's attribute raises it."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


_ALONE = """
import sys
import numpy as np
from chemtensor_gb300 import native
from test_gpu_qr_values import _factors
m, n, cplx = int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3])
rng = np.random.default_rng(0)
a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
q, r = _factors(native.lib(), a, "qr")
assert np.abs(q @ r - a).max() <= 8 * max(m, n) * 2.3e-16 * np.abs(a).max() * np.sqrt(min(m, n))
"""


@pytest.mark.parametrize("m,n,cplx", [(48, 126, 0), (32, 190, 0), (48, 62, 1), (32, 94, 1)])
def test_first_call_just_below_48_kb(gpu, m, n, cplx):
    """In a process of its own: the shared-memory limit has not been raised by a larger block before."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", _ALONE, str(m), str(n), str(cplx)], cwd=root, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
