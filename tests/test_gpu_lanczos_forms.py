"""The Lanczos vector kernels with the thread counts that they choose by vector length (a few dozen doubles,
some thousand, more than 65536) against the same search with every vector on the grid form (a child process
with CTGPU_LZ_CLUSTER_MAX_N=0): the two differ in rounding alone, 1e-15 per operation, which the search's
energies keep to 1e-10."""

import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = """
import json, sys
import numpy as np
from chemtensor_gb300 import ctstructs as cs, hamiltonians as hm, native
L, D = int(sys.argv[1]), int(sys.argv[2])
H = cs.make_c_mpo(hm.fermi_hubbard_1d(L, 1.0, 4.0, 0.0))
psi = native.random_mps(L, 4, hm.HUBBARD_QSITE, hm.encode_quantum_number_pair(L, 0), D, 11)
ret, en, ent = native.dmrg_twosite(H, psi, 2, 6, 1e-10, D)
print(json.dumps({"ret": ret, "en": list(en)}))
"""


def _search(L, D, **env):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SCRIPT, str(L), str(D)], cwd=root, env=dict(os.environ, **env),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("L,D", [(2, 4), (6, 20), (10, 240)])
def test_lanczos_forms(gpu, L, D):
    a, b = _search(L, D), _search(L, D, CTGPU_LZ_CLUSTER_MAX_N="0")
    assert a["ret"] == 0 and b["ret"] == 0
    np.testing.assert_allclose(a["en"], b["en"], rtol=0, atol=1e-10)
