"""The measured work of this package: ground-state searches and the operations around them, through
the entry points that a caller of the library uses.

A case is a dict of plain values. "kind" names the call:
  twosite    dmrg_twosite from a seeded random start state (FP64, complex128 or mixed precision)
  singlesite dmrg_singlesite from a seeded random start state
  energy     <psi|H|psi> and the norm of a state (ctgpu_mpo_inner_product, ctgpu_mps_norm)
  localh     one application of the local effective Hamiltonian (ctgpu_apply_local_hamiltonian)
  svd        SVD of one dense block in device memory (ctgpu_dense_svd_noalloc)

A state after DMRG is defined up to the gauge of its bonds, and rounding decides which gauge comes
back; a search therefore returns what is defined: the energy after every sweep, the entropies, and
for two-site searches the bond dimensions and every retained Schmidt value of every bond.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from chemtensor_gb300 import ctstructs as cs
from chemtensor_gb300 import hamiltonians as hm
from chemtensor_gb300 import native
from chemtensor_gb300 import workloads as wl

LANCZOS = 5          # Lanczos iterations per local problem, as in every workload of the package
TOL = 1e-10          # truncation tolerance of the split
TC_TILE = 128        # fixed tile width of the reduced-precision products: the same arithmetic every time


def listed():
    return [
        # the smallest request of a serving stream: launches, synchronisations and host work
        dict(name="xxz_L9_D16", kind="twosite", model="xxz", L=9, D=16, sweeps=2, dtype="f64", precision=0),
        # the plain configuration: Heisenberg chain, six sweeps
        dict(name="xxz_L20_D32", kind="twosite", model="xxz", L=20, D=32, sweeps=6, dtype="f64", precision=0),
        # an ordinary request of the stream, of odd sizes
        dict(name="hubbard_L21_D100", kind="twosite", model="hubbard", L=21, D=100, sweeps=2, dtype="f64", precision=0),
        # the headline configuration: Fermi-Hubbard L=32, D=256
        dict(name="hubbard_L32_D256", kind="twosite", model="hubbard", L=32, D=256, sweeps=2, dtype="f64", precision=0),
        # quantum chemistry in FP64: a wide MPO, large block products
        dict(name="molecular_n16_D256", kind="twosite", model="molecular", L=16, D=256, sweeps=1, dtype="f64", precision=0),
        # the same in mixed precision: a split-BF16 sweep on the tensor cores, the last one in FP64
        dict(name="molecular_n10_D128_bf16x3", kind="twosite", model="molecular", L=10, D=128, sweeps=2, dtype="f64",
             precision=1),
        # complex128 tensors
        dict(name="hubbard_L16_D64_c128", kind="twosite", model="hubbard", L=16, D=64, sweeps=1, dtype="c128", precision=0),
        # single-site search at the headline size: QR / RQ moves instead of the SVD split
        dict(name="single_hubbard_L32_D256", kind="singlesite", model="hubbard", L=32, D=256, sweeps=2, dtype="f64",
             precision=0),
        # the energy and norm of a state in hand
        dict(name="energy_hubbard_L32_D256", kind="energy", model="hubbard", L=32, D=256, dtype="f64"),
        # one local-Hamiltonian application on host tensors, D = 1024 over 41 sectors, FP64 and split-BF16
        dict(name="localh_D1024", kind="localh", D=1024, nsec=41, Dw=26, precision=0),
        dict(name="localh_D1024_bf16x3", kind="localh", D=1024, nsec=41, Dw=26, precision=1),
        # one dense block of a bond of the headline size, in device memory
        dict(name="svd_200x150", kind="svd", m=200, n=150),
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["twosite", "twosite", "twosite", "molecular", "mixed", "c128", "singlesite", "energy", "localh", "svd"])
    model = rng.choice(["xxz", "hubbard"])
    if kind == "twosite":
        return dict(kind="twosite", model=model, L=rng.randint(8, 40), D=_log_int(rng, 16, 256), sweeps=2, dtype="f64",
                    precision=0)
    if kind == "molecular":
        return dict(kind="twosite", model="molecular", L=rng.randint(5, 14), D=_log_int(rng, 32, 256), sweeps=1,
                    dtype="f64", precision=0)
    if kind == "mixed":
        return dict(kind="twosite", model="molecular", L=rng.randint(5, 10), D=_log_int(rng, 32, 128), sweeps=2,
                    dtype="f64", precision=1)
    if kind == "c128":
        return dict(kind=rng.choice(["twosite", "singlesite"]), model=model, L=rng.randint(8, 16), D=_log_int(rng, 16, 64),
                    sweeps=1, dtype="c128", precision=0)
    if kind == "singlesite":
        return dict(kind="singlesite", model=model, L=rng.randint(8, 32), D=_log_int(rng, 16, 256), sweeps=2, dtype="f64",
                    precision=0)
    if kind == "energy":
        return dict(kind="energy", model=model, L=rng.randint(8, 40), D=_log_int(rng, 16, 256),
                    dtype=rng.choice(["f64", "c128"]))
    if kind == "localh":
        return dict(kind="localh", D=_log_int(rng, 64, 1024), nsec=rng.choice([21, 31, 41]), Dw=rng.randint(5, 26),
                    precision=rng.choice([0, 0, 1, 3]))
    return dict(kind="svd", m=_log_int(rng, 8, 256), n=_log_int(rng, 8, 256))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------

def _free_chain(c):
    """Release a C chain (MPS or MPO): the site tensors through the library, then the rest."""
    lib = native.lib()
    for i in range(c.nsites if c.a else 0):
        t = c.a[i]
        lib.ctgpu_delete_block_sparse_tensor(C.byref(t))
        t.blocks = None
        t.qnums_blocks = None
        t.qnums_logical = None
        t.axis_dir = None
        t.dim_blocks = None
        t.dim_logical = None
        t.ndim = 0
    cs.free_mps(c)


class _Problem:
    """What a caller holds: the Hamiltonian as a C MPO and the recipe of the start state."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        model, L = case["model"], case["L"]
        self.case = case
        self.mps_seed = int(rng.integers(1, 2**31))
        if model == "xxz":
            # the configuration's coupling at its own size, the stream's couplings elsewhere
            delta = 1.0 if (L, case["D"]) == (20, 32) else float(rng.uniform(0.5, 1.5))
            H, self.d, self.qsite, self.sector = hm.heisenberg_xxz_1d(L, 1.0, delta, 0.0), 2, [1, -1], L % 2
        elif model == "hubbard":
            u = 4.0 if (L, case["D"]) == (32, 256) else float(rng.uniform(1.0, 8.0))
            H, self.d, self.qsite = hm.fermi_hubbard_1d(L, 1.0, u, 0.0), 4, hm.HUBBARD_QSITE
            self.sector = hm.encode_quantum_number_pair(L, L % 2)
        else:
            tkin, vint = wl.molecular_integrals(L, seed)
            H, self.d, self.qsite = hm.spin_molecular(tkin, vint), 4, hm.HUBBARD_QSITE
            self.sector = hm.encode_quantum_number_pair(L, L % 2)
        self.psi0 = None
        if case["dtype"] == "c128":
            m = native.random_mps(L, self.d, self.qsite, self.sector, case["D"], self.mps_seed)
            self.psi0 = wl.complex_gauge(cs.read_mps(m), seed + 1, entry_phases=True)
            _free_chain(m)
            H = wl.complex_gauge(H, seed)
        self.H = H if case["kind"] == "energy" else None
        self.c_mpo = cs.make_c_mpo(H)

    def start(self):
        """A new start state; the search replaces its tensors in place."""
        if self.psi0 is not None:
            return cs.make_c_mps(self.psi0)
        return native.random_mps(self.case["L"], self.d, self.qsite, self.sector, self.case["D"], self.mps_seed)

    def __del__(self):
        c, self.c_mpo = getattr(self, "c_mpo", None), None
        if c is not None:
            _free_chain(c)


class _EnergyProblem(_Problem):
    def __init__(self, case, seed):
        super().__init__(case, seed)
        self.c_mps = self.start()

    def __del__(self):
        c, self.c_mps = getattr(self, "c_mps", None), None
        if c is not None:
            _free_chain(c)
        super().__del__()


class _LocalH:
    """The operands as C tensors, and where the blocks of a result of a's structure lie."""

    def __init__(self, case, seed):
        ops = wl.local_h_microbench(D=case["D"], nsec=case["nsec"], sigma=6.0, Dw=case["Dw"], seed=seed)
        self.case = case
        self.c = []
        for t in ops:
            c = cs.BlockSparseTensor()
            cs.write_bst(t, c)
            self.c.append(c)
        a = ops[0]
        grid = [len(q) for q in a.qnums_blocks]
        self.blocks = [(int(np.ravel_multi_index(i, grid)), int(np.prod(a.block_shape(i)))) for i in a.allowed]

    def __del__(self):
        for c in getattr(self, "c", []):
            native.lib().ctgpu_delete_block_sparse_tensor(C.byref(c))
        self.c = []


def _svd_matrix(case, seed):
    # singular values graded over four decades, as the retained part of a bond's spectrum
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    m, n = case["m"], case["n"]
    k = min(m, n)
    u = torch.linalg.qr(torch.randn(m, k, dtype=torch.float64, device="cuda", generator=g))[0]
    v = torch.linalg.qr(torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g))[0]
    return ((u * torch.logspace(0, -4, k, dtype=torch.float64, device="cuda")) @ v.T).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("twosite", "singlesite"):
        return _Problem(case, seed)
    if kind == "energy":
        return _EnergyProblem(case, seed)
    if kind == "localh":
        return _LocalH(case, seed)
    lib = native.lib()
    lib.ctgpu_dense_svd_noalloc.argtypes = [C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 5
    lib.ctgpu_dense_svd_noalloc.restype = C.c_int
    m, n = case["m"], case["n"]
    k = min(m, n)
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    return dict(case=case, a=_svd_matrix(case, seed), u=new(m, k), s=new(k), vh=new(k, n),
                info=torch.zeros(1, dtype=torch.int32, device="cuda"))


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------

def _search(p):
    case = p.case
    lib = native.lib()
    psi = p.start()
    try:
        if case["kind"] == "singlesite":
            ret, en = native.dmrg_singlesite(p.c_mpo, psi, case["sweeps"], LANCZOS)
            if ret != 0:
                raise RuntimeError(f"dmrg_singlesite: {ret} {native.last_error()}")
            return {"energies": en}
        if case["precision"]:
            lib.ctgpu_set_tc_tile_width(TC_TILE)
        old = native.set_precision(case["precision"])
        ret, en, ent = native.dmrg_twosite(p.c_mpo, psi, case["sweeps"], LANCZOS, TOL, case["D"])
        native.set_precision(old)
        if ret != 0:
            raise RuntimeError(f"dmrg_twosite: {ret} {native.last_error()}")
        sv = [np.sort(native.bond_singular_values(b))[::-1] for b in range(case["L"] - 1)]
        schmidt = np.zeros((len(sv), case["D"]))
        for row, s in zip(schmidt, sv):
            row[:len(s)] = s
        return {"energies": en, "entropies": ent, "bond_dims": np.array([len(s) for s in sv], dtype=np.int64),
                "schmidt": schmidt}
    finally:
        _free_chain(psi)


def run(state):
    if isinstance(state, _EnergyProblem):
        lib = native.lib()
        e, nrm = np.zeros(2 if state.case["dtype"] == "c128" else 1), np.zeros(1)
        if lib.ctgpu_mpo_inner_product(C.byref(state.c_mps), C.byref(state.c_mpo), C.byref(state.c_mps), e.ctypes.data) != 0:
            raise RuntimeError(native.last_error())
        if lib.ctgpu_mps_norm(C.byref(state.c_mps), nrm.ctypes.data) != 0:
            raise RuntimeError(native.last_error())
        return {"energy": e[:1], "norm": nrm}
    if isinstance(state, _Problem):
        return _search(state)
    if isinstance(state, _LocalH):
        lib = native.lib()
        if state.case["precision"]:
            lib.ctgpu_set_tc_tile_width(TC_TILE)
        old = native.set_precision(state.case["precision"])
        out = cs.BlockSparseTensor()
        ret = lib.ctgpu_apply_local_hamiltonian(*[C.byref(c) for c in state.c], C.byref(out))
        native.set_precision(old)
        if ret != 0:
            raise RuntimeError(native.last_error())
        parts = [np.ctypeslib.as_array(C.cast(out.blocks[k].contents.data, C.POINTER(C.c_double)), shape=(n,))
                 for k, n in state.blocks]
        y = np.concatenate(parts)
        lib.ctgpu_delete_block_sparse_tensor(C.byref(out))
        return y
    c = state["case"]
    ret = native.lib().ctgpu_dense_svd_noalloc(state["a"].data_ptr(), c["m"], c["n"], state["u"].data_ptr(),
                                               state["s"].data_ptr(), state["vh"].data_ptr(), state["info"].data_ptr(),
                                               torch.cuda.current_stream().cuda_stream)
    if ret != 0:
        raise RuntimeError("ctgpu_dense_svd_noalloc failed")
    return [state["u"], state["s"], state["vh"], state["info"]]


# ------------------------------------------------------------------------------------------------
# the work a pass cannot do without
# ------------------------------------------------------------------------------------------------

# standard deviation of the bond's charge distribution, in sectors, per conserved quantity
_SIGMA = {"xxz": (1.5,), "hubbard": (1.2, 1.2), "molecular": (1.5, 1.5)}


def _sector_share(sigmas):
    """Share of the entries of a D x D matrix that conserve the charges: sum s_q^2 / D^2 of Gaussian sectors."""
    p = 1.0
    for s in sigmas:
        p *= min(1.0, 1.0 / (2.0 * np.sqrt(np.pi) * s))
    return p


def _local_flops(D, d2, Dw, p):
    """The three block products of one local-Hamiltonian application (d2: local dimension of the vector)."""
    return 2.0 * (2.0 * D**3 * d2 * Dw * p * p) + 2.0 * D**2 * d2 * d2 * Dw * p * 4.0


def _bonds(case):
    """(local problems per sweep) as the bond dimensions min(D, d^i, d^(L-i)) of their bonds."""
    d = 2 if case["model"] == "xxz" else 4
    return d, [min(case["D"], float(d) ** i, float(d) ** (case["L"] - i)) for i in range(case["L"] + 1)]


def _mpo_dim(case, i):
    if case["model"] == "xxz":
        return 5
    if case["model"] == "hubbard":
        return 6
    m = 2 * min(i, case["L"] - i)
    return 2 + 4 * case["L"] + 2 * m * m - m


def work(case):
    kind = case["kind"]
    if kind == "svd":
        m, n = max(case["m"], case["n"]), min(case["m"], case["n"])
        return {"bytes": 8.0 * (m * n + m * n + n * n + n), "flops": 6.0 * m * n * n + 20.0 * n**3}
    if kind == "localh":
        D, Dw = case["D"], case["Dw"]
        p = _sector_share((6.0,))
        return {"bytes": 8.0 * (2 * 16 * D * D + 2 * Dw * D * D) * p, "flops": _local_flops(D, 16, Dw, p)}
    d, b = _bonds(case)
    p = _sector_share(_SIGMA[case["model"]])
    z = 2.0 if case["dtype"] == "c128" else 1.0
    flops = nbytes = 0.0
    for i in range(case["L"]):
        D, Dw = max(b[i], b[i + 1]), _mpo_dim(case, i)
        mps = b[i] * d * b[i + 1] * p
        env = D * D * Dw * p
        step = _local_flops(D, d, Dw, p)
        if kind == "energy":
            flops += z * z * (step + 4 * D**3 * d * p * p)
            nbytes += z * 8.0 * (2 * mps + 2 * env)
            continue
        d2 = d if kind == "singlesite" else d * d
        vec = b[i] * d2 * b[min(i + 2, case["L"]) if kind == "twosite" else i + 1] * p
        per = LANCZOS * _local_flops(D, d2, Dw, p) + step
        split = 20.0 * (D * d) ** 3 * p * p / 4 if kind == "twosite" else 4.0 * D**3 * d * p
        flops += z * z * 2 * case["sweeps"] * (per + split)
        nbytes += z * 8.0 * 2 * case["sweeps"] * (LANCZOS * (2 * vec + 2 * env) + 2 * mps + env)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ------------------------------------------------------------------------------------------------

def _dense(t, dtype):
    out = np.zeros(t.dim_logical, dtype=dtype)
    where = [[np.nonzero(np.asarray(t.qnums_logical[i]) == q)[0] for q in t.qnums_blocks[i]] for i in range(len(t.dim_logical))]
    for idx, blk in t.blocks.items():
        out[np.ix_(*[where[i][j] for i, j in enumerate(idx)])] = blk
    return torch.from_numpy(out).to("cuda" if torch.cuda.is_available() else "cpu")


def _exact_energy(case, seed):
    p = _EnergyProblem(case, seed)
    dtype = np.complex128 if case["dtype"] == "c128" else np.float64
    psi = p.psi0 if p.psi0 is not None else cs.read_mps(p.c_mps)
    e = n = None
    for a, w in zip(psi.tensors, p.H.tensors):
        A, W = _dense(a, dtype), _dense(w, dtype)
        if e is None:
            e = torch.ones(1, 1, 1, dtype=A.dtype, device=A.device)
            n = torch.ones(1, 1, dtype=A.dtype, device=A.device)
        # e[bra, mpo, ket]; W[wl, s (bra), t (ket), wr]
        x = torch.tensordot(e, A, dims=([2], [0]))                     # bra mpo t ket'
        x = torch.tensordot(x, W, dims=([1, 2], [0, 2]))               # bra ket' s wr
        e = torch.tensordot(A.conj(), x, dims=([0, 1], [0, 2])).permute(0, 2, 1).contiguous()
        y = torch.tensordot(n, A, dims=([1], [0]))
        n = torch.tensordot(A.conj(), y, dims=([0, 1], [0, 1]))
    return {"energy": [float(e.real.item())], "norm": [float(np.sqrt(n.real.item()))]}


def _exact_localh(case, seed):
    a, w, l, r = wl.local_h_microbench(D=case["D"], nsec=case["nsec"], sigma=6.0, Dw=case["Dw"], seed=seed)
    A, W, L, R = (_dense(t, np.float64) for t in (a, w, l, r))
    # a[alpha, s, beta], r[beta, wr, beta', 1], w[wl, s', s, wr], l[1, alpha, wl, alpha']
    x = torch.tensordot(A, R[..., 0], dims=([2], [0]))                  # alpha s wr beta'
    x = torch.tensordot(W, x, dims=([2, 3], [1, 2]))                    # wl s' alpha beta'
    y = torch.tensordot(L[0], x, dims=([0, 1], [2, 0])).cpu().numpy()   # alpha' s' beta'
    where = [[np.nonzero(a.qnums_logical[i] == q)[0] for q in a.qnums_blocks[i]] for i in range(3)]
    return np.concatenate([y[np.ix_(*[where[i][j] for i, j in enumerate(idx)])].ravel() for idx in a.allowed])


def exact(case, seed):
    if case["kind"] == "energy":
        v = _exact_energy(case, seed)
        return {k: np.array(x) for k, x in v.items()}
    if case["kind"] == "localh":
        return _exact_localh(case, seed)
    if case["kind"] == "svd":
        # singular vectors have no sign of their own
        return [None, torch.linalg.svdvals(_svd_matrix(case, seed)), None, None]
    return None
