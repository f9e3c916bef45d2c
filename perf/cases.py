"""Performance cases of the Davidson sigma library: what a CIPSI / Davidson run asks of it.

Every case goes through the Python mirror of the C ABI (``Wavefunction``,
``Batch``) or, for the dense Davidson blocks that have no mirror, through the
C ABI itself.  Inputs are seeded as in ``quantum_package_gb300.generate``
(aufbau reference plus random excitations of rank 1 to 4, integrals from 120
Cholesky-like factors), drawn on the GPU so that large sets are made quickly.

Kinds (the ``kind`` of a case) and what they stand for:

* ``sigma``      one application of H and S^2: ``host`` arrays as the Fortran
                 caller passes them, ``device`` arrays in determinant order, or
                 the ``bilinear`` layout of the Davidson's own blocks; FP64,
                 FP32 or float-float; pairs stored or enumerated (``direct``);
* ``dets``       a new determinant set (after ``TOUCH psi_det``): index, pairs,
                 elements and diagonal, then the first sigma on it;
* ``davidson``   a whole diagonalisation from a unit guess;
* ``batch``      many small problems diagonalised together;
* ``select``     one CIPSI selection with its second-order energy;
* ``algebra``    the tall-skinny products of the Davidson on the tensor cores.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

N_FACTORS = 120      # factors of (pq|rs) = sum_k L^k_pq L^k_rs
MAX_RANK = 4         # excitation ranks of the drawn determinants
EXACT_DETS = 500_000  # largest set whose exact sigma stays within the time of exact()


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # psi_energy of a small CIPSI stage: launch and copy latency
        _sigma("sigma_host_1e3", 1_000, 30, 8, 8, 1, "host", "fp64"),
        # the Fortran caller's arrays, open shell, a full 64-bit word, odd sizes
        _sigma("sigma_host_65537_open", 65_537, 64, 12, 11, 3, "host", "fp64"),
        # headline workload: 14a+14b in 80 MOs, 1e6 determinants, 4 states
        _sigma("sigma_1e6_fp64", 1_000_000, 80, 14, 14, 4, "device", "fp64"),
        # the mixed-precision Davidson's sigma on a block of 8 vectors
        _sigma("sigma_5e5_fp32", 500_000, 80, 14, 14, 8, "device", "fp32"),
        # a set handled without stored pairs (the path of sets that do not fit)
        _sigma("sigma_direct_2e5", 200_003, 120, 16, 16, 2, "device", "fp64", "direct"),
        # early CIPSI stage: new determinants every iteration
        _dets("dets_5e3", 5_000, 40, 10, 10),
        # late CIPSI stage: the provider rebuild of the headline set
        _dets("dets_1e6", 1_000_000, 80, 14, 14),
        # smallest quoted Davidson (10a+10b in 40 MOs, 1e4 determinants)
        _davidson("davidson_1e4_fp64", 10_000, 40, 10, 10, 1, 4, "fp64"),
        # two states in mixed precision on a mid-size set
        _davidson("davidson_1e5_mixed", 100_000, 60, 12, 12, 2, 6, "fp32"),
        # independent problems of uneven size
        dict(name="batch_16", kind="batch", problems=16, n_lo=1_000, n_hi=30_000, n_diag=4),
        # CIPSI selection: 8 generators, 2,000 selectors of a 2e4 wave function
        _select("select_2e4", 20_000, 80, 14, 14, 8, 2_000, 1_000, 1),
        # Davidson algebra late in a restart cycle: 10 blocks of 8 vectors
        dict(name="algebra_1e6x80", kind="algebra", rows=1_000_000, blocks=10, n_diag=8),
    ]


def _named(name, case):
    return case if name is None else dict(name=name, **case)


def _sigma(name, n_det, n_mo, na, nb, n_st, form, precision, mode="stored"):
    return _named(name, dict(kind="sigma", n_det=n_det, n_mo=n_mo, n_alpha=na, n_beta=nb, n_st=n_st, form=form,
                             precision=precision, mode=mode))


def _dets(name, n_det, n_mo, na, nb):
    return _named(name, dict(kind="dets", n_det=n_det, n_mo=n_mo, n_alpha=na, n_beta=nb))


def _davidson(name, n_det, n_mo, na, nb, n_st, n_diag, precision):
    return _named(name, dict(kind="davidson", n_det=n_det, n_mo=n_mo, n_alpha=na, n_beta=nb, n_st=n_st,
                             n_diag=n_diag, precision=precision))


def _select(name, n_det, n_mo, na, nb, n_gen, n_sel, buf, n_st):
    return _named(name, dict(kind="select", n_det=n_det, n_mo=n_mo, n_alpha=na, n_beta=nb, n_gen=n_gen,
                             n_sel=n_sel, buf=buf, n_st=n_st))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _space(rng):
    n_mo = rng.randint(30, 120)
    nb = rng.randint(6, min(16, n_mo // 3))
    return n_mo, nb + rng.choice([0, 0, 0, 1, 2]), nb


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "dets", "davidson", "batch", "select", "algebra"])
    n_mo, na, nb = _space(rng)
    if kind == "sigma":
        direct = rng.random() < 0.2
        if direct:
            return _sigma(None, _log(rng, 1_000, 200_000), n_mo, na, nb, rng.randint(1, 4), "device", "fp64", "direct")
        form = rng.choice(["host", "device", "bilinear"])
        precision = "fp64" if form == "host" else rng.choice(["fp64", "fp32"] if form == "device" else
                                                             ["fp64", "fp32", "ff"])
        return _sigma(None, _log(rng, 1_000, 700_000), n_mo, na, nb, rng.randint(1, 8), form, precision)
    if kind == "dets":
        return _dets(None, _log(rng, 1_000, 700_000), n_mo, na, nb)
    if kind == "davidson":
        n_st = rng.randint(1, 2)
        return _davidson(None, _log(rng, 1_000, 100_000), n_mo, na, nb, n_st, rng.randint(n_st + 2, 8),
                         rng.choice(["fp64", "fp64", "fp32"]))
    if kind == "batch":
        return dict(kind="batch", problems=rng.randint(3, 16), n_lo=1_000, n_hi=_log(rng, 2_000, 30_000),
                    n_diag=rng.randint(3, 5))
    if kind == "select":
        n_det = _log(rng, 1_000, 20_000)
        n_sel = _log(rng, 50, min(2_000, n_det))
        return _select(None, n_det, rng.randint(30, 80), min(na, 14), min(nb, 14), rng.randint(1, 8), n_sel,
                       _log(rng, 10, 1_000), rng.randint(1, 3))
    return dict(kind="algebra", rows=_log(rng, 10_000, 1_000_000), blocks=rng.randint(1, 10), n_diag=rng.randint(2, 8))


# ---------------------------------------------------------------------------
# Seeded inputs
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, stream):
    g = torch.Generator(device=_dev())
    g.manual_seed((seed * 1_000_003 + stream * 7919) & 0x7FFFFFFFFFFF)
    return g


def _n_int(n_mo):
    return (n_mo - 1) // 64 + 1


def _integrals(n_mo, seed):
    """(h (n, n), packed (pq|rs)) on the device, in FP64."""
    d, g = _dev(), _gen(seed, 0)
    eps = torch.sort(torch.rand(n_mo, generator=g, device=d, dtype=torch.float64) * 4.0 - 2.0).values
    off = torch.triu(torch.randn(n_mo, n_mo, generator=g, device=d, dtype=torch.float64) * 0.02, 1)
    p2 = n_mo * (n_mo + 1) // 2
    L = torch.randn(N_FACTORS, p2, generator=g, device=d, dtype=torch.float64) * 0.05
    full = L.T @ L
    rows, cols = torch.tril_indices(p2, p2, device=d)  # row-major lower triangle: entry r (r + 1) / 2 + c
    return off + off.T + torch.diag(eps), full[rows, cols]


def _string_masks(g, m, n_mo, n_el, rank, kmax):
    """XOR masks (m, n_int) of `rank` random holes and particles of each row."""
    d, n_int = _dev(), _n_int(n_mo)
    k = min(kmax, n_el, n_mo - n_el)
    holes = torch.rand(m, n_el, generator=g, device=d).topk(k, dim=1).indices
    parts = torch.rand(m, n_mo - n_el, generator=g, device=d).topk(k, dim=1).indices + n_el
    use = (torch.arange(k, device=d)[None, :] < rank[:, None]).to(torch.int64)
    out = torch.zeros(m, n_int, dtype=torch.int64, device=d)
    one = torch.ones((), dtype=torch.int64, device=d)
    for pos in (holes, parts):
        bit = torch.bitwise_left_shift(one, pos % 64) * use
        for w in range(n_int):
            out[:, w] ^= (bit * (pos // 64 == w)).sum(1)  # distinct bits: the sum is their union
    return out


def _mix(x):
    """A 64-bit hash of rows of words (int64, wrapping products)."""
    h = torch.zeros(x.shape[0], dtype=torch.int64, device=x.device)
    for w in range(x.shape[1]):
        h = (h ^ x[:, w]) * -7046029254386353131
        h = h ^ ((h >> 29) & 0x7FFFFFFFF)
        h = h * -4658895280553007687
        h = h ^ ((h >> 32) & 0xFFFFFFFF)
    return h


def _first_of_each(words):
    """Indices of the first occurrence of each distinct row, ascending."""
    h = _mix(words)
    _, inverse = torch.unique(h, return_inverse=True)
    first = torch.full((int(inverse.max()) + 1,), words.shape[0], dtype=torch.int64, device=words.device)
    first.scatter_reduce_(0, inverse, torch.arange(words.shape[0], device=words.device), "amin")
    return first.sort().values


def _reference(n_mo, na, nb):
    n_int = _n_int(n_mo)
    ref = np.zeros((2, n_int), np.uint64)
    for s, ne in enumerate((na, nb)):
        for p in range(ne):
            ref[s, p // 64] |= np.uint64(1) << np.uint64(p % 64)
    return torch.from_numpy(ref.view(np.int64).reshape(1, 2 * n_int).copy()).to(_dev())


def _determinants(n_mo, na, nb, n_det, seed):
    """(n_det, 2, n_int) int64 words on the device: reference first, all distinct."""
    d, g = _dev(), _gen(seed, 1)
    ref = _reference(n_mo, na, nb)
    have = ref
    while have.shape[0] < n_det:
        m = max(4096, int(1.4 * (n_det - have.shape[0])))
        r = torch.randint(1, MAX_RANK + 1, (m,), generator=g, device=d)
        ra = (torch.rand(m, generator=g, device=d) * (r + 1)).to(torch.int64).clamp(max=min(na, n_mo - na))
        rb = (r - ra).clamp(max=min(nb, n_mo - nb))
        x = torch.cat([_string_masks(g, m, n_mo, na, ra, MAX_RANK), _string_masks(g, m, n_mo, nb, rb, MAX_RANK)], 1)
        have = torch.cat([have, x ^ ref])
        have = have[_first_of_each(have)]
    return have[:n_det].reshape(n_det, 2, _n_int(n_mo)).contiguous()


def _vectors(n_st, n_det, seed):
    """Normalised columns of a decaying expansion, u_0(sze, N_st)."""
    g = _gen(seed, 2)
    u = torch.randn(n_st, n_det, generator=g, device=_dev(), dtype=torch.float64)
    u *= torch.rand(n_det, generator=g, device=_dev(), dtype=torch.float64).pow(3) + 1e-3
    return u / torch.linalg.vector_norm(u, dim=1, keepdim=True)


def _guess(n_diag, n_det, seed):
    """Unit vector on the reference, Gaussian vectors after it (the reference's random guesses)."""
    u = torch.randn(n_diag, n_det, generator=_gen(seed, 3), device=_dev(), dtype=torch.float64)
    u[0] = 0.0
    u[0, 0] = 1.0
    return u


def _wavefunction(n_mo, na, nb, n_det, seed, direct=False):
    from quantum_package_gb300 import SIGMA_DIRECT, SIGMA_STORED
    from quantum_package_gb300.sigma import Wavefunction
    h, eri = _integrals(n_mo, seed)
    dets = _determinants(n_mo, na, nb, n_det, seed).cpu().numpy().view(np.uint64)
    return Wavefunction(n_mo, na, nb, h.cpu().numpy(), eri.cpu().numpy(), dets,
                        SIGMA_DIRECT if direct else SIGMA_STORED), dets


def _batch_shapes(case):
    """(n_mo, n_el, n_det, n_st) of each problem of a batch, N_det log-uniform; the shapes are the case's own."""
    rng = np.random.default_rng([case["problems"], case["n_hi"]])
    for _ in range(case["problems"]):
        n_mo, ne = int(rng.integers(30, 61)), int(rng.integers(8, 17))
        n_det = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        yield n_mo, ne, n_det, int(rng.integers(1, 3))


def _selection_inputs(case, seed):
    """Sorted wave function (determinants and coefficients fall together) and its denominators."""
    n, n_st = case["n_det"], case["n_st"]
    dets = _determinants(case["n_mo"], case["n_alpha"], case["n_beta"], n, seed)
    g = _gen(seed, 4)
    c = torch.randn(n_st, n, generator=g, device=_dev(), dtype=torch.float64)
    c *= torch.exp(-torch.arange(n, device=_dev(), dtype=torch.float64) / (0.025 * n + 10.0))
    c[:, 0] += 3.0
    order = torch.argsort((c * c).sum(0), descending=True, stable=True)
    c = c[:, order]
    return dets[order].contiguous(), c / torch.linalg.vector_norm(c, dim=1, keepdim=True)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_sigma(case, seed):
    from quantum_package_gb300 import FF, FP32, FP64
    n, n_st = case["n_det"], case["n_st"]
    wf, _ = _wavefunction(case["n_mo"], case["n_alpha"], case["n_beta"], n, seed, case["mode"] == "direct")
    u = _vectors(n_st, n, seed)
    s = {"wf": wf, "precision": {"fp64": FP64, "fp32": FP32, "ff": FF}[case["precision"]]}
    if case["form"] == "host":
        s.update(u=u.cpu().numpy(), run=lambda t: t["wf"].H_S2_u_0_nstates_openmp(t["u"]))
    elif case["form"] == "device":
        s.update(u=u, v=torch.empty_like(u), s=torch.empty_like(u), run=_run_device)
    else:
        order = torch.from_numpy(wf.bilinear_order()).to(_dev()).to(torch.int64)
        ut = u[:, order].T.contiguous()
        s.update(u=ut, u32=ut.to(torch.float32), v=torch.empty_like(ut), s=torch.empty_like(ut), run=_run_bilinear)
    return s


def _run_device(t):
    t["wf"].h_s2_u0_device(t["v"], t["s"], t["u"], precision=t["precision"], stream=torch.cuda.current_stream())
    return t["v"], t["s"]


def _run_bilinear(t):
    t["wf"].sigma_bilinear(t["v"], t["s"], t["u"], t["u32"], precision=t["precision"],
                           stream=torch.cuda.current_stream())
    return t["v"], t["s"]


def _prepare_dets(case, seed):
    from quantum_package_gb300 import SIGMA_STORED
    from quantum_package_gb300.sigma import Wavefunction
    h, eri = _integrals(case["n_mo"], seed)
    dets = _determinants(case["n_mo"], case["n_alpha"], case["n_beta"], case["n_det"], seed)
    wf = Wavefunction(case["n_mo"], case["n_alpha"], case["n_beta"], h.cpu().numpy(), eri.cpu().numpy(),
                      sigma_mode=SIGMA_STORED)
    return {"wf": wf, "dets": dets.cpu().numpy().view(np.uint64), "u": _vectors(1, case["n_det"], seed).cpu().numpy(),
            "run": _run_dets}


def _run_dets(t):
    wf = t["wf"]
    wf.set_dets(t["dets"])
    info = wf.info()
    h, s = wf.diag()
    return (h, s) + wf.H_S2_u_0_nstates_openmp(t["u"]) + (info["n_pairs"], info["n_s2_pairs"])


def _prepare_davidson(case, seed):
    from quantum_package_gb300 import FP32, FP64
    n, n_diag = case["n_det"], case["n_diag"]
    wf, _ = _wavefunction(case["n_mo"], case["n_alpha"], case["n_beta"], n, seed)
    return {"wf": wf, "u": _guess(n_diag, n, seed).cpu().numpy(), "n_st": case["n_st"],
            "precision": FP64 if case["precision"] == "fp64" else FP32, "run": _run_davidson}


def _run_davidson(t):
    r = t["wf"].davidson_diag_hs2(t["u"], t["n_st"], davidson_sze_max=10, threshold=1e-10, s2_eig=False,
                                  precision=t["precision"], max_iter=60)
    k = t["n_st"]
    return r["energies"][:k], r["energies"][k:], r["s2"], r["vectors"]


def _prepare_batch(case, seed):
    from quantum_package_gb300.batch import Batch
    wfs, guesses, n_st = [], [], []
    for j, (n_mo, ne, n, k) in enumerate(_batch_shapes(case)):
        wf, _ = _wavefunction(n_mo, ne, ne, n, seed + 101 * (j + 1))
        wfs.append(wf)
        guesses.append(_guess(case["n_diag"], n, seed + 101 * (j + 1)).cpu().numpy())
        n_st.append(k)
    return {"batch": Batch(wfs), "guesses": guesses, "n_st": n_st, "run": _run_batch}


def _run_batch(t):
    r = t["batch"].davidson(t["guesses"], t["n_st"], threshold=1e-10, max_iter=40)
    return r["energies"], r["s2"], r["vectors"]


def _prepare_select(case, seed):
    from quantum_package_gb300.sigma import Wavefunction
    h, eri = _integrals(case["n_mo"], seed)
    dets, coef = _selection_inputs(case, seed)
    wf = Wavefunction(case["n_mo"], case["n_alpha"], case["n_beta"], h.cpu().numpy(), eri.cpu().numpy(),
                      dets.cpu().numpy().view(np.uint64))
    return {"wf": wf, "coef": coef.cpu().numpy(), "e0": _denominators(case, h, eri).cpu().numpy(),
            "args": (case["n_gen"], case["n_sel"], case["buf"]), "run": _run_select}


def _denominators(case, h, eri):
    """Energies a little below the reference determinant's, one for each state."""
    occ = [_occupation(_reference(case["n_mo"], case["n_alpha"], case["n_beta"]).reshape(1, 2, -1)[:, s],
                       case["n_mo"]) for s in (0, 1)]
    step = torch.arange(case["n_st"], device=h.device, dtype=torch.float64)
    return _Elements(h, eri).diagonal(*occ)[0] - 0.5 + 0.25 * step


def _run_select(t):
    pt2, dets, vals, n_ext = t["wf"].select_pt2(t["coef"], t["e0"], *t["args"])
    return pt2, vals, dets.view(np.int64), n_ext


def _algebra_inputs(case, seed):
    """A basis as the Gram reads it (rows of all columns) and as the update does (blocks), [W S] and y."""
    n, nb, nsd = case["rows"], case["blocks"], case["n_diag"]
    g, kw = _gen(seed, 5), dict(device=_dev(), dtype=torch.float64)
    basis = torch.randn(nb, n, nsd, generator=g, **kw) / math.sqrt(n)
    return {"basis": basis, "rows": basis.permute(1, 0, 2).reshape(n, nb * nsd).contiguous(),
            "ws": torch.randn(n, 2 * nsd, generator=g, **kw), "coef": torch.randn(nb * nsd, nsd, generator=g, **kw)}


def _prepare_algebra(case, seed):
    from quantum_package_gb300.sigma import Wavefunction
    s = _algebra_inputs(case, seed)
    nb, n, nsd = s["basis"].shape
    s.update(wf=Wavefunction(4, 1, 1), gram=torch.empty(nb * nsd, 2 * nsd, device=_dev(), dtype=torch.float64),
             out=torch.empty(n, nsd, device=_dev(), dtype=torch.float64), run=_run_algebra)
    return s


def _run_algebra(t):
    """U^T [W S] of a basis with interleaved columns and U y of the same basis in blocks."""
    from quantum_package_gb300 import _lib
    L, ctx = _lib.load(), t["wf"].ctx
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream or 1)
    nb, n, nsd = t["basis"].shape
    p = {k: C.c_void_p(t[k].data_ptr()) for k in ("basis", "rows", "ws", "coef", "gram", "out")}
    _lib.check(L.qpgpu_gram_tc(ctx, p["rows"], nb * nsd, nb * nsd, p["ws"], 2 * nsd, 2 * nsd, n, p["gram"], stream),
               ctx)
    _lib.check(L.qpgpu_lincomb_tc(ctx, p["basis"], n * nsd, nb * nsd, nsd, p["coef"], p["out"], nsd, n, stream), ctx)
    return t["gram"], t["out"]


_PREPARE = {"sigma": _prepare_sigma, "dets": _prepare_dets, "davidson": _prepare_davidson, "batch": _prepare_batch,
            "select": _prepare_select, "algebra": _prepare_algebra}


# ---------------------------------------------------------------------------
# work: bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _pairs(n_det):
    """About how many directed connected pairs such a set has (measured: 114 a row at 3e3, 990 at 1e6)."""
    return n_det * 12.0 * n_det ** 0.32


def work(case):
    kind = case["kind"]
    if kind == "algebra":
        n, m, k = case["rows"], case["blocks"] * case["n_diag"], case["n_diag"]
        return {"bytes": 8.0 * n * (2 * m + 3 * k), "flops": 2.0 * n * m * 3 * k}
    if kind == "batch":
        n = case["problems"] * (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        p = case["problems"] * _pairs(n / case["problems"])
        return {"bytes": 15 * 12.0 * p, "flops": 15 * 2.0 * p * case["n_diag"]}
    n = case["n_det"]
    det = 16.0 * _n_int(case["n_mo"]) * n
    if kind == "select":
        na, nb, v = case["n_alpha"], case["n_beta"], case["n_mo"]
        ext = case["n_gen"] * (na * (na - 1) // 2 * (v - na) * (v - na - 1) // 2 + nb * (nb - 1) // 2 * (v - nb) *
                               (v - nb - 1) // 2 + na * nb * (v - na) * (v - nb))
        return {"bytes": det + 8.0 * ext, "flops": 0.01 * ext * case["n_sel"] * case["n_st"] * 2.0}
    p = _pairs(n)
    if kind == "dets":
        return {"bytes": det + 16.0 * p + 12.0 * p, "flops": 2.0 * p}
    n_st, sigmas, per_pair = case.get("n_diag", case["n_st"]), 1, {"fp64": 12.0, "fp32": 8.0, "ff": 12.0}[case["precision"]]
    if kind == "davidson":
        sigmas = 18
    elif case["mode"] == "direct":
        per_pair = 0.0
    return {"bytes": sigmas * (det + per_pair * p + 24.0 * n * n_st), "flops": sigmas * 2.0 * p * n_st}


# ---------------------------------------------------------------------------
# exact: the same results in 64 bits from plain torch
# ---------------------------------------------------------------------------
def _occupation(words, n_mo):
    """(N, n_mo) 0/1 int8 of spin strings (N, n_int)."""
    p = torch.arange(n_mo, device=words.device)
    return (torch.bitwise_right_shift(words[:, p // 64], p % 64) & 1).to(torch.int8)


class _Elements:
    """Slater-Condon rules over occupation rows (phases by the orbital order inside each spin)."""

    def __init__(self, h, eri):
        self.h, self.eri, self.n = h, eri, h.shape[0]
        p = torch.arange(self.n, device=h.device)
        a, b = p[:, None], p[None, :]
        self.jj = self.chem(a, a, b, b)
        self.kk = self.chem(a, b, b, a)
        q = p[None, None, :]
        self.coul = self.chem(p[:, None, None], p[None, :, None], q, q)  # (hp|kk)
        self.exch = self.chem(p[:, None, None], q, q, p[None, :, None])  # (hk|kp)

    def chem(self, p, q, r, s):
        pq = torch.minimum(p, q) + torch.maximum(p, q) * (torch.maximum(p, q) + 1) // 2
        rs = torch.minimum(r, s) + torch.maximum(r, s) * (torch.maximum(r, s) + 1) // 2
        return self.eri[torch.minimum(pq, rs) + torch.maximum(pq, rs) * (torch.maximum(pq, rs) + 1) // 2]

    def diagonal(self, oa, ob):
        a, b = oa.to(torch.float64), ob.to(torch.float64)
        t = a + b
        e = t @ torch.diagonal(self.h)
        return e + 0.5 * ((t @ self.jj * t).sum(1) - (a @ self.kk * a).sum(1) - (b @ self.kk * b).sum(1))

    def _moves(self, oi, oj):
        """First and last hole and particle, and the parity of the move, of rows oi -> oj."""
        n, d = self.n, oi - oj
        up = torch.arange(1, n + 1, device=oi.device, dtype=torch.int16)
        down = torch.arange(n, 0, -1, device=oi.device, dtype=torch.int16)
        out, sign = [], torch.zeros(oi.shape[0], dtype=torch.int64, device=oi.device)
        for o, mask in ((oi, d == 1), (oj, d == -1)):
            out += [n - (mask * down).amax(1).to(torch.int64), (mask * up).amax(1).to(torch.int64) - 1]
            below = torch.cumsum(o, 1, dtype=torch.int16) - o
            sign = sign + (below * mask).sum(1)
        return out, 1.0 - 2.0 * (sign % 2).to(torch.float64)

    def pairs(self, ai, bi, aj, bj):
        """(<I|H|J>, <I|S+S-|J>) of rows one or two excitations apart."""
        da, db = ((ai - aj) == 1).sum(1), ((bi - bj) == 1).sum(1)
        hij = torch.zeros(ai.shape[0], dtype=torch.float64, device=ai.device)
        s2 = torch.zeros_like(hij)
        for same, da_, db_, (oi, oj, other) in ((True, 2, 0, (ai, aj, bi)), (True, 0, 2, (bi, bj, ai)),
                                                (False, 1, 0, (ai, aj, bi)), (False, 0, 1, (bi, bj, ai))):
            k = torch.nonzero((da == da_) & (db == db_)).flatten()
            if not len(k):
                continue
            (h1, h2, p1, p2), ph = self._moves(oi[k], oj[k])
            if same:
                hij[k] = ph * (self.chem(h1, p1, h2, p2) - self.chem(h1, p2, h2, p1))
            else:
                occ = oi[k].to(torch.float64)
                mean = ((occ + other[k].to(torch.float64)) * self.coul[h1, p1]).sum(1) - \
                    (occ * self.exch[h1, p1]).sum(1)
                hij[k] = ph * (self.h[h1, p1] + mean)
        k = torch.nonzero((da == 1) & (db == 1)).flatten()
        if len(k):
            (ha, _, pa, _), fa = self._moves(ai[k], aj[k])
            (hb, _, pb, _), fb = self._moves(bi[k], bj[k])
            hij[k] = fa * fb * self.chem(ha, pa, hb, pb)
            s2[k] = torch.where((pa == hb) & (pb == ha), -fa * fb, torch.zeros_like(fa))
        return hij, s2


def _connected(occ_rows, occ_cols, ne):
    """(I, J) of rows and columns one or two excitations apart (both spins)."""
    t = torch.float16 if occ_rows[0].is_cuda else torch.float32
    ov = sum(r.to(t) @ c.to(t).T for r, c in zip(occ_rows, occ_cols))
    return torch.nonzero((ov >= ne - 2) & (ov <= ne - 1), as_tuple=True)


class _Exact:
    """H and S^2 of a determinant set, block of rows by block of rows."""

    def __init__(self, n_mo, na, nb, dets, h, eri):
        self.el, self.ne = _Elements(h, eri), na + nb
        self.occ = [_occupation(dets[:, s], n_mo) for s in (0, 1)]
        self.n = dets.shape[0]

    def diagonal(self):
        return self.el.diagonal(*self.occ), (self.occ[0] > self.occ[1]).sum(1).to(torch.float64)

    def blocks(self):
        """(I, J, h, s2) of all connected pairs, a bounded number at a time."""
        step = max(1, min(self.n, 400_000_000 // self.n))
        for r0 in range(0, self.n, step):
            I, J = _connected([o[r0:r0 + step] for o in self.occ], self.occ, self.ne)
            for k in range(0, len(I), 2_000_000):
                i, j = I[k:k + 2_000_000] + r0, J[k:k + 2_000_000]
                yield (i, j) + self.el.pairs(self.occ[0][i], self.occ[1][i], self.occ[0][j], self.occ[1][j])

    def apply(self, u):
        hd, sd = self.diagonal()
        v, s = hd * u, sd * u
        n_pairs = n_s2 = 0
        for i, j, hij, s2 in self.blocks():
            for st in range(u.shape[0]):
                v[st].index_add_(0, i, hij * u[st, j])
                s[st].index_add_(0, i, s2 * u[st, j])
            n_pairs += len(i)
            n_s2 += int((s2 != 0).sum())
        return v, s, n_pairs, n_s2

    def lowest(self, k, steps=160):
        """Lowest k eigenvalues: Lanczos with full reorthogonalisation, restarted on what it found."""
        found = list(self.blocks())
        I, J, V = (torch.cat([b[q] for b in found]) for q in (0, 1, 2))
        hd = self.diagonal()[0]
        steps = min(steps, self.n)
        start = torch.randn(self.n, generator=_gen(1, 9), device=hd.device, dtype=torch.float64)
        start[torch.argsort(hd)[:4 * k]] += 3.0 * math.sqrt(self.n)
        Q = torch.zeros(steps, self.n, device=hd.device, dtype=torch.float64)
        q, T = start / torch.linalg.vector_norm(start), torch.zeros(steps, steps, dtype=torch.float64)
        for m in range(steps):
            Q[m] = q
            w = (hd * q).index_add_(0, I, V * q[J])
            c = Q[:m + 1] @ w
            w -= c @ Q[:m + 1]
            w -= (Q[:m + 1] @ w) @ Q[:m + 1]
            T[:m + 1, m] = T[m, :m + 1] = c.cpu()
            norm = torch.linalg.vector_norm(w)
            if float(norm) < 1e-11:
                T = T[:m + 1, :m + 1]
                break
            q = w / norm
        return torch.linalg.eigvalsh(T)[:k]


def _bilinear(dets):
    """Beta-major order by bit pattern (unsigned words, the last word leading)."""
    order = torch.arange(dets.shape[0], device=dets.device)
    for s in (0, 1):  # alpha first, then beta: stable sorts, the leading key last
        for w in range(dets.shape[2]):
            key = dets[order, s, w] ^ torch.iinfo(torch.int64).min
            order = order[torch.sort(key, stable=True).indices]
    return order


def exact(case, seed):
    kind = case["kind"]
    if kind == "algebra":
        s = _algebra_inputs(case, seed)
        return s["rows"].T @ s["ws"], s["rows"] @ s["coef"]
    if kind == "select":
        return _exact_select(case, seed)
    if kind == "batch" or case["n_det"] > EXACT_DETS:
        return _exact_diagonal(case, seed) if kind == "dets" else None
    n, shape = case["n_det"], (case["n_mo"], case["n_alpha"], case["n_beta"])
    dets = _determinants(*shape, n, seed)
    x = _Exact(*shape, dets, *_integrals(case["n_mo"], seed))
    if kind == "davidson":
        return x.lowest(case["n_st"]), None, None, None
    u = _vectors(1 if kind == "dets" else case["n_st"], n, seed)
    v, s, n_pairs, n_s2 = x.apply(u)
    if kind == "dets":
        return x.diagonal() + (v, s, n_pairs, n_s2)
    if case["form"] == "bilinear":
        order = _bilinear(dets)
        return v[:, order].T.contiguous(), s[:, order].T.contiguous()
    return v, s


def _exact_diagonal(case, seed):
    shape = (case["n_mo"], case["n_alpha"], case["n_beta"])
    x = _Exact(*shape, _determinants(*shape, case["n_det"], seed), *_integrals(case["n_mo"], seed))
    return x.diagonal() + (None, None, None, None)


def _external(ref, n_mo):
    """Words of every single and double excitation of one determinant (2, n_int)."""
    d, n_int = ref.device, ref.shape[1]
    bit = torch.zeros(n_mo, n_int, dtype=torch.int64, device=d)
    p = torch.arange(n_mo, device=d)
    bit[p, p // 64] = torch.bitwise_left_shift(torch.ones_like(p), p % 64)
    single, double = [], []
    for s in (0, 1):
        occ = _occupation(ref[None, s], n_mo)[0].bool()
        h, q = bit[occ], bit[~occ]
        single.append((h[:, None] ^ q[None, :]).reshape(-1, n_int))
        i, j = torch.triu_indices(len(h), len(h), 1, device=d)
        k, m = torch.triu_indices(len(q), len(q), 1, device=d)
        double.append(((h[i] ^ h[j])[:, None] ^ (q[k] ^ q[m])[None, :]).reshape(-1, n_int))
    z = torch.zeros_like
    rows = [torch.cat([single[0], z(single[0])], 1), torch.cat([z(single[1]), single[1]], 1),
            torch.cat([double[0], z(double[0])], 1), torch.cat([z(double[1]), double[1]], 1)]
    ab = torch.cat([single[0][:, None].expand(-1, len(single[1]), -1),
                    single[1][None].expand(len(single[0]), -1, -1)], 2)
    return torch.cat(rows + [ab.reshape(-1, 2 * n_int)]) ^ ref.reshape(1, -1)


def _exact_select(case, seed):
    h, eri = _integrals(case["n_mo"], seed)
    el, n_mo, ne = _Elements(h, eri), case["n_mo"], case["n_alpha"] + case["n_beta"]
    dets, coef = _selection_inputs(case, seed)
    e0, words = _denominators(case, h, eri), dets.reshape(dets.shape[0], -1)
    ext = torch.cat([_external(dets[k], n_mo) for k in range(case["n_gen"])])
    ext = ext[_first_of_each(ext)]
    ext = ext[~torch.isin(_mix(ext), _mix(words))].reshape(-1, 2, dets.shape[2])
    sel = [_occupation(dets[:case["n_sel"], s], n_mo) for s in (0, 1)]
    c = coef[:, :case["n_sel"]]
    pt2 = torch.zeros(case["n_st"], dtype=torch.float64, device=h.device)
    vals, n_ext = [], 0
    for k in range(0, len(ext), 100_000):
        occ = [_occupation(ext[k:k + 100_000, s], n_mo) for s in (0, 1)]
        I, J = _connected(occ, sel, ne)
        mat = torch.zeros(case["n_st"], len(occ[0]), dtype=torch.float64, device=h.device)
        for q in range(0, len(I), 2_000_000):
            i, j = I[q:q + 2_000_000], J[q:q + 2_000_000]
            hij, _ = el.pairs(occ[0][i], occ[1][i], sel[0][j], sel[1][j])
            for st in range(case["n_st"]):
                mat[st].index_add_(0, i, hij * c[st, j])
        delta = e0[:, None] - el.diagonal(*occ)[None]
        e = 0.5 * (torch.where(delta < 0, -1.0, 1.0) * torch.sqrt(delta * delta + 4.0 * mat * mat) - delta)
        live = (mat != 0).any(0)
        pt2 += e[:, live].sum(1)
        vals.append(e[:, live].amin(0).clamp(max=0.0))
        n_ext += int(live.sum())
    return pt2, torch.cat(vals).sort().values[:case["buf"]], None, n_ext
