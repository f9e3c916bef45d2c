"""Shapes at which the tensor-core Gram and linear-combination kernels change
course: tiles and chunks that end inside 128 / 32 rows, one tile and several per
block, K steps that end inside 16 columns, blocks of 1 to 16 columns (staged in
16-byte lines, or by the lanes when a block starts between them), all 128
columns, and an operand that starts 8 bytes off a 16-byte line.

Bars: the norm-wise ones of these kernels (a few eps sqrt(m) max|a_r| max|c_j|
for a combination, eps sqrt(N) sum|a b| for a Gram entry) against FP64 products,
whose own rounding is inside them.
"""
import ctypes as C
import math

import numpy as np
import pytest

from quantum_package_gb300 import _lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def wf():
    from quantum_package_gb300.sigma import Wavefunction
    w = Wavefunction(4, 1, 1)
    yield w
    w.close()


@pytest.mark.parametrize("off", [0, 1], ids=["aligned", "off8"])
@pytest.mark.parametrize("N,nb,nsd", [(1, 1, 1), (127, 3, 5), (128, 1, 16), (129, 8, 16), (1000, 128, 1), (999, 64, 2),
                                      (257, 42, 3), (4097, 9, 7), (385, 2, 12), (1001, 8, 4), (40_001, 18, 7),
                                      (60_000, 16, 8)])
def test_lincomb_shapes(wf, N, nb, nsd, off):
    import torch
    rng = np.random.default_rng(N + 7 * nb + nsd)
    A = rng.normal(size=(nb, N, nsd)) * np.exp(rng.uniform(-9, 0, size=(nb, N, 1)))
    A[:, N // 2] = 0.0
    Cm = rng.normal(size=(nb * nsd, nsd)) * np.exp(rng.uniform(-5, 0, size=(1, nsd)))
    buf = torch.zeros(A.size + off + 1, dtype=torch.float64, device="cuda")
    buf[off:off + A.size] = torch.from_numpy(A.ravel()).cuda()
    out = torch.full((N + 2, nsd + off), float("nan"), dtype=torch.float64, device="cuda")
    dC = torch.from_numpy(Cm).cuda()
    L = _lib.load()
    rc = L.qpgpu_lincomb_tc(wf.ctx, C.c_void_p(buf.data_ptr() + 8 * off), N * nsd, nb * nsd, nsd,
                            C.c_void_p(dC.data_ptr()), C.c_void_p(out.data_ptr()), nsd + off, N, None)
    _lib.check(rc, wf.ctx)
    O = out.cpu().numpy()
    rows = np.concatenate(list(A), axis=1)
    bar = 16 * EPS * math.sqrt(nb * nsd) * np.outer(np.abs(rows).max(1), np.abs(Cm).max(0))
    assert (np.abs(O[:N, :nsd] - rows @ Cm) <= bar).all()
    assert np.isnan(O[N:]).all() and np.isnan(O[:, nsd:]).all()  # nothing else is written


@pytest.mark.parametrize("N,m,n", [(1, 1, 1), (31, 2, 3), (33, 97, 1), (129, 128, 16), (4095, 65, 9), (20_001, 31, 2),
                                   (152 * 32 + 1, 80, 16)])
def test_gram_shapes(wf, N, m, n):
    import torch
    rng = np.random.default_rng(N + m)
    A = rng.normal(size=(N, m)) * np.exp(rng.uniform(-9, 0, size=(1, m)))
    B = rng.normal(size=(N, n)) * np.exp(rng.uniform(-5, 2, size=(1, n)))
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    X = torch.empty((m, n), dtype=torch.float64, device="cuda")
    L = _lib.load()
    _lib.check(L.qpgpu_gram_tc(wf.ctx, C.c_void_p(dA.data_ptr()), m, m, C.c_void_p(dB.data_ptr()), n, n, N,
                               C.c_void_p(X.data_ptr()), None), wf.ctx)
    bar = 8 * EPS * math.sqrt(N) * (np.abs(A).T @ np.abs(B))
    assert (np.abs(X.cpu().numpy() - A.T @ B) <= bar).all()
