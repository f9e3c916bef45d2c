"""The coupling feature of a determinant, log10(sum_J H_IJ^2) / 4, which the
set-up forms with the stored elements (csrc/pairs.cu: one sum per row, rows of
more than 2,048 pairs from the sums of their stretches) and the learned step of
the Davidson reads.

No entry point returns it, so the network here is made to return it: weights
that pass feature 4 through both GELU layers in their linear range, so that the
step is (A f + 1) d for the diagonal correction d, with one rounding, that of
A f + 16 to FP32 (A is a power of two, the offset comes off exactly).  After two applications of
sigma the vector is a combination of the guess and that step (the second basis
vector is the step orthonormalised against the guess); both coefficients are
fitted over all rows, and every row has to agree.

Bar: the network runs in FP32 on numbers near 16 (the offset that keeps GELU
linear): 8 roundings of 2^-20 each in A f + 1, hence 8e-6 |d| of a row, doubled
for the fit.  A sum that misses a stretch of the reference's row moves A f by
more than 0.1 there.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_STORED, _lib
from quantum_package_gb300 import generate as G
from test_pair_build_gpu import _star

pytestmark = pytest.mark.gpu

A, OFFSET, BAR = 8.0, 16.0, 1.6e-5


def _pass_feature_4():
    w = np.zeros(_lib.MLP_NPARAM, np.float32)
    b1, w2 = 64 * 8, 64 * 8 + 64
    b2 = w2 + 64 * 64
    w3, b3 = b2 + 64, b2 + 128
    w[4] = A           # W1[0][4]
    w[b1] = OFFSET
    w[w2] = 1.0        # W2[0][0]
    w[w3] = 1.0
    w[b3] = 1.0 - OFFSET
    return w


@pytest.mark.parametrize("n_mo,m", [(30, 40), (30, 2048), (30, 2049), (30, 4096), (30, 4097), (30, 9000), (70, 4500)])
def test_coupling_feature_of_rows_of_one_and_several_stretches(n_mo, m):
    from quantum_package_gb300.sigma import Wavefunction
    ne = 8
    ints = G.make_integrals(n_mo, 5)
    dets = _star(n_mo, ne, m, 23 + m)
    n = m + 1
    wf = Wavefunction(n_mo, ne, ne, ints.h, ints.eri, dets, SIGMA_STORED)
    assert (wf.info()["n_split_rows"] > 0) == (m > 2048)
    o = Oracle(n_mo, ne, ne, ints.h, ints.eri, dets)
    g = wf.connected_pairs()  # the elements themselves are held to the oracle's elsewhere
    f = (np.log10(np.bincount(g["I"], weights=g["hij"] ** 2, minlength=n) + 1e-30) * 0.25).astype(np.float32)
    wf.mlp_init(seed=1)
    wf.mlp_set_weights(_pass_feature_4())
    u = np.random.default_rng(m).normal(size=n)
    u /= np.linalg.norm(u)
    r = wf.davidson_diag_hs2(u[None], n_states=1, threshold=1e-30, s2_eig=False, preconditioner=1, max_iter=2)
    assert r["n_sigma"] == 2
    W, S = (x[0] for x in o.h_s2_u0(u[None]))
    h = np.asarray(o.diag()[0])
    lam, s2 = u @ W, u @ S
    d = (lam * u - W) * (1.0 + s2 * u - S) / np.maximum(h - lam, 1e-2)
    y = (np.float32(A) * f + np.float32(OFFSET)).astype(np.float64) + (1.0 - OFFSET)
    step = y * d
    v = r["vectors"][0]
    M = np.stack([u, step], axis=1)
    c, *_ = np.linalg.lstsq(M, v, rcond=None)
    assert abs(c[1]) > 1e-6
    assert (np.abs(v - M @ c) <= BAR * abs(c[1]) * (np.abs(d) + np.abs(d).max() * 1e-3)).all()
    wf.close()
