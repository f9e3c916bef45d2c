"""Direct sigma of rows that are summed in several stretches of 2,048 pairs, and
of sets large enough that the pair scans run side by side.

Bars: v and s of the longest rows within 1e-12 relative of the oracle, for rows
that end just before, at and after a stretch and for one to eight states; a set
of 33,000 determinants within 1e-12 of the stored pairs; every call of a set
gives the same bits.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_DIRECT, SIGMA_STORED
from quantum_package_gb300 import generate as G
from test_pair_build_gpu import _star

pytestmark = pytest.mark.gpu

REL64 = 1e-12  # the bar of the FP64 sigma


@pytest.mark.parametrize("n_mo", [30, 70])
@pytest.mark.parametrize("m,n_st", [(2047, 1), (2048, 2), (2049, 3), (4097, 8), (6000, 5)])
def test_rows_of_several_stretches(n_mo, m, n_st):
    from quantum_package_gb300.sigma import Wavefunction
    ne = 8
    ints = G.make_integrals(n_mo, 5)
    dets = _star(n_mo, ne, m, 23 + m)
    wf = Wavefunction(n_mo, ne, ne, ints.h, ints.eri, dets, SIGMA_DIRECT)
    assert wf.info()["direct_sigma"] == 1 and wf.info()["n_split_rows"] == 0
    o = Oracle(n_mo, ne, ne, ints.h, ints.eri, dets)
    u = G.random_coefficients(m + 1, n_st, 3)
    rows = np.unique(np.array([0, 1, m // 2, m]))
    v, s = wf.H_S2_u_0_nstates_openmp(u)
    vo, so = o.h_s2_u0_rows(u, rows)
    assert np.abs(v[:, rows] - vo).max() <= REL64 * np.abs(vo).max()
    assert np.abs(s[:, rows] - so).max() <= REL64 * max(1.0, np.abs(so).max())
    v2, s2 = wf.H_S2_u_0_nstates_openmp(u)
    np.testing.assert_array_equal(v, v2)
    np.testing.assert_array_equal(s, s2)


@pytest.mark.parametrize("cfg", [1, 2])
def test_scans_side_by_side(cfg):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(cfg, n_det=33_000)
    u = G.random_coefficients(p.n_det, 2, p.seed)
    vs, ss = Wavefunction.from_problem(p, sigma_mode=SIGMA_STORED).H_S2_u_0_nstates_openmp(u)
    wf = Wavefunction.from_problem(p, sigma_mode=SIGMA_DIRECT)
    for _ in range(2):
        v, s = wf.H_S2_u_0_nstates_openmp(u)
        assert np.abs(v - vs).max() <= REL64 * np.abs(vs).max()
        assert np.abs(s - ss).max() <= REL64 * np.abs(ss).max()
