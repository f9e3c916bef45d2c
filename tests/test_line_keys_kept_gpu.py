"""qpgpu_set_line_keys takes effect at the next qpgpu_set_dets: the tables of
the set in hand, which the direct sigma probes at every call, keep the hash bits
that they were built with.

Bar: equal bits of the direct sigma before and after the call, for fewer and
for more bits than the tables have, and the oracle's values (1e-12); the new
bits hold from the next set on.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_DIRECT
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,n", [(1, 3000), (2, 3000)], ids=["nint1", "nint2"])
@pytest.mark.parametrize("bits,later", [(64, 6), (6, 64)])
def test_the_set_in_hand_keeps_its_tables(cfg, n, bits, later):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(cfg, n_det=n)
    wf = Wavefunction.from_problem(p, sigma_mode=SIGMA_DIRECT, line_keys=(0, 0, bits))
    u = G.random_coefficients(n, 2, p.seed)
    v, s = wf.H_S2_u_0_nstates_openmp(u)
    wf.set_line_keys(0, 0, later)
    v2, s2 = wf.H_S2_u_0_nstates_openmp(u)
    np.testing.assert_array_equal(v2, v)
    np.testing.assert_array_equal(s2, s)
    vo, so = Oracle.from_problem(p).h_s2_u0(u)
    wf.set_dets(p.dets)
    for got in (wf.H_S2_u_0_nstates_openmp(u), (v, s)):
        assert np.abs(got[0] - vo).max() <= 1e-12 * np.abs(vo).max()
        assert np.abs(got[1] - so).max() <= 1e-12 * np.abs(so).max()
    wf.close()
