"""Small sets are scanned once: the hits of a set whose warps hold a row each
fit the pool that set-up takes for them, whatever the rows hold.

The phases of a set-up (QPGPU_PROFILE=1) name each pass of the scans.
Bar: one pass, and the oracle's pairs.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_STORED
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 30, 300, 900, 1440, 1800, 3000])
def test_one_pass_of_the_scans(n, monkeypatch, capfd):
    from quantum_package_gb300.sigma import Wavefunction
    # a small space, so that most rows have partners in every class
    ints = G.make_integrals(9, 11)
    full = G.full_ci_dets(9, 5, 5)
    dets = np.ascontiguousarray(full[np.sort(np.random.default_rng(n).permutation(len(full) // 4)[:n])])
    monkeypatch.setenv("QPGPU_PROFILE", "1")
    wf = Wavefunction(9, 5, 5, ints.h, ints.eri, dets, SIGMA_STORED)
    err = capfd.readouterr().err
    assert err.count("pair scans") == 1, err
    I, J, _ = Oracle(9, 5, 5, ints.h, ints.eri, dets).connected_pairs()
    g = wf.connected_pairs()
    np.testing.assert_array_equal(g["I"], I)
    np.testing.assert_array_equal(g["J"], J)
    wf.close()
