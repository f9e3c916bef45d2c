"""The per-phase timeline of a Davidson run (QPGPU_PROFILE=1).

Orthonormalising a block of 8 vectors against up to 9 others takes dozens of
FP64 operations an element and several passes, the step and its norms a dozen
in one: at 1e5 determinants the first phase is the longer one by any count.
"""
import re

import numpy as np
import pytest

from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


def test_orthonormalisation_is_not_charged_to_the_step(monkeypatch, capfd):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(2, n_det=100_000)
    monkeypatch.setenv("QPGPU_PROFILE", "1")
    wf = Wavefunction.from_problem(p)
    u = np.zeros((8, p.n_det))
    u[np.arange(8), np.arange(8)] = 1.0
    wf.davidson_diag_hs2(u, 4, davidson_sze_max=10, threshold=1e-14, s2_eig=False, max_iter=30)
    capfd.readouterr()
    wf.davidson_diag_hs2(u, 4, davidson_sze_max=10, threshold=1e-14, s2_eig=False, max_iter=30)
    err = capfd.readouterr().err
    ms = {m[0].strip(): float(m[1]) for m in re.findall(r"\[qpgpu davidson\] (.{16})\s+([0-9.]+) ms", err)}
    assert ms["orthonormalise"] > ms["step + norms"], ms
    wf.close()
