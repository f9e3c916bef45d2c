"""Memory that a context's pool keeps between calls is there for the next
allocation, whoever asks: one that fails is tried again after every pool of the
process has given back what is not in use.  QPGPU_MEMORY_LIMIT bounds what a
context holds, so that the failure can be had without filling the device.

Bars: a call whose staging and what the pool keeps exceed the limit together,
but not without the kept part, runs and gives the unlimited context's bits; it
takes the kept memory of another context too; a call that exceeds the limit by
itself is refused as out of memory and leaves the context usable.
"""
import numpy as np
import pytest

from quantum_package_gb300 import SIGMA_STORED, QPGPUError
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def test_kept_memory_serves_the_next_allocation(monkeypatch):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(1, n_det=5_000)
    n_st = 1000  # 120 MB of staging beside the pool, so that the limit leaves room for the pool of hits
    u = G.random_coefficients(p.n_det, 1, 3).repeat(n_st, axis=0)
    free = Wavefunction.from_problem(p, SIGMA_STORED)
    base = free.info()["device_bytes"]
    ref = free.H_S2_u_0_nstates_openmp(u)
    more = free.info()["device_bytes"] - base
    assert more > 20 * MIB
    monkeypatch.setenv("QPGPU_MEMORY_LIMIT", str(base + more - 8 * MIB))
    wf = Wavefunction.from_problem(p, SIGMA_STORED)
    assert wf.info()["device_bytes"] == base
    got = wf.H_S2_u_0_nstates_openmp(u)
    np.testing.assert_array_equal(got[0], ref[0])
    np.testing.assert_array_equal(got[1], ref[1])
    assert wf.info()["device_bytes"] <= base + more - 8 * MIB + 32 * MIB  # the pool's pages
    assert free.info()["device_bytes"] < base + more  # the other context's pool gave its share
    with pytest.raises(QPGPUError):
        wf.H_S2_u_0_nstates_openmp(u.repeat(8, axis=0))
    v, s = wf.H_S2_u_0_nstates_openmp(u[:3])
    np.testing.assert_array_equal(v, ref[0][:3])
    wf.close()
    free.close()
