"""Device memory that a context keeps: what qpgpu_info reports is what the
device has given, and a determinant set that goes gives its memory back.

Bars: the reported bytes of a context are those by which the device's free
memory changed, to 4 MiB an allocation of the driver's granularity (2 MiB) for
each of its larger arrays; after qpgpu_set_integrals drops the set of 2e5
determinants the context holds its integral tables and at most 256 MiB.
"""
import pytest

from quantum_package_gb300 import SIGMA_DIRECT, SIGMA_STORED
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def warm():
    """Kernels loaded and side streams' memory taken before anything is measured."""
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(2, n_det=40_000)
    for mode in (SIGMA_STORED, SIGMA_DIRECT):
        wf = Wavefunction.from_problem(p, mode)
        wf.H_S2_u_0_nstates_openmp(G.random_coefficients(p.n_det, 4, 1))
        wf.close()


@pytest.mark.parametrize("mode", [SIGMA_STORED, SIGMA_DIRECT], ids=["stored", "direct"])
def test_reported_bytes(warm, mode):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(2, n_det=200_000)
    before = _free()
    wf = Wavefunction.from_problem(p, mode)
    held = before - _free()
    assert abs(wf.info()["device_bytes"] - held) <= 64 * MIB, (wf.info()["device_bytes"], held)
    wf.H_S2_u_0_nstates_openmp(G.random_coefficients(p.n_det, 4, 1))
    held = before - _free()
    assert abs(wf.info()["device_bytes"] - held) <= 80 * MIB, (wf.info()["device_bytes"], held)
    wf.close()
    assert before - _free() <= 4 * MIB


def test_new_integrals_give_the_set_back(warm):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(2, n_det=200_000)
    before = _free()
    wf = Wavefunction.from_problem(p, SIGMA_STORED)
    assert before - _free() > 1500 * MIB  # the stored pairs
    wf.set_integrals(p.ints.h, p.ints.eri)
    assert before - _free() <= (256 + 128) * MIB
    wf.close()
