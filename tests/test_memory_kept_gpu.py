"""Device memory that a context keeps: what qpgpu_info reports is what the
device has given.

Bars: the reported bytes of a context are those by which the device's free
memory changed, to 4 MiB an allocation of the driver's granularity (2 MiB) for
each of its larger arrays.
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
