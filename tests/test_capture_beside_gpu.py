"""Calls that free or replace a determinant set beside other work of the process.

A graph that another thread captures (thread-local mode) survives them, and a
sigma in flight on the caller's stream reads its set to the end.  The graph's
values and the sigma's bits are exact.
"""
import threading

import numpy as np
import pytest

from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


def _calls(p):
    from quantum_package_gb300.sigma import Wavefunction
    wf = Wavefunction.from_problem(p)
    u = G.random_coefficients(p.n_det, 2, 3)

    def made_and_closed():
        w = Wavefunction.from_problem(p)
        w.H_S2_u_0_nstates_openmp(u)
        w.close()

    return {"set_dets": lambda: wf.set_dets(p.dets),
            "set_integrals": lambda: wf.set_integrals(p.ints.h, p.ints.eri),
            "context": made_and_closed,
            "memory given back": lambda: _short_of_memory(p)}


def _short_of_memory(p):
    """An allocation that fails under the limit is tried again after the pools gave back."""
    import os
    from quantum_package_gb300 import QPGPUError
    from quantum_package_gb300.sigma import Wavefunction
    os.environ["QPGPU_MEMORY_LIMIT"] = str(1 << 20)
    try:
        with pytest.raises(QPGPUError):
            Wavefunction.from_problem(p)
    finally:
        del os.environ["QPGPU_MEMORY_LIMIT"]


@pytest.mark.parametrize("name", ["set_dets", "set_integrals", "context", "memory given back"])
def test_capture_on_another_thread(name):
    import torch
    call = _calls(G.make_problem(2, n_det=3_000))[name]
    x = torch.arange(1000, device="cuda", dtype=torch.float64)
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    failed = []

    def run():
        try:
            call()
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin(capture_error_mode="thread_local")
        y.copy_(x * 2)
        t = threading.Thread(target=run)
        t.start()
        t.join()
        y.add_(1)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert not failed, failed
    assert torch.equal(y, 2 * x + 1)


def test_set_replaced_behind_a_sigma_in_flight():
    import torch
    from quantum_package_gb300 import FP64
    from quantum_package_gb300.sigma import Wavefunction
    p, q = G.make_problem(2, n_det=20_000), G.make_problem(2, n_det=30_000, seed=9)
    wf = Wavefunction.from_problem(p)
    u = torch.from_numpy(np.ascontiguousarray(G.random_coefficients(p.n_det, 4, 1))).cuda()
    want = [torch.empty_like(u) for _ in range(2)]
    got = [torch.empty_like(u) for _ in range(2)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    wf.h_s2_u0_device(*want, u, precision=FP64, stream=stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # about 50 ms before the sigma starts
    wf.h_s2_u0_device(*got, u, precision=FP64, stream=stream)
    assert not stream.query()
    wf.set_dets(q.dets)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
