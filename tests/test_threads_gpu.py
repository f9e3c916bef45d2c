"""Contexts in threads of one process: every call gives the bits it gives alone.

The problems differ in size and state count, so that their kernels ask for
different amounts of shared memory at the same time.
"""
import threading

import numpy as np
import pytest

from quantum_package_gb300 import FP32
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


def _davidson(p, i):
    from quantum_package_gb300.sigma import Wavefunction
    wf = Wavefunction.from_problem(p)
    n_diag = 4
    u = np.zeros((n_diag, p.n_det))
    u[np.arange(n_diag), np.arange(n_diag)] = 1.0

    def call():
        r = wf.davidson_diag_hs2(u, 2, davidson_sze_max=6 + i, s2_eig=False, threshold=1e-9, precision=FP32,
                                 max_iter=15)
        return r["energies"], r["vectors"]

    return call


def _selection(p, i):
    from quantum_package_gb300.sigma import Wavefunction
    c = G.random_coefficients(p.n_det, 1 + i, 4)
    o = np.argsort(-np.abs(c[0]), kind="stable")
    wf = Wavefunction(p.n_mo, p.n_alpha, p.n_beta, p.ints.h, p.ints.eri, np.ascontiguousarray(p.dets[o]))
    e0 = np.full(1 + i, wf.diag()[0].min() - 0.3)
    c = np.ascontiguousarray(c[:, o])
    return lambda: wf.select_pt2(c, e0, 2, 100, 0)[:1]


@pytest.mark.parametrize("make", [_davidson, _selection], ids=["davidson", "selection"])
def test_calls_side_by_side(make):
    calls = [make(G.make_problem(2, n_det=n, seed=50 + i), i) for i, n in enumerate((700, 3_000, 9_000))]
    want = [f() for f in calls]
    wrong = []

    def run(i):
        try:
            for _ in range(20):
                if not all(np.array_equal(x, y) for x, y in zip(want[i], calls[i]())):
                    wrong.append(f"call {i}: other bits")
        except Exception as e:  # noqa: BLE001 - reported below
            wrong.append(f"call {i}: {e}")

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
