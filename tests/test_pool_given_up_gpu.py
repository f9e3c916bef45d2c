"""A determinant set that fits the device is stored, whatever its context held
before: the pool of hits is sized before the pairs are counted, from the
context's last set, and is given up when the pairs do not fit beside it.

The limit (QPGPU_MEMORY_LIMIT) at which a new context, whose estimate leaves no
room for a pool there, just stores the set is found first, in steps of 4 MB.
Bars: at that limit and in steps of 4 MB above it, past the size of the pool, a
context whose last set was hardly connected stores it too, with the same pairs,
elements and sigma; AUTO takes the direct sigma for both or for none.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_AUTO, SIGMA_STORED, QPGPUError
from quantum_package_gb300 import generate as G
from test_pair_build_gpu import _stored_rows

pytestmark = pytest.mark.gpu
STEP = 4_000_000


@pytest.fixture(scope="module")
def space():
    ints = G.make_integrals(9, 11)
    full = G.full_ci_dets(9, 5, 5)  # 15,876 determinants, 560 pairs a row: 142 MB of pairs
    few = np.concatenate([full[:2], full[3000::3000]])
    return ints, full, few


def _make(space, mode, limit, monkeypatch, first=None):
    """The context with the full set, or None when that does not fit the limit."""
    from quantum_package_gb300.sigma import Wavefunction
    ints, full, _ = space
    monkeypatch.setenv("QPGPU_MEMORY_LIMIT", str(limit))
    wf = Wavefunction(9, 5, 5, ints.h, ints.eri, first, mode)
    try:
        wf.set_dets(full)
    except QPGPUError:
        wf.close()
        return None
    return wf


def test_stored_beside_and_without_the_pool(space, monkeypatch):
    ints, full, few = space
    limit = 140_000_000
    while (fresh := _make(space, SIGMA_STORED, limit, monkeypatch)) is None:
        limit += STEP
        assert limit < 400_000_000
    rows = np.arange(0, len(full), 997)
    want = _stored_rows(fresh, rows)
    u = G.random_coefficients(len(full), 1, 4)
    vo, so = Oracle(9, 5, 5, ints.h, ints.eri, full).h_s2_u0_rows(u, rows)
    for extra in range(0, 9):
        wf = _make(space, SIGMA_STORED, limit + extra * STEP, monkeypatch, few)
        assert wf is not None, (limit, extra)
        assert wf.info()["n_pairs"] == fresh.info()["n_pairs"]
        assert wf.info()["n_s2_pairs"] == fresh.info()["n_s2_pairs"]
        for a, b in zip(_stored_rows(wf, rows), want):
            np.testing.assert_array_equal(a, b)
        if extra == 8:  # room for the sigma's own arrays
            v, s = wf.H_S2_u_0_nstates_openmp(u)
            assert np.abs(v[:, rows] - vo).max() <= 1e-12 * np.abs(vo).max()
            assert np.abs(s[:, rows] - so).max() <= 1e-12 * np.abs(so).max()
        wf.close()
    fresh.close()


def test_auto_decides_by_the_set_alone(space, monkeypatch):
    _, _, few = space
    seen = set()
    for limit in range(120_000_000, 240_000_000, 2 * STEP):
        fresh = _make(space, SIGMA_AUTO, limit, monkeypatch)
        wf = _make(space, SIGMA_AUTO, limit, monkeypatch, few)
        assert fresh is not None and wf is not None, limit
        assert fresh.info()["direct_sigma"] == wf.info()["direct_sigma"], limit
        seen.add(wf.info()["direct_sigma"])
        fresh.close()
        wf.close()
    assert seen == {0, 1}
