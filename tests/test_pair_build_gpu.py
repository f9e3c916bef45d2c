"""Building the stored pairs: the one-pass scans, the per-row sort and the pool
that holds the hits in between, at the sizes where they change course.

Bars: the pairs of the checked rows and their FP64 elements equal the oracle's
bit for bit and stand in ascending bilinear order, for rows of every length at
which the sort takes another path (a warp's registers, blocks of 2 to 16 warps,
the segmented sort); a set whose hits do not fit the pool (sized from the
context's previous set) gives the same pairs and sigma as a fresh context; a
set replaced while a sigma of the old one is in flight on another stream leaves
that sigma untouched.  Deletion-key groups of every length at which they are
read another way, and rows that outgrow their chunks of the pool, give the
oracle's pairs.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import SIGMA_STORED, _lib
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu

REL64 = 1e-12  # the bar of the FP64 sigma


def _star(n_mo, ne, m, seed):
    """The reference and m of its single and double excitations: row 0 holds exactly m pairs."""
    ref = G.reference_det(n_mo, ne, ne)
    found = {ref.tobytes(): ref}
    rng = np.random.default_rng(seed)
    while len(found) <= m:
        k = 4 * (m + 1 - len(found)) + 64
        r = rng.integers(1, 3, k)
        ra = rng.integers(0, r + 1)
        xa = G._random_excitations(rng, k, n_mo, ne, ra, ref.shape[1])
        xb = G._random_excitations(rng, k, n_mo, ne, r - ra, ref.shape[1])
        for a, b in zip(xa, xb):
            d = ref ^ np.stack([a, b])
            found.setdefault(d.tobytes(), d)
            if len(found) > m:
                break
    return np.ascontiguousarray(np.stack(list(found.values())))


def _stored_rows(wf, rows):
    """Records of the rows in stored order: (I, J, hij)."""
    L = _lib.load()
    r = np.ascontiguousarray(rows, np.int32)
    n = C.c_int64()
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    _lib.check(L.qpgpu_connected_pairs_rows(wf.ctx, p(r), len(r), C.byref(n), None, None, None, None, None, None, 0),
               wf.ctx)
    P = n.value
    I, J, cls, ph = np.empty(P, np.int32), np.empty(P, np.int32), np.empty(P, np.int8), np.empty(P, np.int8)
    exc, hij = np.empty((P, 4), np.int16), np.empty(P)
    _lib.check(L.qpgpu_connected_pairs_rows(wf.ctx, p(r), len(r), C.byref(n), p(I), p(J), p(cls), p(ph), p(exc),
                                            p(hij), P), wf.ctx)
    return I, J, hij


@pytest.mark.parametrize("n_mo,m", [(30, m) for m in (1, 31, 32, 33, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048,
                                                      2049, 4096, 4097, 8192, 8193, 16384, 16385, 20000)] +
                         [(70, 33), (70, 1025), (70, 4097), (70, 17000)])
def test_rows_of_every_sort_path(n_mo, m):
    from quantum_package_gb300.sigma import Wavefunction
    ne = 8
    ints = G.make_integrals(n_mo, 5)
    dets = _star(n_mo, ne, m, 17 + m)
    wf = Wavefunction(n_mo, ne, ne, ints.h, ints.eri, dets, SIGMA_STORED)
    o = Oracle(n_mo, ne, ne, ints.h, ints.eri, dets)
    pos = np.empty(m + 1, np.int64)
    pos[wf.bilinear_order()] = np.arange(m + 1)
    rows = np.unique(np.array([0, 1, m // 2, m]))
    I, J, hij = _stored_rows(wf, rows)
    assert (I == 0).sum() == m
    for k in rows:
        assert (np.diff(pos[J[I == k]]) > 0).all()
    order = np.lexsort((J, I))
    Io, Jo, cls = o.connected_pairs_rows(rows)
    np.testing.assert_array_equal(I[order], Io)
    np.testing.assert_array_equal(J[order], Jo)
    np.testing.assert_array_equal(hij[order], o.pair_excitations(Io, Jo, cls)[2])
    u = G.random_coefficients(m + 1, 2, 3)
    v, s = wf.H_S2_u_0_nstates_openmp(u)
    vo, so = o.h_s2_u0_rows(u, rows)
    assert np.abs(v[:, rows] - vo).max() <= REL64 * np.abs(vo).max()
    assert np.abs(s[:, rows] - so).max() <= REL64 * max(1.0, np.abs(so).max())


def test_hits_beyond_the_pool():
    from quantum_package_gb300.sigma import Wavefunction
    ints = G.make_integrals(9, 11)
    full = G.full_ci_dets(9, 5, 5)  # 15,876 determinants, 560 pairs a row
    few = np.concatenate([full[:2], full[3000::3000]])  # hardly connected: a small pool next
    wf = Wavefunction(9, 5, 5, ints.h, ints.eri, few, SIGMA_STORED)
    assert 0 < wf.info()["n_pairs"] <= 12
    wf.set_dets(full)
    fresh = Wavefunction(9, 5, 5, ints.h, ints.eri, full, SIGMA_STORED)
    assert wf.info()["n_pairs"] == fresh.info()["n_pairs"]
    assert wf.info()["n_s2_pairs"] == fresh.info()["n_s2_pairs"]
    rows = np.arange(0, len(full), 997)
    for a, b in zip(_stored_rows(wf, rows), _stored_rows(fresh, rows)):
        np.testing.assert_array_equal(a, b)
    u = G.random_coefficients(len(full), 1, 4)
    o = Oracle(9, 5, 5, ints.h, ints.eri, full)
    vo, so = o.h_s2_u0_rows(u, rows)
    for w in (wf, fresh):
        v, s = w.H_S2_u_0_nstates_openmp(u)
        assert np.abs(v[:, rows] - vo).max() <= REL64 * np.abs(vo).max()
        assert np.abs(s[:, rows] - so).max() <= REL64 * np.abs(so).max()


def test_set_replaced_under_a_running_sigma():
    import torch
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(2, n_det=40_000)
    q = G.make_problem(2, n_det=50_000)
    wf = Wavefunction.from_problem(p, SIGMA_STORED)
    u = torch.from_numpy(G.random_coefficients(p.n_det, 4, 5)).cuda()
    ref, v, s = torch.empty_like(u), torch.empty_like(u), torch.empty_like(u)
    wf.h_s2_u0_device(ref, s, u)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(20):  # about 10 ms of sigma queued when the set goes
        wf.h_s2_u0_device(v, s, u, stream=side)
    wf.set_dets(q.dets)
    torch.cuda.synchronize()
    assert torch.equal(v, ref)


def _all_pairs_match(wf, o):
    I, J, cls = o.connected_pairs()
    g = wf.connected_pairs()
    np.testing.assert_array_equal(g["I"], I)
    np.testing.assert_array_equal(g["J"], J)
    np.testing.assert_array_equal(g["cls"], cls)
    np.testing.assert_array_equal(g["hij"], o.pair_excitations(I, J, cls)[2])


@pytest.mark.parametrize("spin", [0, 1])
@pytest.mark.parametrize("n_mo,bits", [(30, 64), (70, 64), (30, 3)])
@pytest.mark.parametrize("m", [62, 63, 64, 127, 128, 129, 200])
def test_key_groups_of_every_length(m, n_mo, bits, spin):
    """m strings that share a deletion key with the reference's: the group is read
    in whole steps from 64 members on (m + 1 with the reference's own), four at a time."""
    from quantum_package_gb300.sigma import Wavefunction
    ne = 4
    ref = G.reference_det(n_mo, ne, ne)
    two = [(p, q) for p in range(ne, n_mo) for q in range(p + 1, n_mo)]
    pick = np.random.default_rng(m).permutation(len(two))[:m]
    dets = np.repeat(ref[None], m + 1, axis=0)
    for k, t in enumerate(pick):
        s = 0b0011  # two electrons of the reference stay
        for p in two[t]:
            s |= 1 << p
        for w in range(ref.shape[1]):
            dets[k + 1, spin, w] = (s >> (64 * w)) & 0xFFFFFFFFFFFFFFFF
    ints = G.make_integrals(n_mo, 5)
    wf = Wavefunction(n_mo, ne, ne, ints.h, ints.eri, dets, SIGMA_STORED, line_keys=(0, 0, bits))
    _all_pairs_match(wf, Oracle(n_mo, ne, ne, ints.h, ints.eri, dets))


@pytest.mark.parametrize("n_mo", [30, 70])
def test_rows_that_outgrow_their_chunks(n_mo):
    """Chunks sized from a set that is hardly connected: the star's rows move to larger ones."""
    from quantum_package_gb300.sigma import Wavefunction
    ne, m = 8, 3000
    ints = G.make_integrals(n_mo, 5)
    dets = _star(n_mo, ne, m, 41)
    wf = Wavefunction(n_mo, ne, ne, ints.h, ints.eri, dets[:2], SIGMA_STORED, line_keys=(0, 0, 64))
    wf.set_dets(dets)
    _all_pairs_match(wf, Oracle(n_mo, ne, ne, ints.h, ints.eri, dets))
