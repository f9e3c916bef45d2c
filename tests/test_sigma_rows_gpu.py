"""FP64 sigma rows on the GPU: S^2 lists from one to more than 32 partners, any
number of states, host arrays on both sides of the limit up to which they go
through pinned memory, padded host columns.

The oracle's sigma is met within 1e-12 relative (the sums of a row run in
another order); the routes of the same call (host arrays, device arrays,
bilinear rows) share the kernel and agree bit for bit.
"""
import numpy as np
import pytest

from oracle import Oracle
from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu

REL64 = 1e-12


def _flip_set(n_mo=14, n=6, extra=0, seed=3):
    """alpha in 0..5, beta in 6..11, its 36 spin flips and `extra` random determinants."""
    a0, b0 = (1 << n) - 1, ((1 << n) - 1) << n
    out = {(a0, b0)}
    for i in range(n):
        for j in range(n, 2 * n):
            out.add((a0 ^ (1 << i) ^ (1 << j), b0 ^ (1 << i) ^ (1 << j)))
    rng = np.random.default_rng(seed)
    while len(out) < 1 + n * n + extra:
        w = [sum(1 << int(k) for k in rng.choice(n_mo, n, replace=False)) for _ in range(2)]
        out.add((w[0], w[1]))
    order = rng.permutation(len(out))
    d = np.array(sorted(out), dtype=np.uint64)[order]
    return d[:, :, None]


@pytest.fixture(scope="module", params=[0, 4000], ids=["flips", "flips_and_random"])
def flips(request):
    from quantum_package_gb300.sigma import Wavefunction
    ints = G.make_integrals(14, 9)
    dets = _flip_set(extra=request.param)
    return Wavefunction(14, 6, 6, ints.h, ints.eri, dets), Oracle(14, 6, 6, ints.h, ints.eri, dets), len(dets)


@pytest.mark.parametrize("n_st", [1, 2, 3, 4, 5, 6, 7, 8, 11])
def test_rows(flips, n_st):
    import torch
    wf, oracle, n = flips
    u = np.random.default_rng(n_st).normal(size=(n_st, n))
    vo, so = oracle.h_s2_u0(u)
    v, s = wf.H_S2_u_0_nstates_openmp(u)
    assert np.abs(v - vo).max() <= REL64 * np.abs(vo).max()
    assert np.abs(s - so).max() <= REL64 * np.abs(so).max()
    ut = torch.from_numpy(u).cuda()
    vd, sd = torch.empty_like(ut), torch.empty_like(ut)
    wf.h_s2_u0_device(vd, sd, ut)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(vd.cpu().numpy(), v)
    np.testing.assert_array_equal(sd.cpu().numpy(), s)
    if n_st <= 8:
        order = wf.bilinear_order()
        ub = ut[:, torch.from_numpy(order).long().cuda()].T.contiguous()
        vb, sb = torch.empty_like(ub), torch.empty_like(ub)
        wf.sigma_bilinear(vb, sb, ub)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(vb.cpu().numpy().T, v[:, order])
        np.testing.assert_array_equal(sb.cpu().numpy().T, s[:, order])


@pytest.mark.parametrize("n_st", [1, 3, 8])
def test_padded_columns_and_nan(flips, n_st):
    import ctypes as C

    from quantum_package_gb300 import QPGPUError, _lib
    wf, _, n = flips
    u = np.random.default_rng(20 + n_st).normal(size=(n_st, n))
    v, s = wf.H_S2_u_0_nstates_openmp(u)
    ld = n + 3
    up, vp, sp = (np.full((n_st, ld), 7.0) for _ in range(3))
    up[:, :n] = u
    ptr = [x.ctypes.data_as(C.c_void_p) for x in (vp, sp, up)]
    assert _lib.load().qpgpu_h_s2_u0(wf.ctx, *ptr, n_st, ld) == 0
    np.testing.assert_array_equal(vp[:, :n], v)
    np.testing.assert_array_equal(sp[:, :n], s)
    assert (vp[:, n:] == 7.0).all() and (sp[:, n:] == 7.0).all()
    u[n_st - 1, n // 2] = np.nan
    with pytest.raises(QPGPUError, match="NaN"):
        wf.H_S2_u_0_nstates_openmp(u)
    u[n_st - 1, n // 2] = 0.0
    wf.H_S2_u_0_nstates_openmp(u)  # the flag does not outlive its call
