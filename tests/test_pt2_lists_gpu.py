"""A generator's second-order energy does not depend on the list it is called
with: the stochastic PT2 asks for its generators batch by batch, and the same
generator in another batch has to give the same bits.  The work of a call is
split over the device by the load of the whole list; the sums may not follow
that split.

Bar: equal bits, for lists of one generator, of some, of all, in another order
and repeated, over items that are cut by the tile and split by their work.
"""
import numpy as np
import pytest

from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_mo,ne,n_det,n_st", [(40, 8, 600, 1), (67, 5, 400, 2), (80, 6, 300, 8)])
def test_a_generators_bits_in_every_list(n_mo, ne, n_det, n_st):
    from quantum_package_gb300.sigma import Wavefunction
    p = G.make_problem(1, n_det=n_det, n_mo=n_mo, n_alpha=ne, n_beta=ne)
    wf = Wavefunction.from_problem(p)
    rng = np.random.default_rng(n_det)
    c = rng.normal(size=(n_st, n_det)) * np.exp(-np.arange(n_det) / 100.0)
    e0 = wf.diag()[0].min() - 1.0 - 0.1 * np.arange(n_st)
    n_sel = n_det * 3 // 4
    gens = [0, 1, 2, 3, 7, 20, 55, 120, n_sel - 1]
    whole = wf.pt2_generators(c, e0, n_sel, gens)
    assert (whole[0] < 0).all()
    for k, g in enumerate(gens):
        np.testing.assert_array_equal(wf.pt2_generators(c, e0, n_sel, [g])[0], whole[k])
    np.testing.assert_array_equal(wf.pt2_generators(c, e0, n_sel, gens[4:]), whole[4:])
    np.testing.assert_array_equal(wf.pt2_generators(c, e0, n_sel, gens[::-1]), whole[::-1])
    np.testing.assert_array_equal(wf.pt2_generators(c, e0, n_sel, [gens[2]] * 5 + gens)[:6], whole[[2] * 5 + [0]])
    np.testing.assert_array_equal(wf.pt2_generators(c, e0, n_sel, range(60))[[0, 1, 2, 3, 7, 20, 55]], whole[:7])
    wf.close()
