"""A batch whose problems' determinants or integrals were set again after it was
made is refused: its arrays have gone back to the contexts' pools.

Bar: the error is a state error that names the reason, the batch made anew
solves the new sets to the single-problem energies (1e-9 Ha), and other members
are not disturbed.
"""
import numpy as np
import pytest

from quantum_package_gb300 import generate as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["dets", "same dets", "integrals"])
def test_a_batch_of_replaced_sets_is_refused(what):
    from quantum_package_gb300.batch import Batch, BatchError
    from quantum_package_gb300.sigma import Wavefunction
    probs = [G.make_problem(1, n_det=n) for n in (900, 1200)]
    wfs = [Wavefunction.from_problem(p) for p in probs]
    guess = lambda n: np.random.default_rng(n).normal(size=(2, n))  # noqa: E731
    kw = dict(n_states=[1, 1], threshold=1e-12)
    b = Batch(wfs)
    first = b.davidson([guess(900), guess(1200)], **kw)
    new = G.make_problem(1, n_det=1000).dets if what == "dets" else probs[1].dets
    if what == "integrals":
        wfs[1].set_integrals(probs[1].ints.h, probs[1].ints.eri)
    wfs[1].set_dets(new)
    with pytest.raises(BatchError, match="ERR_STATE.*set again"):
        b.davidson([guess(900), guess(len(new))], **kw)
    b.close()
    b = Batch(wfs)
    r = b.davidson([guess(900), guess(len(new))], **kw)
    one = wfs[1].davidson_diag_hs2(guess(len(new)), n_states=1, threshold=1e-12, s2_eig=False)
    assert abs(r["energies"][0, 0] - first["energies"][0, 0]) < 1e-9
    assert abs(r["energies"][1, 0] - one["energies"][0]) < 1e-9
    b.close()
