"""The tensor-core Gram block at the column counts where its splitting changes:
tasks of 2, 4 or 8 rows, and the number of splitting warps that have any.

Bar: as the other shapes of this kernel, 8 eps sqrt(N) sum|a b| against FP64
products; the columns' order changes no bit (the sums are exact integers per
block of rows, whatever tasks cut them).
"""
import ctypes as C
import math

import numpy as np
import pytest

from quantum_package_gb300 import _lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _gram(wf, A, B):
    import torch
    N, m = A.shape
    n = B.shape[1]
    dA, dB = torch.from_numpy(np.ascontiguousarray(A)).cuda(), torch.from_numpy(np.ascontiguousarray(B)).cuda()
    X = torch.empty((m, n), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().qpgpu_gram_tc(wf.ctx, C.c_void_p(dA.data_ptr()), m, m, C.c_void_p(dB.data_ptr()), n, n, N,
                                         C.c_void_p(X.data_ptr()), None), wf.ctx)
    return X.cpu().numpy()


@pytest.mark.parametrize("N", [37, 20_011])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 1), (4, 4), (5, 4), (8, 8), (9, 8), (16, 1), (17, 15), (48, 16), (80, 16),
                                 (96, 1), (96, 16), (128, 16)])
def test_columns_of_every_split(N, m, n):
    from quantum_package_gb300.sigma import Wavefunction
    wf = Wavefunction(4, 1, 1)
    rng = np.random.default_rng(100 * m + n)
    A = rng.normal(size=(N, m)) * np.exp(rng.uniform(-9, 0, size=(1, m)))
    B = rng.normal(size=(N, n)) * np.exp(rng.uniform(-5, 2, size=(1, n)))
    X = _gram(wf, A, B)
    assert (np.abs(X - A.T @ B) <= 8 * EPS * math.sqrt(N) * (np.abs(A).T @ np.abs(B))).all()
    p, q = rng.permutation(m), rng.permutation(n)
    np.testing.assert_array_equal(_gram(wf, A[:, p], B[:, q]), X[np.ix_(p, q)])
    # one column against one: 2 rows a task, the same integers
    np.testing.assert_array_equal(_gram(wf, A[:, :1], B[:, -1:]), X[:1, -1:])
    wf.close()
