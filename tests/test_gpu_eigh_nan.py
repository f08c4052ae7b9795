"""GPU: a NaN anywhere in a matrix reaches its eigenvalues and vectors, in every form of the eigensolver, and no other matrix."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", (3, 12000))  # eight lanes or one thread per matrix
@pytest.mark.parametrize("nb", range(1, 10))
def test_nan(native, nb, batch):
    r = np.random.default_rng(nb)
    M = r.normal(size=(batch, nb, nb)) + 1j * r.normal(size=(batch, nb, nb))
    M = M + np.conj(np.swapaxes(M, -1, -2))
    for i in range(nb):
        for j in range(i + 1):
            A = M.copy()
            A[1, i, j] = np.nan
            w, V = native.eigh_batched(A)
            assert np.isnan(w[1]).all() and np.isnan(V[1]).any()
            ok = np.arange(batch) != 1
            assert np.isfinite(w[ok]).all() and np.isfinite(V[ok]).all()
