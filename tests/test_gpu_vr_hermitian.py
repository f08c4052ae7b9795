"""GPU: the check that V(q) is Hermitian, which decides whether the packed build may run."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dv", (1, 3))
@pytest.mark.parametrize("n1,n2", ((1, 1), (4, 6), (5, 7)))
def test_vr_hermitian(native, n1, n2, dv):
    import torch

    r = np.random.default_rng(n1)
    V = r.normal(size=(n1, n2, dv, dv)) + 1j * r.normal(size=(n1, n2, dv, dv))
    V = V + np.conj(np.swapaxes(V, -1, -2))  # Hermitian at every q
    VR = np.fft.fft2(V, axes=(0, 1))

    def check(X):
        return native._vr_hermitian(torch.from_numpy(np.ascontiguousarray(X)).cuda())

    assert check(VR) and check(0 * VR)
    bad = VR.copy()
    bad[-1, 0, 0, -1] += 1e-9j * np.abs(VR).max()
    assert not check(bad)
    for value in (np.nan, complex(0, np.nan), complex(np.nan, np.inf), complex(np.inf, np.nan), complex(-np.inf, np.nan)):
        bad = VR.copy()
        bad[-1, -1, 0, -1] = value
        assert not check(bad)
