"""GPU: density_from_fock's gradient at the edges of the 8-band tiles, against the divided-difference formula in NumPy."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10  # of the largest entry: the divided differences lose up to gap / eps ~ 1e4 digits' worth at nb = 68


@pytest.mark.parametrize("nb", (1, 2, 3, 7, 8, 9, 16, 17, 24, 25, 32, 33, 41, 48, 49, 57, 64, 65, 68))
def test_gradient(nb):
    import torch

    from cpp_hf_b200 import autograd

    r = np.random.default_rng(nb)
    n1, n2, T, n_e = 3, 7, 0.1, 0.45 * nb

    def herm(X):
        return 0.5 * (X + np.conj(np.swapaxes(X, -1, -2)))

    F = herm(r.normal(size=(n1, n2, nb, nb)) + 1j * r.normal(size=(n1, n2, nb, nb))) / np.sqrt(nb)
    G = r.normal(size=F.shape) + 1j * r.normal(size=F.shape)
    w = r.uniform(0.5, 1.5, size=(n1, n2))
    w /= w.sum()
    Ft = torch.tensor(F, device="cuda", requires_grad=True)
    P, eps, mu = autograd.density_from_fock(Ft, torch.tensor(w, device="cuda"), n_e, T)
    (gF,) = torch.autograd.grad(P, Ft, torch.tensor(G, device="cuda"))
    e, V = np.linalg.eigh(F)
    Te = T + 1e-12
    x = (e - float(mu)) / Te
    f, g = 1.0 / (1.0 + np.exp(x)), 1.0 / (1.0 + np.exp(-x))
    fp = -f * g / Te
    lo, hi = np.minimum(x[..., :, None], x[..., None, :]), np.maximum(x[..., :, None], x[..., None, :])
    d = np.maximum(hi - lo, 1e-300)
    L = np.expm1(-d) / d / Te / (1.0 + np.exp(lo)) / (1.0 + np.exp(-hi))
    M = np.conj(np.swapaxes(V, -1, -2)) @ herm(G) @ V
    A, Z = np.sum(np.real(np.diagonal(M, axis1=-2, axis2=-1)) * fp), np.sum(w[..., None] * fp)
    X = M * L
    i = np.arange(nb)
    X[..., i, i] -= w[..., None] * fp * (A / Z)
    ref = V @ X @ np.conj(np.swapaxes(V, -1, -2))
    got = gF.cpu().numpy()
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
