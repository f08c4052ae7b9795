"""GPU: the mixed-radix exchange passes (mesh sides without a four-step codelet) against the oracle.

Sides cover every radix, single-radix lengths, products of two and three radices,
primes above 13 alone and with cofactors, and lengths of many stages.  The sums of
a transform of n points are exact to a few eps * sqrt(n) of their norm; 1e-13 of
the largest entry is the bar.
"""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import superlattice

pytestmark = pytest.mark.gpu

TOL = 1e-13
SIDES = (7, 10, 11, 13, 14, 15, 17, 19, 20, 22, 26, 28, 30, 31, 34, 42, 49, 51, 54, 75, 77, 97, 98, 100, 104, 121, 143,
         169, 186, 187, 191, 210, 240, 289, 361, 480, 1001, 2016)


@pytest.fixture(scope="module")
def native():
    from cpp_hf_b200 import _native

    return _native


@pytest.fixture(scope="module")
def oracle():
    from oracle import native_np

    return native_np


def field(r, *shape):
    return r.normal(size=shape) + 1j * r.normal(size=shape)


def close(a, b):
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("n", SIDES)
def test_exchange(native, oracle, n):
    r = np.random.default_rng(n)
    for n1, n2, nb, dv in ((n, 6, 3, 3), (5, n, 3, 1), (n, n, 1, 1)) if n < 250 else ((n, 6, 2, 2), (5, n, 3, 1)):
        P, VR = field(r, n1, n2, nb, nb), field(r, n1, n2, dv, dv)
        for shift in (False, True):
            close(native.selfenergy_fft_full(VR, P, shift, False), oracle.selfenergy_fft_full(VR, P, shift, False))
        if dv == 1:  # packed upper triangle: Hermitian density, real V(q)
            P = P + np.conj(np.swapaxes(P, -1, -2))
            VR = np.fft.fft2(r.normal(size=(n1, n2)))[..., None, None]
            close(native.selfenergy_fft_full(VR, P, False, True), oracle.selfenergy_fft_full(VR, P, False, True))


@pytest.mark.parametrize("n1,n2", ((14, 75), (97, 30), (22, 17), (169, 10)))
def test_reference_density_and_gradient(native, oracle, n1, n2):
    import torch

    from cpp_hf_b200 import autograd

    r = np.random.default_rng(n1)
    P, VR, G = field(r, n1, n2, 3, 3), field(r, n1, n2, 3, 3), field(r, n1, n2, 3, 3)
    Pt, Vt = (torch.tensor(x, device="cuda", requires_grad=True) for x in (P, VR))
    S = autograd.exchange(Pt, Vt)
    gP, gV = torch.autograd.grad(S, (Pt, Vt), torch.tensor(G, device="cuda"))
    f, fi = (lambda x: np.fft.fft2(x, axes=(0, 1))), (lambda x: np.fft.ifft2(x, axes=(0, 1)))
    close(S.detach().cpu().numpy(), -fi(f(P) * VR))
    close(gP.cpu().numpy(), -fi(f(G) * np.conj(VR)))
    close(gV.cpu().numpy(), -np.conj(f(P)) * f(G) / (n1 * n2))


@pytest.mark.parametrize("hermitian", (False, True))
@pytest.mark.parametrize("orbital", (False, True))
@pytest.mark.parametrize("nkx,nky,pw", ((5, 3, 4), (7, 5, 7), (11, 2, 5), (17, 5, 3)))
def test_padded_grid(native, oracle, nkx, nky, pw, orbital, hermitian):
    r = np.random.default_rng(nkx)
    g, B = superlattice._triangular_shells(pw)
    lay = superlattice.extended_layout(g, B, nkx, nky, lambda q: 1.0 / (q + 0.3), 1.0 / (nkx * nky))
    rho = field(r, nkx, nky, pw, 2, pw, 2)
    if hermitian:
        rho = rho + np.conj(rho.transpose(0, 1, 4, 5, 2, 3))
    Vo = lay.V_lag_fft[..., None, None] * r.normal(size=(2, 2)) if orbital else None
    if orbital and hermitian:
        Vo = 0.5 * (Vo + np.swapaxes(Vo, -1, -2))
    a = (rho, lay.V_lag_fft, lay.g_a_off, lay.delta_pair_i, lay.delta_pair_j, lay.delta_pair_start, nkx, nky, pw, 2,
         lay.N_ext_x, lay.N_ext_y, Vo, hermitian)
    close(native.selfenergy_superlattice_streamed(*a), oracle.selfenergy_superlattice_streamed(*a))
