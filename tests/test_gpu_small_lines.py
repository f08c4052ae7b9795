"""GPU: exchange passes on both sides of the rule between the mixed-radix stages and the small-pass stages.

The rule looks at the length of the lines, their radices and the points of a pass
(2^14, 2^15, 2^16): every kind of length with the channels just below and at each
limit, along either axis, with fewer and with more tiles than SMs.  1e-13 of the
largest entry is the bar, as for the other exchange tests.
"""

from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-13
SIDES = (7, 10, 11, 13, 14, 15, 17, 19, 22, 26, 31, 34, 37, 41, 45, 49, 75, 98, 100, 143, 169, 193, 240, 243)


def field(r, *shape):
    return r.normal(size=shape) + 1j * r.normal(size=shape)


def close(a, b):
    assert np.abs(a - b).max() <= TOL * np.abs(b).max()


def convolve(P, VR):
    return -np.fft.ifft2(np.fft.fft2(P, axes=(0, 1)) * VR, axes=(0, 1))


def below_and_at(n, lines):
    out = {1}
    for limit in (1 << 14, 1 << 15, 1 << 16):
        nb = math.isqrt(limit // (n * lines))  # n lines nb^2 around the limit
        out |= {max(nb, 1), nb + 1}
    return sorted(out)


@pytest.mark.parametrize("n", SIDES)
def test_limits(native, n):
    r = np.random.default_rng(n)
    for n1, n2 in ((n, 6), (6, n), (n, 24)):
        for nb in below_and_at(n1, n2):
            P, VR = field(r, n1, n2, nb, nb), field(r, n1, n2, 1, 1)
            close(native.selfenergy_fft_full(VR, P, False, False), convolve(P, VR))
    for n1, n2, nb in ((n, 6, 3), (6, n, 16), (n, n, 2)):  # packed upper triangle, shifted output
        P = field(r, n1, n2, nb, nb)
        P = P + np.conj(np.swapaxes(P, -1, -2))
        VR = np.fft.fft2(r.normal(size=(n1, n2)))[..., None, None]
        ref = convolve(P, VR)
        close(native.selfenergy_fft_full(VR, P, False, True), ref)
        close(native.selfenergy_fft_full(VR, P, True, False), np.roll(ref, (-(n1 // 2), -(n2 // 2)), axis=(0, 1)))


@pytest.mark.parametrize("n1,n2,nb", ((7, 13, 2), (15, 17, 3), (19, 45, 8), (45, 75, 4), (100, 11, 8)))
def test_gradient(native, n1, n2, nb):
    import torch

    from cpp_hf_b200 import autograd

    r = np.random.default_rng(n1)
    P, VR, G = field(r, n1, n2, nb, nb), field(r, n1, n2, nb, nb), field(r, n1, n2, nb, nb)
    Pt, Vt = (torch.tensor(x, device="cuda", requires_grad=True) for x in (P, VR))
    gP, gV = torch.autograd.grad(autograd.exchange(Pt, Vt), (Pt, Vt), torch.tensor(G, device="cuda"))
    f = lambda x: np.fft.fft2(x, axes=(0, 1))  # noqa: E731
    close(gP.cpu().numpy(), convolve(G, np.conj(VR)))
    close(gV.cpu().numpy(), -np.conj(f(P)) * f(G) / (n1 * n2))
