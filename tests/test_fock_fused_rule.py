"""CPU: which Fock build a kernel takes (host-side rules of the library; no launch is made)."""

from __future__ import annotations

import ctypes as C

import pytest

from cpp_hf_b200 import _lib


def kind(n1, n2, nb, dv=1, hcp=1, packing=0, precision=64, exchange=1):
    K = _lib.Kernel()
    K.nk1, K.nk2, K.nb, K.dv = n1, n2, nb, dv
    K.exchange_hcp, K.hermitian_packing, K.exchange_precision, K.include_exchange = hcp, packing, precision, exchange
    return _lib.load().cpphf_build_fock_fused(C.byref(K))


@pytest.mark.parametrize("nb", (2, 5, 8))
def test_packed_needs_codelets_on_both_sides(nb):
    assert kind(24, 36, nb, packing=1) == 1 and kind(24, 36, nb, dv=nb, hcp=0, packing=1) == 1
    assert kind(24, 36, nb, packing=0) == 0
    assert kind(75, 36, nb, packing=1) == 0 and kind(36, 100, nb, packing=1) == 0


def test_many_bands_need_a_large_field_and_a_codelet_along_ky():
    assert kind(72, 72, 64) == 2 and kind(75, 72, 64) == 2
    assert kind(72, 75, 64) == 0 and kind(6, 8, 64) == 0
    assert kind(72, 72, 64, hcp=0) == 0 and kind(72, 72, 64, dv=64, hcp=0) == 0
    assert kind(72, 72, 64, precision=32) == 0 and kind(72, 72, 64, exchange=0) == 0


@pytest.mark.parametrize("n1,n2,limit", ((1, 288, 8), (288, 1, 8), (1, 6, 16), (24, 256, 16), (75, 16, 16)))
def test_many_bands_stay_within_a_launch_grid(n1, n2, limit):
    """Chunks of `limit` channels lie along grid.y, which takes 65535 of them."""
    for nb in range(960, 1500):
        t = (nb + 3) // 4
        fits = 8 * t * (t + 1) // limit <= 65535
        assert kind(n1, n2, nb) == (2 if fits else 0)
