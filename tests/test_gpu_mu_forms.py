"""GPU: the chemical-potential solvers at the limits of their forms (one block, one cluster, a grid), against the oracle.

The levels of the bisection are exact counts, so its result is the oracle's to
rounding; the in-loop Newton is stopped before the rounding-sensitive end game.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native():
    from cpp_hf_b200 import _native

    return _native


@pytest.fixture(scope="module")
def oracle():
    from oracle import native_np

    return native_np


def bands(nk, nb):
    r = np.random.default_rng(nk)
    return np.sort(3 * r.normal(size=(nk, nb)), axis=1), np.full(nk, 1.0 / nk)


@pytest.mark.parametrize("nk,nb", ((1, 1), (512, 2), (205, 5), (32768, 2), (65537, 1), (36864, 8), (20736, 20)))
def test_forms(native, oracle, nk, nb):
    import torch

    from cpp_hf_b200 import _lib

    e, w = bands(nk, nb)
    n_e = 0.47 * nb
    mu = native.find_mu_bisection(e, w, n_e, 0.05)
    ref = oracle.find_mu_bisection(e, w, n_e, 0.05)
    assert abs(mu - ref) <= 1e-12 * max(1.0, abs(ref))
    lib = _lib.load()
    dev = [torch.from_numpy(x).cuda() for x in (e, w, np.zeros(1), np.zeros(1))]
    ws = native._ws(lib.cpphf_mu_workspace_bytes(nk, nb))
    _lib.check(lib.cpphf_solve_mu_inloop(native._ptr(dev[0]), native._ptr(dev[1]), nk, nb, n_e, native._ptr(dev[2]), 0.05,
                                         6, native._ptr(dev[3]), native._ptr(ws), ws.numel(), native._stream()))
    ref = oracle._solve_mu_inloop(e, w, n_e, 0.0, 0.05, 6)
    assert abs(float(dev[3]) - ref) <= 1e-9 * max(1.0, abs(ref))


def test_more_rounds_than_slots(native):
    """A step occupation (T = 1e-9) takes exact rounds for all 150 levels: the grid reuses its slots.
    1.4 electrons fill whole levels (56000 of 40000 x 3), so mu may lie anywhere between two of them."""
    e, w = bands(40000, 3)
    mu = native.find_mu_bisection(e, w, 1.4, 1e-9, 150)

    def count(m):
        return float(np.sum(w[:, None] * (e < m)))

    assert count(mu - 1e-7) <= 1.4 + 1e-12
    assert count(mu + 1e-7) >= 1.4 - 1e-12
