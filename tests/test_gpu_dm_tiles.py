"""GPU: the tensor-core per-k kernels of the solvers at the edges of their 8-band tiles, against the oracle.

A few iterations from P0 = 0 on a small mesh.  Perturbing h in its last bits
moves the oracle's own results by up to 1e-13 relative over as many iterations
(fillings that leave mu inside a band); 1e-10 is the bar.
"""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu

TOL = 1e-10
SIZES = (1, 3, 5, 7, 9, 16, 17, 24, 25, 33, 40, 41, 48, 49, 56, 57, 64, 65, 68)


@pytest.fixture(scope="module")
def native():
    from cpp_hf_b200 import _native

    return _native


@pytest.fixture(scope="module")
def oracle():
    from oracle import native_np

    return native_np


def model(nb, n1=3, n2=2):
    r = np.random.default_rng(nb)
    A = r.normal(size=(n1, n2, nb, nb)) + 1j * r.normal(size=(n1, n2, nb, nb))
    h = (A + np.conj(np.swapaxes(A, -1, -2))) / (2 * np.sqrt(nb))
    k1, k2 = np.meshgrid(np.arange(n1) - n1 // 2, np.arange(n2) - n2 // 2, indexing="ij")
    V = (1.0 / (0.5 + np.hypot(k1, k2)))[..., None, None]
    args = problem.kernel_args(np.full((n1, n2), 1.0 / (n1 * n2)), h, V, 0.1)
    return args, np.zeros_like(h), 0.45 * nb


def close(a, b):
    a, b = np.asarray(a), np.asarray(b)
    assert a.shape == b.shape
    assert np.abs(a - b).max() <= TOL * max(1.0, np.abs(b).max())


def dm(mod, nb, bt_max):
    args, P0, n_e = model(nb)
    none = np.empty((0,) + P0.shape, complex)
    return mod.solve_dm(args, P0, n_e, 3, 0.0, 0.0, 0.6, 0.5, 1e-3, bt_max, 10, 5, 25, 0, 0.5, 20, none, 0.0, 1.0, [],
                        None, True, True, True)


@pytest.mark.parametrize("bt_max", (8, 0))  # 0: the step no trial has formed the factor of
@pytest.mark.parametrize("nb", SIZES)
def test_direct_minimisation(native, oracle, nb, bt_max):
    got, ref = dm(native, nb, bt_max), dm(oracle, nb, bt_max)
    for i in (1, 2, 3, 4, 5, 8, 9):
        close(got[i], ref[i])
    Q = got[0]
    close(np.conj(np.swapaxes(Q, -1, -2)) @ Q, np.broadcast_to(np.eye(nb), Q.shape))
    D = got[2]
    assert np.array_equal(D, np.conj(np.swapaxes(D, -1, -2)))


@pytest.mark.parametrize("acceleration", ("linear", "diis"))
@pytest.mark.parametrize("nb", SIZES)
def test_scf(native, oracle, nb, acceleration):
    args, P0, n_e = model(nb)
    out = [m.solve_scf(args, P0, n_e, 4, 0.0, 0.0, 0.5, 0.1, None, [], acceleration, 6, 2, 1.0, 0.0, True, True)
           for m in (native, oracle)]
    for i in (0, 1, 2, 3, 6, 7, 8):
        close(out[0][i], out[1][i])


@pytest.mark.parametrize("nb", (3, 5, 7))
def test_newton_odd_band_counts(native, oracle, nb):
    args, P0, n_e = model(nb)
    none = np.empty((0,) + P0.shape, complex)
    out = [m.solve_dm(args, P0, n_e, 2, 0.0, 1e-9, 0.6, 0.5, 1e-3, 8, 10, 5, 25, 1, 0.5, 20, none, 0.0, 1.0, [], None,
                      False, True, True) for m in (native, oracle)]
    for i in (1, 2, 3, 4, 5, 8, 9):
        close(out[0][i], out[1][i])
