"""GPU: the weighted density sum with the Hartree diagonal and the contact terms against the oracle.

Meshes of one point, of fewer points than a block's lanes and of several blocks per
slice; band counts of one slice of channels, of a partly filled last slice and of many.
"""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu

TOL = 1e-12  # of the largest entry: sums of up to 2e4 points and nb^2 products


@pytest.fixture(scope="module")
def native():
    from cpp_hf_b200 import _native

    return _native


@pytest.fixture(scope="module")
def oracle():
    from oracle import native_np

    return native_np


def herm(X):
    return 0.5 * (X + np.conj(np.swapaxes(X, -1, -2)))


@pytest.mark.parametrize("hartree", (False, True))
@pytest.mark.parametrize("nb,n1,n2", ((1, 1, 1), (1, 130, 140), (2, 3, 5), (5, 29, 31), (7, 101, 97), (15, 6, 1),
                                      (16, 40, 41), (17, 1, 2), (17, 48, 50), (33, 9, 13), (64, 5, 7), (70, 3, 4)))
def test_hartree_contact(native, oracle, nb, n1, n2, hartree):
    r = np.random.default_rng(1000 * nb + n1)

    def field(*shape):
        return r.normal(size=shape + (nb, nb)) + 1j * r.normal(size=shape + (nb, nb))

    w = r.uniform(0.5, 1.5, size=(n1, n2)) / (n1 * n2)
    HH, O = r.normal(size=(nb, nb)), field(6)
    kw = {}
    if hartree:
        kw = dict(include_hartree=True, hartree_matrix=HH + HH.T, reference_density=herm(field(n1, n2)))
    if nb <= 64:  # the bound of the contact terms
        kw["contact_terms"] = [(0.7, O[0], O[1]), (0.0, O[2], O[3]), (-0.3, O[4], O[5])]
    args = problem.kernel_args(w, herm(field(n1, n2)), r.normal(size=(n1, n2, 1, 1)), 0.1, **kw)
    args["exchange_hcp"] = False  # P is not Hermitian: no packed build
    P = field(n1, n2)
    got, ref = native.build_fock_apply(args, P, None), oracle.build_fock_apply(args, P, None)
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() <= TOL * max(1.0, np.abs(b).max())
    assert abs(got[3] - ref[3]) <= TOL * max(1.0, abs(ref[3]))
