"""GPU: the Fock build of many bands with a scalar V (4 x 4 channel tiles, fused assembly) against the oracle.

Band counts around the tiles of four, all terms, and a density that is not
Hermitian (the exchange then takes its upper triangle, the energy all of it).
"""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu

TOL = 1e-12  # of the largest entry: transforms of a few thousand points and sums of nb^2 nk terms


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


# at least 2^22 entries (2^23 where more of the tiles is unused): channel counts 1.00 to
# 1.57 times the triangle's, lines of 1 to 288 points with and without a codelet along kx,
# tiles of 16 and of 8 channels, and the shapes on either side of the rule
SHAPES = (
    (12, 200, 192),
    (15, 65, 288),
    (17, 202, 144),
    (17, 101, 144),
    (18, 360, 72),
    (27, 21, 288),
    (30, 75, 64),
    (32, 1024, 4),
    (33, 54, 72),
    (64, 5, 256),
    (64, 1030, 1),
    (64, 11, 96),
)


@pytest.mark.parametrize("extras", (False, True))
@pytest.mark.parametrize("nb,n1,n2", SHAPES)
def test_build(native, oracle, nb, n1, n2, extras):
    r = np.random.default_rng(nb * 100 + n1)

    def field():
        return r.normal(size=(n1, n2, nb, nb)) + 1j * r.normal(size=(n1, n2, nb, nb))

    w = r.uniform(0.5, 1.5, size=(n1, n2)) / (n1 * n2)
    kw = {}
    if extras:
        HH = r.normal(size=(nb, nb))
        O = herm(r.normal(size=(4, nb, nb)) + 1j * r.normal(size=(4, nb, nb)))
        kw = dict(include_hartree=True, hartree_matrix=HH + HH.T, reference_density=herm(field()),
                  contact_terms=[(0.7, O[0], O[1]), (-0.3, O[2], O[3])])
    args = problem.kernel_args(w, herm(field()), r.normal(size=(n1, n2, 1, 1)), 0.1, **kw)
    assert args["exchange_hcp"]
    for P in (herm(field()), field()):
        got, ref = native.build_fock_apply(args, P, None), oracle.build_fock_apply(args, P, None)
        for a, b in zip(got[:3], ref[:3]):
            assert np.abs(a - b).max() <= TOL * max(1.0, np.abs(b).max())
        assert abs(got[3] - ref[3]) <= TOL * max(1.0, abs(ref[3]))
