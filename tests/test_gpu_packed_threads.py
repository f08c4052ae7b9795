"""GPU: the packed build's last pass on long lines, with few and many threads to a line, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu

TOL = 1e-12  # of the largest entry: transforms of up to 2304 points in double


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


# more tiles than CTAs in the last two rows; 96 threads at nb = 4, 5, 128 at 6, 7, 160 at 8 (16 lanes)
@pytest.mark.parametrize("n1,n2,nb", ((1, 128, 4), (2, 192, 5), (9, 256, 6), (3, 192, 7), (9, 256, 8), (6, 144, 7),
                                      (288, 144, 8), (256, 192, 6)))
def test_long_lines(native, oracle, n1, n2, nb):
    r = np.random.default_rng(nb * 1000 + n2)

    def field():
        return herm(r.normal(size=(n1, n2, nb, nb)) + 1j * r.normal(size=(n1, n2, nb, nb)))

    w = r.uniform(0.5, 1.5, size=(n1, n2)) / (n1 * n2)
    args = problem.kernel_args(w, field(), r.normal(size=(n1, n2, 1, 1)), 0.1)
    P = field()
    got, ref = native.build_fock_apply(args, P, None), oracle.build_fock_apply(args, P, None)
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() <= TOL * max(1.0, np.abs(b).max())
    assert abs(got[3] - ref[3]) <= TOL * max(1.0, abs(ref[3]))
