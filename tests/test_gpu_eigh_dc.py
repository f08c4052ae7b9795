"""GPU: the eigensolvers against LAPACK: divide and conquer (nb outside 2..8, block structures), QL (nb = 2..8).

Sizes are the edges of its size classes (16, 24, 32, 48, 64, 80) and of its
merge tree.  A backward stable solver has residual, orthogonality and
eigenvalue errors of at most a small multiple of nb * eps * ||A||; 20 nb eps is
the bar.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
SIZES = (1, 9, 10, 15, 16, 17, 24, 25, 32, 33, 48, 49, 63, 64, 65, 80)


@pytest.fixture(scope="module")
def native():
    from cpp_hf_b200 import _native

    return _native


def unitary(r, n):
    return np.linalg.qr(r.normal(size=(n, n)) + 1j * r.normal(size=(n, n)))[0]


def matrices(nb, r):
    """Random, degenerate, clustered, graded, diagonal, zero, tiny off-diagonals, tridiagonal of ones."""
    A = r.normal(size=(nb, nb)) + 1j * r.normal(size=(nb, nb))
    out = [A + A.conj().T]
    for lam in (np.repeat(r.normal(size=(nb + 3) // 4), 4)[:nb], 1.0 + 1e-13 * r.normal(size=nb),
                10.0 ** r.uniform(-14, 0, nb)):
        U = unitary(r, nb)
        out.append((U * lam) @ U.conj().T)
    D = np.diag(np.round(3 * r.normal(size=nb))).astype(complex)
    out += [D, np.zeros((nb, nb), complex), D + 1e-17 * out[0], D + 1e-158 * out[0], 1e-200 * out[0], 1e200 * out[0]]
    out.append(2 * np.eye(nb) + np.eye(nb, k=1) + np.eye(nb, k=-1) + 0j)
    return np.array([0.5 * (M + M.conj().T) for M in out])


def check(M, w, V):
    nb = M.shape[-1]
    for A, wk, Vk in zip(M, w, V):
        scale = np.abs(np.linalg.eigvalsh(A)).max()
        bar = 20 * nb * EPS * scale
        assert np.abs(Vk.conj().T @ Vk - np.eye(nb)).max() <= 20 * nb * EPS
        assert np.abs(A @ Vk - Vk * wk).max() <= bar


@pytest.mark.parametrize("nb", SIZES)
def test_against_lapack(native, nb):
    M = matrices(nb, np.random.default_rng(nb))
    w, V = native.eigh_batched(M)
    check(M, w, V)
    for A, wk in zip(M, w):
        wr = np.linalg.eigvalsh(A)
        assert np.all(np.diff(wk) >= 0)
        assert np.abs(wk - wr).max() <= 20 * nb * EPS * np.abs(wr).max()


@pytest.mark.parametrize("batch", (1, 33, 9300))  # one thread, a partial warp, a batch past every rule
@pytest.mark.parametrize("nb", range(2, 9))
def test_small(native, nb, batch):
    """nb = 2..8: a thread or eight lanes per matrix, by batch."""
    M = matrices(nb, np.random.default_rng(nb))
    M = np.concatenate([M] * (batch // len(M) + 1))[:batch]
    w, V = native.eigh_batched(M)
    n = min(batch, 64)
    check(M[-n:], w[-n:], V[-n:])
    for A, wk in zip(M[-n:], w[-n:]):
        wr = np.linalg.eigvalsh(A)
        assert np.all(np.diff(wk) >= 0)
        assert np.abs(wk - wr).max() <= 20 * nb * EPS * np.abs(wr).max()


@pytest.mark.parametrize("sort", (True, False))
@pytest.mark.parametrize("sizes", ((1, 1), (2, 3), (3, 1, 5), (7, 9), (1, 31, 5), (20, 44)))
def test_blocks(native, sizes, sort):
    nb = sum(sizes)
    M = matrices(nb, np.random.default_rng(nb))
    w, V = native.eigh_block_sizes(M, list(sizes), sort)
    own = np.repeat(np.arange(len(sizes)), sizes)
    B = np.where(own[:, None] == own[None, :], M, 0)
    check(B, w, V)
    for wk, Vk, Bk in zip(w, V, B):
        blk = own[np.abs(Vk).argmax(axis=0)]
        # every vector keeps to the rows of one block
        assert np.all(Vk[own[:, None] != blk[None, :]] == 0)
        if sort:
            assert np.all(np.diff(wk) >= 0)
        else:
            assert np.array_equal(blk, own)
            assert all(np.all(np.diff(wk[own == b]) >= 0) for b in range(len(sizes)))


def test_not_finite(native):
    """A matrix with a NaN or an infinity gives NaN and leaves the others of the batch alone."""
    M = matrices(20, np.random.default_rng(0))[:3].copy()
    M[1, 3, 4] = np.nan
    w, V = native.eigh_batched(M)
    assert np.isnan(w[1]).all() and np.isnan(V[1]).all()
    check(M[[0, 2]], w[[0, 2]], V[[0, 2]])
