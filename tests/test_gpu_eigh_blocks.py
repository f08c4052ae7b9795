"""GPU: block-diagonal eigenproblems of small blocks (solved block by block), and nb = 1, against LAPACK.

Block sizes 1..8 in mixed and uniform structures up to the largest matrix, batches
of one problem, of partial warps and past the rules of the dispatch.  The
bar is that of a backward stable solver, 20 nb eps ||A||.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
STRUCTURES = ((1, 1), (2, 1), (1,) * 16, (4, 4), (2, 2, 2, 2), (3, 1, 5), (7, 1), (6, 6), (8, 8), (5, 4, 8, 1, 2, 7, 3, 6), (8,) * 10,
              (1,) * 80)


def matrices(sizes, batch, r):
    """Random, degenerate (also between blocks), diagonal, graded; entries outside the blocks are to be ignored."""
    nb = sum(sizes)
    n = min(batch, 16)
    A = r.normal(size=(n, nb, nb)) + 1j * r.normal(size=(n, nb, nb))
    A = A + np.conj(np.swapaxes(A, -1, -2))
    if n >= 4:
        A[1] = np.eye(nb) * 2.0
        A[2] = np.diag(np.round(2 * r.normal(size=nb)))
        g = 10.0 ** r.uniform(-8, 0, nb)
        A[3] *= g[:, None] * g[None, :]
    return np.concatenate([A] * (batch // n + 1))[:batch]


@pytest.mark.parametrize("sort", (True, False))
@pytest.mark.parametrize("batch", (1, 70, 9300))
@pytest.mark.parametrize("sizes", STRUCTURES, ids=lambda s: "x".join(map(str, s[:8])) + f"of{sum(s)}")
def test_blocks(native, sizes, batch, sort):
    nb = sum(sizes)
    if batch * nb * nb > 3_000_000:
        batch = 700
    M = matrices(sizes, batch, np.random.default_rng(nb))
    w, V = native.eigh_block_sizes(M, list(sizes), sort)
    own = np.repeat(np.arange(len(sizes)), sizes)
    n = min(batch, 24)
    for A, wk, Vk in zip(M[-n:], w[-n:], V[-n:]):
        B = np.where(own[:, None] == own[None, :], A, 0)
        bar = 20 * nb * EPS * max(np.abs(np.linalg.eigvalsh(B)).max(), 1e-300)
        assert np.abs(Vk.conj().T @ Vk - np.eye(nb)).max() <= 20 * nb * EPS
        assert np.abs(B @ Vk - Vk * wk).max() <= bar
        assert np.abs(np.sort(wk) - np.linalg.eigvalsh(B)).max() <= bar
        blk = own[np.abs(Vk).argmax(axis=0)]
        assert np.all(Vk[own[:, None] != blk[None, :]] == 0)
        if sort:
            assert np.all(np.diff(wk) >= 0)
        else:
            assert np.array_equal(blk, own)
            assert all(np.all(np.diff(wk[own == b]) >= 0) for b in range(len(sizes)))


@pytest.mark.parametrize("bad", (np.nan, np.inf))
@pytest.mark.parametrize("sizes", ((2, 1), (4, 4), (8, 3)))
def test_not_finite(native, sizes, bad):
    """A matrix with a NaN or an infinity inside a block gives NaN and leaves the others of the batch alone."""
    M = matrices(sizes, 12000, np.random.default_rng(0))
    M[5, 0, 1] = bad
    w, V = native.eigh_block_sizes(M, list(sizes))
    assert np.isnan(w[5]).all() and np.isnan(V[5]).all()
    ok = np.arange(len(M)) != 5
    assert np.isfinite(w[ok]).all() and np.isfinite(V[ok]).all()


@pytest.mark.parametrize("batch", (1, 63, 64, 65, 20000))
def test_one_band(native, batch):
    M = np.random.default_rng(batch).normal(size=(batch, 1, 1)) + 1j
    if batch > 2:
        M[2] = np.nan
    w, V = native.eigh_batched(M)
    ok = ~np.isnan(M.real[:, 0, 0])
    assert np.array_equal(w[ok, 0], M.real[ok, 0, 0]) and np.all(V[ok] == 1.0)
    assert np.isnan(w[~ok]).all() and np.isnan(V[~ok]).all()
