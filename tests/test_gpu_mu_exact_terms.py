"""GPU: every form of the chemical-potential solvers evaluates the same occupations.

All the weight is on one eigenvalue, so each sum is that eigenvalue's term
exactly, in whatever order a form adds, and the scalar iteration has to give the
same bits in one block, one cluster and a grid.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (1025, 4608, 32768, 65536, 65537, 294912))
def test_same_bits_in_every_form(native, n):
    import torch

    from cpp_hf_b200 import _lib
    from cpp_hf_b200._native import _ptr, _stream

    lib = _lib.load()
    r = np.random.default_rng(n)
    ws = native._ws(lib.cpphf_mu_workspace_bytes(n, 1))

    def solve(size, e0, T, n_e, mu0):
        e = torch.full((size,), e0, dtype=torch.float64, device="cuda")
        w = torch.zeros(size, dtype=torch.float64, device="cuda")
        w[int(r.integers(size))] = 1.0
        mu = torch.tensor([mu0, 0.0, 0.0], dtype=torch.float64, device="cuda")
        _lib.check(lib.cpphf_solve_mu_inloop(_ptr(e), _ptr(w), size, 1, n_e, _ptr(mu), T, 25, _ptr(mu[1:]), _ptr(ws),
                                             ws.numel(), _stream()))
        _lib.check(lib.cpphf_find_mu_bisection(_ptr(e), _ptr(w), size, 1, n_e, T, 60, _ptr(mu[2:]), _ptr(ws), ws.numel(),
                                               _stream()))
        return mu[1:].tolist()

    for _ in range(40):
        T, n_e, e0 = float(r.uniform(0.03, 0.3)), float(10.0 ** r.uniform(-8, -0.05)), float(r.normal())
        mu0 = e0 + float(r.normal()) * T
        assert solve(n, e0, T, n_e, mu0) == solve(1024, e0, T, n_e, mu0)
