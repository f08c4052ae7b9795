"""GPU: chemical-potential solves of up to 65536 eigenvalues use no scratch, so those that share one may overlap."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = ((512, 2), (205, 5), (2304, 2), (32768, 1), (65536, 1))  # the one-block and cluster forms at their limits


def problem(nk, nb, seed):
    import torch

    r = np.random.default_rng(seed)
    return torch.from_numpy(np.sort(3 * r.normal(size=(nk, nb)), axis=1)).cuda(), \
        torch.full((nk,), 1.0 / nk, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("nk,nb", SIZES)
def test_workspace_is_left_alone(native, nk, nb):
    import torch

    from cpp_hf_b200 import _lib
    from cpp_hf_b200._native import _ptr, _stream

    lib = _lib.load()
    e, w = problem(nk, nb, 1)
    ws = torch.full((lib.cpphf_mu_workspace_bytes(nk, nb),), 0x5A, dtype=torch.uint8, device="cuda")
    mu = torch.zeros(2, dtype=torch.float64, device="cuda")
    _lib.check(lib.cpphf_find_mu_bisection(_ptr(e), _ptr(w), nk, nb, 0.47 * nb, 0.05, 30, _ptr(mu), _ptr(ws), ws.numel(),
                                           _stream()))
    _lib.check(lib.cpphf_solve_mu_inloop(_ptr(e), _ptr(w), nk, nb, 0.47 * nb, _ptr(mu), 0.05, 25, _ptr(mu[1:]), _ptr(ws),
                                         ws.numel(), _stream()))
    assert bool((ws == 0x5A).all())


@pytest.mark.parametrize("nk,nb", SIZES)
def test_overlapping_calls_without_a_workspace(native, nk, nb):
    import torch

    from cpp_hf_b200 import _lib
    from cpp_hf_b200._native import _ptr

    lib = _lib.load()
    cases = [problem(nk, nb, s) for s in range(8)]
    n_e = [nb * (0.3 + 0.05 * i) for i in range(8)]
    ref = [native.find_mu_bisection(e, w, x, 0.05) for (e, w), x in zip(cases, n_e)]
    assert len(set(ref)) == len(ref)
    streams = [torch.cuda.Stream() for _ in cases]
    mu = torch.zeros((20, 8), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for row in mu:
        for i, ((e, w), s) in enumerate(zip(cases, streams)):
            _lib.check(lib.cpphf_find_mu_bisection_noalloc(_ptr(e), _ptr(w), nk, nb, n_e[i], 0.05, 0, _ptr(row[i:]),
                                                           C.c_void_p(s.cuda_stream)))
    torch.cuda.synchronize()
    assert (mu.cpu().numpy() == np.array(ref)).all()
