"""GPU: the fused Fock build of many bands as the solvers run it (no exchange field written), and where it stops applying.

The meshes are past the size from which the build is fused (2^22 entries), so whole
solves go through it; a switched-precision solve goes from the unfused complex64
build to it in one workspace.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu

TOL = 1e-8  # a few iterations of differences at the rounding of a 64 x 64 eigenproblem


def herm(X):
    return 0.5 * (X + np.conj(np.swapaxes(X, -1, -2)))


def model(nb, n1, n2, extras=False):
    r = np.random.default_rng(nb + n1)

    def field(*shape):
        return herm(r.normal(size=shape + (nb, nb)) + 1j * r.normal(size=shape + (nb, nb))) / np.sqrt(nb)

    k1, k2 = np.meshgrid(np.arange(n1) - n1 // 2, np.arange(n2) - n2 // 2, indexing="ij")
    V = (1.0 / (0.5 + np.hypot(k1, k2)))[..., None, None]
    kw = {}
    if extras:
        HH, O = r.normal(size=(nb, nb)), field(4)
        kw = dict(include_hartree=True, hartree_matrix=HH + HH.T, reference_density=field(n1, n2),
                  contact_terms=[(0.7, O[0], O[1]), (-0.3, O[2], O[3])])
    return problem.kernel_args(np.full((n1, n2), 1.0 / (n1 * n2)), field(n1, n2), V, 0.1, **kw), field(n1, n2)


def close(a, b, tol=TOL):
    a, b = np.asarray(a), np.asarray(b)
    assert a.shape == b.shape
    assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())


def fused(native, args):
    from cpp_hf_b200 import _lib

    return _lib.load().cpphf_build_fock_fused(C.byref(native._DeviceKernel(args).K))


@pytest.mark.parametrize("extras", (False, True))
@pytest.mark.parametrize("nb,n1,n2", ((12, 200, 192), (33, 54, 72), (64, 11, 96), (64, 1030, 1)))
def test_build_without_the_exchange_field(native, nb, n1, n2, extras):
    import torch

    from cpp_hf_b200 import _lib
    from cpp_hf_b200._native import _DeviceKernel, _ptr, _stream, _ws

    args, P = model(nb, n1, n2, extras)
    dk, lib = _DeviceKernel(args), _lib.load()
    assert fused(native, args) == 2
    P = torch.from_numpy(np.ascontiguousarray(P)).cuda()
    ws = _ws(lib.cpphf_build_fock_workspace_bytes(dk.ref()))
    out = []
    for sigma in (torch.empty_like(P), None):
        F, hd = torch.empty_like(P), torch.zeros(nb, dtype=torch.float64, device="cuda")
        E = torch.zeros(1, dtype=torch.float64, device="cuda")
        _lib.check(lib.cpphf_build_fock(dk.ref(), _ptr(P), _ptr(sigma), _ptr(F), _ptr(hd), _ptr(E), None, _ptr(ws),
                                        ws.numel(), _stream()))
        out.append((F, hd, E))
    assert all(torch.equal(a, b) for a, b in zip(*out))


def dm(mod, args, P0, n_e, optimizer=0, iters=2):
    none = np.empty((0,) + P0.shape, complex)
    return mod.solve_dm(args, P0, n_e, iters, 0.0, 0.0, 0.6, 0.5, 1e-3, 8, 10, 5, 25, optimizer, 0.5, 4, none, 0.0, 1.0,
                        [], None, False, True, True)


def scf(mod, args, P0, n_e, iters=3):
    return mod.solve_scf(args, P0, n_e, iters, 0.0, 0.0, 0.5, 0.0, None, [], "linear", 6, 2, 1.0, 0.0, True, True)


@pytest.mark.parametrize("solver", ("dm", "scf"))
def test_solves(native, oracle, solver):
    args, _ = model(64, 11, 96)
    P0 = np.zeros_like(args["h"])
    assert fused(native, args) == 2
    run = dm if solver == "dm" else scf
    got, ref = run(native, args, P0, 29.0), run(oracle, args, P0, 29.0)
    for a, b in zip(got, ref):
        if a is not None and not isinstance(a, bool):
            close(a, b)


@pytest.mark.parametrize("solver", ("dm", "newton", "scf"))
def test_solves_match_the_full_channel_build(native, solver):
    """The same solve with the upper-triangle packing off, which is not fused."""
    nb, n1, n2 = (32, 64, 64) if solver == "newton" else (64, 11, 96)  # Newton takes up to 48 bands
    args, _ = model(nb, n1, n2)
    P0, n_e = np.zeros_like(args["h"]), 0.45 * nb
    full = dict(args, exchange_hcp=False)
    assert fused(native, args) == 2 and fused(native, full) == 0
    run = {"dm": dm, "scf": scf, "newton": lambda m, a, P, n: dm(m, a, P, n, optimizer=1)}[solver]
    for a, b in zip(run(native, args, P0, n_e), run(native, full, P0, n_e)):
        if a is not None and not isinstance(a, bool):
            close(a, b)


@pytest.mark.parametrize("solver", ("dm", "scf"))
def test_switched_precision(native, solver):
    """complex64 until the first residual, complex128 from then on: within the first build's single precision."""
    args, _ = model(64, 11, 96)
    P0 = np.zeros_like(args["h"])
    mixed = dict(args, exchange_precision="mixed", mixed_switch=1e3)
    run = dm if solver == "dm" else scf
    for a, b in zip(run(native, mixed, P0, 29.0, iters=4), run(native, args, P0, 29.0, iters=4)):
        if a is not None and not isinstance(a, bool):
            close(a, b, 1e-4)


def test_more_channels_than_a_launch_grid_takes_tiles(native):
    """1446 bands: the tiled packing would need 65703 chunks along grid.y, the rows packing needs 16347."""
    args, P = model(1446, 1, 6)
    assert fused(native, args) == 0
    S, _, F, E = native.build_fock_apply(args, P, None)
    ref = -np.fft.ifft2(np.fft.fft2(P, axes=(0, 1)) * args["VR"], axes=(0, 1))
    close(S, ref, 1e-12)
    close(F, herm(args["h"] + ref), 1e-12)
    w = args["w2d"][..., None, None]
    close(E, np.sum(w * ((args["h"] + 0.5 * ref) * np.swapaxes(P, -1, -2)).real), 1e-11)
