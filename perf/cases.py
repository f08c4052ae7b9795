"""Performance cases: the work that users of this library have it do, through its public entry points.

A case is a dict of plain values.  Its ``kind`` names the entry point:

* ``build``   one Fock build of a device-resident density with a kept ``FockBuilder``: what every
              iteration of a self-consistent loop does (``out`` = "fe": F and E, as the solvers build;
              "sigma": the exchange field too, the public ``build_fock`` triple);
* ``grad``    ``autograd.build_fock`` + ``hf_energy`` and the gradient with respect to P, h and VR:
              fitting model parameters through the energy;
* ``density`` ``autograd.density_from_fock`` (batched eigh, chemical potential, density), with its
              gradient where ``backward`` is set;
* ``dm``      ``_native.solve_dm`` for a fixed number of iterations (direct minimisation, a
              continuation step from a neighbouring parameter takes about as many);
* ``scf``     ``_native.solve_scf`` with linear mixing for a fixed number of iterations;
* ``stream``  ``_native.selfenergy_superlattice_streamed``: the plane-wave exchange of a moire problem.

Meshes, band counts, temperatures and interactions are those of the configurations, tests and the
benchmark: 2-band Dirac models from 36^2 on, layered stacks of up to 8 bands on up to 192^2, Dirac
superlattices of up to 64 bands on up to 144^2, and odd meshes and band counts.  Inputs are made on
the GPU from the seed; fillings of solver cases are not integer (a doped system), so that the
chemical potential is determined by the inputs.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from cpp_hf_b200 import _native, autograd, superlattice
from cpp_hf_b200.fock_builder import FockBuilder

C128, F64 = torch.complex128, torch.float64
# SolverConfig's defaults, as the reference's Python layer passes them
DM = dict(tol_E=0.0, tol_grad=0.0, max_step=0.6, bt_shrink=0.5, denom_scale=1e-3, bt_max=8, cg_restart=10,
          plateau_window=5, mu_maxiter=25)
MIXING = 0.5


def listed():
    return [
        # the smallest solve's build: three short launches of a 2-band Dirac mesh
        dict(name="build_dirac_36", kind="build", n1=36, n2=36, nb=2, v="scalar", hermitian=True, out="fe",
             extras=False, precision=64),
        # the headline build of the 4-layer model, as DM and SCF iterations run it
        dict(name="build_layered_192", kind="build", n1=192, n2=192, nb=8, v="orbital", hermitian=True, out="fe",
             extras=False, precision=64),
        # ragged mesh and odd band count, a density that is not declared Hermitian, with a reference
        # density, Hartree and contact terms and the exchange field written: the general build_fock
        dict(name="build_general_75x98", kind="build", n1=75, n2=98, nb=5, v="orbital", hermitian=False,
             out="sigma", extras=True, precision=64),
        # the complex64 exchange that switched-precision solves start with
        dict(name="build_c64_144", kind="build", n1=144, n2=144, nb=6, v="orbital", hermitian=True, out="fe",
             extras=False, precision=32),
        # the build of the 64-band superlattice in its plain-mesh form (1.4 GB fields)
        dict(name="build_mesh_144_nb64", kind="build", n1=144, n2=144, nb=64, v="scalar", hermitian=True,
             out="sigma", extras=False, precision=64),
        # the differentiation workload: energy gradient of the 4-layer model
        dict(name="grad_layered_96", kind="grad", n1=96, n2=96, nb=8, v="orbital"),
        # density of a 32-band Fock matrix (mid-size plane-wave basis) and its gradient
        dict(name="density_48_nb32", kind="density", n1=48, n2=48, nb=32, T=0.05, fill=0.45, backward=True),
        # a whole small solve, where launches and host work count
        dict(name="dm_dirac_48", kind="dm", n1=48, n2=48, nb=2, v="scalar", T=0.1, U=1.0, fill=0.45, iters=8),
        # direct minimisation of the 4-layer model at the benchmark size
        dict(name="dm_layered_192", kind="dm", n1=192, n2=192, nb=8, v="orbital", T=0.05, U=1.0, fill=0.47,
             iters=6),
        # self-consistent field iterations at the benchmark size
        dict(name="scf_layered_192", kind="scf", n1=192, n2=192, nb=8, v="orbital", T=0.05, U=1.0, fill=0.47,
             iters=8),
        # direct minimisation of the 64-band superlattice in its plain-mesh form
        dict(name="dm_mesh_72_nb64", kind="dm", n1=72, n2=72, nb=64, v="scalar", T=0.05, U=0.5, fill=0.48,
             iters=4),
        # streamed plane-wave exchange of a 16-plane-wave Dirac superlattice
        dict(name="stream_48_pw16", kind="stream", n=48, pw=16, orb=2, hermitian=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
    """A side of a mesh: mostly the configurations' sizes, otherwise any."""
    sizes = [s for s in (24, 36, 48, 72, 96, 144, 192) if lo <= s <= hi]
    return rng.choice(sizes) if sizes and rng.random() < 0.6 else _log_int(rng, lo, hi)


def _bands(rng):
    """Band count: the models' 2..8 mostly (odd ones too), otherwise a plane-wave basis."""
    return rng.choice((2, 3, 4, 5, 6, 7, 8)) if rng.random() < 0.6 else 2 * _log_int(rng, 5, 32)


def draw(rng):
    kind = rng.choice(("build", "build", "grad", "density", "dm", "dm", "scf", "scf", "stream"))
    if kind == "stream":
        return dict(kind=kind, n=_log_int(rng, 12, 48), pw=rng.randint(4, 16), orb=2,
                    hermitian=rng.random() < 0.7)
    nb = rng.choice((2, 4, 5, 6, 8)) if kind == "grad" else _bands(rng)
    # the largest mesh side that keeps a drawn case below the largest listed one of its kind
    if kind in ("build", "grad"):
        top = min(192, int(144 * 64 / nb)) if kind == "build" else 144
    else:
        top = 192 if nb <= 8 else max(24, min(144, int(72 * (56.0 / nb) ** 1.5)))
    n1 = _mesh(rng, 24, top)
    n2 = n1 if rng.random() < 0.7 else _mesh(rng, 24, top)
    v = "scalar" if nb > 8 or rng.random() < 0.4 else "orbital"
    if kind == "build":
        return dict(kind=kind, n1=n1, n2=n2, nb=nb, v=v, hermitian=rng.random() < 0.7,
                    out=rng.choice(("fe", "sigma")), extras=nb <= 8 and rng.random() < 0.3,
                    precision=32 if nb <= 8 and rng.random() < 0.2 else 64)
    if kind == "grad":
        return dict(kind=kind, n1=n1, n2=n2, nb=nb, v=v)
    T, fill = round(rng.uniform(0.05, 0.2), 3), round(rng.uniform(0.3, 0.7), 3)
    if kind == "density":
        return dict(kind=kind, n1=n1, n2=n2, nb=nb, T=T, fill=fill, backward=rng.random() < 0.5)
    U = round(rng.uniform(0.5, 1.5), 2) if nb <= 8 else 0.5
    iters = rng.randint(3, 8) if nb <= 8 else rng.randint(2, 4)
    return dict(kind=kind, n1=n1, n2=n2, nb=nb, v=v, T=T, U=U, fill=fill, iters=iters)


# ---------------------------------------------------------------------------
# models, on the GPU
# ---------------------------------------------------------------------------

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _herm(X):
    return 0.5 * (X + X.mH)


def _cnormal(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=F64),
                         torch.randn(shape, generator=g, device="cuda", dtype=F64))


def _kgrid(n1, n2):
    k1 = -math.pi + 2.0 * math.pi * torch.arange(n1, device="cuda", dtype=F64) / n1
    k2 = -math.pi + 2.0 * math.pi * torch.arange(n2, device="cuda", dtype=F64) / n2
    return torch.meshgrid(k1, k2, indexing="ij")


def _plane_waves(count):
    """The `count` shortest vectors of the triangular lattice, integer and Cartesian."""
    B = np.array([[1.0, 0.5], [0.0, math.sqrt(3.0) / 2.0]])
    r = int(math.ceil(math.sqrt(count))) + 2
    g = np.array([(a, b) for a in range(-r, r + 1) for b in range(-r, r + 1)], dtype=np.int64)
    x = g @ B.T
    order = np.lexsort((np.round(np.mod(np.arctan2(x[:, 1], x[:, 0]), 2 * math.pi), 9),
                        np.round(np.hypot(x[:, 0], x[:, 1]), 9)))[:count]
    return g[order], x[order], B


def _hamiltonian(n1, n2, nb, g):
    """h(k) with seeded Hermitian noise: the 2-band Dirac model, a stack of A/B layers (an odd band
    count leaves the top layer one sublattice), or a Dirac superlattice of nb / 2 plane waves."""
    kx, ky = _kgrid(n1, n2)
    h = torch.zeros((n1, n2, nb + (nb & 1), nb + (nb & 1)), dtype=C128, device="cuda")
    if nb == 2:
        d = -0.5 + 2.0 - torch.cos(kx) - torch.cos(ky)
        h[..., 0, 0], h[..., 1, 1] = d.to(C128), -d.to(C128)
        h[..., 0, 1] = torch.complex(torch.sin(kx), -torch.sin(ky))
        h[..., 1, 0] = torch.complex(torch.sin(kx), torch.sin(ky))
        noise = 0.01
    elif nb <= 8:
        layers = (nb + 1) // 2
        f = 1.0 + torch.polar(torch.ones_like(kx), kx) + torch.polar(torch.ones_like(ky), ky)
        for l in range(layers):
            a, b = 2 * l, 2 * l + 1
            h[..., a, b], h[..., b, a] = f, f.conj()
            ramp = 0.2 * ((l / (layers - 1) if layers > 1 else 0.0) - 0.5)
            h[..., a, a] += ramp
            h[..., b, b] += ramp
            if l + 1 < layers:
                h[..., a + 2, b] += 0.4
                h[..., b, a + 2] += 0.4
        noise = 0.005
    else:
        gi, gc, B = _plane_waves(nb // 2)
        fx, fy = (kx + math.pi) / (2 * math.pi), (ky + math.pi) / (2 * math.pi)
        qx, qy = B[0, 0] * fx + B[0, 1] * fy, B[1, 0] * fx + B[1, 1] * fy
        phase = torch.rand((nb, nb), generator=g, device="cuda", dtype=F64).cpu().numpy() * 2 * math.pi
        for a in range(nb // 2):
            z = torch.complex(qx + gc[a, 0], -(qy + gc[a, 1]))
            h[..., 2 * a, 2 * a + 1], h[..., 2 * a + 1, 2 * a] = z, z.conj()
            for b in range(a + 1, nb // 2):
                if abs(math.hypot(*(gc[a] - gc[b])) - 1.0) < 1e-9:
                    c = 0.1 * complex(math.cos(phase[a, b]), math.sin(phase[a, b]))
                    for s in range(2):
                        h[..., 2 * a + s, 2 * b + s] = c
                        h[..., 2 * b + s, 2 * a + s] = c.conjugate()
        noise = 0.005
    h = h[..., :nb, :nb]
    return (h + noise * _herm(_cnormal(g, n1, n2, nb, nb))).contiguous()


def _coulomb(n1, n2, nb, v, U):
    kx, ky = _kgrid(n1, n2)
    q = torch.hypot(kx, ky)
    if v == "scalar":
        return (2 * math.pi * U / (q + 0.05) * torch.tanh(5 * q))[..., None, None]
    layer = torch.arange(nb, device="cuda") // 2
    dl = (layer[:, None] - layer[None, :]).abs().to(F64)
    return (2 * math.pi * U / (q + 0.05))[..., None, None] * torch.exp(-0.3 * q[..., None, None] * dl)


def _vr(Vq, w):
    """FFT2(w V) with the phase that centres the mesh (the kernel arrays' VR)."""
    n1, n2 = w.shape
    p1 = torch.exp(2j * math.pi * torch.arange(n1, device="cuda", dtype=F64) * (n1 // 2) / n1)
    p2 = torch.exp(2j * math.pi * torch.arange(n2, device="cuda", dtype=F64) * (n2 // 2) / n2)
    VR = torch.fft.fftn((w[..., None, None] * Vq).to(C128), dim=(0, 1))
    return (VR * (p1[:, None] * p2[None, :])[..., None, None]).contiguous()


def _density(g, n1, n2, nb):
    """Hermitian P(k), eigenvalues in [0, 1]: U diag(lam) U^H, U a Cayley unitary or, for many bands, a
    Householder reflection."""
    lam = torch.rand((n1, n2, nb), generator=g, device="cuda", dtype=F64)
    if nb <= 8:
        S = _herm(_cnormal(g, n1, n2, nb, nb))
        I = torch.eye(nb, dtype=C128, device="cuda")
        Q = torch.linalg.solve(I + 0.5j * S, I - 0.5j * S)
        return _herm((Q * lam[..., None, :].to(C128)) @ Q.mH).contiguous()
    u = _cnormal(g, n1, n2, nb)
    u = u / torch.linalg.vector_norm(u, dim=-1, keepdim=True)
    lu = lam.to(C128) * u
    P = torch.diag_embed(lam.to(C128)) - 2 * lu[..., :, None] * u.conj()[..., None, :]
    P -= 2 * u[..., :, None] * lu.conj()[..., None, :]
    P += 4 * (u.conj() * lu).sum(-1)[..., None, None] * u[..., :, None] * u.conj()[..., None, :]
    return _herm(P).contiguous()


def _problem(case, seed):
    """(kernel_args with device tensors, generator) of a mesh problem."""
    n1, n2, nb = case["n1"], case["n2"], case["nb"]
    g = _rng(seed)
    w = torch.full((n1, n2), 1.0 / (n1 * n2), dtype=F64, device="cuda")
    h = _hamiltonian(n1, n2, nb, g)
    VR = _vr(_coulomb(n1, n2, nb, case["v"], case.get("U", 1.0)), w)
    args = dict(h=h, VR=VR, refP=np.empty((0,), np.complex128), has_refP=False, w2d=w, HH=np.zeros((nb, nb)),
                contact_g=np.zeros((1,)), contact_Oi=np.zeros((1, nb, nb), np.complex128),
                contact_Oj=np.zeros((1, nb, nb), np.complex128), weight_sum=1.0, T=float(case.get("T", 0.05)),
                include_hartree=False, include_exchange=True, exchange_hcp=case["v"] == "scalar")
    if case.get("extras"):
        r = np.random.default_rng(seed)
        HH = r.normal(size=(nb, nb))
        O = r.normal(size=(4, nb, nb)) + 1j * r.normal(size=(4, nb, nb))
        O = 0.5 * (O + np.conj(np.swapaxes(O, -1, -2)))
        args.update(refP=_density(g, n1, n2, nb), has_refP=True, include_hartree=True, HH=0.5 * (HH + HH.T),
                    contact_g=r.normal(size=2), contact_Oi=O[:2].copy(), contact_Oj=O[2:].copy())
    return args, g


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "stream":
        n, orb = case["n"], case["orb"]
        g = _rng(seed)
        gi, gc, B = _plane_waves(case["pw"])
        lay = superlattice.extended_layout(gi, B, n, n, lambda q: math.pi / (q + 0.05) * np.tanh(5.0 * q),
                                           1.0 / (n * n))
        D = case["pw"] * orb
        rho = _cnormal(g, n, n, D, D) * 0.1
        if case["hermitian"]:
            rho = _herm(rho)
        return dict(case=case, lay=lay, rho=rho.reshape(n, n, case["pw"], orb, case["pw"], orb).contiguous(),
                    V=torch.from_numpy(lay.V_lag_fft).cuda())
    n1, n2, nb = case["n1"], case["n2"], case["nb"]
    if kind == "density":
        g = _rng(seed)
        w = torch.full((n1, n2), 1.0 / (n1 * n2), dtype=F64, device="cuda")
        F = _hamiltonian(n1, n2, nb, g) + 0.05 * _herm(_cnormal(g, n1, n2, nb, nb))
        return dict(case=case, F=F, w=w, n_e=case["fill"] * nb, gP=_herm(_cnormal(g, n1, n2, nb, nb)).contiguous())
    args, g = _problem(case, seed)
    if kind == "build":
        fb = FockBuilder(args, precision=case["precision"], hermitian_density=case["hermitian"])
        return dict(case=case, args=args, fb=fb, P=_density(g, n1, n2, nb))
    if kind == "grad":
        return dict(case=case, args=args, P=_density(g, n1, n2, nb))
    return dict(case=case, args=args, P0=torch.zeros_like(args["h"]), n_e=case["fill"] * nb,
                none=torch.empty((0, n1, n2, nb, nb), dtype=C128, device="cuda"))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "build":
        out = s["fb"].build(s["P"]) if case["out"] == "sigma" else s["fb"].build_fe(s["P"])
        return list(out)
    if kind == "grad":
        a = s["args"]
        P, h, VR = (x.detach().requires_grad_(True) for x in (s["P"], a["h"], a["VR"]))
        Sigma, H, F = autograd.build_fock(P, h=h, VR=VR, w2d=a["w2d"], include_exchange=True)
        E = autograd.hf_energy(P, h=h, Sigma=Sigma, H=H, weights_b=a["w2d"][..., None, None])
        return [E.detach(), F.detach()] + list(torch.autograd.grad(E, (P, h, VR)))
    if kind == "density":
        F = s["F"].detach().requires_grad_(case["backward"])
        P, eps, mu = autograd.density_from_fock(F, s["w"], s["n_e"], case["T"])
        out = [P.detach(), eps, mu]
        return out + list(torch.autograd.grad(P, F, s["gP"])) if case["backward"] else out
    if kind == "dm":
        r = _native.solve_dm(s["args"], s["P0"], s["n_e"], case["iters"], DM["tol_E"], DM["tol_grad"],
                             DM["max_step"], DM["bt_shrink"], DM["denom_scale"], DM["bt_max"], DM["cg_restart"],
                             DM["plateau_window"], DM["mu_maxiter"], 0, 0.5, 20, s["none"], 0.0, 1.0, [], None,
                             False, True, True)
        return dict(p=r[1], density=r[2], fock=r[3], mu=r[4], energy=r[5], hist_E=r[8], hist_grad=r[9])
    if kind == "scf":
        r = _native.solve_scf(s["args"], s["P0"], s["n_e"], case["iters"], 0.0, 0.0, MIXING, 0.0, None, [],
                              "linear", 6, 2, 1.0, 0.0, True, True)
        return dict(density=r[0], fock=r[1], energy=r[2], mu=r[3], hist_E=r[6], hist_D=r[7], hist_C=r[8])
    lay, n = s["lay"], case["n"]
    return _native.selfenergy_superlattice_streamed(
        s["rho"], s["V"], lay.g_a_off, lay.delta_pair_i, lay.delta_pair_j, lay.delta_pair_start, n, n, case["pw"],
        case["orb"], lay.N_ext_x, lay.N_ext_y, None, case["hermitian"])


def work(case):
    """Bytes: inputs once, outputs once.  Flops: the transforms at 5 N log2 N per channel and direction,
    and 8 flops per complex multiply-add of the per-k products."""
    kind = case["kind"]
    if kind == "stream":
        n, pw, orb = case["n"], case["pw"], case["orb"]
        gi, _, _ = _plane_waves(pw)
        dim = gi.max(axis=0) - gi.min(axis=0) + 1
        N = float(2 * n * dim[0] * 2 * n * dim[1])
        deltas = len({tuple(a - b) for a in gi for b in gi})
        ch = (deltas + 1) / 2 if case["hermitian"] else deltas
        return dict(bytes=2 * 16.0 * n * n * (pw * orb) ** 2 + 16 * N,
                    flops=ch * orb * orb * 10 * N * math.log2(N))
    n1, n2, nb = case["n1"], case["n2"], case["nb"]
    nk = float(n1 * n2)
    field = 16.0 * nk * nb * nb
    v = 16.0 * nk if case.get("v") == "scalar" else field
    fft = 10.0 * nk * math.log2(nk)
    if kind == "density":
        # eigh with vectors about 32 nb^3, the density 8 nb^3, its gradient four products
        per_k = (32 + 8 + (32 if case["backward"] else 0)) * nb ** 3
        return dict(bytes=(4 if case["backward"] else 2) * field + 8 * nk * nb, flops=nk * per_k)
    if kind == "grad":
        return dict(bytes=5 * field + 2 * v, flops=nb * nb * 2.5 * fft)
    half = nb * (nb + 1) / 2
    if kind == "build":
        part = half / nb ** 2 if case["hermitian"] else 1.0
        n_in = 2 + (1 if case["extras"] else 0)
        vb = v if case["v"] == "scalar" else part * v
        return dict(bytes=n_in * part * field + vb + (2 if case["out"] == "sigma" else 1) * field,
                    flops=part * nb * nb * fft)
    # solvers: h, VR and P0 in, density and Fock out; per iteration a build and the per-k products (DM:
    # density, rotation, Cayley step, diagonal, retraction; SCF: eigh, density, commutator)
    per_k = {"dm": 48, "scf": 56}[kind] * nb ** 3
    ends = (72 if kind == "dm" else 40) * nb ** 3 * nk
    return dict(bytes=4 * field + v, flops=(case["iters"] + 1) * (half * fft + nk * per_k) + ends)


# ---------------------------------------------------------------------------
# 64-bit values in plain torch
# ---------------------------------------------------------------------------

def _convolve(R, VR):
    return -torch.fft.ifftn(torch.fft.fftn(R, dim=(0, 1)) * VR, dim=(0, 1))


def _eigh(F):
    w, V = torch.linalg.eigh(_herm(F).cpu())
    return w.cuda(), V.cuda()


def _plain_build(a, P):
    """(Sigma, F, E) of a kernel_args dict."""
    w = a["w2d"]
    R = P - a["refP"] if a["has_refP"] else P
    Sigma = _convolve(R, a["VR"])
    rho = (w[..., None, None] * R).sum(dim=(0, 1))
    for c, Oi, Oj in zip(a["contact_g"], a["contact_Oi"], a["contact_Oj"]):
        if c != 0.0:
            Oi, Oj = torch.from_numpy(Oi).cuda(), torch.from_numpy(Oj).cuda()
            Sigma = Sigma + c * (Oi * (Oj * rho.T).sum() - Oi @ rho @ Oj)
    A = Sigma
    if a["include_hartree"]:
        A = Sigma + torch.diag((torch.from_numpy(a["HH"]).cuda() @ torch.diagonal(rho).real).to(C128))
    tr = lambda X, Y: (w * (X * Y.transpose(-1, -2)).sum(dim=(-2, -1)).real).sum()  # noqa: E731
    return Sigma, _herm(a["h"] + A), tr(a["h"], P) + 0.5 * tr(A, R)


def _fermi(x, T):
    return torch.sigmoid(-x / (T + 1e-12))


def _mu_bisect(eps, w, n_e, T):
    span = float(eps.max() - eps.min()) + 10.0 * max(T, 1e-6)
    lo, hi = float(eps.min()) - span, float(eps.max()) + span
    for _ in range(30):
        mid = 0.5 * (lo + hi)
        if float((w[..., None] * _fermi(eps - mid, T)).sum()) > n_e:
            hi = mid
        else:
            lo = mid
    return 0.5 * (lo + hi)


def _mu_newton(eps, w, n_e, T, mu):
    lo, hi = float(eps.min()) - 50 * T, float(eps.max()) + 50 * T
    mu = min(max(mu, lo), hi)
    for _ in range(DM["mu_maxiter"]):
        p = torch.sigmoid((mu - eps) / T)
        d = float((w[..., None] * p).sum()) - n_e
        Z = float((w[..., None] * p * (1 - p)).sum()) / T
        lo, hi = (mu if d < 0 else lo), (mu if d > 0 else hi)
        new = mu - d / max(Z, 1e-18)
        mu = min(max(new if lo < new < hi else 0.5 * (lo + hi), lo), hi)
    return mu


def _occupied(V, occ):
    return _herm((V * occ[..., None, :].to(C128)) @ V.mH)


def _plain_dm(s):
    a, case, n_e, w = s["args"], s["case"], s["n_e"], s["args"]["w2d"]
    T = max(a["T"], 1e-12)
    ip = lambda X, Y: float((w * (X.conj() * Y).real.flatten(2).sum(-1)).sum())  # noqa: E731

    def omega(e, p):
        p = p.clamp(1e-8, 1 - 1e-8)
        ent = -(p * torch.log(p) + (1 - p) * torch.log1p(-p))
        return float((w[..., None] * (p * e - T * ent)).sum())

    eps, Q = _eigh(_plain_build(a, s["P0"])[1])
    mu = _mu_newton(eps, w, n_e, T, 0.0)
    p = torch.sigmoid((mu - eps) / T)
    I = torch.eye(case["nb"], dtype=C128, device="cuda")
    hist_E, hist_g, prev = [], [], None
    for k in range(case["iters"]):
        _, F, E = _plain_build(a, _occupied(Q, p))
        Ft = Q.mH @ F @ Q
        eps = torch.diagonal(Ft, dim1=-2, dim2=-1).real
        A = (p[..., None, :] - p[..., :, None]) * Ft
        G = 0.5 * (A - A.mH)
        pl = p.clamp(1e-6, 1 - 1e-6)
        gp = eps + T * (torch.log(pl) - torch.log1p(-pl)) - mu
        hist_E.append(float(E))
        hist_g.append(math.sqrt(max(0.0, ip(G, G))))
        lam = max(T, DM["denom_scale"] * math.sqrt(float((eps * eps).mean()) + 1e-30))
        gap = eps[..., :, None] - eps[..., None, :]
        d = G / torch.sqrt(gap * gap + lam * lam)
        ps = p.clamp(1e-8, 1 - 1e-8)
        dp = gp * ps * (1 - ps) / T
        beta = 0.0
        if prev is not None and k % DM["cg_restart"]:
            Gp, gpp, dpr, dpp = prev
            num = ip(G - Gp, d) + float((w[..., None] * (gp - gpp) * dp).sum())
            den = ip(Gp, Gp) + float((w[..., None] * gpp * gpp).sum())
            beta = min(max(0.0, num / den), 5.0) if den > 1e-30 else 0.0
            d, dp = d + beta * dpr, dp + beta * dpp
        tau0 = min(1.0, DM["max_step"] / max(math.sqrt(ip(d, d)), 1e-30))
        start, tau = omega(eps, p), tau0
        step = lambda t: torch.linalg.solve(I + 0.5 * t * d, I - 0.5 * t * d)  # noqa: E731
        value = lambda M: torch.diagonal(M.mH @ Ft @ M, dim1=-2, dim2=-1).real  # noqa: E731
        for _ in range(DM["bt_max"]):
            if omega(value(step(tau)), p - tau * dp) < start:
                break
            tau *= DM["bt_shrink"]
        M = step(tau)
        eps = value(M)
        Q = Q @ M
        mu = _mu_newton(eps, w, n_e, T, mu)
        p = torch.sigmoid((mu - eps) / T)
        prev = (G, gp, d, dp)
    F = _plain_build(a, _occupied(Q, p))[1]
    eps, V = _eigh(Q.mH @ F @ Q)
    Q = Q @ V
    mu = _mu_newton(eps, w, n_e, T, mu)
    p = torch.sigmoid((mu - eps) / T)
    P = _occupied(Q, p)
    _, F, E = _plain_build(a, P)
    return dict(p=p, density=P, fock=F, mu=mu, energy=float(E), hist_E=np.array(hist_E), hist_grad=np.array(hist_g))


def _plain_scf(s):
    a, case, w = s["args"], s["case"], s["args"]["w2d"]
    norm = lambda X: math.sqrt(float((w * (X.abs() ** 2).flatten(2).sum(-1)).sum()))  # noqa: E731
    D, hE, hD, hC = s["P0"], [], [], []
    for it in range(case["iters"] + 1):
        _, F, E = _plain_build(a, D)
        eps, V = _eigh(F)
        mu = _mu_bisect(eps, w, s["n_e"], a["T"])
        if it == case["iters"]:
            break
        Pn = _occupied(V, _fermi(eps - mu, a["T"]))
        hE.append(float(E))
        hD.append(norm(Pn - D))
        hC.append(norm(F @ D - D @ F))
        D = _herm(D + MIXING * (Pn - D))
    return dict(density=D, fock=F, energy=float(E), mu=mu, hist_E=np.array(hE), hist_D=np.array(hD),
                hist_C=np.array(hC))


def exact(case, seed):
    kind = case["kind"]
    if kind != "stream":
        # a batched LAPACK eigh of one core: about 20 nb^3 operations a matrix at a few GFLOP/s
        eighs = {"density": 1, "dm": 2, "scf": case.get("iters", 0) + 1}.get(kind, 0)
        if eighs * case["n1"] * case["n2"] * (20e-9 * case["nb"] ** 3 + 20e-6) > 15.0:
            return None
    s = prepare(case, seed)
    if kind == "build":
        out = _plain_build(s["args"], s["P"])
        out = [out[0], out[1], out[2].reshape(1)]
        return out if case["out"] == "sigma" else out[1:]
    if kind == "grad":
        a = s["args"]
        P, h, VR = (x.detach().requires_grad_(True) for x in (s["P"], a["h"], a["VR"]))
        _, F, E = _plain_build(dict(a, h=h, VR=VR), P)
        return [E.detach(), F.detach()] + list(torch.autograd.grad(E, (P, h, VR)))
    if kind == "density":
        T, w = case["T"], s["w"]
        eps, V = _eigh(s["F"])
        mu = _mu_bisect(eps, w, s["n_e"], T)
        f = _fermi(eps - mu, T)
        out = [_occupied(V, f), eps, torch.tensor([mu], dtype=F64, device="cuda")]
        if not case["backward"]:
            return out
        # divided differences of the Fermi function, n_e held fixed: with x_lo <= x_hi,
        # f_lo - f_hi = f_lo (1 - f_hi) (1 - exp(x_lo - x_hi)), free of cancellation
        Te = T + 1e-12
        G = V.mH @ s["gP"] @ V
        x = (eps - mu) / Te
        lo, hi = torch.minimum(x[..., :, None], x[..., None, :]), torch.maximum(x[..., :, None], x[..., None, :])
        d = (hi - lo).clamp(min=1e-300)
        L = torch.sigmoid(-lo) * torch.sigmoid(hi) * torch.expm1(-d) / d / Te
        fp = -torch.sigmoid(-x) * torch.sigmoid(x) / Te
        A = (torch.diagonal(G, dim1=-2, dim2=-1).real * fp).sum()
        Z = (w[..., None] * fp).sum()
        M = G * L - torch.diag_embed((w[..., None] * fp * (A / Z)).to(C128))
        return out + [V @ M @ V.mH]
    if kind == "dm":
        return _plain_dm(s)
    if kind == "scf":
        return _plain_scf(s)
    lay, n, rho = s["lay"], case["n"], s["rho"]
    sigma = torch.zeros_like(rho)
    for c in range(lay.n_delta):
        a, b = int(lay.delta_pair_start[c]), int(lay.delta_pair_start[c + 1])
        buf = torch.zeros((lay.N_ext_x, lay.N_ext_y, case["orb"], case["orb"]), dtype=C128, device="cuda")
        at = []
        for i, j in zip(lay.delta_pair_i[a:b], lay.delta_pair_j[a:b]):
            x, y = (int(v) * n for v in lay.g_a_off[i])
            at.append((slice(x, x + n), slice(y, y + n), int(i), int(j)))
            buf[at[-1][:2]] = rho[:, :, i, :, j, :]
        buf = _convolve(buf, s["V"][..., None, None])
        for x, y, i, j in at:
            sigma[:, :, i, :, j, :] = buf[x, y]
    return sigma
