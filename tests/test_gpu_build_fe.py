"""GPU: FockBuilder.build_fe on every kind of build: packed, packing asked for on mesh sides without a codelet, many bands."""

from __future__ import annotations

import numpy as np
import pytest

from cpp_hf_b200 import problem

pytestmark = pytest.mark.gpu


def herm(X):
    return 0.5 * (X + np.conj(np.swapaxes(X, -1, -2)))


# shape, width of V, extras, and which build it takes: (packed, fused)
CASES = (
    ((24, 36, 4), 4, False, (True, True)),
    ((75, 98, 5), 5, False, (False, False)),
    ((100, 100, 3), 1, True, (False, False)),
    ((7, 24, 8), 8, True, (False, False)),
    ((24, 7, 2), 1, False, (False, False)),
    ((11, 96, 64), 1, False, (False, True)),
    ((15, 65, 64), 1, True, (False, False)),
    ((9, 8, 12), 1, False, (False, False)),
)


@pytest.mark.parametrize("shape,dv,extras,kind", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_build_fe(oracle, shape, dv, extras, kind):
    import torch

    from cpp_hf_b200.fock_builder import FockBuilder

    n1, n2, nb = shape
    r = np.random.default_rng(nb)

    def field():
        return herm(r.normal(size=(n1, n2, nb, nb)) + 1j * r.normal(size=(n1, n2, nb, nb)))

    w = np.full((n1, n2), 1.0 / (n1 * n2))
    V = r.normal(size=(n1, n2, dv, dv))
    kw = dict(include_hartree=True, hartree_matrix=np.ones((nb, nb)), reference_density=field()) if extras else {}
    args = problem.kernel_args(w, field(), V + np.swapaxes(V, -1, -2), 0.1, **kw)
    P = np.ascontiguousarray(field())
    fb = FockBuilder(args, hermitian_density=True)
    assert (fb.packed, fb.fused) == kind
    Pd = torch.from_numpy(P).cuda()
    _, F0, E0 = (x.clone() for x in fb.build(Pd))
    fb.Sigma.fill_(7.0)
    F1, E1 = fb.build_fe(Pd)
    assert torch.equal(F0, F1) and torch.equal(E0, E1)
    assert bool((fb.Sigma == 7.0).all()) == fb.fused
    ref = oracle.build_fock_apply(args, P, None)
    assert np.abs(F1.cpu().numpy() - ref[2]).max() <= 1e-12 * max(1.0, np.abs(ref[2]).max())
    assert abs(float(E1) - ref[3]) <= 1e-12 * max(1.0, abs(ref[3]))


@pytest.mark.parametrize("shape,dv,extras,kind", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_launches_per_build(native, shape, dv, extras, kind):
    import torch
    from cuda.bindings import runtime as rt

    from cpp_hf_b200.fock_builder import FockBuilder

    n1, n2, nb = shape
    one = np.broadcast_to(np.eye(nb, dtype=complex), (n1, n2, nb, nb)).copy()
    kw = dict(include_hartree=True, hartree_matrix=np.ones((nb, nb))) if extras else {}
    args = problem.kernel_args(np.full((n1, n2), 1.0 / (n1 * n2)), one, np.ones((n1, n2, dv, dv)), 0.1,
                               reference_density=0 * one, **kw)
    fb = FockBuilder(args, hermitian_density=True)
    P = torch.from_numpy(one).cuda()
    fb.build_fe(P)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fb.build_fe(P)
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(raw)
    assert err == rt.cudaError_t.cudaSuccess
    err, nodes, _ = rt.cudaGraphGetNodes(raw, count)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes]
    assert kinds.count(rt.cudaGraphNodeType.cudaGraphNodeTypeKernel) == fb.launches_per_build
