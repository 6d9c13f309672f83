"""A solver built under one streaming kernel and run under another that needs more partial sums (march -> xp, zp)."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx
from voxel_b200 import _lib, slab
from voxel_b200 import solver as vs
from voxel_b200.batch import BatchedSolver
from voxel_b200.problems import cantilever_equal_split

pytestmark = pytest.mark.gpu
KE = vx.quadrature([1.0, 1.0, 1.0], 0.3)
SHAPE = (3, 300, 1500)      # more partial sums under xp than any scratch that a solver has for other uses


@pytest.fixture(autouse=True)
def march():
    prev = _lib.set_stream_kernel("march")
    yield
    _lib.set_stream_kernel(prev)


def problem(shape):
    g = torch.Generator("cuda").manual_seed(9)
    E = 0.1 + torch.rand(int(np.prod(shape)), dtype=torch.float64, device="cuda", generator=g)
    mask, force = cantilever_equal_split(shape)
    return E, mask, vx.node_mask_from_dofs(mask), force


def counts(shape):
    n = {}
    for kind in ("march", "xp", "zp"):
        _lib.set_stream_kernel(kind)
        n[kind] = vx.VoxelOperator(shape, KE).partials_size
    _lib.set_stream_kernel("march")
    return n


def run(build, shape, kinds):
    """The results of one solver under the kernels `kinds` in turn, and of solvers built under each of them."""
    E, mask, nm, force = problem(shape)
    s = build(E, mask, nm)
    got, want = [], []
    for kind in kinds:
        _lib.set_stream_kernel(kind)
        got.append([v.clone() if torch.is_tensor(v) else v for v in s(force)])
        want.append([v.clone() if torch.is_tensor(v) else v for v in build(E, mask, nm)(force)])
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            assert torch.equal(a, b) if torch.is_tensor(a) else a == b


def test_the_selections_need_different_scratch():
    n = counts(SHAPE)
    assert n["xp"] > max(n["march"], 2 * 1184)                # 2368: vx_jacobi_step's partials
    m = counts((32, 16, 16))
    assert len(set(m.values())) > 1


@pytest.mark.parametrize("shape", [(32, 16, 16), SHAPE])
def test_jacobi_fcg(shape):
    def build(E, mask, nm):
        op = vx.VoxelOperator(shape, KE)
        s = vs.FCGSolver(op, E, nm, vs.JacobiPreconditioner(op, E, nm), tol=1e-12, maxiter=20, check_every=5, graph=False)
        return lambda f: tuple(s.solve(f))
    run(build, shape, ["xp", "march", "zp", "xp"])


def test_graph_captured_after_the_switch_and_tail_under_another_kernel():
    E, mask, nm, force = problem(SHAPE)
    op = vx.VoxelOperator(SHAPE, KE)
    s = vs.FCGSolver(op, E, nm, vs.JacobiPreconditioner(op, E, nm), tol=1e-12, maxiter=23, check_every=10)
    _lib.set_stream_kernel("xp")
    want = s.solve(force).x.clone()
    _lib.set_stream_kernel("march")
    s.solve(force)                                            # loop: the captured xp kernel; tail: march
    _lib.set_stream_kernel("xp")
    assert torch.equal(s.solve(force).x, want)


def test_donor_solvers():
    def pcg(E, mask, nm):
        s = vs.JacobiPCG(vx.VoxelOperator(SHAPE, KE), E, nm, tol=1e-12, maxiter=20, check_every=5, graph=False)
        return lambda f: tuple(s.solve(f))

    def ir(E, mask, nm):
        s = vs.PCGIR(vx.VoxelOperator(SHAPE, KE), E, nm, tol=1e-12, max_outer=3, inner_maxiter=10, check_every=5, graph=False)
        return lambda f: tuple(s.solve(f))
    for build in (pcg, ir):
        run(build, SHAPE, ["xp", "march", "zp"])


def test_batch_and_slabs():
    shape = (64, 48, 48)

    def batch(E, mask, nm):
        s = BatchedSolver(shape, 2, precision="fp64", maxiter=6, chunk=3)
        def go(f):
            s.admit([(0, E, f, 1e-8), (1, E, 2 * f, 1e-8)])
            s.run(2)                                          # not the captured chunk
            s.poll()
            return [s.result(k)[0] for k in (0, 1)]
        return go

    def slabs(E, mask, nm):
        s = slab.SlabSolver(shape, E, mask, 2, precision="fp64", tol=1e-12, maxiter=4, graph=False)

        def go(f):
            r = s.solve(f)
            return [s.gather().clone(), r.iterations, r.rel]
        return go
    for build in (batch, slabs):
        run(build, shape, ["xp", "march", "zp"])


def test_short_partials_are_refused():
    E, mask, nm, force = problem((24, 24, 24))
    op = vx.VoxelOperator((24, 24, 24), KE)
    q, n = torch.empty_like(force), op.partials_size
    part, S = torch.zeros(n - 1, dtype=torch.float64, device="cuda"), torch.zeros(16, dtype=torch.float64, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    for call in (lambda: op.apply_dot(force, E, nm, q, part), lambda: op.true_residual(force, force, E, nm, q, part),
                 lambda: op.apply_dot_fin(force, E, nm, q, part, S, counter, 0),
                 lambda: op.true_residual_fin(force, force, E, nm, q, part, S, counter, 1)):
        with pytest.raises(ValueError, match="partials"):
            call()
