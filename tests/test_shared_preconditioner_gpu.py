"""Solvers that share one JacobiPreconditioner and take turns, and a preconditioner whose emit was replaced."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx
from voxel_b200 import solver as vs
from voxel_b200.problems import cantilever_equal_split

pytestmark = pytest.mark.gpu
KE = vx.quadrature([1.0, 1.0, 1.0], 0.3)
SHAPES = [(12, 6, 6), (52, 46, 46)]          # on both sides of the small systems' iteration (303,104 unknowns)


def problem(shape):
    g = torch.Generator("cuda").manual_seed(5)
    E = 0.1 + torch.rand(int(np.prod(shape)), dtype=torch.float64, device="cuda", generator=g)
    mask, force = cantilever_equal_split(shape)
    other = torch.randn(force.numel(), dtype=torch.float64, device="cuda", generator=g) * mask
    return vx.VoxelOperator(shape, KE), E, vx.node_mask_from_dofs(mask), force, other


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_solvers_sharing_a_preconditioner_take_turns(shape, graph):
    """With the graph, the iterations past the last full body run in finish() (23 = 2 x 10 + 3)."""
    op, E, nm, force, other = problem(shape)
    M = vs.JacobiPreconditioner(op, E, nm)
    a, b = (vs.FCGSolver(op, E, nm, M, tol=1e-12, maxiter=23, check_every=10, graph=graph) for _ in range(2))
    alone = a.solve(force)
    want = (alone.x.clone(), alone.iterations, alone.rel)
    a.launch(force)
    torch.cuda.synchronize()
    b.launch(other)
    torch.cuda.synchronize()
    res = a.finish()
    b.finish()
    assert (res.iterations, res.rel) == want[1:]
    assert torch.equal(res.x, want[0])


@pytest.mark.parametrize("shape", SHAPES)
def test_a_replaced_emit_is_called(shape):
    """z = r instead of d r: plain conjugate gradients."""
    op, E, nm, force, _ = problem(shape)
    M = vs.JacobiPreconditioner(op, E, nm)
    calls = []

    def emit(r):
        calls.append(1)
        M.z.copy_(r)
        return M.z

    class Plain(vs.JacobiPreconditioner):
        def emit(self, r):
            self.z.copy_(r)
            return self.z

    want = vs.FCGSolver(op, E, nm, Plain(op, E, nm), tol=1e-12, maxiter=20, check_every=5, graph=False).solve(force)
    M.emit = emit
    res = vs.FCGSolver(op, E, nm, M, tol=1e-12, maxiter=20, check_every=5, graph=False).solve(force)
    assert len(calls) == 21
    assert torch.equal(res.x, want.x) and res.rel == want.rel
