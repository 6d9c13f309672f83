"""The default streaming operator (parity_march) where its tiling can go wrong: node counts one below,
at and one above the tile edges (14 x 14 nodes a CTA in FP64, 14 x 30 in FP32), a single element in a
direction, x chunks of one plane and of many, fixed DOFs scattered over every edge, cube and brick
elements, every fused form and storage mode.  Against the FP64 oracle on the rounded inputs; tolerances
in max-norm relative: FP64 1e-13, FP32 arithmetic 1e-5, outputs stored in bf16 one rounding (4.5e-3)."""
import numpy as np
import pytest
import torch

from oracle import voxel_oracle as vo

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("voxel_b200")
from voxel_b200 import _lib  # noqa: E402

F64, F32, BF16 = torch.float64, torch.float32, torch.bfloat16
GRIDS = [(2, 12, 12), (3, 13, 13), (6, 14, 27), (1, 5, 29), (2, 4, 28), (3, 6, 30), (4, 13, 59), (5, 14, 60), (70, 12, 1), (1, 1, 64), (9, 27, 2), (40, 29, 89)]
CUBE, BRICK = vo.quadrature([1, 1, 1], 0.3), vo.quadrature([1.0, 0.5, 2.0], 0.25)


def maxrel(t, ref):
    return float(np.max(np.abs(t.double().cpu().numpy() - ref)) / max(np.max(np.abs(ref)), 1e-300))


@pytest.mark.parametrize("shape", GRIDS)
@pytest.mark.parametrize("dtype,aux", [(F64, F64), (F32, F32), (F32, BF16), (BF16, BF16)])
def test_every_form_at_tile_edges(shape, dtype, aux):
    rng = np.random.default_rng(sum(shape))
    ke = CUBE if shape[0] % 2 else BRICK
    cu = lambda v, dt: torch.as_tensor(v, device="cuda").to(dt)
    n = 3 * vo.n_nodes(shape)
    E = cu(1e-3 + rng.random(int(np.prod(shape))), aux)
    u, r = cu(rng.standard_normal(n), dtype), cu(rng.standard_normal(n), aux)
    mask = vo.cantilever_equal_split(shape)[0] * (rng.random(n) > 0.05)
    nm = vx.node_mask_from_dofs(cu(mask, F64))
    Eh, uh, rh = (t.double().cpu().numpy() for t in (E, u, r))
    invd = cu(1 / np.where(mask != 0, vo.product_diagonal(shape, ke, Eh), 1.0), aux)
    dh = invd.double().cpu().numpy()
    A, K = vo.apply_dirichlet(shape, ke, Eh, mask, uh), vo.product_raw(shape, ke, uh, Eh)
    op = vx.VoxelOperator(shape, ke, dtype, aux)
    tol = {F64: 1e-13, F32: 1e-5}
    out = lambda dt: tol.get(dt, 4.5e-3)
    if (dtype, aux) != (F32, BF16):
        t = tol.get(dtype, 1e-5)
        assert maxrel(op.matvec(u, E), K) < t and maxrel(op.matvec(u, E, nm), A) < t
    assert maxrel(op.jacobi(u, r, invd, E, nm, 0.6), uh + 0.6 * dh * (rh - A)) < out(dtype)
    assert maxrel(op.jacobi(u, r, invd, E, None, 0.6), uh + 0.6 * dh * (rh - K)) < out(dtype)
    assert maxrel(op.residual(u, r, E, nm), (rh - A) * mask) < out(aux)
    if dtype == aux and dtype != BF16:
        part = torch.full((op.partials_size,), float("nan"), dtype=F64, device="cuda")
        q = torch.empty_like(u)
        op.apply_dot(u, E, nm, q, part)
        assert maxrel(q, A) < tol[dtype]
        assert abs(float(part.sum()) - float(uh @ A)) <= 10 * tol[dtype] * float(np.abs(uh * A).sum())
        op.true_residual(u, r, E, nm, q, part)
        assert maxrel(q, rh - A) < tol[dtype]
        assert abs(float(part.sum()) - float((rh - A) @ (rh - A))) <= 10 * tol[dtype] * float((rh - A) @ (rh - A))


@pytest.mark.parametrize("dtype,tol", [(F64, 1e-14), (F32, 2e-6)])
def test_agrees_with_the_other_streaming_kernels(dtype, tol):
    """march and xp evaluate the same sums in another order of stages: equal to a few roundings."""
    shape = (150, 40, 70)
    rng = np.random.default_rng(2)
    op = vx.VoxelOperator(shape, CUBE, dtype)
    u = torch.as_tensor(rng.standard_normal(op.ndof), device="cuda").to(dtype)
    E = torch.as_tensor(rng.random(op.n_elem), device="cuda").to(dtype)
    nm = torch.as_tensor(rng.integers(0, 8, op.nodes).astype(np.uint8), device="cuda")
    y = op.matvec(u, E, nm)
    prev = _lib.set_stream_kernel("xp")
    try:
        assert prev == "march"
        ref = op.matvec(u, E, nm)
    finally:
        _lib.set_stream_kernel(prev)
    assert float((y - ref).abs().max()) <= tol * float(ref.abs().max())


def test_noalloc_residual_takes_long_thin_grids():
    """A grid six nodes thin in y needs more FP64 march tiles than the built-in scratch holds, but fits it
    by the xp kernel's: accepted, and equal to the residual with a caller's buffer to rounding."""
    shape = (1, 5, 240000)
    rng = np.random.default_rng(4)
    op = vx.VoxelOperator(shape, CUBE, F64)
    L = _lib.load()
    assert op.partials_size > 16384 >= L.vx_operator_partials(_lib.VX_F64 | _lib.VX_STREAM_XP, *shape)
    x, b = (torch.as_tensor(rng.standard_normal(op.ndof), device="cuda") for _ in range(2))
    E = torch.as_tensor(1e-3 + rng.random(op.n_elem), device="cuda")
    nm = torch.full((op.nodes,), 7, dtype=torch.uint8, device="cuda")
    nm[:36] = 0
    part = torch.empty(op.partials_size, dtype=F64, device="cuda")
    ref, res, n2 = torch.empty_like(x), torch.empty_like(x), torch.zeros(1, dtype=F64, device="cuda")
    op.true_residual(x, b, E, nm, ref, part)
    _lib.call("vx_true_residual_noalloc", op.prec, *shape, op._bp, E.data_ptr(), nm.data_ptr(), x.data_ptr(),
              b.data_ptr(), res.data_ptr(), n2.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert float((res - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
    assert abs(float(n2) - float(ref @ ref)) <= 1e-12 * float(ref @ ref)
