"""Grids few nodes thin in y, on which the default streaming kernel is the element-plane-pair kernel."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx
from oracle import voxel_oracle as vo
from voxel_b200 import _lib

F64, F32, BF16 = _lib.VX_F64, _lib.VX_F32, _lib.VX_BF16_F32
THIN = [(F32, (64, 1, 200)), (F32, (1, 5, 300)), (F32, (512, 5, 1500)), (F32, (300, 14, 800)), (F32, (300, 17, 800)),
        (F32, (300, 28, 800)), (BF16, (8, 5, 8)), (_lib.VX_F32_BF16AUX, (8, 5, 8)), (F64, (512, 5, 1500)), (F64, (24, 1, 5000))]
FULL = [(F32, (64, 6, 200)), (F32, (300, 13, 800)), (F32, (300, 18, 800)), (F32, (300, 30, 800)), (F32, (600, 15, 45)),
        (BF16, (576, 288, 288)), (F64, (512, 6, 1500)), (F64, (300, 5, 300)), (F64, (1, 5, 240000)), (F64, (576, 288, 288))]


@pytest.mark.parametrize("prec,shape", THIN + FULL)
def test_route(prec, shape):
    lib = _lib.load()
    xp, march = (lib.vx_operator_partials(min(prec, F32) | bit, *shape) for bit in (_lib.VX_STREAM_XP, 0x200))
    if prec in (F64, F32):
        assert lib.vx_operator_partials(prec, *shape) == (xp if (prec, shape) in THIN else march)
    kinds = [lib.vx_stream_kernel(prec | bit, *shape) for bit in (0, _lib.VX_STREAM_XP, _lib.VX_STREAM_MARCH)]
    x, m = _lib.STREAM_KERNELS["xp"], _lib.STREAM_KERNELS["march"]
    assert kinds == [x if (prec, shape) in THIN else m, x, m]


def test_bad_arguments():
    lib = _lib.load()
    assert lib.vx_stream_kernel(9, 4, 4, 4) == -1 and lib.vx_stream_kernel(F64, 0, 4, 4) == -1
    with pytest.raises(ValueError):
        vx.VoxelOperator((4, 4, 4), vx.quadrature([1, 1, 1], 0.3), stream="zp")


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(24, 3, 5200), (9, 5, 40), (300, 14, 420)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32, torch.bfloat16])
def test_every_form(shape, dtype):
    """The default is xp, bit for bit, where it routes there, and the forced march kernel agrees to rounding."""
    g = torch.Generator("cuda").manual_seed(sum(shape))
    ke = vo.quadrature([1, 1, 1], 0.3)
    ops = {s: vx.VoxelOperator(shape, ke, dtype, stream=s) for s in (None, "xp", "march")}
    rand = lambda n: torch.randn(n, dtype=torch.float64, device="cuda", generator=g).to(dtype)
    op = ops[None]
    u, r, d = (rand(op.ndof) for _ in range(3))
    E = rand(op.n_elem).abs() + 0.01
    nm = torch.randint(0, 8, (op.nodes,), device="cuda", generator=g).to(torch.uint8)
    tol = {torch.float64: 1e-13, torch.float32: 1e-5, torch.bfloat16: 1e-2}[dtype]
    forms = {"matvec": lambda o: o.matvec(u, E, nm), "free": lambda o: o.matvec(u, E),
             "sweep": lambda o: o.jacobi(u, r, d, E, nm, 0.6), "residual": lambda o: o.residual(u, r, E, nm)}
    if dtype != torch.bfloat16:
        def reduce(o, form):
            q, part = torch.empty_like(u), torch.full((o.partials_size,), float("nan"), dtype=torch.float64, device="cuda")
            form(o, q, part)
            return torch.cat([q.double(), part.sum()[None] / op.ndof ** 0.5])
        forms["apply"] = lambda o: reduce(o, lambda o, q, p: o.apply_dot(u, E, nm, q, p))
        forms["true residual"] = lambda o: reduce(o, lambda o, q, p: o.true_residual(u, r, E, nm, q, p))
    thin = _lib.load().vx_stream_kernel(op.prec, *shape) == _lib.STREAM_KERNELS["xp"]
    assert thin == (dtype != torch.float64 or shape == (24, 3, 5200))
    for name, form in forms.items():
        y, x, m = (form(ops[s]) for s in (None, "xp", "march"))
        assert torch.equal(y, x if thin else m), name
        assert float((x.double() - m.double()).abs().max()) <= tol * float(x.double().abs().max()), name


@pytest.mark.gpu
def test_noalloc_residual_where_only_march_fits():
    """A grid on which the default kernel's FP32 partial sums are more than the built-in scratch holds."""
    shape = (4, 16, 170000)
    lib, op = _lib.load(), vx.VoxelOperator(shape, vo.quadrature([1, 1, 1], 0.3), torch.float32)
    assert lib.vx_operator_partials(F32 | _lib.VX_STREAM_MARCH, *shape) <= 16384 < op.partials_size
    g = torch.Generator("cuda").manual_seed(1)
    x, b = (torch.randn(op.ndof, dtype=torch.float32, device="cuda", generator=g) for _ in range(2))
    E = torch.rand(op.n_elem, dtype=torch.float32, device="cuda", generator=g) + 0.01
    nm = torch.full((op.nodes,), 7, dtype=torch.uint8, device="cuda")
    nm[:17] = 0
    part = torch.empty(op.partials_size, dtype=torch.float64, device="cuda")
    ref, res, n2 = torch.empty_like(x), torch.empty_like(x), torch.zeros(1, dtype=torch.float64, device="cuda")
    op.true_residual(x, b, E, nm, ref, part)
    _lib.call("vx_true_residual_noalloc", op.prec, *shape, op._bp, E.data_ptr(), nm.data_ptr(), x.data_ptr(),
              b.data_ptr(), res.data_ptr(), n2.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert float((res - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
    assert abs(float(n2) - float(ref.double() @ ref.double())) <= 1e-6 * float(n2)
