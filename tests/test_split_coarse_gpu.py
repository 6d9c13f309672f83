"""The coarsest system split at its middle plane (vx_split_factor / vx_split_apply) against a dense FP64 solve:
odd and even numbers of planes (an even number pads one half), bands narrower and wider than a 64-column
block, planes of fewer and more DOFs than a block, masks on every face, each storage mode; a matrix that is
not positive definite is flagged wherever its bad pivot lies; grids too short to split are refused."""
import numpy as np
import pytest
import torch

from oracle import voxel_oracle as vo

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("voxel_b200")
from voxel_b200 import _lib  # noqa: E402

KE = vo.quadrature([1, 1, 1], 0.3)


def _s():
    return torch.cuda.current_stream().cuda_stream


def system(shape, rng):
    E = torch.as_tensor(1e-6 + rng.random(int(np.prod(shape))) ** 3, device="cuda")
    mask = rng.integers(0, 8, vo.n_nodes(shape)).astype(np.uint8)
    mask[rng.random(mask.size) < 0.9] = 7
    mask.reshape(shape[0] + 1, -1)[0] = 0
    nm = torch.as_tensor(mask, device="cuda")
    n = 3 * vo.n_nodes(shape)
    A = torch.empty(n, n, dtype=torch.float64, device="cuda")
    _lib.call("vx_assemble_dense", *shape, _lib.dptr(np.ascontiguousarray(KE)), E.data_ptr(), nm.data_ptr(), A.data_ptr(), _s())
    free = torch.as_tensor(np.stack([(mask >> c) & 1 for c in range(3)], axis=1).ravel().astype(bool), device="cuda")
    return A, nm, free


def factor(shape, A):
    lib = _lib.load()
    F = torch.empty(int(lib.vx_split_factor_size(*shape)), dtype=torch.float64, device="cuda")
    work = torch.empty(int(lib.vx_split_workspace(*shape)), dtype=torch.float64, device="cuda")
    info = torch.full((3,), 7, dtype=torch.int32, device="cuda")
    _lib.call("vx_split_factor", *shape, A.data_ptr(), F.data_ptr(), work.data_ptr(), info.data_ptr(), _s())
    return F, info


@pytest.mark.parametrize("shape", [(4, 1, 1), (5, 1, 2), (6, 2, 3), (7, 3, 2), (9, 4, 4), (10, 5, 5), (16, 8, 8), (13, 6, 7)])
def test_split_solve_matches_the_dense_solve(shape):
    rng = np.random.default_rng(sum(shape))
    A, nm, free = system(shape, rng)
    n, p = A.shape[0], A.shape[0] // (shape[0] + 1)
    F, info = factor(shape, A)
    assert info.tolist() == [0, 0, 0]
    y = torch.full((n + p,), float("nan"), dtype=torch.float64, device="cuda")
    inv = torch.linalg.inv(A)
    for (x, aux), prec in vx.operators.STORAGE.items():
        r = torch.as_tensor(rng.standard_normal(n), device="cuda").to(aux)
        z = torch.full((n,), float("nan"), dtype=x, device="cuda")
        _lib.call("vx_split_apply", prec, *shape, F.data_ptr(), r.data_ptr(), nm.data_ptr(), y.data_ptr(), z.data_ptr(), _s())
        ref = torch.where(free, torch.linalg.solve(A, r.double()), 0.0)
        # FP64: the rounding of a product with the inverse factors, |A^-1| |A| |z| eps-sized
        bound = 64 * 2.3e-16 * float((inv.abs() @ (A.abs() @ ref.abs())).max())
        tol = {torch.float64: 0.0, torch.float32: 1.2e-7, torch.bfloat16: 8e-3}[x]
        assert float((z.double() - ref).abs().max()) <= bound + tol * float(ref.abs().max())


def test_indefinite_matrices_are_flagged_in_each_part():
    shape = (8, 3, 3)
    A, _, _ = system(shape, np.random.default_rng(1))
    p = A.shape[0] // 9
    for plane, part in ((1, 0), (7, 1), (4, 2)):
        B = A.clone()
        B[plane * p + 5, plane * p + 5] = -1.0
        assert (factor(shape, B)[1] != 0).tolist()[part]


def test_short_grids_do_not_split():
    lib = _lib.load()
    for shape in ((3, 4, 4), (1, 1, 1), (4, 0, 1)):
        assert lib.vx_split_factor_size(*shape) == 0 and lib.vx_split_workspace(*shape) == 0
    with pytest.raises(ValueError):
        t = torch.zeros(8, dtype=torch.float64, device="cuda")
        _lib.call("vx_split_factor", 3, 4, 4, t.data_ptr(), t.data_ptr(), t.data_ptr(), t.data_ptr(), _s())
