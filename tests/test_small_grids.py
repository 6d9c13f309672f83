"""The streaming kernel of a multigrid solve is chosen by the job's own grid: the same through every entry point, and
whatever it is stacked with or cut into."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx
from voxel_b200 import _lib, slab
from voxel_b200 import solver as vs
from voxel_b200.batch import BatchedSolver, stack_geometry
from voxel_b200.problems import cantilever_equal_split

F64, F32, AUX = _lib.VX_F64, _lib.VX_F32, _lib.VX_F32_BF16AUX
KE = vx.quadrature([1.0, 1.0, 1.0], 0.3)
# a small grid that eight slots stack beyond the limit; an ordinary one; one whose stack alone counts as thin in y
SHAPES = [(24, 12, 12), (48, 24, 24), (256, 16, 128)]
FLAT = (64, 4, 600)


def test_stacking_would_change_the_choice():
    lib, names = _lib.load(), {v: k for k, v in _lib.STREAM_KERNELS.items()}
    for shape, prec, alone, stacked in ((SHAPES[2], F32, "march", "xp"), (FLAT, F64, "march", "xp"),
                                        (SHAPES[1], F32, "march", "march"), (FLAT, F32, "xp", "xp")):
        grid = stack_geometry(shape, 8).grid
        assert names[lib.vx_default_kernel(prec, *shape)] == alone == vs.level_stream(shape, shape, prec)
        assert names[lib.vx_default_kernel(prec, *grid)] == stacked
    assert vs.small_grid_stream(SHAPES[0]) == "xp" and vs.small_grid_stream(stack_geometry(SHAPES[0], 8).grid) is None
    assert vs.level_stream(SHAPES[0], (12, 6, 6), AUX) == "xp"
    assert lib.vx_default_kernel(9, 4, 4, 4) == -1 and lib.vx_default_kernel(F64, 0, 4, 4) == -1


def test_the_default_is_not_the_selection():
    prev = _lib.set_stream_kernel("zp")
    try:
        assert _lib.load().vx_default_kernel(F64, 48, 24, 24) == _lib.STREAM_KERNELS["march"]
        assert _lib.load().vx_stream_kernel(F64, 48, 24, 24) == _lib.STREAM_KERNELS["zp"]
    finally:
        _lib.set_stream_kernel(prev)


def rough(shape, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    return 1e-9 + (0.01 + 0.99 * torch.rand(int(np.prod(shape)), dtype=torch.float64, device="cuda", generator=g)) ** 3


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", ["mixed", "fp64", "bf16"])
def test_every_entry_point_runs_the_same_kernels(shape, precision):
    mask, _ = cantilever_equal_split(shape)
    E = rough(shape, 3)
    es = vx.ElasticitySolver(shape, E, mask, precision=precision)
    lib = _lib.load()
    pick = lambda op, s: lib.vx_stream_kernel(op._sel, *s)                    # noqa: E731
    want = [(pick(L.op, L.shape), pick(L.op64, L.shape)) for L in es.M.levels]
    outer = pick(es.fcg.op, shape)
    nm = vx.node_mask_from_dofs(mask)
    assert pick(vs.FCGSolver(vx.VoxelOperator(shape, KE), E, nm, es.M).op, shape) == outer
    named = vx.VoxelOperator(shape, KE, stream="march")
    assert vs.FCGSolver(named, E, nm, es.M).op is named
    bs = BatchedSolver(shape, 8, precision=precision)
    assert [(pick(L.op, L.shape), pick(L.op64, L.shape)) for L in bs.M.levels] == want
    assert pick(bs.op, bs.geo.grid) == outer
    sl = slab.SlabSolver(shape, E, mask, 2, precision=precision, graph=False)
    for levels in sl.M.parts.values():
        assert [(pick(L.op, L.shape), pick(L.op64, L.shape)) for L in levels] == want
    assert want[0][1] == outer


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "fp64", "bf16"])
def test_a_small_job_alone_and_among_eight_is_bitwise_equal(precision):
    """On rough moduli, where the iterate at maxiter follows every rounding."""
    shape = SHAPES[0]
    _, force = cantilever_equal_split(shape)
    jobs = [(rough(shape, 20 + k), force, 1e-12) for k in range(8)]
    all_ = BatchedSolver(shape, 8, precision=precision, maxiter=40).solve(jobs)
    for k in (0, 7):
        alone = BatchedSolver(shape, 1, precision=precision, maxiter=40).solve([jobs[k]])[0]
        assert torch.equal(alone[0], all_[k][0]) and alone[1:4] == all_[k][1:4]


def test_the_partials_size_follows_the_selection():
    op = vx.VoxelOperator((32, 16, 16), KE)
    lib, seen = _lib.load(), {}
    prev = _lib.set_stream_kernel("march")
    try:
        for kind in ("march", "xp", "zp", "march", "xp"):
            _lib.set_stream_kernel(kind)
            assert lib.vx_selected_kernel() == _lib.STREAM_KERNELS[kind]
            seen[kind] = op.partials_size
            assert seen[kind] == lib.vx_operator_partials(op._sel, *op.shape)
        _lib.set_stream_kernel("march")
        assert op.on("xp").partials_size == seen["xp"] != seen["march"] == op.partials_size
    finally:
        _lib.set_stream_kernel(prev)
