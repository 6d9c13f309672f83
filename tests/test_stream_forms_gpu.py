"""Every form and storage mode of both streaming kernels that solves run (parity_march and parity_stream_xp) against the
FP64 oracle on the rounded inputs, on ragged grids and on grids whose x chunks are long, where parity_march's inner loop
loads planes without testing them.  Inputs and outputs sit in guard bands.  Tolerances (max-norm relative): FP64 1e-13,
FP32 arithmetic 1e-5, outputs stored in bf16 one rounding (4.5e-3)."""
import numpy as np
import pytest
import torch

from oracle import voxel_oracle as vo
from test_guard_gpu import bands_intact, guarded, out_buf

vx = pytest.importorskip("voxel_b200")
from voxel_b200 import _lib  # noqa: E402

F64, F32, BF16 = torch.float64, torch.float32, torch.bfloat16
KES = {"cube": vo.quadrature([1, 1, 1], 0.3), "brick": vo.quadrature([1.0, 0.5, 2.0], 0.25)}
LONG = [(6000, 1, 1), (300, 30, 31)]
SHAPES = [(1, 1, 1), (3, 13, 13), (5, 14, 60), (9, 27, 2), *LONG]


def chunk(shape, sel):
    """Node planes an x chunk of parity_march."""
    rows, cols = (14, 14) if sel == _lib.VX_F64 else (14, 30)
    tiles = -(-(shape[1] + 1) // rows) * -(-(shape[2] + 1) // cols)
    return -(-(shape[0] + 1) * tiles // _lib.load().vx_operator_partials(sel | _lib.VX_STREAM_MARCH, *shape))


@pytest.mark.gpu
@pytest.mark.parametrize("sel", [_lib.VX_F64, _lib.VX_F32])
def test_the_long_chunks_reach_the_untested_steps(sel):
    for shape in LONG:
        assert chunk(shape, sel) >= 5                        # planes x0 to x0 + cx - 3 of a chunk are such steps


def walk(nx, cx):
    """parity_march's plane offsets: (what, plane wanted, plane read) of every load and store of every chunk."""
    for x0 in range(0, nx + 1, cx):
        x1 = min(x0 + cx, nx + 1)
        n_in, e_in, n_out, held = max(x0 - 1, 0), x0 - 1, x0 - 1, []

        def load_u(ix, inside=False):
            nonlocal n_in
            yield "u", min(max(ix, 0), nx), n_in
            n_in += inside or 0 <= ix < nx

        def load_e(ex, inside=False):
            nonlocal e_in
            if inside or 0 <= ex < nx:
                yield "E", ex, e_in
            e_in += 1

        yield from load_u(x0 - 1)
        yield from load_e(x0 - 1)
        yield from load_u(x0)
        yield from load_u(x0 + 1)
        held = x0 + 1                                        # the plane in flight
        bulk = min(x1, nx - 1) - 2
        for e in range(x0 - 1, x1):
            inside = x0 <= e < bulk
            if inside or e + 2 <= x1:
                yield "ring", e + 2, held
                if inside or e + 3 <= x1:
                    yield from load_u(e + 3, inside)
                    held = e + 3
                yield from load_e(e + 1, inside)
            if e >= x0:
                yield "y", e, n_out
            n_out += 1


def test_plane_offsets_stay_in_the_grid():
    steps = 0
    for nx in (*range(1, 30), 65, 100):
        for cx in range(1, nx + 2):
            stored = []
            for what, want, got in walk(nx, cx):
                assert want == got and (what == "ring" or 0 <= got <= nx - (what == "E")), (nx, cx, what)
                stored += [got] * (what == "y")
                steps += 1
            assert stored == list(range(nx + 1))
    assert steps > 10000


def maxrel(t, ref):
    return float(np.max(np.abs(t.double().cpu().numpy() - ref)) / max(np.max(np.abs(ref)), 1e-300))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("element", KES)
@pytest.mark.parametrize("dtype,aux", [(F64, F64), (F32, F32), (F32, BF16), (BF16, BF16)])
def test_every_form(shape, element, dtype, aux):
    rng = np.random.default_rng(sum(shape))
    ke = KES[element]
    n = 3 * vo.n_nodes(shape)
    E = guarded(1e-3 + rng.random(int(np.prod(shape))), aux)[0]
    u, r = guarded(rng.standard_normal(n), dtype)[0], guarded(rng.standard_normal(n), aux)[0]
    mask = vo.cantilever_equal_split(shape)[0] * (rng.random(n) > 0.05)
    nm = guarded(vx.node_mask_from_dofs(torch.as_tensor(mask, device="cuda")).cpu().numpy(), torch.uint8)[0]
    Eh, uh, rh = (t.double().cpu().numpy() for t in (E, u, r))
    d = guarded(1 / np.where(mask != 0, vo.product_diagonal(shape, ke, Eh), 1.0), aux)[0]
    dh = d.double().cpu().numpy()
    A, K = vo.apply_dirichlet(shape, ke, Eh, mask, uh), vo.product_raw(shape, ke, uh, Eh)
    tol = lambda dt: {F64: 1e-13, F32: 1e-5}.get(dt, 4.5e-3)
    arith = F32 if dtype == BF16 else dtype
    for stream in ("march", "xp"):
        op = vx.VoxelOperator(shape, ke, dtype, aux, stream=stream)

        def check(ref, dt, form, scale=1.0):
            y, whole = out_buf(n, dt)
            form(y)
            assert bands_intact(whole, n) and maxrel(y, ref) < scale * tol(dt), stream
            return y
        if (dtype, aux) != (F32, BF16):
            check(K, arith, lambda y: op.matvec(u, E, out=y))
            check(A, arith, lambda y: op.matvec(u, E, nm, out=y))
        check(uh + 0.6 * dh * (rh - A), dtype, lambda y: op.jacobi(u, r, d, E, nm, 0.6, out=y))
        check(uh + 0.6 * dh * (rh - K), dtype, lambda y: op.jacobi(u, r, d, E, None, 0.6, out=y))
        check((rh - A) * mask, aux, lambda y: op.residual(u, r, E, nm, out=y))
        if dtype == aux and dtype != BF16:
            part, whole = out_buf(op.partials_size, F64)
            check(A, dtype, lambda y: op.apply_dot(u, E, nm, y, part))
            assert abs(float(part.sum()) - float(uh @ A)) <= 10 * tol(dtype) * float(np.abs(uh * A).sum())
            check(rh - A, dtype, lambda y: op.true_residual(u, r, E, nm, y, part))
            assert abs(float(part.sum()) - float((rh - A) @ (rh - A))) <= 10 * tol(dtype) * float((rh - A) @ (rh - A))
            assert bands_intact(whole, part.numel())


@pytest.mark.parametrize("kind", ["march", "xp", "zp"])
def test_noalloc_scratch_covers_the_grids_of_every_kernel(kind):
    prev = _lib.set_stream_kernel(kind)
    try:
        for prec in (_lib.VX_F64, _lib.VX_F32):
            for shape in ((2047, 400, 400), (1, 1, 1), (576, 288, 288), (1, 1500, 1500)):
                assert 1 <= _lib.load().vx_operator_partials(prec, *shape) <= 16384
    finally:
        _lib.set_stream_kernel(prev)
