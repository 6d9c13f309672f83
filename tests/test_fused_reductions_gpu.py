"""Reductions finished by the last CTA of the kernel that forms them, and the fused Jacobi-CG step: the
same bits as the separate kernels (partials summed by the same threads in the same order), from one CTA's
worth of entries to many, repeated launches included (the arrival counter returns to zero)."""
import numpy as np
import pytest
import torch

from oracle import voxel_oracle as vo

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("voxel_b200")
from voxel_b200 import _lib, solver as vs  # noqa: E402

S_ALPHA, S_BETA, S_RZ, S_DONE = vs.S_ALPHA, vs.S_BETA, vs.S_RZ, vs.S_DONE


def _s():
    return torch.cuda.current_stream().cuda_stream


def vec(rng, n):
    return torch.as_tensor(rng.standard_normal(n), device="cuda")


@pytest.mark.parametrize("n", [3, 2047, 2049, 400_000, 2_500_000])
@pytest.mark.parametrize("done", [0.0, 1.0])
def test_dots_and_jacobi_step_equal_the_separate_kernels(n, done):
    rng = np.random.default_rng(n)
    G = int(_lib.load().vx_solver_partials(n))
    part = torch.empty(max(2 * G, int(_lib.load().vx_jacobi_step_partials(n))), dtype=torch.float64, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    S0 = torch.as_tensor(rng.random(16) + 0.5, device="cuda")
    S0[S_DONE], S0[vs.S_BREAK] = done, 0.0
    x, p, r, q, zo = (vec(rng, n) for _ in range(5))
    d = torch.as_tensor(rng.random(n), device="cuda")
    for update in (1, 0):
        Sa, xa, ra, za = S0.clone(), x.clone(), r.clone(), torch.empty_like(r)
        if update:
            _lib.call("vx_cg_update", _lib.VX_F64, n, Sa.data_ptr(), xa.data_ptr(), p.data_ptr(), ra.data_ptr(),
                      q.data_ptr(), 1, _s())
        _lib.call("vx_scaled_product", _lib.VX_F64, n, 1.0, d.data_ptr(), ra.data_ptr(), za.data_ptr(), _s())
        Sd = Sa.clone()
        _lib.call("vx_dots_pr", _lib.VX_F64, _lib.VX_F64, n, ra.data_ptr(), za.data_ptr(), zo.data_ptr(), part.data_ptr(), _s())
        _lib.call("vx_solver_finalize", vs.FIN_BETA_PR, G, part.data_ptr(), Sa.data_ptr(), _s())
        _lib.call("vx_dots_pr_fin", vs.FIN_BETA_PR, _lib.VX_F64, _lib.VX_F64, n, ra.data_ptr(), za.data_ptr(), zo.data_ptr(),
                  part.data_ptr(), Sd.data_ptr(), cnt.data_ptr(), _s())
        assert torch.equal(Sd, Sa) and int(cnt) == 0
        Sb, xb, rb, zb = S0.clone(), x.clone(), r.clone(), zo.clone()
        _lib.call("vx_jacobi_step", n, Sb.data_ptr(), xb.data_ptr(), p.data_ptr(), rb.data_ptr(), q.data_ptr(), d.data_ptr(),
                  zb.data_ptr(), update, part.data_ptr(), cnt.data_ptr(), _s())
        assert torch.equal(xb, xa) and torch.equal(rb, ra) and torch.equal(zb, za) and int(cnt) == 0
        for k in range(16):        # its CTAs are more, so its two sums (r.z, r.(z - z_old) and beta) differ by rounding
            scale = float((ra * za).abs().sum()) if k in (S_RZ, vs.S_RZN) else float((ra * (za - zo)).abs().sum())
            scale = scale / float(S0[S_RZ]) if k == S_BETA else scale
            exact = k not in (S_RZ, vs.S_RZN, vs.S_RZD, S_BETA)
            assert abs(float(Sb[k] - Sa[k])) <= (0.0 if exact else 1e-14 * scale)


@pytest.mark.parametrize("shape", [(1, 1, 1), (20, 9, 33), (64, 40, 64)])
@pytest.mark.parametrize("stream", [None, "xp"])
def test_operator_reductions_equal_the_separate_finalize(shape, stream):
    rng = np.random.default_rng(sum(shape))
    op = vx.VoxelOperator(shape, vo.quadrature([1, 1, 1], 0.3), stream=stream)
    E = torch.as_tensor(0.1 + rng.random(op.n_elem), device="cuda")
    u, b = vec(rng, op.ndof), vec(rng, op.ndof)
    nm = torch.as_tensor(rng.integers(0, 8, op.nodes).astype(np.uint8), device="cuda")
    G = op.partials_size
    part = torch.empty(G, dtype=torch.float64, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    for fin in (vs.FIN_PQ, vs.FIN_TRUE):
        Sa = torch.as_tensor(rng.random(16) + 0.5, device="cuda")
        Sa[S_DONE] = 0.0
        Sb, ya, yb = Sa.clone(), torch.empty_like(u), torch.empty_like(u)
        for _ in range(2):
            if fin == vs.FIN_PQ:
                op.apply_dot(u, E, nm, ya, part)
                _lib.call("vx_solver_finalize", fin, G, part.data_ptr(), Sa.data_ptr(), _s())
                op.apply_dot_fin(u, E, nm, yb, part, Sb, cnt, fin)
            else:
                op.true_residual(u, b, E, nm, ya, part)
                _lib.call("vx_solver_finalize", fin, G, part.data_ptr(), Sa.data_ptr(), _s())
                op.true_residual_fin(u, b, E, nm, yb, part, Sb, cnt, fin)
        assert torch.equal(Sa, Sb) and torch.equal(ya, yb) and int(cnt) == 0


@pytest.mark.parametrize("n", [3, 256, 257, 28_611, 303_104])
def test_small_iteration_equals_the_separate_kernels(n):
    """vx_small_step / vx_small_direction against the separate kernels: vectors to rounding of alpha and beta
    (the sums are grouped differently), scalars likewise; a zero p . q takes no step."""
    rng = np.random.default_rng(n)
    G = 37
    pq = torch.as_tensor(rng.random(G) + 0.1, device="cuda")
    sp = torch.empty(int(_lib.load().vx_jacobi_step_partials(n)), dtype=torch.float64, device="cuda")
    x, p, r, q, z = (vec(rng, n) for _ in range(5))
    d = torch.as_tensor(rng.random(n), device="cuda")
    for scale in (1.0, 0.0):
        S = torch.zeros(16, dtype=torch.float64, device="cuda")
        S[S_RZ] = S[vs.S_RZN] = 2.5
        xs, rs, zs, ps, part = x.clone(), r.clone(), z.clone(), p.clone(), pq * scale
        _lib.call("vx_small_step", n, G, part.data_ptr(), S.data_ptr(), xs.data_ptr(), ps.data_ptr(), rs.data_ptr(),
                  q.data_ptr(), d.data_ptr(), zs.data_ptr(), 1, 1, sp.data_ptr(), _s())
        alpha = 2.5 / float(pq.sum()) if scale else 0.0
        rr = r - alpha * q
        assert torch.allclose(xs, x + alpha * p, rtol=0, atol=1e-14) and torch.allclose(rs, rr, rtol=0, atol=1e-14)
        assert torch.equal(zs, d * rs)
        _lib.call("vx_small_direction", n, sp.data_ptr(), S.data_ptr(), zs.data_ptr(), ps.data_ptr(), _s())
        rz, rd = float(rs @ zs), float(rs @ (zs - z))
        tol = 1e-13 * float((rs * zs).abs().sum() + (rs * z).abs().sum())
        assert abs(float(S[vs.S_RZN]) - rz) <= tol and abs(float(S[vs.S_RZD]) - rd) <= tol and float(S[S_RZ]) == 2.5
        assert float((ps - (zs + float(S[S_BETA]) * p)).abs().max()) <= 1e-15 * float(p.abs().max()) * (1 + abs(float(S[S_BETA])))
        assert float(S[vs.S_IT]) == scale and float(S[vs.S_BREAK]) == 1.0 - scale
