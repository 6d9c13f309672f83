"""The four-entries-a-thread form of the CG vector kernels (long aligned vectors) against the one-entry form
(the same vectors one entry off alignment): bit for bit, at lengths with every remainder by four and at the
length where the form changes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
vx = pytest.importorskip("voxel_b200")
from voxel_b200 import _lib, solver as vs  # noqa: E402

F64, F32, BF16 = torch.float64, torch.float32, torch.bfloat16
WIDE = 1 << 20


def run(name, n, off, dtypes, args, seed):
    """The vectors after one call; off: entries by which every vector is off its allocation."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    S = torch.rand(16, dtype=F64, device="cuda", generator=g)
    S[vs.S_DONE], S[vs.S_BREAK] = 0.0, 0.0
    vecs = {}
    for k, dt in dtypes.items():
        vecs[k] = torch.empty(n + 8, dtype=dt, device="cuda")[off:off + n]
        vecs[k].copy_(torch.randn(n, device="cuda", generator=g))
    _lib.call(name, *[S.data_ptr() if a == "S" else vecs[a].data_ptr() if isinstance(a, str) else n if a is None else a
                      for a in args], torch.cuda.current_stream().cuda_stream)
    return vecs


@pytest.mark.parametrize("n", [WIDE - 1, WIDE, WIDE + 1, WIDE + 2, WIDE + 3])
@pytest.mark.parametrize("prec,x,r", [(_lib.VX_F64, F64, F64), (_lib.VX_F32, F32, F32), (_lib.VX_BF16_F32, BF16, BF16),
                                      (_lib.VX_F32_BF16AUX, F32, BF16)])
def test_wide_and_narrow_forms_agree_bitwise(n, prec, x, r):
    zprec = {F64: _lib.VX_F64, F32: _lib.VX_F32, BF16: _lib.VX_BF16_F32}[x]
    cases = [("vx_cg_direction_update", dict(z=x, p=F64, zo=x, x=F64), (zprec, None, "S", "z", "p", "zo", "x")),
             ("vx_cg_direction", dict(z=x, p=F64, zo=x), (_lib.VX_F64, zprec, None, "S", "z", "p", "zo")),
             ("vx_vcycle_entry_update", dict(r64=F64, q=F64, rm=r, d=r, xo=x), (prec, None, "S", "r64", "q", "rm", "d", 0.6, "xo")),
             ("vx_vcycle_entry", dict(r64=F64, rm=r, d=r, xo=x), (prec, None, "r64", "rm", "d", 0.6, "xo"))]
    if x in (F64, F32) and x == r:
        cases += [("vx_cg_update", dict(x=x, p=x, r=x, q=x), (prec, None, "S", "x", "p", "r", "q", u)) for u in (0, 1)]
    for name, dtypes, args in cases:
        a, b = run(name, n, 0, dtypes, args, 5), run(name, n, 1, dtypes, args, 5)
        for k in dtypes:
            assert torch.equal(a[k], b[k]), (name, k)
