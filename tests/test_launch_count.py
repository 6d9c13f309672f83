"""The count of launched kernels for the entry points whose number follows from their arguments."""
import pytest

from voxel_b200 import _lib


@pytest.mark.parametrize("name", ["vx_apply_dot_fin", "vx_true_residual_fin"])
@pytest.mark.parametrize("kind,sel,shape,kernels", [
    ("march", _lib.VX_F64, (48, 24, 24), 1), ("march", _lib.VX_F64 | _lib.VX_STREAM_XP, (48, 24, 24), 2),
    ("march", _lib.VX_F32, (64, 3, 200), 2), ("march", _lib.VX_F32 | _lib.VX_STREAM_MARCH, (64, 3, 200), 1),
    ("xp", _lib.VX_F64, (48, 24, 24), 2), ("zp", _lib.VX_F32 | _lib.VX_STREAM_MARCH, (48, 24, 24), 2)])
def test_reducing_forms(name, kind, sel, shape, kernels):
    prev = _lib.set_stream_kernel(kind)
    try:
        assert _lib._bind(name)[1] is None and _lib._kernels(name, (0, sel, *shape)) == kernels
    finally:
        _lib.set_stream_kernel(prev)


def test_factors():
    # 65 blocks of 64 columns; halves of 8 planes of 243 and the plane between them
    assert _lib._kernels("vx_coarse_factor", (4131, 275)) == 2 * 65 + 1
    assert _lib._kernels("vx_split_factor", (16, 8, 8)) == 2 * 31 + 2 * 4 + 6
