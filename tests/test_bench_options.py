"""Options of bench.py that reach the library."""
import sys

import pytest

import bench
from voxel_b200 import _lib


@pytest.mark.parametrize("kind", ["march", "xp", "zp"])
def test_stream_kernel_is_selected(kind, monkeypatch):
    seen = []
    monkeypatch.setattr(sys, "argv", ["bench.py", "--kernels", "--stream-kernel", kind])
    monkeypatch.setattr(bench, "run_kernels", lambda args: seen.append(_lib.load().vx_stream_kernel(_lib.VX_F64, 48, 24, 24)))
    prev = _lib.set_stream_kernel("march")
    try:
        bench.main()
    finally:
        _lib.set_stream_kernel(prev)
    assert seen == [_lib.STREAM_KERNELS[kind]]
