"""A process forked after CUDA's initialisation asks torch about it again (which then refuses)."""
import os

from voxel_b200 import operators


def test_the_initialisation_is_not_taken_over(monkeypatch):
    monkeypatch.setattr(operators, "_initialized", True)
    pid = os.fork()
    if pid == 0:
        os._exit(int(operators._initialized))
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0
    assert operators._initialized
