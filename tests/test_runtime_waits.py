"""Waiting for tasks: the wait ends with the task, and the runtime can be restarted the moment a name is known."""
import time

import pytest
import torch

from hipress_b200 import hp_cuda, ops


def submit_and_wait(n, names):
    size = ops.tbq_payload_bytes(n)
    tensors = [(name, torch.randn(n) * 1e-3, torch.zeros(n), torch.zeros(size, dtype=torch.uint8),
                torch.zeros(size, dtype=torch.uint8)) for name in names]
    for t in tensors:
        hp_cuda.submit_task(*t, 0, hp_cuda.COMP_TASK)
    return hp_cuda.wait_for(hp_cuda.COMP_TASK, names)


@pytest.mark.timeout(60)
def test_restart_right_after_a_wait():
    """The caller drops its tensors and restarts the runtime while the worker may still be returning from the last task."""
    names = [f"t{i}" for i in range(4)]
    for _ in range(300):
        assert hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
        assert sorted(submit_and_wait(64, names)) == names
    hp_cuda.end()


@pytest.mark.timeout(60)
def test_wait_ends_on_error_and_on_timeout():
    hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
    bad = torch.zeros(64, dtype=torch.float64)
    u8 = torch.zeros(16, dtype=torch.uint8)
    hp_cuda.submit_task("bad", bad, torch.zeros(64), u8, u8.clone(), 0, hp_cuda.COMP_TASK)
    with pytest.raises(RuntimeError, match="bad"):
        hp_cuda.wait_for(hp_cuda.COMP_TASK, ["bad"], timeout_s=30)
    t0 = time.monotonic()
    with pytest.raises(TimeoutError):
        hp_cuda.wait_for(hp_cuda.COMP_TASK, ["never"], timeout_s=0.3)
    assert 0.2 < time.monotonic() - t0 < 10
    hp_cuda.end()
