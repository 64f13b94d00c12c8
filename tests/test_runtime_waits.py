"""Waiting for tasks: the wait ends with the task, and the runtime can be restarted the moment a name is known."""
import subprocess
import sys
import time
import weakref
from pathlib import Path

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


@pytest.mark.timeout(60)
def test_wait_for_an_unknown_kind_of_task_sleeps():
    hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
    cpu = time.process_time()
    with pytest.raises(TimeoutError):
        hp_cuda.wait_for(99, ["never"], timeout_s=1.0)
    assert time.process_time() - cpu < 0.5
    hp_cuda.end()


@pytest.mark.timeout(60)
def test_names_do_not_wait_for_the_interpreter():
    """A name is out when its task is done, also while some Python code keeps the interpreter lock."""
    hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
    n, names = 64, {"a", "b", "c"}
    size = ops.tbq_payload_bytes(n)
    tensors = [(name, torch.randn(n) * 1e-3, torch.zeros(n), torch.zeros(size, dtype=torch.uint8),
                torch.zeros(size, dtype=torch.uint8)) for name in sorted(names)]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(20.0)
    try:
        for t in tensors:
            hp_cuda.submit_task(*t, 0, hp_cuda.COMP_TASK)
        seen, t0 = set(), time.monotonic()
        while seen < names and time.monotonic() < t0 + 5:
            seen.update(hp_cuda.getResults(hp_cuda.COMP_TASK))
    finally:
        sys.setswitchinterval(interval)
    assert seen == names
    hp_cuda.end()


@pytest.mark.timeout(60)
@pytest.mark.parametrize("collect", ["getResults", "getErrors", "submit_task", "end"])
def test_tensors_are_let_go_with_the_next_call(collect):
    """Of a task that worked and of one that failed."""
    hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
    size = ops.tbq_payload_bytes(64)

    def submit(dtype):
        t = (torch.zeros(64, dtype=dtype), torch.zeros(64), torch.zeros(size, dtype=torch.uint8),
             torch.zeros(size, dtype=torch.uint8))
        hp_cuda.submit_task("x", *t, 0, hp_cuda.COMP_TASK)
        return [weakref.ref(x) for x in t]

    held = submit(torch.float32) + submit(torch.float64)
    deadline = time.monotonic() + 20
    while any(x() is not None for x in held) and time.monotonic() < deadline:
        time.sleep(0.01)
        if collect == "getResults":
            hp_cuda.getResults(hp_cuda.COMP_TASK)
        elif collect == "getErrors":
            hp_cuda.getErrors()
        elif collect == "submit_task":
            submit(torch.float32)
        else:
            hp_cuda.end()
    assert all(x() is None for x in held)
    hp_cuda.end()


EXIT_AFTER_NAME = """
import torch
from hipress_b200 import hp_cuda, ops
size = ops.tbq_payload_bytes(64)
assert hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
for i in range(200):
    hp_cuda.submit_task("x", torch.zeros(64), torch.zeros(64), torch.zeros(size, dtype=torch.uint8),
                        torch.zeros(size, dtype=torch.uint8), 0, hp_cuda.COMP_TASK)
hp_cuda.wait_for(hp_cuda.COMP_TASK, ["x"])
"""


@pytest.mark.timeout(90)
def test_exit_with_tasks_in_the_workers():
    """The program ends without end(), while workers still finish tasks that own the last reference to their tensors."""
    root = Path(__file__).resolve().parent.parent
    done = subprocess.run([sys.executable, "-c", EXIT_AFTER_NAME], cwd=root, capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, (done.returncode, done.stderr[-2000:])


RESTART_BESIDE_SUBMIT = """
import sys, threading, time
import torch
from hipress_b200 import hp_cuda, ops

n, size = 64, ops.tbq_payload_bytes(64)
stop = time.monotonic() + 3.0
failures = []

def submit(k):
    try:
        while time.monotonic() < stop:
            t = (torch.randn(n) * 1e-3, torch.zeros(n), torch.zeros(size, dtype=torch.uint8),
                 torch.zeros(size, dtype=torch.uint8))
            assert hp_cuda.submit_task(f"t{k}", *t, 0, hp_cuda.COMP_TASK)
            hp_cuda.getResults(hp_cuda.COMP_TASK)
            hp_cuda.numThreads()
    except Exception as e:
        failures.append(repr(e))

assert hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
threads = [threading.Thread(target=submit, args=(k,)) for k in range(2)]
for t in threads:
    t.start()
while time.monotonic() < stop:
    assert hp_cuda.init("tbq", {"threshold": 2e-3}, 0, 0, 1)
for t in threads:
    t.join()
assert not failures and not hp_cuda.getErrors(), failures
hp_cuda.end()
print("ended")
"""


@pytest.mark.timeout(90)
def test_restart_beside_submitting_threads():
    """Two threads hand in tasks while a third restarts the runtime; in a process of its own, whose end is looked at."""
    root = Path(__file__).resolve().parent.parent
    done = subprocess.run([sys.executable, "-c", RESTART_BESIDE_SUBMIT], cwd=root, capture_output=True, text=True, timeout=60)
    assert done.returncode == 0 and "ended" in done.stdout, (done.returncode, done.stderr[-2000:])
