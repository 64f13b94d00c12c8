"""The reference's module API (init / submit_task / getResults / end) on CUDA tensors with the
CPU staging buffer ``C`` of the original contract."""
import struct
import time

import pytest
import torch

from hipress_b200 import hp_cuda, ops

pytestmark = pytest.mark.gpu


@pytest.fixture()
def runtime():
    yield hp_cuda
    hp_cuda.end()


def gauss(n, std=0.01, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(n, generator=g) * std


def test_terngrad_tasks_on_gpu_match_cpu_codec(runtime):
    runtime.init("terngrad", {"enable_random": 0, "bitwidth": 2}, 0, 0, 1)
    names = [f"t{i}" for i in range(16)]
    grads = {k: gauss(20000 + 37 * i, seed=i) for i, k in enumerate(names)}
    dev = {k: g.cuda() for k, g in grads.items()}
    Bs = {k: torch.zeros(ops.terngrad_payload_bytes(g.numel(), 2), dtype=torch.uint8, device="cuda") for k, g in grads.items()}
    Cs = {k: torch.zeros(b.numel(), dtype=torch.uint8).pin_memory() for k, b in Bs.items()}
    for k in names:
        assert runtime.submit_task(k, dev[k], Bs[k], Cs[k], 0, runtime.COMP_TASK)
    assert sorted(runtime.wait_for(runtime.COMP_TASK, names)) == sorted(names)
    for k in names:
        assert torch.equal(Cs[k], ops.terngrad_compress(grads[k], 2, False)), k
    outs = {k: torch.zeros_like(v) for k, v in dev.items()}
    for k in names:
        Bs[k].zero_()
        runtime.submit_task(k, outs[k], Bs[k], Cs[k], 0, runtime.DECOMP_TASK)
    runtime.wait_for(runtime.DECOMP_TASK, names)
    for k in names:
        ref = torch.empty_like(grads[k])
        ops.terngrad_decompress(Cs[k], ref)
        assert torch.equal(outs[k].cpu(), ref), k
    assert runtime.getErrors() == []


def test_tbq_root_task_on_gpu(runtime):
    world, rank, n, t = 4, 2, 30001, 0.01
    runtime.init("tbq", {"threshold": t}, 0, rank, world)
    size = ops.tbq_payload_bytes(n)
    payloads = [ops.tbq_compress(gauss(n, 0.02, seed=r), torch.zeros(n), t) for r in range(world)]
    C = torch.cat(payloads).pin_memory()
    own = gauss(n, 0.02, seed=50)
    tensor, resid = own.cuda(), torch.zeros(n, device="cuda")
    B = torch.zeros(size, dtype=torch.uint8, device="cuda")
    assert runtime.submit_task("w", tensor, resid, B, C, 1, runtime.ROOT_DECOMP_COMP_TASK)
    runtime.wait_for(runtime.ROOT_DECOMP_COMP_TASK, ["w"])
    acc = own.clone()
    for r in range(world):
        if r != rank:
            ops.tbq_decompress(payloads[r], acc, t, add=True)
    assert torch.equal(tensor.cpu(), acc)
    r2 = torch.zeros(n)
    expect = ops.tbq_compress(acc, r2, t)
    assert torch.equal(B.cpu(), expect) and torch.equal(C[:size], expect)
    assert torch.equal(resid.cpu(), r2)


def test_graddrop_tasks_on_gpu(runtime):
    n, drop = 200000, 0.999
    runtime.init("graddrop", {"drop_ratio": drop, "sample_rate": 0.01, "seed": 3}, 0, 0, 1)
    g = gauss(n, seed=1)
    gd, resid = g.cuda(), torch.zeros(n, device="cuda")
    cap = ops.sparse_payload_bytes(n, 1 - drop)
    B = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    C = torch.zeros(cap, dtype=torch.uint8).pin_memory()
    runtime.submit_task("g", gd, resid, B, C, 0, runtime.COMP_TASK)
    runtime.wait_for(runtime.COMP_TASK, ["g"])
    total = struct.unpack("<i", bytes(C[:4].tolist()))[0]
    assert 4 < total <= cap
    out = torch.zeros(n, device="cuda")
    runtime.submit_task("g", out, resid, torch.zeros_like(B), C, 0, runtime.DECOMP_TASK)
    runtime.wait_for(runtime.DECOMP_TASK, ["g"])
    torch.testing.assert_close(out.cpu() + resid.cpu(), g, atol=0, rtol=0)


def test_powersgd_tasks_on_gpu(runtime):
    runtime.init("powersgd", {"matrix_approximation_rank": 4}, 0, 0, 1)
    n, m, r = 256, 1024, 4
    torch.manual_seed(1)
    grad = torch.randn(n * m, device="cuda")
    g0 = grad.clone()
    resid = torch.zeros(n * m, device="cuda")
    M, P = torch.zeros(n, m, device="cuda"), torch.zeros(n, r, device="cuda")
    Q = torch.randn(m, r, device="cuda")
    Q0 = Q.clone()
    runtime.submit_task("p", grad, resid, M, P, Q, runtime.POWERSGD_ENCODE1)
    runtime.wait_for(runtime.POWERSGD_ENCODE1, ["p"])
    ref = g0.view(n, m).double() @ Q0.double()
    assert ((P.double() - ref).norm() / ref.norm()).item() < 5e-3
    runtime.submit_task("p", grad, resid, M, P, Q, runtime.POWERSGD_ENCODE2)
    runtime.wait_for(runtime.ROOT_DECOMP_COMP_TASK, ["p"])
    eye = P.double().T @ P.double()
    torch.testing.assert_close(eye, torch.eye(r, dtype=torch.float64, device="cuda"), atol=1e-4, rtol=0)
    runtime.submit_task("p", grad, resid, M, P, Q, runtime.POWERSGD_DECODE)
    runtime.wait_for(runtime.DECOMP_TASK, ["p"])
    approx = (P @ Q.T).view(-1)
    torch.testing.assert_close(grad, approx, atol=1e-3, rtol=1e-3)
    torch.testing.assert_close(resid, g0 - approx, atol=1e-3, rtol=1e-3)
    assert runtime.getErrors() == []


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("task", ["compress", "decompress"])
def test_names_of_a_backlog_come_one_by_one(runtime, pinned, task):
    """One worker and a backlog: a name is out when its task is done, and not together with those behind it."""
    n, count = 1 << 26, 20
    runtime.init("tbq", {"threshold": 0.02}, 0, 0, 1)
    size = ops.tbq_payload_bytes(n)
    x, r = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    B = torch.zeros(size, dtype=torch.uint8, device="cuda")
    C = torch.zeros(size, dtype=torch.uint8)
    C = C.pin_memory() if pinned else C
    kind = runtime.COMP_TASK if task == "compress" else runtime.DECOMP_TASK
    for warm in (True, False):
        torch.cuda.synchronize()
        t0, came = time.monotonic(), []
        for i in range(count):
            runtime.submit_task(f"t{i}", x, r, B, C, 0, kind)
        while len(came) < count and time.monotonic() < t0 + 30:
            came += [(k, time.monotonic() - t0) for k in runtime.getResults(kind)]
    assert [k for k, _ in came] == [f"t{i}" for i in range(count)]
    when = [t for _, t in came]
    assert when[9] - when[0] > 0.25 * (when[-1] - when[0]), when   # 9 of 19 steps if all take the same time


def medians_beside_matrix_products(*calls):
    """Median time of each call, started while products that fill the chip run on another stream."""
    a = torch.randn(16384, 16384, device="cuda").bfloat16()
    c = torch.empty_like(a)
    side = torch.cuda.Stream()
    medians = []
    for call in calls:
        call()
        times = []
        for _ in range(9):
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                for _ in range(4):
                    torch.matmul(a, a, out=c)
            time.sleep(0.002)
            t = time.monotonic()
            call()
            times.append(time.monotonic() - t)
        medians.append(sorted(times)[4])
    return medians


@pytest.mark.parametrize("n", [65536, 1 << 20])
def test_terngrad_tasks_do_not_wait_for_a_free_gpu(runtime, n):
    """Beside matrix products that fill the chip, a task starts on what is left of it (about a third of the time of the
    forms that want eight or all SMs at once, which the op takes)."""
    runtime.init("terngrad", {"enable_random": 0, "bitwidth": 2}, 0, 0, 1)
    g = gauss(n).cuda()
    B = torch.zeros(ops.terngrad_payload_bytes(n, 2), dtype=torch.uint8, device="cuda")
    C = torch.zeros(B.numel(), dtype=torch.uint8).pin_memory()
    high = torch.cuda.Stream(priority=-1)

    def task():
        runtime.submit_task("t", g, B, C, 0, runtime.COMP_TASK)
        runtime.wait_for(runtime.COMP_TASK, ["t"])

    def op():
        with torch.cuda.stream(high):
            ops.terngrad_compress(g, 2, False, out=B)
            C.copy_(B, non_blocking=True)
        high.synchronize()

    task()
    assert torch.equal(C, ops.terngrad_compress(g.cpu(), 2, False))
    of_task, of_op = medians_beside_matrix_products(task, op)
    assert of_task < 0.75 * of_op


def test_graddrop_decode_tasks_do_not_wait_for_a_free_gpu(runtime):
    """The same for the sparse decode, whose op works in tiles."""
    n, drop = 1 << 20, 0.999
    runtime.init("graddrop", {"drop_ratio": drop, "sample_rate": 0.01, "seed": 3}, 0, 0, 1)
    r = gauss(n, seed=1).cuda()
    B = ops.graddrop_compress(torch.zeros_like(r), r, 0.01, drop, 3)
    C = torch.zeros(B.numel(), dtype=torch.uint8).pin_memory()
    C.copy_(B)
    out, want = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    high = torch.cuda.Stream(priority=-1)
    torch.cuda.synchronize()

    def task():
        runtime.submit_task("t", out, r, B, C, 0, runtime.DECOMP_TASK)
        runtime.wait_for(runtime.DECOMP_TASK, ["t"])

    def op():
        with torch.cuda.stream(high):
            B.copy_(C, non_blocking=True)
            ops.sparse_decompress(B, want)
        high.synchronize()

    of_task, of_op = medians_beside_matrix_products(task, op)
    assert torch.equal(out, want)
    assert of_task < 0.75 * of_op


@pytest.mark.parametrize("alg", ["tbq", "terngrad"])
@pytest.mark.parametrize("n", [1, 1003, 4 * ((1 << 20) - 10), 4 * (1 << 20) + 4, 5000001])
@pytest.mark.parametrize("host", ["pinned", "off_a_word", "pageable", "longer"])
def test_payload_reaches_the_staging_buffer(runtime, alg, n, host):
    """Stored by the kernel into pinned memory, up to a size, or copied: B and C hold the same payload, and nothing
    behind it is touched."""
    if alg == "tbq":
        runtime.init("tbq", {"threshold": 0.01}, 0, 0, 1)
        size = ops.tbq_payload_bytes(n)
    else:
        runtime.init("terngrad", {"enable_random": 0, "bitwidth": 2}, 0, 0, 1)
        size = ops.terngrad_payload_bytes(n, 2)
    g, r = gauss(n, seed=n), gauss(n, 0.004, seed=n + 1)
    buf = torch.full((size + 64,), 9, dtype=torch.uint8)
    if host != "pageable":
        buf = buf.pin_memory()
    first = 1 if host == "off_a_word" else 0
    C = buf[first:first + size + (32 if host == "longer" else 0)]
    B = torch.zeros(size, dtype=torch.uint8, device="cuda")
    rc, dev, rg = r.clone(), g.cuda(), r.cuda()
    if alg == "tbq":
        want = ops.tbq_compress(g, rc, 0.01)
        runtime.submit_task("t", dev, rg, B, C, 0, runtime.COMP_TASK)
    else:
        want = ops.terngrad_compress(g, 2, False)
        runtime.submit_task("t", dev, B, C, 0, runtime.COMP_TASK)
    runtime.wait_for(runtime.COMP_TASK, ["t"])
    assert torch.equal(C[:size], want) and torch.equal(B.cpu(), want)
    assert int((buf[:first] != 9).sum()) == 0 and int((buf[first + size:] != 9).sum()) == 0
    if alg == "tbq":
        assert torch.equal(rg.cpu(), rc)
    assert runtime.getErrors() == []
