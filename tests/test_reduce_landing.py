"""Landing-reduce kernel against PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype.is_floating_point:
        return (torch.rand(n, generator=g, device="cuda") * 2 - 1).to(dtype)
    return torch.randint(-100, 100, (n,), generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16, torch.float64, torch.int32,
                                   torch.int64, torch.int8, torch.uint8])
@pytest.mark.parametrize("count", [1, 17, 4096, 100003])
def test_two_address_sum(dtype, count):
    from hylink_b200.ops import reduce_landing

    a, b = _rand(count, dtype, 1), _rand(count, dtype, 2)
    if dtype == torch.uint8:
        a, b = a.abs().to(dtype), b.abs().to(dtype)
    dst = a.clone()
    reduce_landing(dst, [b], accumulate=True)
    torch.cuda.synchronize()
    if dtype in (torch.bfloat16, torch.float16):
        ref = (a.float() + b.float()).to(dtype)
    else:
        ref = a + b
    assert torch.equal(dst, ref)


@pytest.mark.parametrize("op", ["sum", "max", "min"])
@pytest.mark.parametrize("k", [1, 3, 8])
def test_k_way_three_address(op, k):
    from hylink_b200.ops import reduce_landing

    count = 70001
    srcs = [_rand(count, torch.bfloat16, 10 + i) for i in range(k)]
    dst = torch.empty(count, dtype=torch.bfloat16, device="cuda")
    reduce_landing(dst, srcs, op=op, scale=0.5 if op == "sum" else 1.0)
    torch.cuda.synchronize()
    acc = srcs[0].float()
    for s in srcs[1:]:
        acc = {"sum": acc + s.float(), "max": torch.maximum(acc, s.float()), "min": torch.minimum(acc, s.float())}[op]
    if op == "sum":
        acc = acc * 0.5
    assert torch.equal(dst, acc.to(torch.bfloat16))


# one, two, up to four and up to nine operands; one packet per thread and four, whole packets and a rest, off the boundary
@pytest.mark.parametrize("op", ["max", "min", "prod"])
@pytest.mark.parametrize("k,accumulate", [(1, False), (1, True), (2, False), (3, True), (4, True), (8, False)])
@pytest.mark.parametrize("dtype,count,off", [(torch.bfloat16, 4097, 0), (torch.float16, 9_700_003, 0), (torch.int8, 100_003, 0), (torch.float32, 3001, 1)])
def test_operators_in_every_operand_class(op, k, accumulate, dtype, count, off):
    from hylink_b200.ops import reduce_landing

    srcs = [_rand(count + off, dtype, 20 + i)[off:] for i in range(k)]
    dst = _rand(count + off, dtype, 5)[off:]
    up = (lambda t: t.float()) if dtype in (torch.bfloat16, torch.float16) else (lambda t: t)
    parts = ([up(dst)] if accumulate else []) + [up(s) for s in srcs]
    want = parts[0].clone()
    for p in parts[1:]:
        want = {"max": torch.maximum, "min": torch.minimum, "prod": torch.mul}[op](want, p)
    reduce_landing(dst, srcs, op=op, accumulate=accumulate)
    assert torch.equal(dst, want.to(dtype))


def test_pinned_host_source_and_unaligned():
    from hylink_b200.ops import reduce_landing

    count = 50001
    host = torch.randn(count + 1).pin_memory()
    dev = torch.randn(count + 1, device="cuda")
    dst = dev.clone()
    reduce_landing(dst[1:], [host[1:]], accumulate=True)  # 4-byte offset: element-wise path
    torch.cuda.synchronize()
    torch.testing.assert_close(dst[1:], dev[1:] + host[1:].cuda(), rtol=0, atol=0)
    dst2 = dev.clone()
    reduce_landing(dst2[:count], [host[:count]], accumulate=True)  # aligned: vector path over PCIe
    torch.cuda.synchronize()
    assert torch.equal(dst2[:count], dev[:count] + host[:count].cuda())


def test_other_threads_run_while_a_launch_waits():
    """A stream whose queue is full makes the next launch wait; the interpreter must not wait with it."""
    import threading
    import time

    from hylink_b200.ops import reduce_landing

    src, dst = (torch.ones(16, device="cuda") for _ in range(2))
    reduce_landing(dst, [src])
    torch.cuda.synchronize()

    def fill():
        torch.cuda._sleep(1_000_000_000)                 # about half a second
        for _ in range(4000):
            reduce_landing(dst, [src])

    t = threading.Thread(target=fill)
    t.start()
    worst, last = 0.0, time.perf_counter()
    while t.is_alive():
        now = time.perf_counter()
        worst, last = max(worst, now - last), now
    t.join()
    torch.cuda.synchronize()
    assert worst < 0.2, worst


def test_folds_captured_in_a_graph():
    """A chain of folds whose launches overlap, with an ordinary kernel and a copy between them."""
    from hylink_b200.ops import reduce_landing

    a, b = (torch.zeros(1 << 18, device="cuda") for _ in range(2))
    x = torch.ones(1 << 18, device="cuda")

    def chain():
        reduce_landing(a, [x, b])
        reduce_landing(b, [a], accumulate=True, scale=0.5)
        a.mul_(2)
        reduce_landing(b, [a])
        x.copy_(b)
        reduce_landing(a, [x], accumulate=True)

    chain()
    torch.cuda.synchronize()
    for t, v in ((a, 0), (b, 0), (x, 1)):
        t.fill_(v)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    va, vb, vx = 0.0, 0.0, 1.0
    for _ in range(6):
        graph.replay()
        va = vx + vb
        va *= 2
        vb = vx = va
        va += vx
        assert bool((a == va).all()) and bool((b == vb).all()) and bool((x == vx).all())
