"""Streamed push kernels (large messages between ranks of one GPU: a ring of pieces instead of staging of the message's
size) against PyTorch, bit for bit: ascending rank order, fp32 accumulation, one rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(count, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype.is_floating_point:
        return torch.randn(count, generator=g, device="cuda").to(dtype)
    return torch.randint(-50, 50, (count,), generator=g, device="cuda").to(dtype)


def _sum(ts, dtype):
    acc = ts[0].float() if dtype.is_floating_point else ts[0].clone()
    for t in ts[1:]:
        acc = acc + (t.float() if dtype.is_floating_point else t)
    return acc.to(dtype)


# whole pieces, ragged ends, every rank-count class and counts between the classes, a strided prefix of wider segments,
# segments that start inside a packet (these keep the plain kernels)
@pytest.mark.parametrize("n,seg,dtype,offset", [(2, (9 << 20) + 4, torch.float32, 0), (3, 3 * 1000003 + 1, torch.float32, 0),
                                                (4, 3 << 20, torch.bfloat16, 0), (8, 448 * 8 * 200 + 5, torch.bfloat16, 0),
                                                (8, (1 << 19) + 3, torch.int32, 0), (5, 1500001, torch.bfloat16, 1)])
def test_streamed_collectives(n, seg, dtype, offset, monkeypatch):
    from hylink_b200.ops import EmuGroup

    monkeypatch.setenv("HYLINK_KERNEL_TIMELINE", "1")
    g = EmuGroup(n)
    kinds = lambda: {launch["kind"] for launch in g.kernel_timeline()}  # noqa: E731
    pad = 16

    def outs(elems):
        return [torch.full((offset + elems + pad,), 7, dtype=dtype, device="cuda") for _ in range(n)]

    def body(bufs, elems):
        return [b[offset:offset + elems] for b in bufs]

    stride = (seg + 31) // 8 * 8
    wide = [_rand(offset + n * stride, dtype, 900 + r)[offset:] for r in range(n)]
    sums = [_sum([w[r * stride:r * stride + seg] for w in wide], dtype) for r in range(n)]
    for _ in range(2):                                # back to back: the ring and its flags carry over
        o = outs(seg)
        g.run("reduce_scatter", wide, body(o, seg), seg, in_seg_stride=stride)
        for b, want in zip(o, sums):
            assert torch.equal(b[offset:offset + seg], want) and bool((b[offset + seg:] == 7).all())
    o = outs(n * stride)
    g.run("all_gather", [w[:seg] for w in wide], body(o, n * stride), seg, out_seg_stride=stride)
    for b in o:
        for q in range(n):
            at = offset + q * stride
            assert torch.equal(b[at:at + seg], wide[q][:seg]) and bool((b[at + seg:at + stride] == 7).all())
    o = outs(n * stride)
    g.run("all_to_all", wide, body(o, n * stride), seg, in_seg_stride=stride, out_seg_stride=stride)
    for r, b in enumerate(o):
        for q in range(n):
            at = offset + q * stride
            assert torch.equal(b[at:at + seg], wide[q][r * stride:r * stride + seg]) and bool((b[at + seg:at + stride] == 7).all())
    want = {"allgather_streamed", "alltoall_streamed"} | ({"reducescatter_streamed"} if n <= 4 else set())
    assert {k for k in kinds() if k.endswith("streamed")} == (want if offset == 0 else set())
    # in place: the result into the own segment of the input, the input out of the own segment of the output, one buffer
    work = [w.clone() for w in wide]
    g.run("reduce_scatter", work, [w[r * stride:r * stride + seg] for r, w in enumerate(work)], seg, in_seg_stride=stride)
    assert all(torch.equal(w[r * stride:r * stride + seg], sums[r]) for r, w in enumerate(work))
    work = [w.clone() for w in wide]
    g.run("all_gather", [w[r * stride:r * stride + seg] for r, w in enumerate(work)], work, seg, out_seg_stride=stride)
    assert all(torch.equal(w[q * stride:q * stride + seg], wide[q][q * stride:q * stride + seg]) for w in work for q in range(n))
    work = [w.clone() for w in wide]
    g.run("all_to_all", work, work, seg, in_seg_stride=stride, out_seg_stride=stride)
    assert all(torch.equal(w[q * stride:q * stride + seg], wide[q][r * stride:r * stride + seg]) for r, w in enumerate(work) for q in range(n))
    assert g.status(0)[0] == 0
    g.close()


# two whole pieces for every CTA (a piece: 448 threads of eight, four or two packets), one packet more or less, ragged ends
@pytest.mark.parametrize("n,extra", [(2, 0), (2, 5), (3, 1), (4, -8), (4, 0), (4, 8), (8, -1), (8, 0), (8, 9)])
def test_streamed_all_gather_at_the_edges_of_its_pieces(n, extra, monkeypatch):
    from hylink_b200.ops import EmuGroup

    monkeypatch.setenv("HYLINK_KERNEL_TIMELINE", "1")
    g = EmuGroup(n)
    seg = 148 // n * 448 * (8 if n <= 2 else 4 if n <= 4 else 2) * 2 * 8 + extra
    stride = (seg + 7) // 8 * 8
    for rep in range(3):                              # back to back: a slow reader of one call, a fast writer of the next
        ins = [_rand(seg, torch.bfloat16, 10 * rep + r) for r in range(n)]
        outs = [torch.full((n * stride + 8,), 7, dtype=torch.bfloat16, device="cuda") for _ in range(n)]
        g.run("all_gather", ins, outs, seg, out_seg_stride=stride)
        for o in outs:
            assert all(torch.equal(o[q * stride:q * stride + seg], ins[q]) and bool((o[q * stride + seg:(q + 1) * stride] == 7).all()) for q in range(n))
    assert "allgather_streamed" in {launch["kind"] for launch in g.kernel_timeline()}
    g.close()


def test_streamed_wait_is_bounded():
    from hylink_b200.ops import EmuGroup

    n, seg = 4, 2 << 20
    g = EmuGroup(n, timeout_ms=200)
    ins = [_rand(n * seg, torch.float32, r) for r in range(n)]
    outs = [torch.zeros(seg, device="cuda") for _ in range(n)]
    g.set_active_ranks(n - 1)
    g.run("reduce_scatter", ins, outs, seg, in_seg_stride=seg)
    torch.cuda.synchronize()                          # returns: the wait was bounded
    code, _, peer, _ = g.status(0)
    assert code == 1 and peer == n - 1
    g.set_active_ranks(n)
    g.reset()
    g.run("reduce_scatter", ins, outs, seg, in_seg_stride=seg)
    torch.cuda.synchronize()
    assert g.status(0)[0] == 0
    assert all(torch.equal(o, _sum([t[r * seg:(r + 1) * seg] for t in ins], torch.float32)) for r, o in enumerate(outs))
    g.close()


# the smallest message that streams, ragged ends, a message of more than one launch, outputs that keep the plain kernel
@pytest.mark.parametrize("n,count,dtype,offset", [(2, (12 << 20) - 3, torch.bfloat16, 0), (3, (4 << 20) + 9, torch.float32, 0),
                                                  (8, (4 << 20) + 1, torch.bfloat16, 0), (4, (8 << 20) + 5, torch.bfloat16, 3),
                                                  (2, (17 << 20) + 2, torch.int32, 0)])
def test_streamed_broadcast(n, count, dtype, offset, monkeypatch):
    from hylink_b200.ops import EmuGroup

    monkeypatch.setenv("HYLINK_KERNEL_TIMELINE", "1")
    g = EmuGroup(n)
    outs = [torch.full((offset + count + 16,), 7, dtype=dtype, device="cuda") for _ in range(n)]
    bufs = [o[offset:offset + count] for o in outs]
    for rep in range(3):                              # back to back, from different roots, in place
        root = (rep + 1) % n
        data = _rand(count, dtype, rep)
        srcs = [data if r == root else bufs[r] for r in range(n)]
        if rep == 2:
            bufs[root].copy_(data)
            srcs = bufs
        g.run("broadcast", srcs, bufs, count, root=root)
        assert all(torch.equal(b, data) and bool((o[offset + count:] == 7).all()) for o, b in zip(outs, bufs))
    assert ("broadcast_streamed" in {launch["kind"] for launch in g.kernel_timeline()}) == (offset == 0)
    g.close()


@pytest.mark.parametrize("least,kind", [(None, "allgather_streamed"), (str(192 << 20), "allgather_streamed"), (str(160 << 20), "allgather_lanes")])
def test_the_lane_kernel_can_be_asked_for(least, kind):
    """HYLINK_AG_LANES_MIN_BYTES counts between ranks of one GPU too, where it is set; without it they stream, at any size."""
    import os
    import subprocess
    import sys

    code = """
import torch
from hylink_b200.ops import EmuGroup
g = EmuGroup(2)
seg = 40 << 20
ins = [torch.arange(seg, device="cuda").add(r).to(torch.bfloat16) for r in range(2)]
outs = [torch.zeros(2 * seg, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
g.run("all_gather", ins, outs, seg, out_seg_stride=seg)
torch.cuda.synchronize()
assert all(torch.equal(o, torch.cat(ins)) for o in outs)
print("kinds", *{launch["kind"] for launch in g.kernel_timeline()})
"""
    env = {**os.environ, "HYLINK_KERNEL_TIMELINE": "1"}
    env.pop("HYLINK_AG_LANES_MIN_BYTES", None)
    if least:
        env["HYLINK_AG_LANES_MIN_BYTES"] = least
    out = subprocess.run([sys.executable, "-c", code], check=True, timeout=120, env=env, capture_output=True, text=True).stdout
    assert f"kinds {kind}" in out
