"""The sharded AdamW kernel and the fused mixture-of-experts layer on one GPU (a one-rank job), against plain PyTorch."""
import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def one_rank_job():
    from hylink_b200.parallel.trainer import init_distributed

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    yield
    if fresh:
        dist.destroy_process_group()


# fewer elements than a packet, one over a CTA's, many CTAs
@pytest.mark.parametrize("count", [3, 2049, 300001])
@pytest.mark.parametrize("dtype,master", [(torch.float32, False), (torch.bfloat16, True), (torch.float16, False)])
def test_sharded_adamw_matches_adamw(count, dtype, master):
    from hylink_b200.parallel.zero import ShardedAdamW

    torch.manual_seed(count)
    p = torch.nn.Parameter(torch.randn(count, device="cuda").to(dtype))
    ref = torch.nn.Parameter(p.detach().double())
    opt = ShardedAdamW([p], lr=1e-2, weight_decay=0.1, master_fp32=master)
    ropt = torch.optim.AdamW([ref], lr=1e-2, weight_decay=0.1)
    for _ in range(3):
        g = (1e-3 * torch.randn(count, device="cuda")).to(dtype)
        p.grad.copy_(g)
        ref.grad = g.double()
        opt.step()
        ropt.step()
        if dtype != torch.float32 and not master:
            ref.data.copy_(ref.data.to(dtype))       # 16-bit weights without a master copy are rounded every step
    if master:
        torch.testing.assert_close(opt.master[:count].double(), ref.detach(), rtol=1e-5, atol=1e-6)
    ulp = {torch.float32: 1e-5, torch.bfloat16: 8e-3, torch.float16: 1e-3}[dtype]
    torch.testing.assert_close(p.detach().double(), ref.detach(), rtol=ulp, atol=1e-5)
    st = ropt.state[ref]
    torch.testing.assert_close(opt.m[:count].double(), st["exp_avg"], rtol=1e-5, atol=1e-8)
    torch.testing.assert_close(opt.v[:count].double(), st["exp_avg_sq"], rtol=1e-5, atol=1e-12)
    assert not opt.flat[count:].any() and not opt.m[count:].any()


# one token; tokens that fill no warp; overflowing experts; more than a CTA of tokens; experts in and beyond registers
@pytest.mark.parametrize("tokens,width,experts,capacity", [(1, 8, 1, 1), (37, 64, 4, 5), (1500, 264, 8, 200), (2100, 1024, 16, 256), (515, 2048, 24, 30)])
def test_moe_matches_the_dense_layer(tokens, width, experts, capacity):
    from hylink_b200.parallel.moe import ExpertParallelMLP

    torch.manual_seed(tokens)
    layer = ExpertParallelMLP(width, 4 * width, experts_per_rank=experts, capacity=capacity).cuda().to(torch.bfloat16)
    with torch.no_grad():
        layer.router.weight.mul_(2)
    ref = ExpertParallelMLP(width, 4 * width, experts_per_rank=experts, capacity=capacity).cuda()
    ref.load_state_dict({k: v.float() for k, v in layer.state_dict().items()})
    # the choice of expert is a step function: both layers have to start from the same 16-bit logits
    class Rounded(torch.autograd.Function):
        @staticmethod
        def forward(ctx, z):
            return z.to(torch.bfloat16).float()

        @staticmethod
        def backward(ctx, g):
            return g

    plain = ref.router.forward
    ref.router.forward = lambda z: Rounded.apply(plain(z))
    x = torch.randn(tokens, width, device="cuda").to(torch.bfloat16).requires_grad_(True)
    with torch.no_grad():
        close = (layer.router(x).float() - ref.router(x.float())).abs().amax(1) > 0     # rounded another way: leave those tokens out
        x[close] = x[~close][0] if bool((~close).any()) else x[close]
    xr = x.detach().float().requires_grad_(True)
    assert layer._fusable(x)
    y, yr = layer(x), ref(xr)
    dy = torch.randn_like(y)
    y.backward(dy)
    yr.backward(dy.float())

    def rel(a, b):
        return float((a.float() - b).norm() / b.norm().clamp_min(1e-12))

    assert rel(y, yr) < 5e-3 and rel(x.grad, xr.grad) < 1e-2
    for (n, p), q in zip(layer.named_parameters(), ref.parameters()):
        if float(q.grad.norm()) > 1e-6:
            assert rel(p.grad, q.grad) < 2e-2, n


def _off_boundary(t):
    """A contiguous copy of `t` that starts inside a 16-byte packet."""
    out = torch.empty(t.numel() + 3, dtype=t.dtype, device=t.device)[3:].view(t.shape)
    assert out.is_contiguous() and out.data_ptr() % 16
    return out.copy_(t)


# experts whose gradients a warp holds in registers, and more
@pytest.mark.parametrize("tokens,width,experts,capacity", [(37, 64, 4, 11), (300, 264, 20, 17)])
@pytest.mark.parametrize("pieces", [False, True])
def test_moe_takes_tensors_off_the_packet_boundary(tokens, width, experts, capacity, pieces):
    """Weights that a parameter of three elements shifts in ShardedAdamW's flat buffer; tokens and gradients that are views."""
    import copy

    from hylink_b200.parallel.moe import ExpertParallelMLP
    from hylink_b200.parallel.zero import ShardedAdamW

    torch.manual_seed(tokens)
    plain = ExpertParallelMLP(width, 4 * width, experts_per_rank=experts, capacity=capacity).cuda().to(torch.bfloat16)
    layer = copy.deepcopy(plain)
    lead = torch.nn.Parameter(torch.zeros(3, device="cuda", dtype=torch.bfloat16))
    ShardedAdamW([lead, *layer.parameters()])
    assert layer.router.weight.data_ptr() % 16
    if pieces:                                       # the form in which tokens travel: weights of another type take it on one rank too
        for m in (plain, layer):
            m.w1.data = m.w1.data.float()
            m.w1.grad = None
    x, dy = (torch.randn(tokens, width, device="cuda").to(torch.bfloat16) for _ in range(2))
    results = []
    for m, place in ((plain, lambda t: t.clone()), (layer, _off_boundary)):
        xi = place(x).requires_grad_()
        assert m._fusable(xi)
        y = m(xi)
        y.backward(place(dy))
        results.append([y.detach(), xi.grad, *(p.grad for p in m.parameters())])
    for a, b in zip(*results):
        assert float((a.float() - b.float()).norm()) <= 1e-2 * float(a.float().norm()) + 1e-6


def test_sharded_adamw_takes_a_gradient_off_the_packet_boundary():
    from hylink_b200.parallel.zero import ShardedAdamW

    torch.manual_seed(1)
    start, grad = torch.randn(1003, device="cuda").to(torch.bfloat16), torch.randn(1003, device="cuda").to(torch.bfloat16)
    weights = []
    for place in (lambda t: t.clone(), _off_boundary):
        opt = ShardedAdamW([torch.nn.Parameter(start.clone())], lr=1e-2)
        opt.flat_grad[:1003].copy_(grad)
        opt.flat_grad = opt.grad_shard = place(opt.flat_grad)
        opt.step()
        weights.append(opt.master.clone())
    torch.testing.assert_close(*weights, rtol=1e-5, atol=1e-6)


def test_the_routers_own_forward_is_called():
    from hylink_b200.parallel.moe import ExpertParallelMLP

    layer, seen = ExpertParallelMLP(64, 128, experts_per_rank=4, capacity=16).cuda().to(torch.bfloat16), []
    plain = layer.router.forward
    layer.router.forward = lambda x: (seen.append(1), plain(x))[1]
    layer(torch.randn(10, 64, device="cuda", dtype=torch.bfloat16))
    assert len(seen) == 1


def test_moe_under_modes_and_hooks_runs_as_modules():
    from torch.utils._python_dispatch import TorchDispatchMode

    from hylink_b200.parallel.moe import ExpertParallelMLP

    class Seen(TorchDispatchMode):
        names = set()

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.add(str(func))
            return func(*args, **(kwargs or {}))

    torch.manual_seed(2)
    layer = ExpertParallelMLP(64, 128, experts_per_rank=4, capacity=16).cuda().to(torch.bfloat16)
    x = torch.randn(10, 64, device="cuda", dtype=torch.bfloat16)
    with Seen() as seen:
        layer(x)
    assert any("gelu" in n for n in seen.names)
    calls = []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, a, o: calls.append(m))
    try:
        layer(x)
    finally:
        handle.remove()
    assert layer.router in calls


@pytest.mark.parametrize("pieces", [False, True])
def test_moe_can_be_differentiated_again(pieces):
    """A gradient penalty, against the same layer as modules; the third expert overflows."""
    import copy

    from hylink_b200.parallel.moe import ExpertParallelMLP

    torch.manual_seed(3)
    layer = ExpertParallelMLP(64, 128, experts_per_rank=4, capacity=9).cuda().to(torch.bfloat16)
    with torch.no_grad():
        layer.router.weight.mul_(4)
        layer.w1.mul_(5)
        layer.w2.mul_(5)
    if pieces:
        layer.w1.data = layer.w1.data.float()
    plain = copy.deepcopy(layer)
    plain._fusable = lambda x: False
    x0, dy = (torch.randn(40, 64, device="cuda").to(torch.bfloat16) for _ in range(2))
    results = []
    for m in (layer, plain):
        x = x0.clone().requires_grad_()
        assert m is plain or m._fusable(x)
        y = m(x * 1)                                 # not a leaf
        grads = torch.autograd.grad(y, [x, *m.parameters()], dy, create_graph=True)
        sum(g.float().square().sum() for g in grads).backward()
        results.append([*(g.detach().float() for g in grads), x.grad.float(), *(p.grad.float() for p in m.parameters())])
    for i, (a, b) in enumerate(zip(*results)):       # the plain layer rounds every step to 16 bits, the dot products of the gate among them
        assert float((a - b).norm()) <= 3e-2 * float(b.norm()) + 1e-6, i


@pytest.mark.parametrize("frozen,products", [([], 4), (["w1", "w2"], 2), (["x"], 3), (["x", "router.weight"], 3), (["x", "router.weight", "w1"], 1),
                                             (["x", "w1", "w2"], 0)])
def test_moe_leaves_the_products_of_frozen_weights_out(frozen, products):
    from torch.utils._python_dispatch import TorchDispatchMode

    from hylink_b200.parallel.moe import ExpertParallelMLP

    class Products(TorchDispatchMode):
        count = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.count += func is torch.ops.aten.bmm.default
            return func(*args, **(kwargs or {}))

    torch.manual_seed(5)
    layer = ExpertParallelMLP(64, 128, experts_per_rank=4, capacity=12).cuda().to(torch.bfloat16)
    x, dy = (torch.randn(40, 64, device="cuda").to(torch.bfloat16) for _ in range(2))
    leaves = {"x": x, **dict(layer.named_parameters())}
    for t in leaves.values():
        t.requires_grad_(True)
    want = dict(zip(leaves, torch.autograd.grad(layer(x), list(leaves.values()), dy)))
    for n, t in leaves.items():
        t.requires_grad_(n not in frozen)
    y = layer(x)
    with Products() as seen:
        y.backward(dy)
    assert seen.count == products
    for n, t in leaves.items():
        assert t.grad is None if n in frozen else torch.equal(t.grad, want[n]), n


def test_sizes_beyond_the_moe_kernels_run_as_modules():
    from hylink_b200.ops.extension import ops
    from hylink_b200.parallel.moe import ExpertParallelMLP

    layer = ExpertParallelMLP(64, 128, experts_per_rank=4, capacity=5).cuda().to(torch.bfloat16)
    x = torch.randn(10, 64, device="cuda", dtype=torch.bfloat16)
    for capacity, fits in ((0, False), (5, True), (ops().max_rows // 4, True), (ops().max_rows // 4 + 1, False)):
        layer.cap = capacity
        assert layer._fusable(x) == fits
    layer.cap, layer.n_experts = 5, 3
    assert not layer._fusable(x)


@pytest.mark.parametrize("wanted", [False, True])
def test_dispatched_rows_want_a_gradient_when_the_tokens_do(wanted):
    """As on the plain path: every rank then takes part in the same number of exchanges, whichever path it is on."""
    from hylink_b200.ops.extension import ops

    x = torch.randn(10, 64, device="cuda", dtype=torch.bfloat16).requires_grad_(wanted)
    router = torch.randn(4, 64, device="cuda", dtype=torch.bfloat16).requires_grad_()
    _, send, gate, row_of, token_of = ops().moe_dispatch(x, router, 5)
    assert send.requires_grad == wanted and gate.requires_grad and not row_of.requires_grad and not token_of.requires_grad
    gate.sum().backward()
    assert bool(router.grad.isfinite().all()) and (x.grad is not None) == wanted


def test_the_gates_gradient_is_whole():
    """Zero for a token beyond the capacity, whatever the memory held before."""
    from hylink_b200.ops.extension import ops

    x = torch.randn(40, 64, device="cuda", dtype=torch.bfloat16)
    router = torch.randn(1, 64, device="cuda", dtype=torch.bfloat16).requires_grad_()
    x1, send, gate, row_of, token_of = ops().moe_dispatch(x, router, 5)
    for _ in range(3):
        trash = [torch.full((40,), float("nan"), device="cuda") for _ in range(8)]
        del trash
        y = ops().moe_combine(x1, gate, send, row_of, token_of)
        dgate, = torch.autograd.grad(y, gate, torch.ones_like(y), retain_graph=True)
        assert bool((dgate[row_of < 0] == 0).all()) and bool(dgate[row_of >= 0].isfinite().all())


def test_routing_of_equal_infinite_and_nan_logits():
    """Expert and gate of every token are the maximum of the softmax, as torch finds it."""
    from hylink_b200.ops.extension import ops

    torch.manual_seed(6)
    router, x = (torch.randn(n, 64, device="cuda") for n in (8, 40))
    router[5] = router[2]                            # equal logits
    x[:8] *= 1e-9                                    # different logits, one probability
    x[8:16] *= 1e38                                  # infinite ones of either sign
    x[16, 3], x[17, 9] = float("nan"), float("inf")
    x[18] = 0
    broken = router.clone()
    broken[3, 0] = float("nan")                      # one expert's logits are NaN for every token
    x = x.to(torch.bfloat16)
    for w in (router.to(torch.bfloat16), broken.to(torch.bfloat16)):
        want, expert = torch.softmax((x @ w.t()).float(), -1).max(-1)
        _, _, gate, row_of, _ = ops().moe_dispatch(x, w, 40)
        assert torch.equal(row_of.long() // 40, expert)
        torch.testing.assert_close(gate, want, rtol=1e-6, atol=0, equal_nan=True)


def test_gelu_over_all_16_bit_values():
    """Every finite bf16 value, through experts whose two products are the identity: the bits of torch's own kernel."""
    from hylink_b200.ops.extension import ops

    x = torch.arange(1 << 16, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = x[x.isfinite()]
    x = x[:x.numel() // 8 * 8].view(1, -1, 8)
    eye = torch.eye(8, device="cuda", dtype=torch.bfloat16)[None]
    got = ops().moe_experts(x, eye, eye)
    want = torch.nn.functional.gelu(x, approximate="tanh")
    assert torch.equal(got, want), [(float(a), float(b), float(c)) for a, b, c in zip(x[got != want], got[got != want], want[got != want])][:20]


def _plain_experts(h, w1, w2, dy):
    """Forward and gradients in fp64, rounded where the layer stores a 16-bit tensor."""
    r = [t.detach().double() for t in (h, w1, w2, dy)]
    at = lambda t: t.to(h.dtype).double()                                   # noqa: E731
    u = at(torch.bmm(r[0], r[1])).requires_grad_()
    act = torch.nn.functional.gelu(u, approximate="tanh")
    a = at(act.detach())
    dact = at(torch.bmm(r[3], r[2].transpose(1, 2)))
    du = at(torch.autograd.grad(act, u, dact)[0])
    return torch.bmm(a, r[2]), torch.bmm(du, r[1].transpose(1, 2)), torch.bmm(r[0].transpose(1, 2), du), torch.bmm(a.transpose(1, 2), r[3])


# tiles are 256 x 256, an operand's box 64, k goes in blocks of 64 and steps of 16, rows in steps of 32
@pytest.mark.parametrize("experts,rows,width,hidden", [(1, 512, 256, 1024), (3, 257, 264, 1032), (2, 31, 512, 2048), (40, 33, 136, 520), (2, 320, 1000, 72),
                                                       (1, 1, 4096, 4096), (5, 129, 320, 1288)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["dense", "off the boundary", "transposed", "strided"])
def test_expert_products_at_the_edges_of_their_tiles(experts, rows, width, hidden, dtype, form):
    from hylink_b200.ops.extension import ops

    assert experts * rows * width * hidden >= 1 << 24                       # these go through the own kernel
    torch.manual_seed(rows)
    place = {"dense": lambda t: t, "off the boundary": _off_boundary, "transposed": lambda t: t.transpose(1, 2).contiguous().transpose(1, 2),
             "strided": lambda t: torch.cat([t, t], 2)[:, :, :t.shape[2]]}[form]
    h, dy = (torch.randn(experts, rows, width, device="cuda").to(dtype) for _ in range(2))
    w1 = (torch.randn(experts, width, hidden, device="cuda") * width ** -0.5).to(dtype)
    w2 = (torch.randn(experts, hidden, width, device="cuda") * hidden ** -0.5).to(dtype)
    want = _plain_experts(h, w1, w2, dy)
    leaves = [place(t).requires_grad_() for t in (h, w1, w2)]
    y = ops().moe_experts(*leaves)
    got = (y.detach(), *torch.autograd.grad(y, leaves, place(dy)))
    # a result is rounded once, and where an fp32 sum falls on the other side of a tie an intermediate is one step off: under one
    # step (2^-8 or 2^-11 of the value) in all, in the mean; a single entry is off by sums of such steps
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for name, a, b in zip(("y", "dh", "dw1", "dw2"), got, want):
        diff = (a.double() - b).abs()
        assert float(diff.norm() / b.norm()) < step, name
        assert float((diff / (b.abs() + b.square().mean().sqrt())).max()) < 8 * step, name


# an expert without tokens, with one, with a full and with an overflowing queue; capacities off every step
@pytest.mark.parametrize("capacity", [1, 31, 300, 513])
def test_experts_of_any_load(capacity):
    """Rows beyond an expert's tokens are not computed: whatever memory held there must not be seen."""
    from hylink_b200.ops.extension import ops

    torch.manual_seed(capacity)
    experts, width, hidden = 5, 256, 1 << 14
    load = torch.tensor([0, 1, min(capacity, 40), capacity, capacity + 70])
    expert = torch.repeat_interleave(torch.arange(experts), load)[torch.randperm(int(load.sum()))].cuda()
    router = torch.zeros(experts, width, device="cuda")
    router[:, :experts] = 30 * torch.eye(experts, device="cuda")
    x = torch.randn(expert.numel(), width, device="cuda")
    x[:, :experts] = torch.nn.functional.one_hot(expert, experts).float()
    w1, w2 = (torch.randn(experts, *s, device="cuda") * s[0] ** -0.5 for s in ((width, hidden), (hidden, width)))
    leaves = [t.to(torch.bfloat16).requires_grad_() for t in (x, router, w1, w2)]
    dy = torch.randn_like(leaves[0])
    trash = [torch.full((experts, capacity, hidden), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(6)]
    del trash
    y = ops().moe_layer(*leaves, capacity)
    got = (y.detach(), *torch.autograd.grad(y, (leaves[0], leaves[2], leaves[3]), dy))
    fx, fw1, fw2 = (t.detach().double().requires_grad_() for t in (leaves[0], leaves[2], leaves[3]))
    out = fx.clone()
    for e in range(experts):
        mine = (expert == e).nonzero().squeeze(1)[:capacity]
        out[mine] = fx[mine] + torch.nn.functional.gelu(fx[mine] @ fw1[e], approximate="tanh") @ fw2[e]     # the gate is one
    want = (out, *torch.autograd.grad(out, (fx, fw1, fw2), dy.double()))
    for name, a, b in zip(("y", "dx", "dw1", "dw2"), got, want):
        assert bool(a.isfinite().all()), name
        assert float((a.double() - b).norm()) < 3 * 2.0 ** -8 * float(b.norm()), name      # three roundings on the way


# a warp's 256 columns, a CTA's 1024, rows that leave warps without work; fewer tokens than CTAs, more than a CTA's threads; one to all experts
@pytest.mark.parametrize("tokens,width,experts", [(1, 8, 1), (147, 264, 8), (149, 768, 3), (600, 1032, 8), (40000, 256, 2), (1200, 2048, 5)])
def test_the_routers_gradient_at_the_edges_of_its_blocks(tokens, width, experts):
    from hylink_b200.ops.extension import ops

    torch.manual_seed(tokens)
    capacity = max(1, tokens // experts)             # some tokens have no row
    x, dy = (torch.randn(tokens, width, device="cuda").to(torch.bfloat16) for _ in range(2))
    router = (torch.randn(experts, width, device="cuda") * width ** -0.5).to(torch.bfloat16)
    w1, w2 = (torch.randn(experts, *s, device="cuda").mul(s[0] ** -0.5).to(torch.bfloat16) for s in ((width, 64), (64, width)))
    leaves = [t.clone().requires_grad_() for t in (x, router)]
    y = ops().moe_layer(*leaves, w1, w2, capacity)
    dx, drouter = torch.autograd.grad(y, leaves, dy)
    # the same pieces, with the router's share left to a product and the sums to fp64
    alone = [x.clone().requires_grad_(), router]
    plain = torch.autograd.grad(ops().moe_layer(*alone, w1, w2, capacity), alone[0], dy)[0]
    assert torch.equal(dx, plain)                    # without the router's gradient the tokens' comes from the kernel of its own
    x1, send, gate, row_of, _ = ops().moe_dispatch(x, router, capacity)
    p = torch.softmax((x @ router.t()).double(), -1)
    expert = p.argmax(-1)
    h = torch.bmm(torch.nn.functional.gelu(torch.bmm(send.view(experts, capacity, width).double(), w1.double()), approximate="tanh"), w2.double())
    dgate = torch.where(row_of >= 0, (dy.double() * h.view(-1, width)[row_of.long().clamp_min(0)]).sum(1), 0.)
    onehot = torch.nn.functional.one_hot(expert, experts)
    dlogits = (dgate * p.gather(1, expert[:, None]).squeeze(1))[:, None] * (onehot - p)
    want = dlogits.t() @ x.double()
    # 16-bit logits' gradients from rows that were rounded three times: two steps of 2^-8 in the mean
    if float(want.norm()) > 0:
        assert float((drouter.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8
    else:
        assert not drouter.any()


def test_hooks_on_the_experts_saved_tensors():
    """Hooks see rows out of use too, and may keep a tensor in any form: what they see is finite, what one that scales by the largest value gives
    back is good for the gradients, and a tensor that comes back in another type is an error."""
    from hylink_b200.ops.extension import ops

    torch.manual_seed(3)
    tokens, width, hidden, experts, capacity = 300, 256, 1024, 4, 500           # most rows are out of use; 2^29
    leaves = [(torch.randn(*s, device="cuda") * scale).to(torch.bfloat16).requires_grad_()
              for s, scale in (((tokens, width), 1.0), ((experts, width), width ** -0.5), ((experts, width, hidden), width ** -0.5),
                               ((experts, hidden, width), hidden ** -0.5))]
    dy = torch.randn(tokens, width, device="cuda").to(torch.bfloat16)

    def spoil():                                                                # memory that the next tensors will get
        trash = [torch.full((experts, capacity, n), float("nan"), device="cuda", dtype=torch.bfloat16) for n in (hidden, width) for _ in range(4)]
        del trash

    def through(pack, unpack):
        spoil()
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            y = ops().moe_layer(*leaves, capacity)
        spoil()
        return torch.autograd.grad(y, leaves, dy)

    want = torch.autograd.grad(ops().moe_layer(*leaves, capacity), leaves, dy)
    seen = []

    def scaled(t):
        if not t.is_floating_point():
            return t
        seen.append(bool(t.isfinite().all()))
        top = t.abs().max().float().clamp_min(1e-30)
        return (t.float() / top * 32767).round().to(torch.int16), top, t.dtype

    got = through(scaled, lambda k: k if isinstance(k, torch.Tensor) else (k[0].float() * (k[1] / 32767)).to(k[2]))
    assert len(seen) >= 9 and all(seen)
    for name, a, b in zip(("dx", "drouter", "dw1", "dw2"), got, want):
        assert bool(a.isfinite().all()), name
        # kept to 2^-16 of the largest value, which is some eight times the mean: under two steps of bf16 on the way
        assert float((a.double() - b.double()).norm()) < 2 * 2.0 ** -8 * float(b.double().norm()), name
    big = experts * capacity * hidden
    with pytest.raises(RuntimeError, match="hylink"):
        through(lambda t: t, lambda t: t.float() if t.numel() == big and t.dim() == 3 else t)


# below and from the 2^33 multiplications on from which the own products are the faster ones on the GPU
@pytest.mark.parametrize("rows,own", [(2000, False), (2048, True)])
def test_recorded_experts_take_the_faster_products(rows, own):
    """Recorded into a graph, a layer costs the GPU's time alone. An eager layer of the same size is issued faster by the own products,
    whatever its size, and its backward pass goes the way of its forward pass, recorded or not."""
    from hylink_b200.ops.extension import ops

    torch.manual_seed(rows)
    h, w1, w2, dy = ((torch.randn(1, *s, device="cuda") * 0.03).to(torch.bfloat16).requires_grad_(i < 3)
                     for i, s in enumerate(((rows, 1024), (1024, 4096), (4096, 1024), (rows, 1024))))
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):                    # a backward pass runs where its forward pass did
        eager = ops().moe_experts(h, w1, w2)
        want = torch.autograd.grad(eager, (h, w1, w2), dy, retain_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        y = ops().moe_experts(h, w1, w2)
        got = torch.autograd.grad(y, (h, w1, w2), dy)
        mixed = torch.autograd.grad(eager, (h, w1, w2), dy)
    graph.replay()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    # a replay: two launches forward and two backward, and two of `mixed`, the backward pass of an eager layer (a profiler may miss one)
    assert (sum("kExpertGemm" in n for n in names) > 6) == own, names
    assert torch.equal(y, eager)
    for a, b, c in zip(got, mixed, want):
        assert torch.equal(a, c) and torch.equal(b, c)


@pytest.mark.parametrize("experts", [1, 4, 12])
def test_operators_without_tokens(experts):
    """A rank may have no tokens: outputs are empty, the weights' gradients zero."""
    from hylink_b200.ops.extension import ops

    make = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16).requires_grad_()      # noqa: E731
    x, router, w1, w2 = make(0, 64), make(experts, 64), make(experts, 64, 128), make(experts, 128, 64)
    y = ops().moe_layer(x, router, w1, w2, 8)
    grads = torch.autograd.grad(y, (x, router, w1, w2), torch.zeros_like(y))
    x1, send, gate, row_of, token_of = ops().moe_dispatch(x, router, 8)
    grads += torch.autograd.grad((x1, send, gate), (x, router), (torch.zeros_like(x1), torch.randn_like(send), torch.zeros_like(gate)))
    assert y.shape == x1.shape == (0, 64) and not send.any() and bool((token_of == -1).all())
    for g, t in zip(grads, (x, router, w1, w2, x, router)):
        assert g.shape == t.shape and not g.any()
