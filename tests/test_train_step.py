"""The fused training-step operators against the same model in fp32 through plain PyTorch modules."""
import contextlib
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _grads(model, idx, targets):
    model.zero_grad(set_to_none=True)
    loss = model(idx, targets)
    loss.backward()
    return loss.detach().float(), {n: p.grad.detach().float() for n, p in model.named_parameters()}


# a row narrower than a warp, one that ends inside a chunk, whole chunks; head widths 8 to 64; rows that fill no CTA;
# vocabularies with and without padding behind them
@pytest.mark.parametrize("width,heads,vocab,batch,seq", [(64, 8, 101, 1, 5), (264, 3, 1000, 3, 37), (768, 12, 1024, 2, 64), (1024, 16, 3001, 2, 129)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_fused_step_matches_fp32(width, heads, vocab, batch, seq, dtype):
    from hylink_b200.models.gpt2 import GPT2, GPT2Config

    torch.manual_seed(width + seq)
    ref = GPT2(GPT2Config(n_layer=2, n_head=heads, d_model=width, vocab_size=vocab, n_ctx=256)).cuda()
    for p in ref.parameters():                       # gains and biases away from one and zero, weights as the 16-bit model has them
        p.data = (p.data + 0.05 * torch.randn_like(p)).to(dtype).float()
    model = copy.deepcopy(ref).to(dtype)
    idx = torch.randint(0, vocab, (batch, seq), device="cuda")
    targets = torch.randint(0, vocab, (batch, seq), device="cuda")
    targets[0, ::3] = -100                           # rows that do not count
    assert model._fusable(torch.empty(1, device="cuda", dtype=dtype), targets)
    loss, got = _grads(model, idx, targets)
    want_loss, want = _grads(ref, idx, targets)
    eager = copy.deepcopy(model)
    eager._fusable = lambda x, t: False
    eager_loss, plain = _grads(eager, idx, targets)
    assert abs(loss - want_loss) <= max(2 * abs(eager_loss - want_loss), 2e-3 * abs(want_loss))
    for n, w in want.items():
        err, base = ((g[n] - w).norm() / w.norm() for g in (got, plain))
        assert err <= max(1.3 * base, 1e-3), (n, float(err), float(base))


def test_fused_step_takes_parameters_off_the_packet_boundary():
    """As views into one flat buffer, behind a parameter of three elements."""
    from hylink_b200.models.gpt2 import GPT2, GPT2Config

    torch.manual_seed(4)
    plain = GPT2(GPT2Config(n_layer=2, n_head=3, d_model=264, vocab_size=1024, n_ctx=64)).cuda().to(torch.bfloat16)
    model = copy.deepcopy(plain)
    flat = torch.empty(3 + sum(p.numel() for p in model.parameters()), device="cuda", dtype=torch.bfloat16)
    at = 3
    for p in model.parameters():
        p.data = flat[at:at + p.numel()].view(p.shape).copy_(p.data)
        at += p.numel()
        assert p.data_ptr() % 16
    idx, targets = (torch.randint(0, 1024, (2, 37), device="cuda") for _ in range(2))
    assert model._fusable(torch.empty(1, device="cuda", dtype=torch.bfloat16), targets)
    want_loss, want = _grads(plain, idx, targets)
    loss, got = _grads(model, idx, targets)
    assert abs(loss - want_loss) <= 2e-3 * abs(want_loss)
    for n, w in want.items():                        # other places are other kernels of the library for the products
        assert float((got[n] - w).norm() / w.norm()) < 2e-2, n


def _head_case(rows, width, vocab):
    g = torch.Generator(device="cuda").manual_seed(1)
    h = torch.randn(rows, width, generator=g, device="cuda").to(torch.bfloat16).requires_grad_()
    w = (0.02 * torch.randn(vocab, width, generator=g, device="cuda")).to(torch.bfloat16).requires_grad_()
    return h, w, torch.randint(0, vocab, (rows,), generator=g, device="cuda")


@pytest.mark.parametrize("reduced", [True, False])
@pytest.mark.parametrize("rows,width,vocab", [(5, 64, 101), (100, 768, 50257), (2048, 264, 3001), (6144, 1024, 8191)])
def test_head_gradient_over_an_odd_vocabulary(rows, width, vocab, reduced):
    """No further from fp64 than the library's product over the same 16-bit operands; where reduced-precision reductions
    are switched off, the sum adds no error to the two roundings (operand and result, half a unit of 2^-8 each)."""
    from hylink_b200.ops.extension import ops

    h, w, t = _head_case(rows, width, vocab)
    p = torch.softmax((h.detach().float() @ w.detach().float().t()).to(torch.bfloat16).double(), -1)
    p[torch.arange(rows, device="cuda"), t] -= 1
    p /= rows
    want = p @ w.detach().double()
    flag = torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
    try:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = reduced
        got, = torch.autograd.grad(ops().head_loss(h, w, t), h)
        plain = p.to(torch.bfloat16) @ w.detach()
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = flag
    err, base = (float((x.double() - want).norm() / want.norm()) for x in (got, plain))
    assert err <= 1.05 * base + 1e-4, (err, base)
    if not reduced:
        assert err < 3e-3, err


def test_head_gradient_is_one_product_of_the_library():
    """Bit for bit. With the identity for h, the weight's gradient is the transposed gradient of the logits."""
    from hylink_b200.ops.extension import ops

    n, vocab, padded = 2560, 8191, 8192
    _, w, t = _head_case(n, n, vocab)
    h = torch.eye(n, device="cuda", dtype=torch.bfloat16).requires_grad_()
    got, dw = torch.autograd.grad(ops().head_loss(h, w, t), (h, w))
    d = torch.zeros(n, padded, device="cuda", dtype=torch.bfloat16)
    d[:, :vocab] = dw.t()
    assert torch.equal(got, d[:, :vocab] @ w.detach())


@pytest.mark.parametrize("targets", [(2, 7), (1, 8), (2, 9)])
def test_as_many_targets_as_tokens(targets):
    """Another number of targets is the plain loss's error, and the operator's own."""
    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.ops.extension import ops

    model = GPT2(GPT2Config(n_layer=1, n_head=2, d_model=64, vocab_size=100, n_ctx=16)).cuda().to(torch.bfloat16)
    idx, t = torch.zeros(2, 8, dtype=torch.int64, device="cuda"), torch.zeros(targets, dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError):
        model(idx, t)
    with pytest.raises(ValueError):
        ops().head_loss(torch.zeros(2, 8, 64, device="cuda", dtype=torch.bfloat16), model.wte.weight, t)
    assert model.step_signature(idx, t) is None
    assert model.step_signature(idx, idx) is not None and bool(model(idx, idx.reshape(-1)).isfinite())


def test_out_of_range_target_gives_nan_and_large_logits_stay_finite():
    from hylink_b200.ops.extension import ops

    h = torch.full((4, 8), 30.0, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(33, 8, device="cuda").mul_(10).to(torch.bfloat16)
    t = torch.tensor([0, 5, 32, 7], device="cuda")
    want = torch.nn.functional.cross_entropy((h @ w.t()).float(), t)
    torch.testing.assert_close(ops().head_loss(h, w, t), want, rtol=1e-4, atol=1e-4)
    t[1] = 33
    assert bool(ops().head_loss(h, w, t).isnan())


# all packets of a thread, or the first of several, a warp, a row; a value among others, a packet of them
@pytest.mark.parametrize("value", [float("-inf"), float("nan"), float("inf")])
@pytest.mark.parametrize("vocab", [13, 4000, 4104 + 3])
def test_infinite_and_nan_logits(value, vocab):
    """Loss and gradient as the plain loss has them. With a unit vector for h the logits are the weight's first column."""
    from hylink_b200.ops.extension import ops

    torch.manual_seed(vocab)
    base = torch.randn(vocab, device="cuda").to(torch.bfloat16)
    h = torch.zeros(2, 8, device="cuda", dtype=torch.bfloat16)
    h[:, 0] = 1
    for lo, hi in ((0, 8), (0, 256), (3, 4), (8, 13), (0, vocab), (vocab - 1, vocab)):
        w = torch.zeros(vocab, 8, device="cuda", dtype=torch.bfloat16)
        w[:, 0] = base
        w[lo:min(hi, vocab), 0] = value
        for targets in ((1, vocab - 2), (lo, 9)):
            t = torch.tensor(targets, device="cuda")
            z = w[:, 0].float().expand(2, vocab).clone().requires_grad_()
            want = torch.nn.functional.cross_entropy(z, t)
            dz, = torch.autograd.grad(want, z)
            wg = w.clone().requires_grad_()
            got = ops().head_loss(h, wg, t)
            dw, = torch.autograd.grad(got, wg)
            torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5, equal_nan=True)
            torch.testing.assert_close(dw[:, 0].float(), dz.to(torch.bfloat16).float().sum(0), rtol=2e-2, atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("name,batch,seq", [("tiny", 3, 64), ("gpt2-small", 2, 100)])
def test_replayed_steps_train_like_eager_ones(name, batch, seq, monkeypatch):
    """Forward and backward from a graph from the second step on, against the same steps run eagerly: with a learning rate
    that changes, gradients that the caller drops, another batch shape in between, and a hook that has to be called."""
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    cfg = GPT2Config.by_name(name)
    torch.manual_seed(3)
    first = GPT2(cfg)
    g = torch.Generator().manual_seed(5)
    tokens = [torch.randint(0, cfg.vocab_size, (batch, (seq if i != 6 else seq // 2) + 1), generator=g).pin_memory() for i in range(14)]

    def train(replay):
        monkeypatch.setenv("HYLINK_TRAIN_GRAPH", "1" if replay else "0")
        model = copy.deepcopy(first)
        t = DDPTrainer(model, torch.device("cuda", 0))
        losses, replayed, seen = [], [], []
        for i, tok in enumerate(tokens):
            t.opt.param_groups[0]["lr"] = 1e-3 / (1 + i)
            if i == 5:
                t.opt.zero_grad(set_to_none=True)
            if i == 12:
                model.ln_f.register_forward_hook(lambda *a: seen.append(1))
            losses.append(t.step(tok))
            replayed.append(t._graph is not None)
        assert len(seen) == 2
        out = torch.cat([p.detach().float().reshape(-1) for p in model.parameters()]), [p.grad.float() for p in model.parameters()]
        t.close()
        return losses, replayed, out

    losses, replayed, (weights, grads) = train(True)
    want_losses, never, (want, want_grads) = train(False)
    # steps 1 to 5 replay; a batch of another shape; three eager steps of the old one (its recording was short-lived)
    # before it is recorded again; hooked
    assert replayed == [False] + [True] * 5 + [False] * 4 + [True] * 2 + [False] * 2 and not any(never)
    torch.testing.assert_close(torch.tensor(losses), torch.tensor(want_losses), rtol=5e-3, atol=0)
    assert float((weights - want).norm() / want.norm()) < 1e-2
    if fresh:
        dist.destroy_process_group()


@pytest.mark.parametrize("change", ["no affine", "no bias", "wide norm", "odd hidden", "heads"])
def test_other_layers_run_as_modules(change):
    """Layers of the plain classes that the fused operators do not take."""
    from hylink_b200.models.gpt2 import GPT2, GPT2Config

    torch.manual_seed(7)
    ref = GPT2(GPT2Config(n_layer=2, n_head=4, d_model=64, vocab_size=100, n_ctx=16)).cuda()
    b = ref.blocks[1]
    nn = torch.nn
    with torch.device("cuda"):
        if change == "no affine":
            b.ln1, ref.ln_f = nn.LayerNorm(64, elementwise_affine=False), nn.LayerNorm(64, elementwise_affine=False)
        elif change == "no bias":
            b.ln2 = nn.LayerNorm(64, bias=False)
        elif change == "wide norm":
            b.ln1 = nn.LayerNorm((8, 64))
        elif change == "odd hidden":
            b.fc, b.out = nn.Linear(64, 101), nn.Linear(101, 64)
        else:
            b.n_head = 16
    model = copy.deepcopy(ref).to(torch.bfloat16)
    ref = copy.deepcopy(model).float()
    idx = torch.randint(0, 100, (2, 8), device="cuda")
    loss, got = _grads(model, idx, idx)
    want_loss, want = _grads(ref, idx, idx)
    assert abs(loss - want_loss) <= 5e-3 * abs(want_loss)
    for n, w in want.items():                        # two layers of 16-bit modules
        assert float((got[n] - w).norm()) <= 3e-2 * float(w.norm()) + 1e-6, n


def _small(dtype=torch.bfloat16):
    from hylink_b200.models.gpt2 import GPT2, GPT2Config

    torch.manual_seed(9)
    model = GPT2(GPT2Config(n_layer=2, n_head=2, d_model=64, vocab_size=100, n_ctx=16)).cuda().to(dtype)
    return model, torch.randint(0, 100, (2, 8), device="cuda"), torch.randint(0, 100, (2, 8), device="cuda")


def test_tracing_and_compilation_see_the_modules():
    model, idx, targets = _small()
    want = model(idx, targets)
    traced = torch.jit.trace(model, (targets, idx), check_trace=False)
    torch.testing.assert_close(traced(idx, targets), want, rtol=2e-3, atol=0)
    torch.testing.assert_close(torch.compile(model, backend="eager", fullgraph=True)(idx, targets), want, rtol=2e-3, atol=0)


def test_transforms_and_modes_see_the_modules():
    import torch.autograd.forward_ad as fwd
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        names = set()

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.add(str(func))
            return func(*args, **(kwargs or {}))

    model, idx, targets = _small()
    want_loss, want = _grads(model, idx, targets)
    params = dict(model.named_parameters())
    got = torch.func.grad(lambda p: torch.func.functional_call(model, p, (idx, targets)))(params)
    for n, w in want.items():
        assert float((got[n].float() - w).norm() / w.norm()) < 2e-2, n
    # the derivative along the gradient is its squared norm
    with sdpa_kernel(SDPBackend.MATH), fwd.dual_level():
        dual = {n: fwd.make_dual(p.detach(), want[n].to(p.dtype)) for n, p in params.items()}
        slope = fwd.unpack_dual(torch.func.functional_call(model, dual, (idx, targets))).tangent
    squared = sum(float(w.double().square().sum()) for w in want.values())
    assert abs(float(slope) - squared) < 2e-2 * squared
    with Seen() as seen:
        model(idx, targets)
    assert any("gelu" in n for n in seen.names)
    fake = FakeTensorMode()
    stand_ins, *tokens = [{n: fake.from_tensor(p.detach()) for n, p in params.items()}, fake.from_tensor(idx), fake.from_tensor(targets)]
    with fake:
        assert torch.func.functional_call(model, stand_ins, tuple(tokens)).shape == ()
    with torch.device("cuda"):                       # a default device is no reason
        assert model._fusable(torch.empty(1, dtype=torch.bfloat16), targets)


def test_a_step_can_be_differentiated_again():
    """The gradient of the squared length of the gradient; the same gradients with a graph behind them."""
    from torch.nn.attention import SDPBackend, sdpa_kernel

    def penalty(model, idx, targets):
        model.zero_grad(set_to_none=True)
        with sdpa_kernel(SDPBackend.MATH):
            loss = model(idx, targets)
            grads = torch.autograd.grad(loss, list(model.parameters()), create_graph=True)
            sum(g.float().square().sum() for g in grads).backward()
        return [g.detach().float() for g in grads], [p.grad.float() for p in model.parameters()]

    model, idx, targets = _small()
    ref = copy.deepcopy(model).float()
    names = [n for n, _ in model.named_parameters()]
    for tol, got, want in zip((2e-2, 5e-2), penalty(model, idx, targets), penalty(ref, idx, targets)):
        for n, a, b in zip(names, got, want):
            assert float((a - b).norm()) <= tol * float(b.norm()) + 1e-4, n


# frozen parameters by the end of their name, and how many of the step's products for gradients remain: 2 blocks x 8 and the head's 2
@pytest.mark.parametrize("frozen,products", [([], 18), (["fc.weight", "out.weight", "qkv.weight", "proj.weight"], 10), (["wte.weight", "wpe.weight"], 17),
                                             (["blocks."], 10), (["wte.weight", "wpe.weight", "blocks."], 1)])
def test_products_of_frozen_weights_are_left_out(frozen, products):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Products(TorchDispatchMode):
        count = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.count += func is torch.ops.aten.mm.default
            return func(*args, **(kwargs or {}))

    model, idx, targets = _small()
    _, want = _grads(model, idx, targets)
    model.zero_grad(set_to_none=True)
    left = []
    for n, p in model.named_parameters():
        p.requires_grad_(not any(f in n for f in frozen))
        left += [n] * p.requires_grad
    loss = model(idx, targets)
    with Products() as seen:
        loss.backward()
    assert seen.count == products
    for n, p in model.named_parameters():
        assert (p.grad is None) == (n not in left)
        if n in left and n != "wte.weight":
            assert torch.equal(p.grad.float(), want[n]), n


def _counted(module, seen):
    plain = module.forward
    module.forward = lambda *a: (seen.append(1), plain(*a))[1]


@pytest.mark.parametrize("where", ["blocks.1", "blocks.0.fc", "blocks.0.ln2", "ln_f", "wte", "wpe", ""])
def test_a_forward_of_an_instance_is_called(where):
    """On the model, its blocks and their layers: in every step, recorded ones included."""
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    model, seen = GPT2(GPT2Config.tiny()), []
    t = DDPTrainer(model, torch.device("cuda", 0))
    _counted(model.get_submodule(where), seen)
    tokens = torch.randint(0, 1024, (2, 33)).pin_memory()
    for _ in range(4):
        t.step(tokens)
    assert len(seen) == 4
    t.close()
    if fresh:
        dist.destroy_process_group()


@pytest.mark.parametrize("what", ["hook on wpe", "subclass", "accumulation", "accumulation, before", "accumulation, later", "saved tensors"])
def test_a_step_with_effects_is_not_replayed(what):
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    seen = []

    class Counting(GPT2):
        def forward(self, *a):
            seen.append(1)
            return super().forward(*a)

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    model = (Counting if what == "subclass" else GPT2)(GPT2Config.tiny())
    if what == "hook on wpe":
        model.wpe.register_forward_hook(lambda *a: seen.append(1))
    t = DDPTrainer(model, torch.device("cuda", 0))
    tokens = torch.randint(0, 1024, (2, 33)).pin_memory()
    if what.endswith("later"):
        for _ in range(3):
            t.step(tokens)
        assert t._graph is not None
    if what.startswith("accumulation"):
        p = model.blocks[1].fc.weight
        node = p.expand_as(p).grad_fn.next_functions[0][0]
        (node.register_prehook if what.endswith("before") else node.register_hook)(lambda *a: seen.append(1))
    context = contextlib.nullcontext()
    if what == "saved tensors":
        first = []
        context = torch.autograd.graph.saved_tensors_hooks(lambda x: (first.append(1), x)[1], lambda x: x)
    with context:
        for _ in range(4):
            t.step(tokens)
            if what == "saved tensors":
                seen += [1] * bool(first)
                first.clear()
    assert len(seen) == 4 and t._graph is None
    t.close()
    if fresh:
        dist.destroy_process_group()


def test_a_wrapper_of_the_callers_own():
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    model, seen = GPT2(GPT2Config.tiny()), []
    t = DDPTrainer(model, torch.device("cuda", 0))
    tokens = torch.randint(0, 1024, (2, 33)).pin_memory()
    for _ in range(3):
        t.step(tokens)
    t.ddp = lambda idx, targets: (seen.append(1), model(idx, targets))[1]
    for _ in range(3):
        t.step(tokens)
    assert len(seen) == 3
    t.close()
    if fresh:
        dist.destroy_process_group()


@pytest.mark.parametrize("where", ["before", "inside"])
def test_a_failed_capture_leaves_eager_steps(where, monkeypatch, capsys):
    """Raised on the host, before the capture begins and in the middle of the recorded forward pass: one message, the steps go on."""
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel import trainer
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    fresh = not dist.is_initialized()
    if fresh:
        init_distributed("hylink")
    torch.manual_seed(8)
    first = GPT2(GPT2Config.tiny())
    tokens = torch.randint(0, 1024, (2, 33)).pin_memory()
    plain = GPT2._fused_loss

    def fails(self, x, targets):
        loss = plain(self, x, targets)
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("no room")
        return loss

    def train(broken):
        with monkeypatch.context() as m:
            m.setenv("HYLINK_TRAIN_GRAPH", "1" if broken else "0")
            if broken and where == "before":
                m.setattr(trainer._StepGraph, "_capture", lambda self, model: (_ for _ in ()).throw(RuntimeError("no room")))
            elif broken:
                m.setattr(GPT2, "_fused_loss", fails)
            t = DDPTrainer(copy.deepcopy(first), torch.device("cuda", 0))
            losses = [t.step(tokens) for _ in range(4)]
            assert t._graph is None and not t._use_graph
            grads = [p.grad for p in t.model.parameters()]
            t.close()
            return losses, grads

    losses, grads = train(True)
    assert capsys.readouterr().out.count("not replayed") == 1
    want, want_grads = train(False)
    torch.testing.assert_close(torch.tensor(losses), torch.tensor(want), rtol=5e-3, atol=0)
    for a, b in zip(grads, want_grads):
        assert float((a.float() - b.float()).norm()) <= 3e-2 * float(b.float().norm()) + 1e-6
    if fresh:
        dist.destroy_process_group()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_multi_tensor_adamw_matches_torch(dtype):
    """Tensors shorter than a packet, of a ragged length, unaligned, of several chunks; more of them than one launch takes."""
    from hylink_b200.ops.extension import ops

    g = torch.Generator(device="cuda").manual_seed(2)
    sizes = [1, 7, 8, 8193, 40000] + [5 + i for i in range(500)]
    ps = [torch.randn(n + 1, generator=g, device="cuda").to(dtype)[1 if i == 3 else 0:n + (1 if i == 3 else 0)] for i, n in enumerate(sizes)]
    ref = [p.double().clone().requires_grad_() for p in ps]
    ms, vs = [torch.zeros_like(p) for p in ps], [torch.zeros_like(p) for p in ps]
    steps = [torch.zeros((), device="cuda") for _ in ps]
    opt = torch.optim.AdamW(ref, lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1)
    for _ in range(3):
        gs = [(0.1 * torch.randn(p.shape, generator=g, device="cuda")).to(dtype) for p in ps]
        assert ops().multi_adamw(ps, gs, ms, vs, steps, 1e-2, 0.9, 0.95, 0.1, 1e-8)
        for r, x in zip(ref, gs):
            r.grad = x.double()
        opt.step()
        for p, r, m, v in zip(ps, ref, ms, vs):                 # both go on from the rounded weights and moments
            tol = {torch.bfloat16: 1e-2, torch.float16: 2e-3, torch.float32: 1e-5}[dtype]
            torch.testing.assert_close(p.double(), r.detach(), rtol=tol, atol=tol * 1e-1)
            r.data.copy_(p)
            opt.state[r]["exp_avg"].copy_(m)
            opt.state[r]["exp_avg_sq"].copy_(v)
    assert all(float(s) == 3 for s in steps)
    assert not ops().multi_adamw(ps[:1], [gs[0].cpu()], ms[:1], vs[:1], steps[:1], 1e-2, 0.9, 0.95, 0.1, 1e-8)


# the smallest MLP whose products carry gelu themselves (2^33 multiplications), rows off the steps of 32 and of a tile's 256, fp16
@pytest.mark.parametrize("rows,width,hidden,dtype", [(2048, 1024, 4096, torch.bfloat16), (2049, 1024, 4096, torch.bfloat16), (4100, 520, 4104, torch.bfloat16),
                                                     (2300, 1024, 4096, torch.float16)])
def test_gelu_inside_the_products_of_an_mlp(rows, width, hidden, dtype):
    from hylink_b200.ops.extension import ops

    assert rows * width * hidden >= 1 << 33
    torch.manual_seed(rows)
    make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(dtype)            # noqa: E731
    x, a, dx2, dy2 = (make(1, rows, width) for _ in range(4))
    wp, bp, gamma, beta = make(width, width, scale=width ** -0.5), make(width, scale=0.1), 1 + make(width, scale=0.1), make(width, scale=0.1)
    wf, bf = make(hidden, width, scale=width ** -0.5), make(hidden, scale=0.1)
    wo, bo = make(width, hidden, scale=hidden ** -0.5), make(width, scale=0.1)
    leaves = [t.requires_grad_() for t in (x, a, wp, bp, gamma, beta, wf, bf, wo, bo)]
    x2, y2 = ops().block_post(*leaves, 1e-5)
    got = (x2.detach(), y2.detach(), *torch.autograd.grad((x2, y2), leaves, (dx2, dy2)))
    r = [t.detach().double().requires_grad_() for t in leaves]
    F = torch.nn.functional
    rx2 = r[0] + F.linear(r[1], r[2], r[3])
    ry2 = F.linear(F.gelu(F.linear(F.layer_norm(rx2, (width,), r[4], r[5], 1e-5), r[6], r[7]), approximate="tanh"), r[8], r[9])
    want = (rx2, ry2, *torch.autograd.grad((rx2, ry2), r, (dx2.double(), dy2.double())))
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for i, (g, w) in enumerate(zip(got, want)):      # up to six roundings one after the other, each half a step at most
        assert float((g.double() - w).norm() / w.norm()) < 3 * step, i


# every 16-bit pattern in some order, in the element-wise kernels (one row) and in the products' epilogues (2^33 multiplications)
@pytest.mark.parametrize("rows,width", [(1, 64), (512, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_of_a_value_beside_any_others(rows, width, dtype):
    """gelu has torch's bits in bf16, and it and its slope are those of the value alone: infinities, NaN and far values beside it change nothing."""
    from hylink_b200.ops.extension import ops

    hidden = 1 << 16
    zeros = lambda *s: torch.zeros(*s, device="cuda", dtype=dtype)             # noqa: E731
    values = torch.arange(hidden, device="cuda").to(torch.int16).view(dtype)

    def through(u):                                                            # pre-activations are the bias, the outputs' gradient picks row 0
        x, a, wp, bp, gamma, beta, wf, wo, bo = (zeros(1, rows, width), zeros(1, rows, width), zeros(width, width), zeros(width), 1 + zeros(width),
                                                 zeros(width), zeros(hidden, width), zeros(width, hidden), zeros(width))
        wo[0], bf, dy = 1, u.clone().requires_grad_(), zeros(1, rows, width)
        dy[0, 0, 0] = 1
        x2, y2 = ops().block_post(x, a, wp, bp, gamma, beta, wf, bf, wo.requires_grad_(), bo, 1e-5)
        act, slope = torch.autograd.grad(y2, (wo, bf), dy)
        return act[0], slope

    act, slope = through(values)
    want = torch.nn.functional.gelu(values, approximate="tanh")
    fin, step, least = want.isfinite(), *((2.0 ** -8, 0.0) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25))    # half a step of the type, of its least
    if dtype == torch.bfloat16:
        assert torch.equal(act[fin], want[fin])
    else:                                                                      # rounded to the other side of a tie
        assert bool(((act - want).abs()[fin].double() <= 2 * step * want.abs()[fin].double() + 2 * least).all())
    u = values.double().requires_grad_()
    (exact,) = torch.autograd.grad(torch.nn.functional.gelu(u, approximate="tanh").sum(), u)
    near = values.abs() < 1e4                                                  # further out u^3 leaves fp32's range, in torch's kernel too
    # one rounding to the type, and the fp32 operations before it: some 2^-22 of terms up to 2
    assert bool(((slope.double() - exact).abs()[near] <= step * exact.abs()[near] + 2.0 ** -21 + least).all())
    for seed in range(6):
        order = torch.randperm(hidden, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        a, s = through(values[order])
        for got, one in ((a, act[order]), (s, slope[order])):
            assert torch.equal(got[one.isfinite()], one[one.isfinite()])


def test_a_product_that_gives_up_is_reported(monkeypatch):
    """A wait inside a product that runs out (its operands never arrive) is an error for whoever waits for the results: in the step that
    it happens in, replayed from a graph or not, once; and for launches until then."""
    import math

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.ops import check_products
    from hylink_b200.ops.extension import ops
    from hylink_b200.parallel.trainer import DDPTrainer, init_distributed

    monkeypatch.setenv("MASTER_PORT", "29575")
    init_distributed("hylink")
    a = torch.randn(264, 136, device="cuda").to(torch.bfloat16)
    h, w1, w2 = (torch.randn(2, *s, device="cuda").to(torch.bfloat16) for s in ((256, 256), (256, 512), (512, 256)))     # 2^26: the own products

    def gives_up():
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="ran out"):
            check_products()
        check_products()                             # reported once

    check_products()
    ops().product_without_operands(a, 20.0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="ran out"):
        ops().moe_experts(h, w1, w2)
    gives_up()
    ops().moe_experts(h, w1, w2)                     # and the next one works
    # recorded: the host enters no launch function when the graph runs
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        ops().product_without_operands(a, 20.0)
    torch.cuda.synchronize()
    check_products()
    graph.replay()
    gives_up()
    # a trainer's step, eager and replayed
    torch.manual_seed(0)
    trainer = DDPTrainer(GPT2(GPT2Config.tiny()), torch.device("cuda", 0))
    tokens = torch.randint(0, 1024, (2, 65)).pin_memory()
    for step in range(5):
        trainer.step(tokens)
        real = trainer._opt_step

        def after_a_product(real=real):
            ops().product_without_operands(a, 20.0)
            real()

        trainer._opt_step = after_a_product
        with pytest.raises(RuntimeError, match="ran out"):
            trainer.step(tokens)
        trainer._opt_step = real
        assert math.isfinite(trainer.step(tokens))
    assert trainer._graph is not None                # the later ones were replayed
    ops().product_without_operands(a, 20.0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="ran out"):
        trainer.step_device(tokens[:, :-1].cuda(), tokens[:, 1:].cuda())
    trainer.close()


_PRODUCTS = """
import sys, torch
from hylink_b200.ops.extension import ops
out, dtype = {}, torch.bfloat16
g = torch.Generator("cuda").manual_seed(5)
make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=g) * scale).to(dtype)
for rows, width, hidden in ((8192, 1024, 4096), (4096, 768, 3072)):       # MLPs of the two larger models
    x, a, dx2, dy2 = (make(1, rows, width) for _ in range(4))
    wp, bp, gamma, beta = make(width, width, scale=width ** -0.5), make(width, scale=0.1), 1 + make(width, scale=0.1), make(width, scale=0.1)
    wf, bf = make(hidden, width, scale=width ** -0.5), make(hidden, scale=0.1)
    wo, bo = make(width, hidden, scale=hidden ** -0.5), make(width, scale=0.1)
    leaves = [t.requires_grad_() for t in (x, a, wp, bp, gamma, beta, wf, bf, wo, bo)]
    def go():
        x2, y2 = ops().block_post(*leaves, 1e-5)
        return (x2.detach(), y2.detach(), *torch.autograd.grad((x2, y2), leaves, (dx2, dy2)))
    for name, t in zip("x2 y2 dx da dwp dbp dgamma dbeta dwf dbf dwo dbo".split(), go()):
        out[f"mlp {rows} {name}"] = t.cpu()
for tokens, width, experts in ((8192, 1024, 8), (500, 512, 2)):
    capacity = tokens * 5 // 4 // experts
    leaves = [t.requires_grad_() for t in (make(tokens, width), make(experts, width, scale=width ** -0.5), make(experts, width, 4 * width, scale=width ** -0.5),
                                           make(experts, 4 * width, width, scale=0.5 * width ** -0.5))]
    dy = make(tokens, width)
    def go():
        y = ops().moe_layer(*leaves, capacity)
        return (y.detach(), *torch.autograd.grad(y, leaves, dy))
    for name, t in zip("y dx drouter dw1 dw2".split(), go()):
        out[f"moe {tokens} {name}"] = t.cpu()
with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
    go()
    torch.cuda.synchronize()
out["own"] = any("kExpertGemm" in e.name for e in p.events())
torch.save(out, sys.argv[1])
"""


def test_the_products_bits_are_the_librarys(tmp_path):
    """Without the own products, switched off or not available, the same calls give the same results: the training step's forward
    pass rests on that."""
    import os
    import subprocess
    import sys

    got = []
    for own in ("1", "0"):
        path = tmp_path / own
        subprocess.run([sys.executable, "-c", _PRODUCTS, str(path)], check=True, timeout=300, env={**os.environ, "HYLINK_OWN_PRODUCTS": own})
        got.append(torch.load(path))
    assert got[0].pop("own") and not got[1].pop("own")
    for name, a in got[0].items():
        b = got[1][name]
        if name.endswith("dbf"):                     # fp32 partials, added up in another order: a step of the result at most
            assert bool(((a - b).abs().double() <= 2.0 ** -7 * b.abs().double() + 2.0 ** -16).all()), name
        else:
            assert torch.equal(a, b), name


def test_products_of_a_job_of_several_ranks_are_the_librarys(monkeypatch):
    """The own products deal their tiles out to an empty GPU's multiprocessors; gradient all-reduces of other ranks hold some of them."""
    import torch.distributed as dist

    from hylink_b200.models.gpt2 import GPT2, GPT2Config
    from hylink_b200.parallel.moe import ExpertParallelMLP
    from hylink_b200.parallel.trainer import init_distributed

    monkeypatch.setenv("MASTER_PORT", "29576")
    init_distributed("hylink")
    torch.manual_seed(0)
    with torch.device("cuda"):
        model = GPT2(GPT2Config(n_layer=1, vocab_size=1024)).to(torch.bfloat16)                              # 2048 tokens: 2^33
        layer = ExpertParallelMLP(512, 2048, experts_per_rank=2, capacity=128).to(torch.bfloat16)            # 2^28
    idx = torch.randint(0, 1024, (2, 1024), device="cuda")
    x = torch.randn(200, 512, device="cuda").to(torch.bfloat16)

    def step():
        model.zero_grad(set_to_none=True)
        layer.zero_grad(set_to_none=True)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            loss = model(idx, idx)
            loss.backward()
            y = layer(x)
            y.sum().backward()
            torch.cuda.synchronize()
        return (loss.detach(), y.detach(), *(q.grad for m in (layer, model.blocks) for q in m.parameters())), sum("kExpertGemm" in e.name for e in p.events())

    one, launches = step()
    assert launches > 3                              # MLP: one each way; experts: two each way
    monkeypatch.setattr(dist, "get_world_size", lambda group=None: 2)
    two, launches = step()
    assert launches == 0
    assert torch.equal(one[0], two[0]) and torch.equal(one[1], two[1])
    for a, b in zip(one[2:], two[2:]):               # attention's own backward pass adds up in any order
        assert float((a - b).float().norm()) <= 2.0 ** -7 * float(b.float().norm())
