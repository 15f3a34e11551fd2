"""The fused training-step operators against the same model in fp32 through plain PyTorch modules."""
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


def test_out_of_range_target_gives_nan_and_large_logits_stay_finite():
    from hylink_b200.ops.extension import ops

    h = torch.full((4, 8), 30.0, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(33, 8, device="cuda").mul_(10).to(torch.bfloat16)
    t = torch.tensor([0, 5, 32, 7], device="cuda")
    want = torch.nn.functional.cross_entropy((h @ w.t()).float(), t)
    torch.testing.assert_close(ops().head_loss(h, w, t), want, rtol=1e-4, atol=1e-4)
    t[1] = 33
    assert bool(ops().head_loss(h, w, t).isnan())
