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
