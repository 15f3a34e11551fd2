"""GPT-2 (the benchmark workload): decoder-only transformer with learned
positions, pre-LayerNorm blocks, GELU MLP and a tied output head.

``GPT2Config.medium()`` is the configuration the headline benchmark names:
24 layers, d_model 1024, 16 heads, vocabulary 50257, context 1024. Weights are
random-initialised (no checkpoints are available offline); the model exists so
that the collective library can be measured under a real DDP training step,
with gradient buckets overlapping the backward pass.
"""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch
import torch.nn as nn
import torch.nn.functional as F

from ..ops.extension import alone, global_module_hooks, ops, overridden, plain_eager, traced


@dataclass
class GPT2Config:
    n_layer: int = 24
    n_head: int = 16
    d_model: int = 1024
    vocab_size: int = 50257
    n_ctx: int = 1024
    dropout: float = 0.0

    @staticmethod
    def medium() -> "GPT2Config":
        return GPT2Config()

    @staticmethod
    def tiny() -> "GPT2Config":
        return GPT2Config(n_layer=2, n_head=4, d_model=128, vocab_size=1024, n_ctx=128)

    @staticmethod
    def by_name(name: str) -> "GPT2Config":
        return {"gpt2-medium": GPT2Config.medium, "medium": GPT2Config.medium, "tiny": GPT2Config.tiny,
                "gpt2-small": lambda: GPT2Config(n_layer=12, n_head=12, d_model=768)}[name]()


class Block(nn.Module):
    def __init__(self, c: GPT2Config):
        super().__init__()
        self.ln1 = nn.LayerNorm(c.d_model)
        self.qkv = nn.Linear(c.d_model, 3 * c.d_model)
        self.proj = nn.Linear(c.d_model, c.d_model)
        self.ln2 = nn.LayerNorm(c.d_model)
        self.fc = nn.Linear(c.d_model, 4 * c.d_model)
        self.out = nn.Linear(4 * c.d_model, c.d_model)
        self.n_head = c.n_head

    def forward(self, x):
        b, t, d = x.shape
        q, k, v = self.qkv(self.ln1(x)).view(b, t, 3, self.n_head, d // self.n_head).permute(2, 0, 3, 1, 4)
        a = F.scaled_dot_product_attention(q, k, v, is_causal=True)
        x = x + self.proj(a.transpose(1, 2).reshape(b, t, d))
        return x + self.out(F.gelu(self.fc(self.ln2(x)), approximate="tanh"))


class GPT2(nn.Module):
    def __init__(self, c: GPT2Config):
        super().__init__()
        self.config = c
        self.wte = nn.Embedding(c.vocab_size, c.d_model)
        self.wpe = nn.Embedding(c.n_ctx, c.d_model)
        self.blocks = nn.ModuleList([Block(c) for _ in range(c.n_layer)])
        self.ln_f = nn.LayerNorm(c.d_model)
        self.apply(self._init)
        for blk in self.blocks:  # scaled init of the residual projections
            for p in (blk.proj.weight, blk.out.weight):
                nn.init.normal_(p, mean=0.0, std=0.02 / math.sqrt(2 * c.n_layer))

    @staticmethod
    def _init(m):
        if isinstance(m, (nn.Linear, nn.Embedding)):
            nn.init.normal_(m.weight, mean=0.0, std=0.02)
        if isinstance(m, nn.Linear) and m.bias is not None:
            nn.init.zeros_(m.bias)

    def forward(self, idx: torch.Tensor, targets: torch.Tensor | None = None):
        b, t = idx.shape
        pos = torch.arange(t, device=idx.device)
        x = self.wte(idx) + self.wpe(pos)
        if targets is not None and not traced() and self._sizes_fit(idx, targets) and self._fusable(x, targets):
            return self._fused_loss(x, targets)
        for blk in self.blocks:
            x = blk(x)
        x = self.ln_f(x)
        logits = F.linear(x, self.wte.weight)  # tied head
        if targets is None:
            return logits
        return F.cross_entropy(logits.float().view(-1, logits.size(-1)), targets.reshape(-1))

    @staticmethod
    def _sizes_fit(idx: torch.Tensor, targets: torch.Tensor) -> bool:
        """A target per token, where the tokens are (anything else is an error that the plain loss reports), and no more rows
        than the fused operators take."""
        return targets.numel() == idx.numel() and targets.device == idx.device and (not idx.is_cuda or idx.numel() <= ops().max_rows)

    def _fusable(self, x: torch.Tensor, targets: torch.Tensor) -> bool:
        """Whether the loss can go through the fused operators: a 16-bit model on a GPU, made of the plain modules
        above (no hooks, nothing replaced, no `forward` of an instance's own), of the shapes they have here, at
        widths that the layer norm's backward kernel takes."""
        c = self.config
        if not (x.is_cuda and x.dtype in (torch.bfloat16, torch.float16) and x.numel() and targets.is_cuda and targets.dtype == torch.int64):
            return False
        d = c.d_model
        if d > ops().max_norm_width or d % 8 or torch.is_autocast_enabled("cuda"):
            return False
        if global_module_hooks() or not plain_eager(x, targets):
            return False
        mods = [(self.ln_f, nn.LayerNorm, d, 0), (self.wte, nn.Embedding, 0, d)]
        for blk in self.blocks:
            if type(blk) is not Block or overridden(blk) or d % blk.n_head or (d // blk.n_head) % 8:
                return False
            mods += ((blk.ln1, nn.LayerNorm, d, 0), (blk.qkv, nn.Linear, 3 * d, d), (blk.proj, nn.Linear, d, d), (blk.ln2, nn.LayerNorm, d, 0),
                     (blk.fc, nn.Linear, 0, d), (blk.out, nn.Linear, d, 0))
        for m, kind, rows, cols in mods:     # 0: any number
            if type(m) is not kind or overridden(m):
                return False
            tensors = (m.weight,) if kind is nn.Embedding else (m.weight, m.bias)
            if any(type(t) not in (nn.Parameter, torch.Tensor) or t.dtype != x.dtype for t in tensors):
                return False
            shape = m.weight.shape
            if len(shape) != (1 if kind is nn.LayerNorm else 2) or (rows and shape[0] != rows) or (cols and shape[1] != cols):
                return False
        return all(blk.fc.weight.shape[0] % 8 == 0 for blk in self.blocks)

    def step_signature(self, idx: torch.Tensor, targets: torch.Tensor):
        """What a recorded training step depends on besides its inputs' values: equal signatures may share a recording.
        None when a step has effects that a recording would not repeat (hooks of any kind) or does not take the fused operators."""
        if not self._sizes_fit(idx, targets) or not self._fusable(self.wte.weight, targets) or not torch.is_grad_enabled():
            return None
        if type(self) is not GPT2 or type(self.wpe) is not nn.Embedding or overridden(self) or overridden(self.wpe):
            return None
        ps = list(self.parameters())
        if any(p._backward_hooks or p._post_accumulate_grad_hooks for p in ps) or ops().accumulation_hooks(ps):
            return None
        if torch._C._autograd._top_saved_tensors_default_hooks(False) is not None:
            return None
        cuda = torch.backends.cuda
        flags = (alone(), torch.are_deterministic_algorithms_enabled(), cuda.flash_sdp_enabled(), cuda.mem_efficient_sdp_enabled(), cuda.cudnn_sdp_enabled(),
                 cuda.math_sdp_enabled(), cuda.fp16_bf16_reduction_math_sdp_allowed(), tuple(torch._C._get_sdp_priority_order()),
                 torch._C._get_cublas_allow_bf16_reduced_precision_reduction(), torch._C._get_cublas_allow_fp16_reduced_precision_reduction(),
                 cuda.matmul.allow_fp16_accumulation, torch._C._get_blas_preferred_backend())
        eps = tuple(m.eps for blk in self.blocks for m in (blk.ln1, blk.ln2)) + (self.ln_f.eps,)
        heads = tuple(blk.n_head for blk in self.blocks)
        return tuple((p.data_ptr(), p.requires_grad, p.shape) for p in ps), eps, heads, flags

    def _fused_loss(self, x: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
        f = ops()
        b, t, d = x.shape
        by_itself = alone()
        branch = None      # what the block before adds to the residual stream: the next layer norm reads both
        for blk in self.blocks:
            x, q, k, v = f.block_pre(x, branch, blk.ln1.weight, blk.ln1.bias, blk.qkv.weight, blk.qkv.bias, blk.n_head, blk.ln1.eps)
            a = F.scaled_dot_product_attention(q, k, v, is_causal=True)
            x, branch = f.block_post(x, a.transpose(1, 2).reshape(b, t, d), blk.proj.weight, blk.proj.bias, blk.ln2.weight, blk.ln2.bias,
                                     blk.fc.weight, blk.fc.bias, blk.out.weight, blk.out.bias, blk.ln2.eps, by_itself)
        h = f.add_norm(x, branch, self.ln_f.weight, self.ln_f.bias, self.ln_f.eps)
        return f.head_loss(h, self.wte.weight, targets)

    def num_params(self) -> int:
        return sum(p.numel() for p in self.parameters())


def smoke_step() -> float:
    """One tiny forward + backward + fused all-reduce of the gradients on cuda:0."""
    from ..ops import EmuGroup

    dev = torch.device("cuda", 0)
    torch.manual_seed(0)
    model = GPT2(GPT2Config.tiny()).to(dev, torch.bfloat16)
    idx = torch.randint(0, 1024, (2, 64), device=dev)
    loss = model(idx, idx)
    loss.backward()
    # the gradients of two emulated ranks go through the NVLink all-reduce kernel
    flat = torch.cat([p.grad.reshape(-1) for p in model.parameters()])
    g = EmuGroup(2, stage_bytes=16 << 20)
    ins = [flat.clone(), flat.clone()]
    outs = [torch.empty_like(flat), torch.empty_like(flat)]
    g.run("all_reduce", ins, outs, flat.numel(), scale=0.5, algo="twoshot")
    torch.cuda.synchronize()
    assert torch.equal(outs[0], ((flat.float() + flat.float()) * 0.5).to(torch.bfloat16))
    g.close()
    return float(loss.detach())
