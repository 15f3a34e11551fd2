"""A small data-parallel trainer on the ``hylink`` backend.

``DDPTrainer`` is the user-facing entry for the benchmark workload: it wraps
the model in ``DistributedDataParallel`` over this library's process group
(25 MB gradient buckets by default), owns a fused AdamW, and exposes
``step(tokens)`` which takes a pinned host batch, copies it to the device,
runs forward / backward (gradient all-reduces overlap the backward pass on the
backend's own stream) / optimizer, and returns the loss as a Python float.

A job of one rank has no gradient to reduce: the model is not wrapped then (the
buckets would only cost a copy of every gradient), and models that can say when
a step may be replayed (``step_signature``, as :class:`~hylink_b200.models.gpt2.GPT2`
does) run forward and backward from a CUDA graph from the second step of a
batch shape on. Issuing the thousand launches of a step takes the host
longer than the GPU needs for a small batch. The graph holds the memory of one
step; ``HYLINK_TRAIN_GRAPH=0`` or :meth:`DDPTrainer.close` gives it back.
"""
from __future__ import annotations

import gc
import os

import torch
import torch.distributed as dist
from torch.nn.parallel import DistributedDataParallel as DDP
from torch.optim import optimizer as _optimizer

from ..ops.extension import check_products, ops

_global_hooks = (_optimizer._global_optimizer_pre_hooks, _optimizer._global_optimizer_post_hooks)


def init_distributed(backend: str = "hylink"):
    """Initialise ``torch.distributed`` from torchrun's environment (or as a single rank)."""
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    local = int(os.environ.get("LOCAL_RANK", rank))
    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29533")
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if backend == "hylink":
        from .backend import register_backend

        register_backend()
    if not dist.is_initialized():
        dist.init_process_group(backend, rank=rank, world_size=world, device_id=dev)
    return rank, world, dev


class _StepGraph:
    """Forward and backward of one batch shape as a CUDA graph. Inputs are copied into place, the loss and the
    gradients are where the capture put them."""

    def __init__(self, model: torch.nn.Module, params: list, idx: torch.Tensor, targets: torch.Tensor):
        self.idx, self.targets = idx.clone(), targets.clone()
        self.params = params
        old = [p.grad for p in params]
        try:
            for p in params:
                p.grad = None
            self._capture(model)
        except BaseException:
            for p, g in zip(params, old):
                p.grad = g
            raise

    def _capture(self, model: torch.nn.Module) -> None:
        self.graph, self.replays = torch.cuda.CUDAGraph(), 0
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        collecting = gc.isenabled()
        gc.disable()                      # whatever a collection would free must not be freed inside the capture
        try:
            with torch.cuda.stream(side):
                # other threads may go on calling CUDA; the memory of earlier steps stays in the allocator's cache
                self.graph.capture_begin(capture_error_mode="thread_local")
                try:
                    loss = model(self.idx, self.targets)
                    loss.backward()
                    self.loss = loss.detach()
                finally:
                    self.graph.capture_end()
        finally:
            if collecting:
                gc.enable()
        self.grads = [p.grad for p in self.params]

    def run(self, idx: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
        self.idx.copy_(idx)
        self.targets.copy_(targets)
        self.graph.replay()
        self.replays += 1
        for p, g in zip(self.params, self.grads):
            if p.grad is not g:
                p.grad = g
        return self.loss.clone()


class DDPTrainer:
    def __init__(self, model: torch.nn.Module, device: torch.device, lr: float = 3e-4, bucket_cap_mb: int = 25,
                 dtype: torch.dtype = torch.bfloat16, cta_budget: int | None = None):
        self.device = device
        # gradient all-reduces overlap the backward pass: they get a CTA budget (the GEMMs keep the other SMs)
        self._old_budget = None
        if dist.get_backend() == "hylink":
            from .backend import set_cta_budget

            if cta_budget is None:
                cta_budget = int(os.environ.get("HYLINK_DDP_CTA_BUDGET", "32"))
            self._old_budget = set_cta_budget(cta_budget)
        self.model = model.to(device=device, dtype=dtype)
        self.registered_buckets = False
        self._pool = None
        self._steps = 0
        pool = None
        if dist.get_backend() == "hylink" and dist.get_world_size() > 1 and os.environ.get("HYLINK_DDP_REGISTERED", "1") != "0":
            # Gradient buckets in registered memory: the bucket all-reduces then run zero-copy, in place in every
            # rank's bucket (multimem load-reduce / store through NVSwitch), on a few SMs beside the backward GEMMs.
            try:
                from .backend import registered_mem_pool

                dist.barrier()                       # the group's communicator (and its allocator) exists after this
                pool = registered_mem_pool()
            except Exception as ex:  # noqa: BLE001 - an older PyTorch without pluggable pools: buckets are staged
                print(f"hylink: gradient buckets stay unregistered ({type(ex).__name__}: {ex})", flush=True)
        self._ddp = None
        self._bucket_cap_mb = bucket_cap_mb
        self._graph, self._graph_key, self._key_seen, self._patience = None, None, 0, 2
        self._use_graph = os.environ.get("HYLINK_TRAIN_GRAPH", "1") != "0"
        if pool is not None:
            with torch.cuda.use_mem_pool(pool):
                self.ddp  # noqa: B018 - wrapped here, under the registered pool
            self.registered_buckets = True
            self._pool = pool
        elif dist.get_world_size() > 1:
            self.ddp  # noqa: B018
        self._params = list(self.model.parameters())
        self.opt = torch.optim.AdamW(self._params, lr=lr, betas=(0.9, 0.95), weight_decay=0.1, fused=True)
        self._loss_host = torch.zeros(1, dtype=torch.float32).pin_memory()
        self._dev_batch = None

    @property
    def ddp(self) -> DDP:
        """The ``DistributedDataParallel`` wrapper. A one-rank job makes it when it is asked for, and uses it from then on."""
        if self._ddp is None:
            self._graph = None
            self._ddp = DDP(self.model, device_ids=[self.device.index], bucket_cap_mb=self._bucket_cap_mb, gradient_as_bucket_view=True,
                            static_graph=False)
        return self._ddp

    @ddp.setter
    def ddp(self, wrapper) -> None:
        """A wrapper of the caller's own, which every step goes through from now on."""
        self._graph, self._ddp = None, wrapper

    def _opt_step(self) -> None:
        """``self.opt.step()``, through this library's kernel where the optimizer is what the constructor made and nobody
        watches its steps (a scheduler replaces ``step``, hooks want to be called); its state stays where it is."""
        opt = self.opt
        g = opt.param_groups[0]
        plain = (type(opt) is torch.optim.AdamW and len(opt.param_groups) == 1 and "step" not in opt.__dict__
                 and not (opt._optimizer_step_pre_hooks or opt._optimizer_step_post_hooks or _global_hooks[0] or _global_hooks[1])
                 and not (g["amsgrad"] or g["maximize"] or g["differentiable"] or g["capturable"])
                 and isinstance(g["lr"], float) and isinstance(g["betas"][0], float) and isinstance(g["betas"][1], float)
                 and getattr(opt, "grad_scale", None) is None and getattr(opt, "found_inf", None) is None)
        if plain:
            ps, gs, ms, vs, steps = [], [], [], [], []
            state = opt.state
            for p in g["params"]:
                grad = p.grad
                if grad is None:
                    continue
                st = state.get(p)
                if not st:                 # the first step: the optimizer sets its state up itself
                    plain = False
                    break
                ps.append(p)
                gs.append(grad)
                ms.append(st["exp_avg"])
                vs.append(st["exp_avg_sq"])
                steps.append(st["step"])
        if not plain or not ops().multi_adamw(ps, gs, ms, vs, steps, g["lr"], g["betas"][0], g["betas"][1], g["weight_decay"], g["eps"]):
            opt.step()

    def _replayable(self, idx: torch.Tensor, targets: torch.Tensor) -> bool:
        """Whether this step runs from the graph; captures it when the same step has been run before."""
        signature = getattr(self.model, "step_signature", None)
        if not self._use_graph or signature is None or not (idx.is_cuda and targets.is_cuda) or torch.is_anomaly_enabled():
            return False
        sig = signature(idx, targets)
        key = None if sig is None else (sig, idx.shape, idx.dtype, targets.shape, targets.dtype)
        if key != self._graph_key:
            if self._graph is not None and self._graph.replays < 16:   # a capture costs a few steps: shapes that keep changing
                self._patience = min(2 * self._patience, 1 << 20)      # have to prove themselves for longer and longer
            self._graph, self._graph_key, self._key_seen = None, key, 0
        if key is None:
            return False
        self._key_seen += 1
        if self._graph is None and self._key_seen >= self._patience:   # an eager step has loaded and sized everything
            try:
                self._graph = _StepGraph(self.model, self._params, idx, targets)
            except RuntimeError as ex:   # out of memory among them
                print(f"hylink: training steps are not replayed from a graph ({type(ex).__name__}: {ex})", flush=True)
                self._use_graph = False
                torch.cuda.empty_cache()
        return self._graph is not None

    def close(self) -> None:
        """Gives the process group its previous CTA budget back, and the memory of the step graph."""
        self._graph, self._graph_key = None, None
        if self._old_budget is not None:
            from .backend import set_cta_budget

            set_cta_budget(self._old_budget)
            self._old_budget = None

    def step_device(self, idx: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
        """One optimisation step on device-resident tokens; returns the loss tensor (no host sync)."""
        if self._pool is not None and self._steps == 1:
            # DDP re-buckets its gradients once, before the second forward pass, in the order they became ready:
            # do that here, under the registered pool, so that the new buckets are registered too.
            with torch.cuda.use_mem_pool(self._pool):
                if self._ddp.reducer._rebuild_buckets():
                    self._ddp._has_rebuilt_buckets = True
        self._steps += 1
        check_products(self.device.index)     # of steps that nobody has waited for
        if self._ddp is not None:
            loss = self._ddp(idx, targets)
        elif self._replayable(idx, targets):
            loss = self._graph.run(idx, targets)
            self._opt_step()
            return loss
        else:
            loss = self.model(idx.to(self.device), targets.to(self.device))
        self.opt.zero_grad(set_to_none=True)
        loss.backward()
        self._opt_step()
        return loss

    def step(self, tokens: torch.Tensor) -> float:
        """``tokens``: pinned host tensor [batch, seq + 1] of token ids. Returns the loss. An error of a kernel in this step is raised
        here; the weights have been updated by then."""
        if self._dev_batch is None or self._dev_batch.shape != tokens.shape:
            self._dev_batch = torch.empty(tokens.shape, dtype=tokens.dtype, device=self.device)
        self._dev_batch.copy_(tokens, non_blocking=True)
        loss = self.step_device(self._dev_batch[:, :-1], self._dev_batch[:, 1:])
        self._loss_host.copy_(loss.detach().float().reshape(1), non_blocking=True)
        torch.cuda.current_stream().synchronize()
        check_products(self.device.index)     # a replayed graph reports nothing by itself
        return float(self._loss_host[0])
