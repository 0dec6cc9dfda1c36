"""AdamW for bf16 parameters with fp32 master weights and moments, one fused kernel per step."""
from __future__ import annotations

from typing import Optional

import torch

from .. import runtime


class FusedAdamW:
    """``step()`` updates every parameter that has a gradient. ``step_param`` updates one parameter
    from an explicit gradient tensor, optionally on another stream: the MoE layer uses it to apply a
    weight's update as soon as its gradient exists, under the remaining backward GEMMs
    (optimizer-in-backward); such parameters are then skipped by the next ``step()``."""

    def __init__(self, params, lr=1e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.0):
        self.params = [p for p in params if p.requires_grad]
        self.lr, self.betas, self.eps, self.wd = lr, betas, eps, weight_decay
        self.state = {}
        self.steps = {}
        self._stepped_early = set()
        for p in self.params:
            assert p.dtype == torch.bfloat16 and p.numel() % 8 == 0 and p.is_contiguous(), "FusedAdamW wants contiguous bf16 tensors (numel % 8 == 0)"
            self.state[p] = (p.detach().float().clone(), torch.zeros_like(p, dtype=torch.float32), torch.zeros_like(p, dtype=torch.float32))
            self.steps[p] = 0

    def owns(self, p) -> bool:
        return p in self.state

    def zero_grad(self, set_to_none: bool = True):
        for p in self.params:
            if set_to_none:
                p.grad = None
            elif p.grad is not None:
                p.grad.zero_()

    def _update(self, params, grads, grad_scale: float) -> None:
        if len(set(params)) < len(params):
            # One launch updates its tensors side by side: a parameter that is listed twice is updated twice, one after the other.
            for p, g in zip(params, grads):
                self._update([p], [g], grad_scale)
            return
        state = [self.state[p] for p in params]
        for p in params:
            self.steps[p] += 1
        runtime.ext().adamw_step([p.data for p in params], [s[0] for s in state], [s[1] for s in state], [s[2] for s in state],
                            [g.to(torch.bfloat16).contiguous() for g in grads], [self.steps[p] for p in params], self.lr, self.betas[0], self.betas[1], self.eps, self.wd,
                            grad_scale)

    @torch.no_grad()
    def step_param(self, p, grad: torch.Tensor, grad_scale: float = 1.0, stream: Optional[torch.cuda.Stream] = None, early: bool = False):
        if stream is None:
            self._update([p], [grad], grad_scale)
        else:
            with torch.cuda.stream(stream):
                self._update([p], [grad], grad_scale)
        if early:
            self._stepped_early.add(p)

    @torch.no_grad()
    def step(self, grad_scale: float = 1.0):
        due = [p for p in self.params if p not in self._stepped_early and p.grad is not None]
        if due:
            self._update(due, [p.grad for p in due], grad_scale)
        self._stepped_early.clear()
