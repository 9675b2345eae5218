"""Mixture-of-experts feed-forward block under expert parallelism.

    logits = x @ w_router.T                                  (tcgen05 GEMM)
    route: softmax + top-k                                   (one kernel)
    dispatch: tokens -> their experts' GPUs, expert-major    (one kernel over peer memory)
    experts: SwiGLU MLP per local expert on its rows         (two grouped tcgen05 GEMMs over contiguous row ranges)
    combine: gate-weighted sum of the top-k outputs          (one kernel over peer memory)

DeepSeek-V3-like shapes are the defaults of the benchmark: hidden 7168, 256 experts (32 per GPU at 8 GPUs), top-8.
Weights are random N(0, 0.02) from a seed; there is no checkpoint loading here. ``w_gu`` and ``w_down`` are best one contiguous
tensor each, expert after expert: then the experts are two launches. A list of tensors, or a stack with gaps between the experts,
is computed expert by expert.
"""
from __future__ import annotations

from typing import Optional

import torch

from ..ops.gemm import gemm, gemm_swiglu, grouped_gemm, interleave_gate_up
from ..parallel.expert_parallel import ExpertParallelContext


class ExpertParallelMoE:
    def __init__(self, hidden: int = 7168, intermediate: int = 2048, experts: int = 256, topk: int = 8, max_tokens: int = 4096,
                 group=None, device=None, seed: int = 11, ep: Optional[ExpertParallelContext] = None, capacity_factor: float = 2.0):
        self.ep = ep or ExpertParallelContext(group, device, max_tokens=max_tokens, hidden=hidden, experts=experts, topk=topk,
                                              capacity_factor=capacity_factor)
        self.hidden, self.intermediate, self.experts, self.topk = hidden, intermediate, experts, topk
        dev = self.ep.device
        g = torch.Generator(device=dev).manual_seed(seed)                      # the router is replicated: same seed everywhere
        self.w_router = (torch.randn(experts, hidden, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        ge = torch.Generator(device=dev).manual_seed(seed * 1000 + 1 + self.ep.rank)
        n = self.ep.experts_per_rank
        def init(*shape):
            return (torch.randn(*shape, generator=ge, device=dev) * 0.02).to(torch.bfloat16)
        self.w_gate, self.w_up = init(n, intermediate, hidden), init(n, intermediate, hidden)
        self.w_down = init(n, hidden, intermediate)
        self.w_gu = torch.stack([interleave_gate_up(self.w_gate[e], self.w_up[e]) for e in range(n)])
        self._h = torch.empty(self.ep.capacity_rows, intermediate, dtype=torch.bfloat16, device=dev)

    def forward(self, x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        t = x.shape[0]
        self.ep._route_bf16(gemm(x, self.w_router))
        recv, counts = self.ep.dispatch(x)
        outb = self.ep.out_rows()
        w_gu, w_down = self._in_one_block(self.w_gu), self._in_one_block(self.w_down)
        if w_gu is not None and w_down is not None:
            # one launch per projection; the row counts stay on the device (rows per expert when every rank brings as many tokens)
            average = -(-t * self.topk * self.ep.world // self.experts)
            report = {"status_ptr": self.ep.status_ptr, "timeout_ns": self.ep.timeout_ns}     # ep.check() covers the experts too
            h = grouped_gemm(recv, w_gu, counts, average, self._h, swiglu=True, **report)
            grouped_gemm(h, w_down, counts, average, outb, **report)
        else:
            self._expert_by_expert(recv, counts, outb)
        return self.ep.combine(t, out)

    __call__ = forward

    def _in_one_block(self, w):
        """The weights of this rank's experts as one contiguous [experts, N, K], as the grouped GEMM reads them, or None: a list
        with a tensor per expert, or a stack of which only the slices are contiguous."""
        n = self.ep.experts_per_rank
        if not isinstance(w, torch.Tensor) or w.dim() != 3 or len(w) < n:
            return None
        w = w if len(w) == n else w[:n]
        return w if w.is_contiguous() else None

    def _expert_by_expert(self, recv, counts, outb):
        """The experts when their weights are not one block: two GEMMs each, for which the host has to read the row counts."""
        offs = [0] + torch.cumsum(counts[: self.ep.experts_per_rank], 0).tolist()
        for e in range(self.ep.experts_per_rank):
            a, b = offs[e], offs[e + 1]
            if b > a:
                gemm(gemm_swiglu(recv[a:b], self.w_gu[e], self._h[a:b]), self.w_down[e], outb[a:b])

    def reference(self, x: torch.Tensor, all_gate=None, all_up=None, all_down=None) -> torch.Tensor:
        """fp32 PyTorch result for a world of one (all experts local)."""
        xf = x.float()
        probs = torch.softmax((x.float() @ self.w_router.float().t()).to(torch.bfloat16).float(), dim=-1)
        w, idx = torch.topk(probs, self.topk, dim=-1)
        w = w / w.sum(-1, keepdim=True)
        y = torch.zeros_like(xf)
        for e in range(self.experts):
            tok, k = (idx == e).nonzero(as_tuple=True)
            if tok.numel() == 0:
                continue
            xe = xf[tok]
            h = torch.nn.functional.silu(xe @ self.w_gate[e].float().t()) * (xe @ self.w_up[e].float().t())
            o = (h.to(torch.bfloat16).float() @ self.w_down[e].float().t()).to(torch.bfloat16).float()
            y.index_add_(0, tok, o * w[tok, k].unsqueeze(-1))
        return y
