"""``FusedMoeGGUF``: routing plus the three grouped expert matmuls of a quantized mixture-of-experts block.

Mirrors candle-transformers/src/fused_moe.rs:222-301 (``FusedMoeGGUF::forward``): router logits -> softmax -> the
``num_experts_per_tok`` largest weights per token (optionally renormalised) -> (token, expert) pairs sorted by expert ->
``moe_gemm_gguf`` for gate and up, ``up * act(gate)``, ``moe_gemm_gguf`` for down with the routing weights applied ->
sum over the token's experts.  The router is a dense f32 linear layer (candle de-quantizes it at load).  The block runs as a few
launches of libcandle_q_b200 (`_block`); shapes and formats outside of those take the single calls with tensor operations between them.

Expert parallelism: a rank may own a contiguous range of experts.  Pairs routed elsewhere write nothing (the kernels
skip expert ids outside their range), every pair is produced by exactly one rank, so summing the pair outputs across
ranks adds one value and zeros - exact in any order.  Which of the two forms runs, and which kernels inside, depends on the layer and
on the number of pairs only, so the result has the same bits for any number of ranks.
"""
from __future__ import annotations

import torch
import torch.distributed as dist

from . import capi
from .capi import CandleQError
from .moe import _CODE, moe_gemm_gguf
from .quantized import GgmlDType, QTensor


def route(router_logits: torch.Tensor, num_experts_per_tok: int, norm_topk_prob: bool):
    """fused_moe.rs:233-247: softmax over experts, the top-k of each token (descending), optional renormalisation.
    Returns (topk_weights f32 [tokens, k], topk_ids int64 [tokens, k])."""
    weights = torch.softmax(router_logits.to(torch.float32), dim=-1)
    order = torch.argsort(weights, dim=-1, descending=True, stable=True)
    topk_ids = order[:, :num_experts_per_tok].contiguous()
    topk_weights = weights.gather(-1, topk_ids)
    if norm_topk_prob:
        topk_weights = topk_weights / topk_weights.sum(dim=-1, keepdim=True)
    return topk_weights, topk_ids


def sort_pairs(topk_ids: torch.Tensor):
    """fused_moe.rs:249-260: the flattened (token, slot) pairs sorted by expert id.
    Returns (expert_ids int32 [pairs] ascending, sorted_token_ids int32 [pairs] = pair indices in that order)."""
    expert_ids, sorted_token_ids = torch.sort(topk_ids.reshape(-1), stable=True)
    return expert_ids.to(torch.int32), sorted_token_ids.to(torch.int32)


class FusedMoeGGUF:
    def __init__(self, gate: torch.Tensor, gate_experts: QTensor, up_experts: QTensor, down_experts: QTensor,
                 num_experts_per_tok: int, norm_topk_prob: bool = True, prefill_dtype: torch.dtype = torch.bfloat16,
                 expert_offset: int = 0, group=None, world: int = 1):
        """gate: router weight f32 [num_experts, hidden].  *_experts: rank-3 QTensors [local experts, n, k] holding the
        experts [expert_offset, expert_offset + local experts) of the layer."""
        for w in (gate_experts, up_experts, down_experts):
            if w.rank() != 3:
                raise CandleQError("FusedMoeGGUF expects expert weights of rank 3 [experts, n, k]")
        if gate_experts.shape != up_experts.shape or down_experts.shape[1] != gate_experts.shape[2] or \
                down_experts.shape[2] != gate_experts.shape[1]:
            raise CandleQError("FusedMoeGGUF: expert weight shapes do not fit together")
        self.gate, self.gate_experts, self.up_experts, self.down_experts = gate, gate_experts, up_experts, down_experts
        self.num_experts_per_tok, self.norm_topk_prob, self.prefill_dtype = num_experts_per_tok, norm_topk_prob, prefill_dtype
        self.expert_offset, self.group, self.world = expert_offset, group, world

    def _block(self, x: torch.Tensor, is_prefill: bool) -> torch.Tensor | None:
        """The block as a few launches of libcandle_q_b200; None: the general path has to run.  The expert products are those of
        `moe_gemm_gguf` - same kernels, same rule for which of them a prompt takes, on the layer's experts, not this rank's."""
        local, ffn, hidden = self.gate_experts.shape
        experts, tokens, k = self.gate.shape[0], x.shape[0], self.num_experts_per_tok
        gu, down = self.gate_experts.dtype, self.down_experts.dtype
        if experts > 1024 or not 0 < k <= min(32, experts) or tokens == 0 or not x.is_cuda or self.up_experts.dtype != gu or \
                gu not in _CODE or down not in _CODE or x.shape[1] != hidden or \
                any(w.device != x.device for w in (self.gate_experts, self.up_experts, self.down_experts)):
            return None
        pairs, dev, lib = tokens * k, x.device, capi.lib()
        kind = {torch.float16: capi.F16, torch.bfloat16: capi.BF16}.get(self.prefill_dtype)
        if is_prefill:
            need = lib.cq_moe_block_prompt_scratch_bytes(pairs, local, hidden, ffn)
            if kind is None or need == 0 or self._few_pairs(pairs) or {gu, down} - {GgmlDType.Q4K, GgmlDType.Q6K}:
                return None
        else:
            need = lib.cq_moe_block_decode_scratch_bytes(tokens, k, hidden, ffn)
            if pairs > 65535:
                return None
        part = self.world > 1 or self.expert_offset != 0 or local != experts       # pairs of other ranks must read as zero
        with capi.on_device(dev):
            st = capi.stream_of(dev)
            ids = torch.empty((3, pairs), dtype=torch.int32, device=dev)        # by token; then experts and pairs, sorted
            weights = torch.empty((tokens, k), dtype=torch.float32, device=dev)
            scratch = torch.empty(need, dtype=torch.uint8, device=dev)
            norm, gate = 1 if self.norm_topk_prob else 0, self.gate
            floats = lib.cq_moe_route_rows_floats(tokens, experts, hidden) if is_prefill else 0
            if floats and gate.dtype == torch.float32 and gate.device == dev and gate.is_contiguous() and not (gate.data_ptr() | x.data_ptr()) & 15 and \
                    not torch.is_autocast_enabled("cuda"):
                logits = torch.empty(floats, dtype=torch.float32, device=dev)
                lib.cq_moe_route_rows_f32(x.data_ptr(), gate.data_ptr(), logits.data_ptr(), ids.data_ptr(), weights.data_ptr(), tokens, experts, hidden, k, norm, st)
            else:
                logits = torch.nn.functional.linear(x, gate).to(torch.float32).contiguous()      # autocast gives 16 bits
                lib.cq_moe_route_f32(logits.data_ptr(), ids.data_ptr(), weights.data_ptr(), tokens, experts, k, norm, st)
            if self.expert_offset:
                ids[0] -= self.expert_offset        # ids outside [0, local) are skipped by the kernels
            g, u, d = (w.device_ptr() for w in (self.gate_experts, self.up_experts, self.down_experts))
            if is_prefill or part:
                y = (torch.zeros if part else torch.empty)((pairs, hidden), dtype=torch.float32, device=dev)
            if is_prefill:
                lib.cq_moe_sort_pairs(ids.data_ptr(), pairs, local, ids[1].data_ptr(), ids[2].data_ptr(), st)
                lib.cq_moe_block_prompt(int(gu), int(down), x.data_ptr(), kind, g, u, d, ids[2].data_ptr(), ids[1].data_ptr(),
                                        weights.data_ptr(), y.data_ptr(), scratch.data_ptr(), local, k, pairs, hidden, ffn, st)
            elif part:
                lib.cq_moe_block_decode_pairs(int(gu), int(down), x.data_ptr(), g, u, d, ids.data_ptr(), y.data_ptr(), scratch.data_ptr(),
                                              local, k, tokens, hidden, ffn, st)
            else:
                out = torch.empty((tokens, hidden), dtype=torch.float32, device=dev)
                lib.cq_moe_block_decode(int(gu), int(down), x.data_ptr(), g, u, d, ids.data_ptr(), weights.data_ptr(), out.data_ptr(),
                                        scratch.data_ptr(), local, k, tokens, hidden, ffn, st)
            if self.world > 1:
                capi.check("moe block")
                dist.all_reduce(y, op=dist.ReduceOp.SUM, group=self.group)      # one value plus zeros per element: exact
            if is_prefill:
                out = y.view(tokens, k, hidden).sum(dim=1)
            elif part:
                out = torch.empty((tokens, hidden), dtype=torch.float32, device=dev)
                lib.cq_moe_weighted_sum_f32(y.data_ptr(), weights.data_ptr(), out.data_ptr(), tokens, k, hidden, st)
        capi.check("moe block")
        return out

    def _few_pairs(self, pairs: int) -> bool:
        """The rule of `moe_gemm_gguf_prefill` for prompts that stay on the GEMV, counted on the layer's experts so that it does not
        depend on how many ranks share them."""
        return pairs < max(64, 4 * self.gate.shape[0]) or self.gate.shape[0] > 1024

    def forward(self, xs: torch.Tensor, is_prefill: bool) -> torch.Tensor:
        batch, seq_len, hidden = xs.shape
        original_dtype = xs.dtype
        x = xs.reshape(-1, hidden).to(torch.float32).contiguous()
        num_tokens, k = x.shape[0], self.num_experts_per_tok
        out = self._block(x, is_prefill)
        if out is not None:
            return out.to(original_dtype).reshape(batch, seq_len, hidden)
        topk_weights, topk_ids = route(torch.nn.functional.linear(x, self.gate), k, self.norm_topk_prob)
        expert_ids, sorted_token_ids = sort_pairs(topk_ids)
        local_ids = expert_ids - self.expert_offset          # ids outside [0, local experts) are skipped by the kernels
        cast = (lambda t: t.to(self.prefill_dtype)) if is_prefill else (lambda t: t)      # the reference casts for its prefill kernel (moe.rs:310-333)
        if is_prefill and self.world > 1 and self._few_pairs(num_tokens * k) and self.prefill_dtype in (torch.float16, torch.bfloat16):
            # With this rank's experts alone the prompt entry point could take the tensor cores where one rank takes the GEMV; the
            # decode entry point on the cast values is that GEMV.
            cast, is_prefill = (lambda t: t.to(self.prefill_dtype).to(torch.float32)), False
        xin = cast(x)
        zero = self.world > 1                                 # pairs of other ranks must read as zero
        gate = moe_gemm_gguf(xin, self.gate_experts, None, sorted_token_ids, local_ids, k, is_prefill, zero_init=zero)
        up = moe_gemm_gguf(xin, self.up_experts, None, sorted_token_ids, local_ids, k, is_prefill, zero_init=zero)
        down_in = cast(up * torch.nn.functional.silu(gate))   # [pairs, intermediate]
        ys = moe_gemm_gguf(down_in, self.down_experts, topk_weights, sorted_token_ids, local_ids, k, is_prefill, zero_init=zero)
        if self.world > 1:
            dist.all_reduce(ys, op=dist.ReduceOp.SUM, group=self.group)      # one value plus zeros per element: exact
        ys = ys.reshape(num_tokens, k, hidden).sum(dim=1)
        return ys.to(original_dtype).reshape(batch, seq_len, hidden)
