"""Ragged-batch inference model for the Llama family (Llama-2/3, Mistral: dense; Mixtral / Qwen2-MoE: sparse MLP).

Reference: ``inference/v2/model_implementations/{llama_v2,mistral,mixtral,qwen_v2,qwen_v2_moe}/model.py`` — per layer:
RMSNorm -> fused QKV GEMM -> rotary + KV-cache append -> blocked flash attention -> output GEMM -> RMSNorm ->
gated MLP (or top-k MoE) -> residual; final norm, last-token gather, unembedding.

Here: GEMMs are the tcgen05 kernel (``ops.functional.linear``), norms/activations the fused elementwise kernels,
rotary + cache append ``sxb_kv_rotary_blocked``, attention ``sxb_paged_attention``, MoE routing
``sxb_top_k_gating / moe_scatter / moe_gather`` with one GEMM per expert over its contiguous row range.
Weights come from a training :class:`~shuffle_exchange_b200.models.llama.LlamaForCausalLM` (same fused
``wqkv`` / ``w_gate_up`` layout) or from a HuggingFace state dict via that class's ``load_hf_state_dict``.
"""
from __future__ import annotations

import array
import math
from typing import List, Optional

import torch

from ....native import lib as _n
from ....ops import functional as F
from ....ops import moe_ops
from ..kernels import ragged_ops as R


class RaggedLlamaModel:
    def __init__(self, causal_lm, state_manager, moe_layers: Optional[List[dict]] = None, top_k: int = 2):
        self.lm = causal_lm
        self.cfg = causal_lm.cfg
        self.state_manager = state_manager
        self.moe_layers = moe_layers       # per layer: {"gate": [E, H], "w_gate_up": [E, 2F, H], "w_down": [E, H, F]} or None
        self.top_k = top_k

    # memory the engine must plan for ------------------------------------------------------------
    def kv_cache_config(self, block_size: int):
        from ..ragged.kv_cache import KVCacheConfig
        c = self.cfg
        return KVCacheConfig(block_size=block_size, cache_shape=(c.num_hidden_layers, c.num_key_value_heads, c.head_dim),
                             cache_dtype=self.lm.model.embed_tokens.dtype)

    def get_kv_requirements(self, sequence, max_new_tokens: int, max_new_blocks: int):
        bs = self.state_manager.kv_block_size
        total = sequence.seen_tokens + max_new_tokens
        need = (total + bs - 1) // bs - sequence.cur_allocated_blocks
        if need > max_new_blocks:
            fit = (sequence.cur_allocated_blocks + max_new_blocks) * bs - sequence.seen_tokens
            return max(0, fit), max_new_blocks
        return max_new_tokens, max(0, need)

    def maybe_allocate_kv(self, sequence, n_new_tokens: int) -> None:
        _, need = self.get_kv_requirements(sequence, n_new_tokens, self.state_manager.free_blocks)
        if need > 0:
            sequence.extend_kv_cache(self.state_manager.allocate_blocks(need))

    # forward -----------------------------------------------------------------------------------------
    def _mlp(self, layer_idx: int, layer, x: torch.Tensor) -> torch.Tensor:
        moe = self.moe_layers[layer_idx] if self.moe_layers is not None else None
        if moe is None:
            return F.linear(F.swiglu(F.linear(x, layer.w_gate_up)), layer.w_down)
        logits = F.linear(x, moe["gate"])
        scores, assign, offsets, counts = moe_ops.top_k_gating(logits, self.top_k, renormalize=True)
        from ....moe import fused_ep
        if fused_ep.grouped_inference_ok(x, moe["w_gate_up"], moe["w_down"]):
            return fused_ep.grouped_experts_inference(x, scores, assign, offsets, counts, moe["w_gate_up"],
                                                      moe["w_down"], F.swiglu, self.top_k, gate_act="silu")
        moe_in, cumsum, slots = moe_ops.moe_scatter(x, assign, offsets, counts)
        ends = cumsum.tolist()
        out = torch.empty_like(moe_in)
        lo = 0
        for e, hi in enumerate(ends):
            if hi > lo:
                h = F.swiglu(F.linear(moe_in[lo:hi], moe["w_gate_up"][e]))
                out[lo:hi] = F.linear(h, moe["w_down"][e])
            lo = hi
        return moe_ops.moe_gather(out, scores, slots)

    def _native_plan(self, batch):
        """Operands of ``sxb_ragged_llama_forward`` for ``batch``, looked at afresh in every call, or None where the operators
        below would not all run on the kernels that it issues (or have more to do than launch them)."""
        c, m = self.cfg, self.lm.model
        H, nq, nkv, d = c.hidden_size, c.num_attention_heads, c.num_key_value_heads, c.head_dim
        Fw, bf16, dev = c.intermediate_size, torch.bfloat16, m.embed_tokens.device
        # (a subclass or an object with a feed-forward of its own has it called)
        if (self.moe_layers is not None or getattr(self._mlp, "__func__", None) is not RaggedLlamaModel._mlp
                or F.flop_sink is not None or dev.type != "cuda" or not hasattr(batch, "atoms")
                or batch.current_tokens == 0 or batch.atoms().shape[0] == 0 or H % 8 or Fw % 8 or not _n.no_tape()):
            return None
        head = self.lm.head_weight()
        ptrs = 0

        def matrix(w, n, k, lds):
            nonlocal ptrs
            if w.dtype != bf16 or w.device != dev or w.shape != (n, k):
                return None
            ld, inner = w.stride()
            if inner != 1 or ld % 8 or hasattr(w, "_sxb_gate") or hasattr(w, "_sxb_grad_ready"):
                return None
            p = w.data_ptr()
            ptrs |= p
            lds.append(ld)
            return p

        def vector(w):
            return (w.data_ptr() if w.dtype == bf16 and w.device == dev and w.shape == (H,) and w.stride(0) == 1
                    and not hasattr(w, "_sxb_grad_ready") else None)

        rows = []
        for li, layer in enumerate(m.layers):
            cache = self.state_manager.get_cache(li)
            if (not isinstance(cache, torch.Tensor) or cache.device != dev or not R.atoms_layout_ok(cache, d)
                    or cache.shape[3:] != (nkv, d)):
                return None
            lds = []
            row = [vector(layer.input_layernorm), matrix(layer.wqkv, (nq + 2 * nkv) * d, H, lds), matrix(layer.wo, H, nq * d, lds),
                   vector(layer.post_attention_layernorm), matrix(layer.w_gate_up, 2 * Fw, H, lds),
                   matrix(layer.w_down, H, Fw, lds), cache.data_ptr()]
            ptrs |= row[-1]
            if None in row:
                return None
            rows += row
            rows += lds
        emb = m.embed_tokens
        top = [matrix(emb, emb.shape[0], H, []), vector(m.norm), matrix(head, head.shape[0], H, [])]
        if not rows or None in top or not emb.is_contiguous() or head.shape[0] % 8 or ptrs % 16:
            return None
        return rows, top, head, cache

    def _native_forward(self, batch, plan) -> torch.Tensor:
        layers, (embed, norm, head_ptr), head, cache = plan
        c = self.cfg
        H, nq, nkv, d, Fw = c.hidden_size, c.num_attention_heads, c.num_key_value_heads, c.head_dim, c.intermediate_size
        T, last, tables, atoms = batch.current_tokens, batch.last_token_index(), batch.block_tables(), batch.atoms()
        n_rows, vocab, dev = last.shape[0], head.shape[0], head.device
        # activations of one layer after the other in one allocation; those of attention and feed-forward take turns
        sizes = [T * H] * 4 + [n_rows * H, T * (nq + 2 * nkv) * d, T * nq * d]
        wide = (T * 2 * Fw + 127) // 128 * 128
        at = [0]
        for n in sizes:
            at.append(at[-1] + (n + 127) // 128 * 128)
        work = torch.empty(max(at[-1], at[5] + wide + T * Fw), dtype=torch.bfloat16, device=dev)
        b0, b1, b2, x, rows, qkv, ctx = (work.data_ptr() + 2 * a for a in at[:-1])
        logits = torch.empty((n_rows, vocab), dtype=torch.bfloat16, device=dev)
        n_packed, n_few, few_keys = R.atoms_split(batch, atoms.shape[0], nq, nkv, True, dev.index)
        model = array.array("q", [
            batch.input_ids().data_ptr(), batch.token_to_seq().data_ptr(), batch.token_positions().data_ptr(), tables.data_ptr(),
            last.data_ptr(), atoms.data_ptr(), embed, norm, head_ptr, b0, b1, b2, x, qkv, ctx, qkv, qkv + 2 * wide, rows,
            logits.data_ptr(), head.stride(0), T, H, nq, nkv, d, Fw, vocab, n_rows, tables.shape[1], cache.shape[0],
            cache.shape[1], atoms.shape[0], n_packed, n_few, *few_keys, 0])
        table = array.array("q", layers)
        n_layers = len(layers) // 11
        _n.attn_call("sxb_ragged_llama_forward", model.buffer_info()[0], table.buffer_info()[0], n_layers,
                     float(c.rms_norm_eps), float(c.rope_theta), 1.0 / math.sqrt(d), _n.stream_ptr())
        _n.count_launches(model[-1] - 1)          # the entry points that the call stood for, itself counted as one
        return logits

    @torch.no_grad()
    def forward(self, batch) -> torch.Tensor:
        """``batch``: finalized :class:`RaggedBatchWrapper`.  Returns logits [n_seqs, vocab] of every sequence's last
        in-flight token."""
        c, m = self.cfg, self.lm.model
        plan = self._native_plan(batch)
        if plan is not None:
            return self._native_forward(batch, plan)
        ids, t2s, pos = batch.input_ids(), batch.token_to_seq(), batch.token_positions()
        tables = batch.block_tables()
        h = R.ragged_embed(ids, m.embed_tokens)
        residual = None
        nq, nkv, d = c.num_attention_heads, c.num_key_value_heads, c.head_dim
        for li, layer in enumerate(m.layers):
            x, residual = F.rms_norm(h, layer.input_layernorm, c.rms_norm_eps, residual)
            qkv = F.linear(x, layer.wqkv)
            cache = self.state_manager.get_cache(li)
            R.kv_rotary_blocked(qkv, cache, t2s, pos, tables, nq, nkv, d, d, c.rope_theta)
            q = qkv.view(qkv.shape[0], nq + 2 * nkv, d)[:, :nq]
            o = R.ragged_attention(q, cache, batch)
            h = F.linear(o.reshape(o.shape[0], nq * d), layer.wo)
            x, residual = F.rms_norm(h, layer.post_attention_layernorm, c.rms_norm_eps, residual)
            h = self._mlp(li, layer, x)
        x, _ = F.rms_norm(h, m.norm, c.rms_norm_eps, residual)
        last = R.logits_gather(x, batch.last_token_index())
        return F.linear(last, self.lm.head_weight())
