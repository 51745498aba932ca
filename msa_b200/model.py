"""Decoder stack around ``MemorySparseAttention`` for inference (mirror of ``src/msa/model.py``:
``MSADeocoderLayer`` :53-135, ``MSAModel`` :137-262, ``MSAForCausalLM`` :264-330).

Only what the stage-1 worker and the generation loop call: embeddings, N pre-norm decoder layers whose attention
is this package's ``MemorySparseAttention`` (``doc_ids`` handed down to every layer), final norm, ``lm_head``.
Module and parameter names follow the reference (``model.embed_tokens``, ``model.layers.<i>.self_attn.*``,
``model.layers.<i>.mlp.*``, ``model.norm``, ``lm_head``), so a reference checkpoint's state dict loads with
``load_state_dict``.  MLP, RMSNorm and rotary embedding are transformers' Qwen3 modules, as in the reference.  In bf16
inference (``fused_ops``) what they do between the matrix products runs on this package's kernels: the projections are called
as modules, the norms with the residual adds, ``act(gate) * up`` and the angles of the rotation are one launch each.
The training losses of the reference's ``MSAForCausalLM.forward`` are out of scope.
"""
from __future__ import annotations

from types import SimpleNamespace

import torch
import torch.nn as nn
import torch.nn.functional as F
from transformers.activations import ACT2FN
from transformers.models.qwen3.modeling_qwen3 import Qwen3MLP, Qwen3RMSNorm, Qwen3RotaryEmbedding

from . import _cabi as A
from . import ops
from .attention import MemorySparseAttention, fused_ops, nn_module, plain_module
from .cache import create_cache

SILU = type(ACT2FN["silu"])


def add_norm(x, branch, norm):
    """``(x + branch, norm(x + branch))`` of ``[B, S, hidden]``, in one launch where the operands allow it."""
    if not (fused_ops(x, norm.weight) if branch is None else fused_ops(x, norm.weight, branch) and branch.shape == x.shape):
        x = x if branch is None else x + branch
        return x, norm(x)
    flat = lambda t: t if t is None else t.reshape(-1, t.shape[-1]).contiguous()
    x_new, h = ops.add_rmsnorm(flat(x), flat(branch), norm.weight, norm.variance_epsilon)
    return x_new.view(x.shape), h.view(x.shape)


class MSADecoderLayer(nn.Module):
    def __init__(self, config, layer_idx: int):
        super().__init__()
        self.layer_idx = layer_idx
        self.self_attn = MemorySparseAttention(config=config, layer_idx=layer_idx)
        self.mlp = Qwen3MLP(config)
        self.input_layernorm = Qwen3RMSNorm(config.hidden_size, eps=config.rms_norm_eps)
        self.post_attention_layernorm = Qwen3RMSNorm(config.hidden_size, eps=config.rms_norm_eps)

    def takes_fused(self, x) -> bool:
        """Whether ``fused`` computes what ``forward`` does on ``x``: nobody watches or replaced the modules it steps over (the
        layer itself is asked about by the caller: a module in its place knows neither method)."""
        norms, mlp = (self.input_layernorm, self.post_attention_layernorm), self.mlp
        return (plain_module(mlp, Qwen3MLP) and plain_module(mlp.act_fn, SILU)
                and all(plain_module(n, Qwen3RMSNorm) and fused_ops(x, n.weight) for n in norms)
                and x.shape[-1] % 2 == 0 and x.shape[-1] <= 12288)

    def fused(self, x, pending, attention_mask, past_key_value, position_embeddings, doc_ids):
        """``forward`` on the stream ``x`` with a branch ``pending`` (or None) that has not joined it yet; returns the same pair,
        so that every residual add is part of the norm that follows it."""
        x, h = add_norm(x, pending, self.input_layernorm)
        attn, _ = self.self_attn(h, doc_ids, attention_mask=attention_mask, position_embeddings=position_embeddings,
                                 past_key_value=past_key_value)
        return self._behind(x, attn)

    def native(self, parts, x, pending, attention_mask, past_key_value, position_embeddings, doc_ids):
        """``fused`` with the modules' weights in hand (``parts``): the same launches from native code, where the operands allow it."""
        n = A.native()
        at = n.front(parts, x, pending, *position_embeddings)
        if at is None:
            if self.takes_fused(x):
                return self.fused(x, pending, attention_mask, past_key_value, position_embeddings, doc_ids)
            return self(x if pending is None else x + pending, attention_mask=attention_mask, past_key_value=past_key_value,
                        position_embeddings=position_embeddings, doc_ids=doc_ids), None
        x, h, q, k, v = at
        attn = self.self_attn.attend(h, doc_ids, attention_mask, past_key_value, q, k, v)
        return n.back(parts, x, attn) or self._behind(x, self.self_attn.o_proj(attn))

    def _behind(self, x, attn):
        """The stream and the feed-forward's branch behind the attention's."""
        x, h = add_norm(x, attn, self.post_attention_layernorm)
        gate, up = self.mlp.gate_proj(h), self.mlp.up_proj(h)
        if fused_ops(gate, up) and gate.shape == up.shape and gate.shape[-1] % 2 == 0:
            act = ops.silu_mul_parts(gate.flatten(0, 1), up.flatten(0, 1)).view(gate.shape)
        else:
            act = F.silu(gate) * up
        return x, self.mlp.down_proj(act)

    def forward(self, hidden_states, attention_mask=None, past_key_value=None, position_embeddings=None, doc_ids=None):
        attn, _ = self.self_attn(self.input_layernorm(hidden_states), doc_ids, attention_mask=attention_mask,
                                 position_embeddings=position_embeddings, past_key_value=past_key_value)
        hidden_states = hidden_states + attn
        return hidden_states + self.mlp(self.post_attention_layernorm(hidden_states))


# what a layer's native pass steps over, in the order that it asks for
STEPPED_OVER = (MSADecoderLayer, MemorySparseAttention, Qwen3MLP, SILU, Qwen3RMSNorm, nn.Linear)


class MSAModel(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.config = config
        self.embed_tokens = nn.Embedding(config.vocab_size, config.hidden_size, getattr(config, "pad_token_id", None))
        self.layers = nn.ModuleList([MSADecoderLayer(config, i) for i in range(config.num_hidden_layers)])
        self.norm = Qwen3RMSNorm(config.hidden_size, eps=config.rms_norm_eps)
        self.rotary_emb = Qwen3RotaryEmbedding(config=config)

    def _native_layers(self, hidden):
        """The layers' weights for their native pass, or None where a module of some layer is not what that pass steps over."""
        if not hidden.is_cuda or torch.is_grad_enabled() or nn_module._has_any_global_hook() or any(
                c.forward.__module__ != c.__module__ for c in STEPPED_OVER) or not ops.own():
            return None
        return A.native().layers(tuple(self.layers), STEPPED_OVER)

    def _angles(self, hidden, position_ids):
        rot = self.rotary_emb
        if hidden.is_cuda and hidden.dtype == torch.bfloat16 and plain_module(rot, Qwen3RotaryEmbedding) and rot.rope_type == "default" and (
                position_ids.get_device() == hidden.get_device()) and ops.own("rope_table"):
            both = A.native().angles(position_ids, rot.inv_freq, rot.attention_scaling)
            if both is not None:
                return both
        if (plain_module(rot, Qwen3RotaryEmbedding) and rot.rope_type == "default" and fused_ops(hidden) and position_ids.is_cuda
                and position_ids.device == hidden.device == rot.inv_freq.device and position_ids.dtype == torch.int64
                and position_ids.dim() == 2 and rot.inv_freq.dtype == torch.float32):
            return ops.rope_table(position_ids, rot.inv_freq, rot.attention_scaling)
        return rot(hidden, position_ids)

    def forward(self, input_ids=None, attention_mask=None, position_ids=None, past_key_values=None, inputs_embeds=None,
                use_cache=True, doc_ids=None, **unused):
        """Same call as the reference's ``MSAModel.forward`` (the flags it only forwards to outputs are accepted and
        ignored).  ``past_key_values`` must carry the stage of every layer (``cache_kwargs[layer]["stage"]``)."""
        if (input_ids is None) == (inputs_embeds is None):
            raise ValueError("You must specify exactly one of input_ids or inputs_embeds")
        hidden = self.embed_tokens(input_ids) if inputs_embeds is None else inputs_embeds
        if past_key_values is None:
            past_key_values = create_cache()
        if position_ids is None:
            position_ids = torch.arange(hidden.shape[1], device=hidden.device).unsqueeze(0)
        position_embeddings = self._angles(hidden, position_ids)
        layers = self._native_layers(hidden)
        if layers is not None:
            pending = None
            for layer, parts in zip(self.layers, layers):
                hidden, pending = layer.native(parts, hidden, pending, attention_mask, past_key_values, position_embeddings, doc_ids)
            last = A.native().add_norm(hidden, pending, self.norm, Qwen3RMSNorm)
            if last is None:
                last = add_norm(hidden, pending, self.norm) if plain_module(self.norm, Qwen3RMSNorm) else (
                    None, self.norm(hidden if pending is None else hidden + pending))
            return SimpleNamespace(last_hidden_state=last[1], past_key_values=past_key_values if use_cache else None)
        if plain_module(self.norm, Qwen3RMSNorm) and fused_ops(hidden, self.norm.weight) and all(
                plain_module(layer, MSADecoderLayer) and layer.takes_fused(hidden) for layer in self.layers):
            pending = None
            for layer in self.layers:
                hidden, pending = layer.fused(hidden, pending, attention_mask, past_key_values, position_embeddings, doc_ids)
            _, hidden = add_norm(hidden, pending, self.norm)
            return SimpleNamespace(last_hidden_state=hidden, past_key_values=past_key_values if use_cache else None)
        for layer in self.layers:
            hidden = layer(hidden, attention_mask=attention_mask, past_key_value=past_key_values,
                           position_embeddings=position_embeddings, doc_ids=doc_ids)
        return SimpleNamespace(last_hidden_state=self.norm(hidden), past_key_values=past_key_values if use_cache else None)


class MSAForCausalLM(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.config = config
        self.model = MSAModel(config)
        self.lm_head = nn.Linear(config.hidden_size, config.vocab_size, bias=False)

    def forward(self, input_ids=None, attention_mask=None, position_ids=None, past_key_values=None, doc_ids=None,
                use_cache=True, logits_to_keep: int = 0, **unused):
        out = self.model(input_ids=input_ids, attention_mask=attention_mask, position_ids=position_ids,
                         past_key_values=past_key_values, use_cache=use_cache, doc_ids=doc_ids)
        # contiguous: as a batch of strided rows the product would read the head's weights once per sequence
        hidden = out.last_hidden_state[:, -logits_to_keep:].contiguous() if logits_to_keep else out.last_hidden_state
        return SimpleNamespace(logits=self.lm_head(hidden), past_key_values=out.past_key_values)
