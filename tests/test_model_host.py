"""When ``MSAModel`` steps over its modules' calls, on fake CUDA tensors: never where a module was replaced."""
import pytest
import torch
import torch.nn as nn
from torch._subclasses.fake_tensor import FakeTensorMode
from transformers.models.qwen3.modeling_qwen3 import Qwen3MLP, Qwen3RMSNorm, Qwen3RotaryEmbedding

pytestmark = pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
BF16 = torch.bfloat16


class Wrapped(nn.Module):
    """What an offload, quantisation or debug wrapper puts in a layer's place."""

    def __init__(self, layer, seen):
        super().__init__()
        self.layer, self.seen = layer, seen

    def forward(self, hidden_states, **kwargs):
        self.seen.append(sorted(kwargs))
        return hidden_states


def small_model(hidden_act="silu"):
    from msa_b200.configuration import MSAConfig
    from msa_b200.model import MSAModel
    cfg = MSAConfig(
        msa_config=dict(router_layer_idx="1", aux_loss=False, aux_loss_method="INFONCE", decouple_router=True, top_k_docs=4, pooling_kernel_size=64,
                        head_reduce_method="mean", query_reduce_method="max", chunk_reduce_method="max", decouple_pooling_mode="mean"),
        hidden_size=256, num_attention_heads=4, num_key_value_heads=2, head_dim=128, num_hidden_layers=2, intermediate_size=520, vocab_size=64,
        max_position_embeddings=4096, rms_norm_eps=1e-6, hidden_act=hidden_act)
    cfg._attn_implementation = "eager"
    return MSAModel(cfg).to(BF16).eval()


def test_a_layer_in_another_layers_place_is_called(monkeypatch):
    from msa_b200 import model as M
    seen, fused = [], []
    net = small_model()
    for i in range(2):
        net.layers[i] = Wrapped(net.layers[i], seen)
    # a forward on the CPU, with the operands answered for as if they were on a GPU
    monkeypatch.setattr(M, "fused_ops", lambda *t: True)
    monkeypatch.setattr(M.ops, "add_rmsnorm", lambda *a: fused.append(a))
    with torch.no_grad():
        out = net(input_ids=torch.zeros(1, 3, dtype=torch.long), attention_mask=torch.ones(1, 3, dtype=torch.long))
    assert seen == [["attention_mask", "doc_ids", "past_key_value", "position_embeddings"]] * 2 and not fused
    assert out.last_hidden_state.shape == (1, 3, 256)


@pytest.mark.parametrize("cls", [Qwen3RMSNorm, Qwen3MLP, Qwen3RotaryEmbedding])
def test_a_forward_put_in_a_class_is_called(monkeypatch, cls):
    from msa_b200.attention import plain_module
    net = small_model()
    m = {Qwen3RMSNorm: net.norm, Qwen3MLP: net.layers[0].mlp, Qwen3RotaryEmbedding: net.rotary_emb}[cls]
    assert plain_module(m, cls)
    monkeypatch.setattr(cls, "forward", lambda self, *a: a[0])
    assert not plain_module(m, cls)


def test_operands_on_two_devices_are_not_fused():
    from msa_b200 import attention
    with FakeTensorMode(), torch.no_grad():
        at = lambda d: torch.empty(4, 64, dtype=BF16, device=d)
        plain = type(at("cuda:0"))
        real, attention.torch = attention.torch, type("T", (), {"Tensor": plain, "bfloat16": BF16, "is_grad_enabled": staticmethod(lambda: False)})
        try:
            assert attention.fused_ops(at("cuda:0"), at("cuda:0"))
            assert not attention.fused_ops(at("cuda:0"), at("cuda:1")) and not attention.fused_ops(at("cuda:0"), at("cpu"))
            assert not attention.fused_ops(at("cpu"), at("cuda:0"))
        finally:
            attention.torch = real


@pytest.mark.parametrize("act,fused", [("silu", True), ("gelu", False), ("relu", False)])
def test_the_fused_pass_asks_a_layer_for_nothing_of_its_own(monkeypatch, act, fused):
    """A layer that was saved whole before the fused pass was there holds nothing but its modules."""
    from msa_b200 import model as M
    monkeypatch.setattr(M, "fused_ops", lambda *t: True)
    layer = small_model(hidden_act=act).layers[0]
    for name in set(vars(layer)) - set(vars(nn.Module())) - {"hidden_size", "layer_idx"}:
        delattr(layer, name)
    with torch.no_grad():
        assert layer.takes_fused(torch.zeros(1, 3, 256, dtype=BF16)) is fused
