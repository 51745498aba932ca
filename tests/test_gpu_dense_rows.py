"""Elementwise kernels of the memory model (head norm + rotation, add + RMSNorm, silu * up, rotation tables) at the edges of
their variants, against plain fp32 / fp64 torch; and the model's forward with them against the eager modules."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16
# an fp32 result rounded once to bf16 (8 significant bits) is at most 2^-9 of its size off; 2^-8 leaves room for the fp32 sums
STEP = 2.0 ** -8


def randn(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(BF16).to(DEV)


# rows * ceil(heads / 8) on both sides of the line between the narrow and the wide variant (9472), odd head counts
@pytest.mark.parametrize("pad", [0, 4])                                       # rows that are 16- or only 8-byte aligned
@pytest.mark.parametrize("rows,hq,hkv,tables", [(1, 1, 1, 1), (6, 3, 2, 3), (1894, 32, 8, 947), (1895, 32, 8, 1895), (9472, 5, 2, 9472), (4736, 7, 5, 2368)])
def test_heads_norm_rope(rows, hq, hkv, tables, pad):
    from msa_b200 import ops
    wide = randn(rows, (hq + hkv) * 128 + pad, seed=rows)
    q, k = wide[:, :hq * 128], wide[:, hq * 128:(hq + hkv) * 128]
    qw, kw = 1 + randn(128, seed=1, scale=0.1), 1 + randn(128, seed=2, scale=0.1)
    cos, sin = randn(tables, 128, seed=3), randn(tables, 128, seed=4)         # nothing relies on the halves being alike
    got = ops.heads_norm_rope(q, k, qw, kw, 1e-6, cos, sin)
    for x, w, y in ((q, qw, got[0]), (k, kw, got[1])):
        x = x.double().reshape(rows, -1, 128)
        x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
        c, s = (t.double().repeat(rows // tables, 1).unsqueeze(1) for t in (cos, sin))
        turned = torch.cat([-x[..., 64:], x[..., :64]], -1)
        bound = STEP * (x * c).abs() + STEP * (turned * s).abs()
        assert ((y.double().view_as(x) - (x * c + turned * s)).abs() <= bound + 1e-6).all()


@pytest.mark.parametrize("rows", [1, 1183, 1185])                             # a block per row up to 1183 rows, then a warp
@pytest.mark.parametrize("hidden", [8, 1024, 1032, 2560, 2568, 3080, 4096, 4104, 12288, 2562])
def test_add_rmsnorm(rows, hidden):
    from msa_b200 import ops
    x, y, w = randn(rows, hidden, seed=rows), randn(rows, hidden, seed=hidden), 1 + randn(hidden, seed=5, scale=0.1)
    for branch in (y, None):
        x_new, h = ops.add_rmsnorm(x, branch, w, 1e-6)
        assert torch.equal(x_new, x if branch is None else x + branch)
        f = x_new.double()
        want = f * torch.rsqrt(f.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
        assert ((h.double() - want).abs() <= STEP * want.abs() + 1e-6).all()


@pytest.mark.parametrize("rows,ffn,offset", [(1, 2, 0), (3, 8, 0), (5, 1022, 0), (7, 4096, 0), (4, 1024, 2), (257, 264, 8)])
def test_silu_mul_parts(rows, ffn, offset):
    from msa_b200 import ops
    wide = randn(rows, 2 * ffn + 2 * offset, seed=ffn, scale=3.0)
    gate, up = wide[:, offset:offset + ffn], wide[:, offset + ffn:offset + 2 * ffn]
    want = F.silu(gate.double()) * up.double()
    assert ((ops.silu_mul_parts(gate, up).double() - want).abs() <= STEP * want.abs() + 1e-6).all()
    assert torch.equal(ops.silu_mul(wide[:, offset:], ffn), ops.silu_mul_parts(gate, up))


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (2, 1000)])
def test_rope_table(shape):
    from msa_b200 import ops
    pos = torch.randint(0, 100_000_000, shape, generator=torch.Generator().manual_seed(7)).to(DEV)
    inv = (1.0 / 1e6 ** (torch.arange(0, 128, 2, dtype=torch.float64) / 128)).float().to(DEV)
    cos, sin = ops.rope_table(pos, inv, 1.25)
    ang = (pos.float()[..., None] * inv).double()
    for got, want in ((cos, ang.cos()), (sin, ang.sin())):
        want = 1.25 * torch.cat([want, want], -1)
        assert ((got.double() - want).abs() <= STEP * want.abs() + 1e-9).all()


def small_model():
    from msa_b200.configuration import MSAConfig
    from msa_b200.model import MSAForCausalLM
    cfg = MSAConfig(
        msa_config=dict(router_layer_idx="1", aux_loss=False, aux_loss_method="INFONCE", decouple_router=True, top_k_docs=4, pooling_kernel_size=64,
                        head_reduce_method="mean", query_reduce_method="max", chunk_reduce_method="max", decouple_pooling_mode="mean"),
        hidden_size=256, num_attention_heads=4, num_key_value_heads=2, head_dim=128, num_hidden_layers=2, intermediate_size=520, vocab_size=64,
        max_position_embeddings=4096, rms_norm_eps=1e-6)
    cfg._attn_implementation = "eager"
    torch.manual_seed(3)
    return MSAForCausalLM(cfg).to(BF16).to(DEV).eval()


@pytest.mark.parametrize("masked", [False, True])
def test_model_forward_matches_the_eager_modules(masked):
    """Stage 1 of a small stack; a hook on any module that the fused pass steps over sends the forward to the eager modules."""
    from msa_b200 import ops
    from msa_b200.cache import SparseCache
    model = small_model()
    doc = torch.tensor([[-2] * 3 + [1] * 200 + [2] * 77], device=DEV)
    pos = torch.tensor([list(range(3)) + list(range(200)) + list(range(77))], device=DEV)
    mask = torch.ones_like(doc)
    if masked:
        mask[0, 50:60] = 0
    ids = torch.randint(0, 64, doc.shape, generator=torch.Generator().manual_seed(1)).to(DEV)

    def run():
        cache = SparseCache()
        for i in range(2):
            cache.record_kwargs(i, {"stage": "prefill_stage1"})
        with torch.no_grad():
            out = model.model(input_ids=ids, attention_mask=mask, position_ids=pos, past_key_values=cache, doc_ids=doc)
        return [out.last_hidden_state, *cache.get_kvcache(1), cache.get_router_kcache(1)]

    counted, fused = [], ops.add_rmsnorm
    try:
        ops.add_rmsnorm = lambda *a: (counted.append(1), fused(*a))[1]
        got = run()
        assert len(counted) == 5                            # two per layer and the final norm
        seen = []
        model.model.layers[1].post_attention_layernorm.register_forward_hook(lambda m, a, o: seen.append(o.shape))
        want = run()
        assert len(counted) == 5 and len(seen) == 1
    finally:
        ops.add_rmsnorm = fused
    rows = mask[0] == 1
    for g, w in zip(got, want):
        g, w = (t.float()[:, rows] if t.dim() == 3 else t.float() for t in (g, w))
        # both round bf16 activations, the eager modules about a dozen times per layer: a few 2^-9 each
        assert float((g - w).norm() / w.norm()) < 2e-2


def test_grad_mode_keeps_the_eager_modules():
    """Outside no_grad the norms and feed-forwards stay differentiable modules."""
    from msa_b200.attention import fused_ops
    x = torch.zeros(1, 8, dtype=BF16, device=DEV)
    assert not fused_ops(x)
    with torch.no_grad():
        assert fused_ops(x) and not fused_ops(x.float()) and not fused_ops(x[:, 1:])
