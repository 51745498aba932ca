"""The memory model's layers through native code: the bits of the pass through the modules, and that pass wherever a module is not plain."""
import ctypes
import subprocess

import pytest
import torch
import torch.nn as nn

from test_model_host import small_model

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda:0", torch.bfloat16


def model(seed=0):
    torch.manual_seed(seed)
    net = small_model().to(DEV)
    net.rotary_emb.inv_freq = net.rotary_emb.inv_freq.float()
    return net


def block(net):
    """Documents of 150 and 41 tokens behind a template of 3."""
    from msa_b200.cache import SparseCache
    cache = SparseCache()
    for i in range(2):
        cache.record_kwargs(i, {"stage": "prefill_stage1"})
    doc = torch.tensor([[-2] * 3 + [1] * 150 + [2] * 41], device=DEV)
    pos = torch.tensor([list(range(3)) + list(range(150)) + list(range(41))], device=DEV)
    ids = torch.randint(0, 64, doc.shape, generator=torch.Generator().manual_seed(1)).to(DEV)
    out = net(input_ids=ids, attention_mask=torch.ones_like(doc), position_ids=pos, past_key_values=cache, doc_ids=doc)
    kw = cache.cache_kwargs
    return [out.last_hidden_state, *cache.get_kvcache(1), cache.get_router_kcache(1), kw[0]["template_prefix_kcache"], kw[1]["template_prefix_vcache"]]


def token(net, steps=2, batch=3):
    from msa_b200.cache import SparseCache
    g = torch.Generator().manual_seed(2)
    cache, lengths = SparseCache(), torch.tensor([90, 33, 71][:batch], device=DEV)
    for i in range(2):
        kv = [torch.randn(batch, 2, 90, 128, generator=g).to(BF16).to(DEV) for _ in range(2)]
        cache.record_kwargs(i, {"stage": "generate", "compacked_key_cache": kv[0], "compacked_value_cache": kv[1], "kv_lengths": lengths.clone()})
    out = []
    for t in range(steps):
        ids = torch.randint(0, 64, (batch, 1), generator=g).to(DEV)
        y = net(input_ids=ids, attention_mask=torch.ones_like(ids), position_ids=lengths[:, None] + t, past_key_values=cache, doc_ids=torch.full_like(ids, -1))
        out.append(y.last_hidden_state)
    kw = cache.cache_kwargs
    return out + [kw[i][n] for i in range(2) for n in ("compacked_key_cache", "compacked_value_cache", "kv_lengths")] + [kw[0]["_msa_b200_store"][3]]


def through_modules(monkeypatch, run, net):
    from msa_b200 import _cabi as A
    with monkeypatch.context() as m:
        none = type("N", (), {n: staticmethod(lambda *a: None) for n in ("layers", "add_norm", "angles", "decode")})
        m.setattr(A, "native", lambda: none)
        return run(net)


@pytest.mark.parametrize("run", [block, token])
def test_the_same_bits(monkeypatch, run):
    from msa_b200 import model as M
    net, calls = model(), []
    real = M.MSADecoderLayer.native
    with torch.no_grad():
        want = through_modules(monkeypatch, run, net)
        monkeypatch.setattr(M.MSADecoderLayer, "native", lambda self, *a: calls.append(self) or real(self, *a))
        got = run(net)
    assert len(calls) == (2 if run is block else 4)
    assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))


class Scaled(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


def hooked(net, seen):
    net.layers[1].self_attn.v_proj.register_forward_hook(lambda m, a, y: seen.append(m))


def hooked_norm(net, seen):
    net.layers[0].post_attention_layernorm.register_forward_pre_hook(lambda m, a: seen.append(m))


def replaced(net, seen):
    old = net.layers[0].mlp.down_proj
    new = Scaled(old.in_features, old.out_features, bias=False).to(DEV, BF16)
    new.load_state_dict(old.state_dict())
    new.register_forward_hook(lambda m, a, y: seen.append(m))
    net.layers[0].mlp.down_proj = new


def own_forward(net, seen):
    m = net.layers[1].mlp.gate_proj
    real = m.forward
    m.forward = lambda x: seen.append(m) or real(x)


def biased(net, seen):
    m = net.layers[0].self_attn.o_proj
    m.bias = nn.Parameter(torch.full((256,), 0.5, device=DEV, dtype=BF16))
    seen.append(m)


@pytest.mark.parametrize("change", [hooked, hooked_norm, replaced, own_forward, biased])
def test_a_module_that_is_not_plain_is_called(monkeypatch, change):
    from msa_b200 import model as M
    net, seen = model(), []
    with torch.no_grad():
        change(net, seen)
        want = through_modules(monkeypatch, token, net)
        seen[:] = seen[:1] if change is biased else []
        monkeypatch.setattr(M.MSADecoderLayer, "native", lambda *a: pytest.fail("stepped over a module"))
        got = token(net)
    assert seen and all(torch.equal(a, b) for a, b in zip(got, want))


def test_what_else_goes_through_the_modules(monkeypatch):
    """Gradients, autocast, function modes and operands off the 16-byte boundary."""
    from msa_b200 import _cabi as A
    from msa_b200 import model as M
    net = model()
    layers = lambda: A.native().layers(tuple(net.layers), M.STEPPED_OVER)
    assert layers() is None                                      # gradients are recorded
    with torch.no_grad():
        assert len(layers()) == 2
        with torch.autocast("cuda", dtype=torch.float16):
            assert layers() is None
        with torch.device(DEV):
            assert layers() is None                              # a function mode
        net.train()
        assert layers() is None
        net.eval()
        parts = layers()[0]
        x = torch.randn(1, 5, 256, device=DEV).to(BF16)
        cos = sin = torch.ones(1, 5, 128, device=DEV, dtype=BF16)
        assert A.native().front(parts, x, None, cos, sin) is not None
        shifted = torch.empty(5 * 256 + 1, device=DEV, dtype=BF16)[1:].view(1, 5, 256).copy_(x)
        for a in ((shifted, None, cos, sin), (x, x[:, :4], cos, sin), (x.float(), None, cos, sin), (x.cpu(), None, cos, sin), (x, None, cos[:, :4], sin[:, :4]),
                  (x.transpose(0, 1), None, cos, sin), (x[:, :0], None, cos[:, :0], sin[:, :0])):
            assert A.native().front(parts, *a) is None
        assert A.native().back(parts, x, x) is None              # the attention's rows are 512 wide
        own = net.layers[0].self_attn.q_proj
        own.weight = nn.Parameter(own.weight.float())
        assert layers() is None


@pytest.mark.parametrize("name,run", [("add_rmsnorm", block), ("silu_mul_parts", block), ("heads_norm_rope", block), ("rope_table", token),
                                      ("sparse_decode_attn", token)])
def test_a_function_put_in_the_place_of_an_op_is_called(monkeypatch, name, run):
    from msa_b200 import ops
    net, calls, real = model(), [], getattr(ops, name)
    with torch.no_grad():
        want = run(net)
        monkeypatch.setattr(ops, name, lambda *a, **k: calls.append(1) or real(*a, **k))
        got = run(net)
    assert calls and all(torch.equal(a, b) for a, b in zip(got, want))


STUB = """
int PyGILState_Check(void);
int calls, held;
static int seen(void) { ++calls; held += PyGILState_Check(); return 0; }
const char* msa_last_error(void) { return "stub"; }
long long msa_decode_workspace_bytes(void) { return 0; }
int msa_add_rmsnorm(void) { return seen(); }
int msa_heads_norm_rope(void) { return seen(); }
int msa_silu_mul_parts(void) { return seen(); }
int msa_rope_table(void) { return seen(); }
int msa_sparse_decode_attn_next(void) { return seen(); }
"""


def test_python_goes_on_meanwhile(tmp_path):
    """Allocations and launches happen without Python's lock: asked where the launches would be."""
    from msa_b200 import _cabi as A
    from msa_b200 import model as M
    (tmp_path / "stub.c").write_text(STUB)
    path = str(tmp_path / "stub.so")
    subprocess.run(["gcc", "-shared", "-fPIC", str(tmp_path / "stub.c"), "-o", path], check=True)
    stub, n, net = ctypes.CDLL(path), A.native(), model()
    of = lambda *s: torch.ones(*s, device=DEV, dtype=BF16)
    count = lambda name: ctypes.c_int.in_dll(stub, name).value
    with torch.no_grad():
        parts = n.layers(tuple(net.layers), M.STEPPED_OVER)[0]
        x, one, store, angle = of(1, 5, 256), of(3, 2, 1, 128), of(3, 2, 90, 128), of(1, 5, 128)
        rows = of(1, 5, net.layers[0].self_attn.o_proj.weight.shape[1])
        pos, ints = torch.zeros(1, 5, device=DEV, dtype=torch.int64), torch.ones(3, device=DEV, dtype=torch.int32)
        calls = [lambda: n.add_norm(x, x, net.norm, M.Qwen3RMSNorm), lambda: n.front(parts, x, x, angle, angle), lambda: n.back(parts, x, rows),
                 lambda: n.angles(pos, net.rotary_emb.inv_freq, 1.0), lambda: n.decode(one, one, one, store, store, ints, ints, ints.long(), 1)]
        n.bind(path)
        try:
            for call in calls:
                before = count("calls")
                assert call() is not None and count("calls") > before and count("held") == 0
        finally:
            n.bind(A.LIB_PATH)
