"""The work this package is measured by: what its users have it do, through its public entry points.

Two families.  The memory model: questions against a bank of pooled documents (``MSAService.doc_query``, ``MSAService.route``)
and the three forward passes of ``MSAForCausalLM`` (a block of documents, a batch of questions, a decode token).  The layered
decoders: prompts, steps that mix a portion of a prompt with decode tokens, and decode steps from a CUDA graph, of both designs.

``exact`` restates each path in plain torch at 64 bits; nothing of the package is used there.  Everything random comes from the
seed, drawn on the GPU in a fixed order, so that ``prepare`` and ``exact`` see the same inputs.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

DEV = "cuda:0"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
HQ, HKV, D = 32, 8, 128                      # the memory model's heads
HIDDEN, FFN, VOCAB, TEMPLATE = 2560, 9728, 32768, 3
TOP_K, POOL = 16, 64
THETA, EPS = 1_000_000.0, 1e-6
PLANTED = 24                                 # documents per question that are about it, each a little less than the one before


def listed():
    return [
        # one question of 64 tokens against a 1M-token memory in 32 bits: the smallest call, all latency
        dict(name="query-one-fp32", kind="query", docs=2000, chunks=8, batch=1, tokens=64, dtype="float32"),
        # a batch of questions against a 1M-token memory
        dict(name="query-1m", kind="query", docs=2048, chunks=8, batch=32, tokens=128, dtype="bfloat16"),
        # the largest: a batch of long questions against one GPU's eighth of a 100M-token memory
        dict(name="query-12m", kind="query", docs=24414, chunks=8, batch=48, tokens=200, dtype="bfloat16"),
        # routing inside a decode step: one token of every sequence against the same shard, keys laid out for it
        dict(name="route-token", kind="route", docs=24414, chunks=8, batch=32),
        # building the memory: a block of documents through the model, attention inside documents, pooled keys and values out
        dict(name="block", kind="block", docs=64, doc_tokens=500),
        # answering: left-padded questions through the model, routed, fetched and attended in the upper layer
        dict(name="question", kind="question", docs=2048, chunks=8, batch=16, tokens=96),
        # ... and the next token of every answer
        dict(name="token", kind="token", batch=32, context=2179),
        # ragged prompts of a layered decoder with experts
        dict(name="mutuvik-prompt", kind="step", design="Mutuvik", width=2048, window=1024, portions="2048,1500,1911,777", past=0, decode=0),
        # continuous batching: a portion of a long prompt beside the tokens of the sequences that decode
        dict(name="mutuvik-mixed", kind="step", design="Mutuvik", width=2048, window=1024, portions="1024", past=2048, decode=31),
        # a decode step
        dict(name="mutuvik-tokens", kind="tokens", design="Mutuvik", width=2048, window=1024, batch=32),
        # the same of the other design: prompts, and the decode step of a lightly loaded server
        dict(name="nazerax-prompt", kind="step", design="Nazerax", width=2048, window=1024, portions="2048,1500,1911,777", past=0, decode=0),
        dict(name="nazerax-tokens", kind="tokens", design="Nazerax", width=2048, window=1024, batch=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "route", "block", "question", "token", "step", "step", "tokens", "tokens"])
    if kind == "query":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        batch = _log(rng, 1, 48 if dtype == "bfloat16" else 4)
        docs = _log(rng, PLANTED * batch + 100, 24414 if dtype == "bfloat16" else 2500)
        return dict(kind=kind, docs=docs, chunks=rng.randint(2, 8), batch=batch, tokens=_log(rng, 4, 200), dtype=dtype)
    if kind == "route":
        batch = _log(rng, 1, 128)
        return dict(kind=kind, docs=_log(rng, PLANTED * batch + 100, 24414), chunks=rng.randint(2, 8), batch=batch)
    if kind == "block":
        tokens = _log(rng, 150, 1500)
        return dict(kind=kind, docs=max(2, _log(rng, 4000, 32000) // tokens), doc_tokens=tokens)
    if kind == "question":
        batch = _log(rng, 1, 32)
        return dict(kind=kind, docs=_log(rng, PLANTED * batch + 100, 4096), chunks=rng.randint(2, 8), batch=batch, tokens=_log(rng, 8, 128))
    if kind == "token":
        return dict(kind=kind, batch=_log(rng, 1, 48), context=_log(rng, 100, 3000))
    design, width = rng.choice(["Mutuvik", "Nazerax"]), rng.choice([1024, 2048])
    window = rng.choice([512, 777, 1024])
    if kind == "tokens":
        return dict(kind=kind, design=design, width=width, window=window, batch=_log(rng, 1, 64))
    portions = [_log(rng, 33, 2048) for _ in range(rng.randint(1, 4))]
    past, decode = rng.choice([(0, 0), (0, 0), (_log(rng, 20, 3000), _log(rng, 1, 48))])
    return dict(kind=kind, design=design, width=width, window=window, portions=",".join(map(str, portions)), past=past, decode=decode)


def tolerance(case):
    if case["kind"] == "query" and case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    if case["kind"] in ("query", "route"):
        return {"rel": 5e-4, "max": 2e-2, "differ": 0.002}       # bf16 folded queries (1e-4 seen); whole values: ids of near ties
    if case["kind"] in ("step", "tokens"):
        return {"rel": 2.5e-2, "max": 0.5, "differ": 0.0}        # bf16 activations through five layer runs, experts that tie (8e-3 seen)
    return {"rel": 2e-2, "max": 0.3, "differ": 0.002}            # bf16 activations through two layers (6e-3 seen)


# ------------------------------------------------------------------------------------------------------------------ draws
class _Draw:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF16):
        return (torch.randn(shape, generator=self.g, device=DEV, dtype=F32) * std + mean).to(dtype)

    def below(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=self.g, device=DEV)

    def some(self, n, k):
        return torch.randperm(n, generator=self.g, device=DEV)[:k]


def _rms(x, w, eps):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


# ------------------------------------------------------------------------------------------------------------------ the bank
def _bank(d, case, about, dtype):
    """Documents of 1 .. 2 * chunks - 1 chunks; ``about`` [B, S, HKV, D]: what the tokens of every question ask for.  Document
    number j of a question's PLANTED ones has the direction of one of its tokens, blurred more with every j."""
    n, b = case["docs"], about.shape[0]
    lens = d.below(1, 2 * case["chunks"], n)
    mean = d.normal(n, HKV, D, std=0.5, dtype=F32)
    docs = d.some(n, b * PLANTED).view(b, PLANTED)
    lens[docs.reshape(-1)] = case["chunks"]                                # so that every question fetches as much
    lens_host = lens.tolist()
    place = torch.arange(PLANTED, device=DEV)
    token = about.shape[1] - 1 - place % max(1, about.shape[1] // 2)       # questions are padded on the left, by half at most
    blur = d.normal(b, PLANTED, HKV, D, std=D ** -0.5, dtype=F32)
    mean[docs.reshape(-1)] = (F.normalize(about[:, token].float(), dim=-1) + blur * (0.3 + 0.06 * place)[:, None, None]).view(-1, HKV, D) * 4.0
    mean = torch.repeat_interleave(mean, lens, dim=0)
    c = mean.shape[0]
    rk = F.normalize(mean + d.normal(c, HKV, D, std=0.125, dtype=F32), dim=-1).to(dtype)
    return lens_host, rk, d.normal(c, HKV, D, dtype=dtype), d.normal(c, HKV, D, std=0.5, dtype=dtype)


def _service(lens, rk, k, v, layers, router, dtype):
    from msa_b200.memory import AttentionGeometry, Document, ModelConfig
    from msa_b200.service import MSAService
    geo = AttentionGeometry(num_hidden_layers=layers, num_attention_heads=HQ, num_key_value_heads=HKV, head_dim=D, dtype=dtype)
    svc = MSAService(0, None, ModelConfig(doc_top_k=TOP_K, pooling_kernel_size=POOL, router_layer_idx=str(router)), None, geo,
                     world_size=1, rank=0)
    svc.load_pooled([Document(doc_id=1000 + i, num_chunks=n) for i, n in enumerate(lens)], {router: (k, v, rk)})
    svc.publish_directory()
    return svc


def _query_inputs(case, seed):
    """Questions of tokens // 2 .. tokens tokens, padded on the left; unit rows per head, as the layer passes them."""
    d, dtype = _Draw(seed), getattr(torch, case.get("dtype", "bfloat16"))
    b, s = case["batch"], case.get("tokens", 1)
    q = d.normal(b, HKV, 1, s, D, dtype=F32) + 0.7 * d.normal(b, HKV, HQ // HKV, s, D, dtype=F32)     # a group's heads agree in part
    q = F.normalize(q, dim=-1).view(b, HQ, s, D)
    first = s - d.below(max(1, s // 2), s + 1, b)
    first[0] = 0
    mask = torch.arange(s, device=DEV)[None] >= first[:, None]
    q = q.to(dtype)
    about = q.float().view(b, HKV, HQ // HKV, s, D).sum(2).permute(0, 2, 1, 3)
    return (q, mask) + _bank(d, case, about, dtype)


def _routed(folded, mask, lens, rk, top):
    """64-bit routing.  folded [B, S, HKV * D] sums over a group's heads; returns the winners' scores and numbers (from 1)."""
    b, s, _ = folded.shape
    c = rk.shape[0]
    doc = torch.repeat_interleave(torch.arange(len(lens), device=DEV), torch.tensor(lens, device=DEV))
    best = torch.full((b, len(lens)), -torch.inf, dtype=F64, device=DEV)
    keys = rk.reshape(c, -1).to(F64)
    for i in range(0, b, 8):
        rows = folded[i:i + 8].to(F64)
        hidden = ~mask[i:i + 8, :, None]
        for lo in range(0, c, 1 << 15):
            z = (rows @ keys[lo:lo + (1 << 15)].T / HQ).masked_fill(hidden, -torch.inf).amax(1)
            best[i:i + 8].scatter_reduce_(1, doc[lo:lo + (1 << 15)].expand(z.shape[0], -1), z, "amax")
    score, at = best.topk(min(top, len(lens)), dim=1)
    return score, at + 1


def _rows_of(at, lens):
    """The bank rows of the winners of every question, in the order of their documents."""
    lens = torch.tensor(lens, device=DEV)
    off = F.pad(lens.cumsum(0), (1, 0))
    out = []
    for row in at.sort(dim=1).values - 1:
        out.append(torch.cat([torch.arange(int(off[i]), int(off[i + 1]), device=DEV) for i in row.tolist()]))
    return out


# ------------------------------------------------------------------------------------------------------------------ the memory model
def _model_weights(d, layers=2, router=1):
    w = {"model.embed_tokens.weight": d.normal(VOCAB, HIDDEN), "lm_head.weight": d.normal(VOCAB, HIDDEN, std=HIDDEN ** -0.5),
         "model.norm.weight": d.normal(HIDDEN, std=0.1, mean=1.0)}
    for i in range(layers):
        p, a = f"model.layers.{i}.", f"model.layers.{i}.self_attn."
        mats = {a + "q_proj": (HQ * D, HIDDEN), a + "k_proj": (HKV * D, HIDDEN), a + "v_proj": (HKV * D, HIDDEN), a + "o_proj": (HIDDEN, HQ * D),
                p + "mlp.gate_proj": (FFN, HIDDEN), p + "mlp.up_proj": (FFN, HIDDEN), p + "mlp.down_proj": (HIDDEN, FFN)}
        if i == router:
            mats.update({a + "router_q_proj.0": (HQ * D, HIDDEN), a + "router_k_proj.0": (HKV * D, HIDDEN)})
        for n, (r, c) in mats.items():
            w[n + ".weight"] = d.normal(r, c, std=c ** -0.5)
        for n, size in ((a + "q_norm", D), (a + "k_norm", D), (p + "input_layernorm", HIDDEN), (p + "post_attention_layernorm", HIDDEN)):
            w[n + ".weight"] = d.normal(size, std=0.1, mean=1.0)
    return w


def _model(w, layers=2, router=1):
    from msa_b200.configuration import MSAConfig
    from msa_b200.model import MSAForCausalLM
    cfg = MSAConfig(
        msa_config=dict(router_layer_idx=str(router), aux_loss=False, aux_loss_method="INFONCE", decouple_router=True, top_k_docs=TOP_K,
                        pooling_kernel_size=POOL, head_reduce_method="mean", query_reduce_method="max", chunk_reduce_method="max",
                        decouple_pooling_mode="mean"),
        hidden_size=HIDDEN, num_attention_heads=HQ, num_key_value_heads=HKV, head_dim=D, num_hidden_layers=layers, intermediate_size=FFN,
        vocab_size=VOCAB, max_position_embeddings=65536, rms_norm_eps=EPS, rope_parameters={"rope_type": "default", "rope_theta": THETA})
    cfg._attn_implementation = "eager"
    with torch.device(DEV):
        default = torch.get_default_dtype()
        torch.set_default_dtype(BF16)
        try:
            model = MSAForCausalLM(cfg).eval()
        finally:
            torch.set_default_dtype(default)
    model.load_state_dict(w)
    model.requires_grad_(False)
    # the angles of the rotation are 32-bit whatever the model's type
    rot = model.model.rotary_emb
    rot.inv_freq = _inv_freq(F32)
    return model


def _inv_freq(dtype):
    return 1.0 / THETA ** (torch.arange(0, D, 2, device=DEV, dtype=F64) / D).to(dtype)


def _turn(x, pos):
    """x [..., n, D], pos [..., n]: first and second half of a head form the planes."""
    ang = pos.to(x.dtype)[..., None] * _inv_freq(x.dtype)
    cos, sin = torch.cat([ang.cos()] * 2, -1), torch.cat([ang.sin()] * 2, -1)
    return x * cos + torch.cat([-x[..., D // 2:], x[..., :D // 2]], -1) * sin


def _heads(w, i, h, pos):
    """(q, k, v) of layer i for rows h [B, n, HIDDEN] at positions pos [B, n], as [B, heads, n, D]."""
    a, at = f"model.layers.{i}.self_attn.", lambda n: w[f"model.layers.{i}.self_attn.{n}.weight"].to(h.dtype)
    split = lambda t: t.view(*h.shape[:2], -1, D).transpose(1, 2)
    q = _turn(_rms(split(h @ at("q_proj").T), at("q_norm"), EPS), pos[:, None])
    k = _turn(_rms(split(h @ at("k_proj").T), at("k_norm"), EPS), pos[:, None])
    return q, k, split(h @ at("v_proj").T)


def _rest(w, i, x, attn):
    p = f"model.layers.{i}."
    at = lambda n: w[p + n + ".weight"].to(x.dtype)
    x = x + attn @ at("self_attn.o_proj").T
    h = _rms(x, at("post_attention_layernorm"), EPS)
    return x + (F.silu(h @ at("mlp.gate_proj").T) * (h @ at("mlp.up_proj").T)) @ at("mlp.down_proj").T


def _look(q, k, v, see):
    """q [HQ, n, D], k and v [HKV, m, D], see [n, m] -> [n, HQ * D]."""
    k, v = (t.repeat_interleave(HQ // HKV, 0) for t in (k, v))
    z = (q @ k.transpose(1, 2) * D ** -0.5).masked_fill(~see, -torch.inf)
    return (torch.softmax(z, -1) @ v).transpose(0, 1).reshape(q.shape[1], -1)


def _block_inputs(case, seed):
    d = _Draw(seed)
    size, n = case["doc_tokens"], case["docs"]
    lens = [size // 2 + (7919 * i + 13 * size) % (size + 1) for i in range(n)]       # half to one and a half times the size
    doc = [-2] * TEMPLATE + [i + 1 for i, n in enumerate(lens) for _ in range(n)]
    pos = list(range(TEMPLATE)) + [j for n in lens for j in range(n)]
    ids = d.below(0, VOCAB, 1, len(doc))
    return d, lens, ids, torch.tensor([doc], device=DEV), torch.tensor([pos], device=DEV)


def _exact_block(case, seed):
    d, lens, ids, doc, pos = _block_inputs(case, seed)
    w = _model_weights(d)
    x = w["model.embed_tokens.weight"][ids].to(F64)
    spans = [(0, TEMPLATE)]
    for n in lens:
        spans.append((spans[-1][1], spans[-1][1] + n))
    out = {}
    for i in range(2):
        h = _rms(x, w[f"model.layers.{i}.input_layernorm.weight"].to(F64), EPS)
        q, k, v = _heads(w, i, h, pos)
        attn = torch.cat([_look(q[0, :, a:b], k[0, :, a:b], v[0, :, a:b], torch.ones(b - a, b - a, dtype=torch.bool, device=DEV).tril())
                          for a, b in spans])[None]
        out[f"template_{i}"] = [k[:, :, :TEMPLATE], v[:, :, :TEMPLATE]]
        if i == 1:
            raw = (h @ w["model.layers.1.self_attn.router_k_proj.0.weight"].to(F64).T).view(1, -1, HKV, D).transpose(1, 2)
            cuts = [(a, min(a + POOL, hi)) for lo, hi in spans[1:] for a in range(lo, hi, POOL)]
            mean = lambda t: torch.stack([t[:, :, a:b].mean(2) for a, b in cuts], 2)
            out["pooled"] = [mean(k), mean(v), F.normalize(mean(raw), dim=-1)]
        x = _rest(w, i, x, attn)
    out["hidden"] = _rms(x, w["model.norm.weight"].to(F64), EPS)
    return out


def _question_inputs(case, seed):
    """Left-padded questions; the bank of the routing layer knows what they ask: its planted documents follow the routing
    queries of a 32-bit restatement of the layers below."""
    d = _Draw(seed)
    w = _model_weights(d)
    b, s = case["batch"], case["tokens"]
    first = s - d.below(max(1, s // 2), s + 1, b)
    first[0] = 0
    mask = (torch.arange(s, device=DEV)[None] >= first[:, None]).long()
    pos = (torch.arange(s, device=DEV)[None] - first[:, None]).clamp(min=0) + TEMPLATE + TOP_K
    ids = d.below(0, VOCAB, b, s) * mask
    prefix = {i: (d.normal(1, HKV, TEMPLATE, D), d.normal(1, HKV, TEMPLATE, D, std=0.5)) for i in range(2)}
    about = _ask(w, ids, mask, pos, prefix, F32)[1]
    return (w, ids, mask, pos, prefix) + _bank(d, case, about.view(b, s, HKV, D), BF16)


def _ask(w, ids, mask, pos, prefix, dtype, bank=None):
    """The questions' pass in plain torch.  Without ``bank`` up to the routing layer: (None, folded routing queries); else the
    logits of the last column and both layers' compact caches."""
    b, s = ids.shape
    x = w["model.embed_tokens.weight"][ids].to(dtype)
    caches, lengths = [], []
    for i in range(2):
        h = _rms(x, w[f"model.layers.{i}.input_layernorm.weight"].to(dtype), EPS)
        found = [None] * b
        if i == 1:
            rq = F.normalize((h @ w["model.layers.1.self_attn.router_q_proj.0.weight"].to(dtype).T).view(b, s, HKV, HQ // HKV, D), dim=-1)
            folded = rq.sum(3).reshape(b, s, -1)
            if bank is None:
                return None, folded
            lens, rk, bk, bv = bank
            found = _rows_of(_routed(folded, mask.bool(), lens, rk, TOP_K)[1], lens)
        q, k, v = _heads(w, i, h, pos)
        attn, rows = x.new_zeros(b, s, HQ * D), []
        for j in range(b):
            n = int(mask[j].sum())
            ks, vs = [prefix[i][0][0].to(dtype)], [prefix[i][1][0].to(dtype)]
            if found[j] is not None:
                ks.append(bk[found[j]].transpose(0, 1).to(dtype))
                vs.append(bv[found[j]].transpose(0, 1).to(dtype))
            kk, vv = torch.cat(ks + [k[j, :, s - n:]], 1), torch.cat(vs + [v[j, :, s - n:]], 1)
            see = torch.ones(n, kk.shape[1], dtype=torch.bool, device=DEV).tril(kk.shape[1] - n)
            attn[j, s - n:] = _look(q[j, :, s - n:], kk, vv, see)
            rows.append((kk, vv))
        if bank is not None:
            longest = max(kk.shape[1] for kk, _ in rows)
            caches.append([torch.stack([F.pad(r[c], (0, 0, longest - r[c].shape[1], 0)) for r in rows]) for c in (0, 1)])
        x = _rest(w, i, x, attn)
    return (_rms(x[:, -1:], w["model.norm.weight"].to(dtype), EPS) @ w["lm_head.weight"].to(dtype).T), caches


def _token_inputs(case, seed):
    """Two tokens for every sequence over caches of 2/3 .. 1 of ``context`` entries, padded on the left."""
    d = _Draw(seed)
    w = _model_weights(d)
    b, n = case["batch"], case["context"]
    length = d.below(max(1, n * 2 // 3), n + 1, b)
    length[0] = n
    kv = []
    for _ in range(2):
        empty = (torch.arange(n, device=DEV)[None] < n - length[:, None])[:, None, :, None]
        kv.append([d.normal(b, HKV, n, D).masked_fill(empty, 0), d.normal(b, HKV, n, D, std=0.5).masked_fill(empty, 0)])
    return w, length, kv, [d.below(0, VOCAB, b, 1) for _ in range(2)], length[:, None] + 5000


def _exact_token(case, seed):
    w, length, kv, ids, pos = _token_inputs(case, seed)
    n = case["context"]
    kv = [[t.to(F64) for t in layer] for layer in kv]
    for t in range(2):
        x = w["model.embed_tokens.weight"][ids[t]].to(F64)
        see = torch.arange(n + t + 1, device=DEV)[None] >= (n - length)[:, None]
        for i in range(2):
            h = _rms(x, w[f"model.layers.{i}.input_layernorm.weight"].to(F64), EPS)
            q, k, v = _heads(w, i, h, pos + t)
            kv[i] = [torch.cat([kv[i][0], k], 2), torch.cat([kv[i][1], v], 2)]
            attn = torch.stack([_look(q[j], kv[i][0][j], kv[i][1][j], see[j][None]) for j in range(case["batch"])])
            x = _rest(w, i, x, attn)
    return {"logits": _rms(x, w["model.norm.weight"].to(F64), EPS) @ w["lm_head.weight"].to(F64).T, "caches": kv}


# ------------------------------------------------------------------------------------------------------------------ layered decoders
def _config(case):
    """Three layers, the upper two looped: five layer runs, two of them attention."""
    width, heads, window = case["width"], case["width"] // 128, case["window"]
    rot = {"base": 10000.0, "dims": 64}
    dense = {"kind": "dense", "ff": 3 * width}
    if case["design"] == "Mutuvik":
        delta = {"type": "delta", "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
        latent = {"type": "latent_attention", "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                                                        "rot": rot, "mask": {"size": window}}}
        moe = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": 3 * width // 4, "limit": 7.0}}
        layers, more = [{**delta, "mlp": dense}, {**latent, "mlp": moe}, {**delta, "mlp": dense}], {}
    else:
        wkv = {"type": "wkv", "mixer": {"heads": width // 64, "dim": 64}}
        att = {"type": "attention", "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "conv": 4, "scale": 128 ** -0.5,
                                              "rot": rot, "mask": {"size": window}}}
        ssd = {"type": "mamba2", "mixer": {"heads": width // 32, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4}}
        layers = [{**wkv, "mlp": dense}, {**att, "mlp": dense}, {**ssd, "mlp": dense}]
        more = {"logit_softcap": 30.0, "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}}}
    return {"architecture": case["design"], "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "layers": layers,
            "loop": {"start": 1, "stop": 3, "times": 2}, **more}


RUNS = [(0, None), (1, 0), (2, 0), (1, 1), (2, 1)]       # (layer, pass) of _config's layers in order of execution


def _layered_weights(d, cfg):
    w, width, par = {}, cfg["width"], cfg["architecture"] == "Nazerax"
    mat = lambda n, r, c: w.__setitem__(n, d.normal(r, c, std=c ** -0.5))
    vec = lambda n, *shape, std=0.1, mean=0.0: w.__setitem__(n, d.normal(*shape, std=std, mean=mean))
    norm = lambda n: vec(n, width, mean=0.0 if par else 1.0)          # the parallel frame stores its norms around zero
    vec("embed", VOCAB, width, std=1.0)
    if par:
        mat("head", VOCAB, width)
        vec("bigram", cfg["embedding"]["bigram"]["buckets"] + 1, width, std=1.0)
    else:
        mat("loop.in", width, 2 * width)
        vec("loop.step", cfg["loop"]["times"], width, std=1.0)
    for i, layer in enumerate(cfg["layers"]):
        p, x, m, kind = f"l{i}.", f"l{i}.mix.", layer["mixer"], layer["type"]
        for n in ("norm1", "norm2"):
            norm(p + n)
        for n in () if par else ("norm1b", "norm2b"):                 # every branch moves the stream a little
            vec(p + n, width, std=0.02, mean=0.2)
        if kind in ("delta", "attention"):
            qk, v = (m["kv_heads"] * m["dim"],) * 2, m["heads"] * m["vdim"]
            if kind == "attention":
                qk, v = (m["heads"] * m["dim"], m["kv_heads"] * m["dim"]), m["kv_heads"] * m["vdim"]
            for n, r in (("q", qk[0]), ("k", qk[1]), ("v", v)):
                mat(x + n, r, width)
                vec(x + n + ".conv", r, m["conv"], std=0.6)
        if kind == "delta":
            mat(x + "g", m["heads"] * m["vdim"], width)
            mat(x + "b", m["heads"], width)
            mat(x + "a", m["heads"], width)
            vec(x + "A_log", m["heads"], std=1.0, mean=-1.0)
            vec(x + "dt_bias", m["heads"], std=1.0)
            vec(x + "norm", m["vdim"], mean=1.0)
        elif kind == "attention":
            mat(x + "g", m["heads"], width)
        elif kind == "latent_attention":
            mat(x + "q", m["heads"] * (m["dim"] + m["rot_dim"]), width)
            mat(x + "dkv", m["kv_rank"] + m["rot_dim"], width)
            vec(x + "dkv.norm", m["kv_rank"], mean=1.0)
            mat(x + "uk", m["heads"] * m["dim"], m["kv_rank"])
            mat(x + "uv", m["heads"] * m["vdim"], m["kv_rank"])
        elif kind == "wkv":
            inner = m["heads"] * m["dim"]
            for n in "rkvgw":
                w[x + "mu." + n] = torch.rand(width, generator=d.g, device=DEV).to(BF16)
            for n in "rkvg":
                mat(x + n, inner, width)
            mat(x + "w1", 64, width)
            mat(x + "w2", inner, 64)
            vec(x + "w0", inner, std=1.0, mean=-2.0)
            vec(x + "u", m["heads"], m["dim"], std=1.0)
            vec(x + "norm", inner, mean=1.0)
        else:
            inner = m["heads"] * m["vdim"]
            chan = inner + 2 * m["groups"] * m["state"]
            mat(x + "in", inner + chan + m["heads"], width)
            vec(x + "conv", chan, m["conv"], std=0.6)
            vec(x + "conv.b", chan, std=0.3)
            vec(x + "dt_bias", m["heads"], std=1.0)
            vec(x + "A_log", m["heads"], std=1.0, mean=-1.0)
            vec(x + "D", m["heads"], std=1.0)
            vec(x + "norm", inner, mean=1.0)
        mat(x + "o", width, m["heads"] * m.get("vdim", m.get("dim")))
        f = layer["mlp"]
        if f["kind"] == "dense":
            for n, r, c in (("gate", f["ff"], width), ("up", f["ff"], width), ("down", width, f["ff"])):
                mat(p + "mlp." + n, r, c)
        else:
            mat(p + "mlp.router", f["router"]["experts"], width)
            vec(p + "mlp.router.b", f["router"]["experts"])
            e_ff = f["expert"]["ff"]
            for e in range(f["router"]["experts"]):
                for n, r, c in (("gate", e_ff, width), ("up", e_ff, width), ("down", width, e_ff)):
                    mat(f"{p}mlp.e{e}.{n}", r, c)
    norm("final.norm")
    return w


def _channels(kind, m):
    if kind == "mamba2":
        return m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
    if kind == "delta":
        return 2 * m["kv_heads"] * m["dim"] + m["heads"] * m["vdim"]
    return (m["heads"] + m["kv_heads"]) * m["dim"] + m["kv_heads"] * m["vdim"] if kind == "attention" else 0


def _past(d, cfg, slots):
    """What the sequences left behind: per layer run its ring or matrix, convolution inputs and previous row."""
    runs = []
    for i, _ in RUNS:
        kind, m = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"]
        s, chan = {}, _channels(kind, m)
        if kind in ("latent_attention", "attention"):
            row = m["kv_rank"] + m["rot_dim"] if kind == "latent_attention" else m["kv_heads"] * (m["dim"] + m["vdim"])
            s["ring"] = d.normal(slots, m["mask"]["size"], row)
        else:
            s["state"] = d.normal(slots, m["heads"], m.get("state", m.get("dim")), m.get("vdim", m.get("dim")), std=0.1, dtype=F32)
        if chan:
            s["conv"] = d.normal(slots, m["conv"] - 1, chan)
        if kind == "wkv":
            s["shift"] = d.normal(slots, cfg["width"])
        runs.append(s)
    return runs, d.below(0, VOCAB, slots)


def _layered_inputs(case, seed):
    """(config, weights, past, previous tokens, [(tokens, positions before them)]): decode tokens first, each past its window."""
    d, cfg = _Draw(seed), _config(case)
    w = _layered_weights(d, cfg)
    window, n_dec = case["window"], case.get("batch", case.get("decode", 0))
    lens = [1] * n_dec + [int(x) for x in case.get("portions", "").split(",") if x]
    past, last = _past(d, cfg, len(lens))
    ahead = d.below(0, 3000, max(n_dec, 1)).tolist()
    ids = d.below(0, VOCAB, sum(lens)).tolist()
    seqs, at = [], 0
    for i, n in enumerate(lens):
        seqs.append((ids[at:at + n], window + 3 + ahead[i] if i < n_dec else case["past"]))
        at += n
    return cfg, w, past, last, seqs


def _conv(x, before, taps, bias=None):
    """x [n, channels] behind its ``before`` [taps - 1, channels]."""
    x, n = torch.cat([before, x]), x.shape[0]
    y = sum(x[j:j + n] * taps[:, j] for j in range(taps.shape[1]))
    return y if bias is None else y + bias


def _turn_pairs(x, pos, base):
    """x [n, ..., dims]: neighbours form the planes."""
    dims = x.shape[-1]
    ang = pos.to(F64)[:, None] * base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEV) / dims)
    ang = ang.view([x.shape[0]] + [1] * (x.dim() - 2) + [dims // 2])
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).flatten(-2)


def _seen(ring, rows, p0, n, window):
    """The rows a portion's queries may look at (those before it from the ring) and the mask; the ring takes the new rows."""
    old = torch.arange(max(0, p0 - window + 1), p0, device=DEV)
    keys = torch.cat([ring[old % ring.shape[0]], rows])
    at = torch.cat([old, torch.arange(p0, p0 + n, device=DEV)])
    back = torch.arange(p0, p0 + n, device=DEV)[:, None] - at[None]
    new = torch.arange(max(p0, p0 + n - ring.shape[0]), p0 + n, device=DEV)
    ring[new % ring.shape[0]] = rows[new - p0]
    return keys, (back >= 0) & (back < window)


def _latent_mixer(h, w, m, s, j, p0, eps):
    n, heads, dim, rank, base = h.shape[0], m["heads"], m["dim"], m["kv_rank"], m["rot"]["base"]
    pos = torch.arange(p0, p0 + n, device=DEV)
    q = (h @ w["q"].T).view(n, heads, -1)
    down = h @ w["dkv"].T
    rows = torch.cat([_rms(down[:, :rank], w["dkv.norm"], eps), _turn_pairs(down[:, rank:], pos, base)], 1)
    keys, see = _seen(s["ring"][j], rows, p0, n, m["mask"]["size"])
    k, v = (keys[:, :rank] @ w["uk"].T).view(-1, heads, dim), (keys[:, :rank] @ w["uv"].T).view(-1, heads, m["vdim"])
    qr, out = _turn_pairs(q[..., dim:], pos, base), []
    for i in range(heads):
        z = (q[:, i, :dim] @ k[:, i].T + qr[:, i] @ keys[:, rank:].T) * m["scale"]
        out.append(torch.softmax(z.masked_fill(~see, -torch.inf), -1) @ v[:, i])
    return torch.cat(out, 1) @ w["o"].T


def _grouped_mixer(h, w, m, s, j, p0, eps):
    n, heads, groups, dim, dims = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["rot"]["dims"]
    pos = torch.arange(p0, p0 + n, device=DEV)
    before = (s["conv"][j] if p0 else torch.zeros_like(s["conv"][j])).split([heads * dim, groups * dim, groups * m["vdim"]], 1)
    q, k, v = (_conv(h @ w[x].T, b, w[x + ".conv"]) for x, b in zip("qkv", before))
    turn = lambda t: torch.cat([_turn_pairs(t[..., :dims], pos, m["rot"]["base"]), t[..., dims:]], -1)
    q, k = turn(q.view(n, heads, dim)), turn(k.view(n, groups, dim)).reshape(n, -1)
    keys, see = _seen(s["ring"][j], torch.cat([k, v], 1), p0, n, m["mask"]["size"])
    k, v, out = keys[:, :groups * dim].view(-1, groups, dim), keys[:, groups * dim:].view(-1, groups, m["vdim"]), []
    gate = torch.sigmoid(h @ w["g"].T)
    for i in range(heads):
        z = (q[:, i] @ k[:, i * groups // heads].T * m["scale"]).masked_fill(~see, -torch.inf)
        z = torch.softmax(torch.cat([z, z.new_zeros(n, 1)], 1), -1)[:, :-1]           # a silent entry of score 0
        out.append(z @ v[:, i * groups // heads] * gate[:, i:i + 1])
    return torch.cat(out, 1) @ w["o"].T


def _delta_mixer(h, w, m, s, j, p0, eps):
    n, heads, groups, dim, vdim = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    before = (s["conv"][j] if p0 else torch.zeros_like(s["conv"][j])).split([groups * dim, groups * dim, heads * vdim], 1)
    q, k, v = (F.silu(_conv(h @ w[x].T, b, w[x + ".conv"])) for x, b in zip("qkv", before))
    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(t.view(n, groups, dim)).repeat_interleave(heads // groups, 1) for t in (q, k))
    q, v = q * dim ** -0.5, v.view(n, heads, vdim)
    beta = torch.sigmoid(h @ w["b"].T)[:, :, None]
    g = torch.exp(-torch.exp(w["A_log"]) * F.softplus(h @ w["a"].T + w["dt_bias"]))[:, :, None, None]
    st, out = s["state"][j] if p0 else torch.zeros_like(s["state"][j]), []
    for t in range(n):
        st = st * g[t]
        u = beta[t] * (v[t] - (k[t][:, None] @ st)[:, 0])
        st = st + k[t][:, :, None] * u[:, None]
        out.append((q[t][:, None] @ st)[:, 0])
    s["state"][j] = st
    o = _rms(torch.stack(out), w["norm"], eps) * F.silu(h @ w["g"].T).view(n, heads, vdim)
    return o.reshape(n, -1) @ w["o"].T


def _wkv_mixer(h, w, m, s, j, p0, eps):
    n, heads, dim = h.shape[0], m["heads"], m["dim"]
    first = s["shift"][j][None] if p0 else torch.zeros_like(h[:1])
    back = torch.cat([first, h[:-1]]) - h
    mix = {x: h + back * w["mu." + x] for x in "rkvgw"}
    r, k, v = ((mix[x] @ w[x].T).view(n, heads, dim) for x in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"])).view(n, heads, dim, 1)
    st, out = s["state"][j] if p0 else torch.zeros_like(s["state"][j]), []
    for t in range(n):
        kv = k[t][:, :, None] * v[t][:, None]
        out.append((r[t][:, None] @ (st + w["u"][:, :, None] * kv))[:, 0])
        st = st * decay[t] + kv
    s["state"][j] = st
    o = _rms(torch.stack(out), None, eps).reshape(n, -1) * w["norm"]
    return (o * F.silu(mix["g"] @ w["g"].T)) @ w["o"].T


def _ssd_mixer(h, w, m, s, j, p0, eps):
    n, heads, vdim, ns, groups = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = heads * vdim
    z, xbc, dt = torch.split(h @ w["in"].T, [inner, inner + 2 * groups * ns, heads], 1)
    xbc = F.silu(_conv(xbc, s["conv"][j] if p0 else torch.zeros_like(s["conv"][j]), w["conv"], w["conv.b"]))
    x, b, c = torch.split(xbc, [inner, groups * ns, groups * ns], 1)
    x = x.reshape(n, heads, vdim)
    b, c = (t.reshape(n, groups, ns).repeat_interleave(heads // groups, 1) for t in (b, c))
    step = F.softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * step)[:, :, None, None]
    st, out = s["state"][j] if p0 else torch.zeros_like(s["state"][j]), []
    for t in range(n):
        st = st * decay[t] + (b[t] * step[t][:, None])[:, :, None] * x[t][:, None]
        out.append((c[t][:, None] @ st)[:, 0])
    s["state"][j] = st
    y = (torch.stack(out) + w["D"][:, None] * x).reshape(n, inner) * F.silu(z)
    return (_rms(y.view(n, m["norm_groups"], -1), None, eps).view(n, -1) * w["norm"]) @ w["o"].T


def _feed(h, w, spec):
    if spec["kind"] == "dense":
        return (F.silu(h @ w["gate"].T) * (h @ w["up"].T)) @ w["down"].T
    top, limit, out = spec["router"]["top"], spec["expert"]["limit"], torch.zeros_like(h)
    z, idx = torch.topk(h @ w["router"].T + w["router.b"], top, dim=-1)
    mix = torch.softmax(z, -1)
    for e in range(spec["router"]["experts"]):
        row, k = torch.nonzero(idx == e, as_tuple=True)
        if row.numel():
            g = torch.clamp(h[row] @ w[f"e{e}.gate"].T, max=limit)
            u = torch.clamp(h[row] @ w[f"e{e}.up"].T, -limit, limit)
            out[row] += mix[row, k][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[f"e{e}.down"].T)
    return out


MIXERS = {"latent_attention": _latent_mixer, "attention": _grouped_mixer, "delta": _delta_mixer, "wkv": _wkv_mixer, "mamba2": _ssd_mixer}


def _exact_layered(case, seed):
    cfg, w, past, last, seqs = _layered_inputs(case, seed)
    eps, par = cfg["norm"]["eps"], cfg["architecture"] == "Nazerax"
    for s in past:
        for k in s:
            s[k] = s[k].to(F64)
    sub = lambda p: {k[len(p):]: t.to(F64) for k, t in w.items() if k.startswith(p)}
    norm = lambda x, name: _rms(x, w[name].to(F64) + (1.0 if par else 0.0), eps)
    ids = torch.tensor([t for toks, _ in seqs for t in toks], device=DEV)
    cut = [0]
    for toks, _ in seqs:
        cut.append(cut[-1] + len(toks))
    x = w["embed"][ids].to(F64)
    if par:
        pair = cfg["embedding"]["bigram"]
        rows = []
        for j, (toks, p0) in enumerate(seqs):
            before = [int(last[j]) if p0 else None] + toks[:-1]
            rows += [pair["buckets"] if a is None else (a * pair["mul_prev"] + b * pair["mul_cur"]) % pair["buckets"] for a, b in zip(before, toks)]
        x = x + w["bigram"][torch.tensor(rows, device=DEV)].to(F64)
    x0 = x
    for run, (i, t) in enumerate(RUNS):
        layer, p = cfg["layers"][i], f"l{i}."
        if t is not None and i == cfg["loop"]["start"]:
            if not par:
                x = torch.cat([x, x0], 1) @ w["loop.in"].to(F64).T + w["loop.step"][t].to(F64)
            elif t:
                x = x + x0
        wm, h = sub(p + "mix."), norm(x, p + "norm1")
        mixed = torch.cat([MIXERS[layer["type"]](h[cut[j]:cut[j + 1]], wm, layer["mixer"], past[run], j, p0, eps)
                           for j, (_, p0) in enumerate(seqs)])
        del wm
        wf = sub(p + "mlp.")
        if par:
            x = x + mixed + _feed(norm(x, p + "norm2"), wf, layer["mlp"])
        else:
            x = x + norm(mixed, p + "norm1b")
            x = x + norm(_feed(norm(x, p + "norm2"), wf, layer["mlp"]), p + "norm2b")
    z = norm(x[torch.tensor(cut[1:], device=DEV) - 1], "final.norm") @ w["head" if par else "embed"].to(F64).T
    if par:
        z = cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
    return {"logits": z, "ring": [s["ring"] for s in past if "ring" in s], "state": [s["state"] for s in past if "state" in s]}


def _prepare_layered(case, seed):
    from msa_b200.hybrid import GraphedDecode, HybridForCausalLM
    from msa_b200.hybrid_config import HybridConfig
    cfg, w, past, last, seqs = _layered_inputs(case, seed)
    model = HybridForCausalLM(HybridConfig.parse(cfg), w, DEV, BF16)
    del w
    n = len(seqs)
    cache = model.new_cache(n, 1 << 20)          # every ring is as long as the window
    graph = GraphedDecode(model, cache, n) if case["kind"] == "tokens" else None
    p0 = torch.tensor([p for _, p in seqs], device=DEV)
    for run, s in enumerate(past):
        for name, t in s.items():
            if name == "conv":                   # the inputs before position p are kept in half p & 1
                cache.conv[run][torch.arange(n, device=DEV), p0 & 1] = t
            else:
                getattr(cache, name)[run][:n] = t
    cache.last_token[:n] = last
    return dict(kind=case["kind"], model=model, cache=cache, graph=graph, seqs=seqs, n=n, pos=[p for _, p in seqs])


def _run_layered(s):
    cache, n = s["cache"], s["n"]
    if s["kind"] == "tokens":                    # a decode loop: every pass is the next position
        logits = s["graph"].run([toks[0] for toks, _ in s["seqs"]], s["pos"], range(n))
        s["pos"] = [p + 1 for p in s["pos"]]
    else:                                        # the sequences come anew, in the same slots
        for j in reversed(range(n)):
            if j in cache:
                cache.release(j)
        for j, (_, p0) in enumerate(s["seqs"]):
            cache.acquire(j)
            cache.advance(j, p0)
        logits = s["model"].run([(j, toks, [len(toks) - 1]) for j, (toks, _) in enumerate(s["seqs"])], cache)
    return {"logits": logits, "ring": [t[:n] for t in cache.ring.values()], "state": [t[:n] for t in cache.state.values()],
            "shift": [t[:n] for t in cache.shift.values()]}


# ------------------------------------------------------------------------------------------------------------------ the contract
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "tokens"):
        return _prepare_layered(case, seed)
    if kind in ("query", "route"):
        q, mask, lens, rk, k, v = _query_inputs(case, seed)
        svc = _service(lens, rk, k, v, 1, 0, rk.dtype)
        if kind == "route":
            svc.block_router_keys()
        return dict(kind=kind, svc=svc, q=q, mask=mask)
    if kind == "block":
        d, _, ids, doc, pos = _block_inputs(case, seed)
        return dict(kind=kind, model=_model(_model_weights(d)), ids=ids, doc=doc, pos=pos, mask=torch.ones_like(ids))
    if kind == "question":
        w, ids, mask, pos, prefix, lens, rk, k, v = _question_inputs(case, seed)
        model, svc = _model(w), _service(lens, rk, k, v, 2, 1, BF16)
        svc.template_prefix_kvcache = prefix
        svc.setup_memory_client(model)
        return dict(kind=kind, model=model, svc=svc, ids=ids, mask=mask, pos=pos, doc=torch.where(mask == 1, 0, -1))
    from msa_b200.cache import SparseCache
    w, length, kv, ids, pos = _token_inputs(case, seed)
    s = dict(kind=kind, model=_model(w), cache=SparseCache(), ids=ids[0], pos=pos, n=case["context"] + 2)
    s.update(doc=torch.full_like(ids[0], -1), mask=torch.ones_like(ids[0]))
    for i in range(2):
        s["cache"].record_kwargs(i, {"stage": "generate", "compacked_key_cache": kv[i][0], "compacked_value_cache": kv[i][1],
                                     "kv_lengths": length.clone()})
    s["at"] = {}
    _run_token(s)                                # the first token moves the caches to storage with room behind them
    s.update(at={i: dict(s["cache"].cache_kwargs[i]) for i in range(2)}, ids=ids[1], pos=pos + 1)
    return s


def _run_token(s):
    for i, kw in s["at"].items():
        s["cache"].cache_kwargs[i] = dict(kw)    # every pass continues the same prefix
    out = s["model"](input_ids=s["ids"], attention_mask=s["mask"], position_ids=s["pos"], past_key_values=s["cache"], doc_ids=s["doc"])
    kw = s["cache"].cache_kwargs
    return {"logits": out.logits, "caches": [[kw[i]["compacked_key_cache"], kw[i]["compacked_value_cache"]] for i in range(2)]}


def run(state):
    with torch.no_grad():
        return _run(state)


def _run(s):
    kind = s["kind"]
    if kind in ("step", "tokens"):
        return _run_layered(s)
    if kind == "query":
        k, v, scores, n_sel, ids = s["svc"].doc_query(s["q"], s["mask"], 0)
        return {"k": k, "v": v, "scores": scores, "n_sel": n_sel, "ids": ids}
    if kind == "route":
        scores, local, ids, rank = s["svc"].route(s["q"], s["mask"], 0, l2_normalize=True, all_valid=True)
        return {"scores": scores, "local": local, "ids": ids, "rank": rank}
    if kind == "token":
        return _run_token(s)
    from msa_b200.cache import SparseCache
    cache = SparseCache()
    for i in range(2):
        cache.record_kwargs(i, {"stage": "prefill_stage1" if kind == "block" else "prefill_stage2"})
    if kind == "block":
        out = s["model"].model(input_ids=s["ids"], attention_mask=s["mask"], position_ids=s["pos"], past_key_values=cache, doc_ids=s["doc"])
        kw = cache.cache_kwargs
        return {"hidden": out.last_hidden_state, "pooled": [*cache.get_kvcache(1), cache.get_router_kcache(1)],
                **{f"template_{i}": [kw[i]["template_prefix_kcache"], kw[i]["template_prefix_vcache"]] for i in range(2)},
                "doc_ids": kw[1]["pooled_doc_ids"]}
    out = s["model"](input_ids=s["ids"], attention_mask=s["mask"], position_ids=s["pos"], past_key_values=cache, doc_ids=s["doc"], logits_to_keep=1)
    kw = cache.cache_kwargs
    return {"logits": out.logits, "caches": [[kw[i]["compacked_key_cache"], kw[i]["compacked_value_cache"]] for i in range(2)],
            "lengths": [kw[i]["kv_lengths"] for i in range(2)]}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("step", "tokens"):
            return _exact_layered(case, seed)
        if kind in ("query", "route"):
            q, mask, lens, rk, k, v = _query_inputs(case, seed)
            q = q.to(F64) if kind == "query" else F.normalize(q.to(F64), dim=-1)
            b, s = mask.shape
            folded = q.view(b, HKV, HQ // HKV, s, D).sum(2).permute(0, 2, 1, 3).reshape(b, s, -1)
            score, at = _routed(folded, mask, lens, rk, TOP_K)
            if kind == "route":
                return {"scores": score, "local": None, "ids": None, "rank": None}
            rows = torch.cat(_rows_of(at, lens))
            return {"k": k[rows].transpose(0, 1).to(F64), "v": v[rows].transpose(0, 1).to(F64), "scores": score, "n_sel": None, "ids": None}
        if kind == "block":
            return {**_exact_block(case, seed), "doc_ids": None}
        if kind == "question":
            w, ids, mask, pos, prefix, *bank = _question_inputs(case, seed)
            logits, caches = _ask(w, ids, mask, pos, prefix, F64, bank)
            return {"logits": logits, "caches": caches, "lengths": [None, None]}
        return _exact_token(case, seed)


def _layered_work(case):
    cfg = _config(case)
    lens = [1] * case.get("batch", case.get("decode", 0)) + [int(x) for x in case.get("portions", "").split(",") if x]
    n, seqs, width, window = sum(lens), len(lens), cfg["width"], case["window"]
    flops = bytes_ = 0.0
    weights, active = VOCAB * width, 0.0
    for i, t in RUNS:
        kind, m, f = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"]
        first = not t
        if f["kind"] == "dense":
            used = held = 3 * width * f["ff"]
        else:
            one = 3 * width * f["expert"]["ff"]
            used = one * f["router"]["top"]
            held = one * min(f["router"]["experts"], n * f["router"]["top"])
        inner = m["heads"] * m.get("vdim", m.get("dim"))
        if kind == "latent_attention":
            mix = width * (m["heads"] * 192 + 576 + inner)
            row, pair, ctx = 576, 2 * m["heads"] * (192 + 128), 2 * 512 * m["heads"] * 256
        elif kind == "attention":
            mix = width * (_channels(kind, m) + m["heads"] + inner)
            row, pair, ctx = m["kv_heads"] * 256, 2 * m["heads"] * 256, 0
        else:
            mix = width * inner + width * (_channels(kind, m) + inner if kind != "wkv" else 4 * inner)
            state = m["heads"] * m.get("state", m.get("dim")) * m.get("vdim", m.get("dim"))
            flops += 6.0 * n * state
            bytes_ += 8.0 * seqs * state
        if kind in ("latent_attention", "attention"):
            for j, length in enumerate(lens):
                p0 = window if j < seqs - len([x for x in lens if x > 1]) or length == 1 else case.get("past", 0)
                old = min(p0, window - 1)
                flops += pair * sum(min(old + t_ + 1, window) for t_ in range(length)) + ctx * (old + length if length > 1 else 0)
                bytes_ += 2.0 * row * (old + min(length, window))
        active += mix + used
        if first:
            weights += mix + held
    flops += 2.0 * n * active + 2.0 * seqs * VOCAB * width
    bytes_ += 2.0 * weights + 2.0 * n * width + 4.0 * seqs * VOCAB
    return {"bytes": bytes_, "flops": flops}


def work(case):
    """Bytes and operations of one pass that no implementation can do without: weights, bank and state once, products of the
    tokens that are there, pairs that see each other.  Fetched documents count as one read and one write; they come over PCIe."""
    kind = case["kind"]
    if kind in ("step", "tokens"):
        return _layered_work(case)
    row = HKV * D
    per_layer = HIDDEN * (2 * HQ * D + 2 * row) + 3 * HIDDEN * FFN
    if kind in ("query", "route"):
        e = 4 if case.get("dtype") == "float32" else 2
        c = case["docs"] * case["chunks"]
        tokens = case["batch"] * max(1, 0.75 * case.get("tokens", 1))
        fetched = 0 if kind == "route" else case["batch"] * TOP_K * case["chunks"] * 2 * row * e * 2
        return {"bytes": c * row * e + tokens * HQ * D * e + fetched, "flops": 2.0 * tokens * c * row}
    if kind == "block":
        n, length = case["docs"] * case["doc_tokens"], case["doc_tokens"]
        flops = 2.0 * n * (2 * per_layer + HIDDEN * row) + 2 * n * (length * 13 / 12) / 2 * 4 * HQ * D
        return {"bytes": 2.0 * (2 * per_layer + n * HIDDEN * 2 + n / POOL * 3 * row), "flops": flops}
    if kind == "question":
        n, found = 0.75 * case["batch"] * case["tokens"], TOP_K * case["chunks"]
        c = case["docs"] * case["chunks"]
        flops = 2.0 * n * (2 * per_layer + HIDDEN * HQ * D + c * row) + n * (found + 0.75 * case["tokens"]) * 4 * HQ * D
        flops += 2.0 * case["batch"] * HIDDEN * VOCAB
        return {"bytes": 2.0 * (2 * per_layer + HIDDEN * HQ * D + VOCAB * HIDDEN + c * row + case["batch"] * found * 4 * row), "flops": flops}
    n = case["batch"] * case["context"] * 5 / 6
    return {"bytes": 2.0 * (2 * per_layer + VOCAB * HIDDEN + 2 * n * 2 * row), "flops": 2.0 * case["batch"] * (2 * per_layer + VOCAB * HIDDEN) + 2 * n * 4 * HQ * D}
