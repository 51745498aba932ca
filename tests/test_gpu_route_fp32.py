"""Routing in fp32 (``route_fp32_kernel``: 16-row blocks, 64 chunks, 32 k a step) at the edges of its tiles, against fp64 torch, and the
forms it leaves to the general kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def setting(b, s, hkv, d, chunks, kind, pad=0):
    g = torch.Generator().manual_seed(b * 1000 + s + chunks)
    doc = torch.repeat_interleave(torch.arange(1, chunks + 1), torch.randint(1, 6, (chunks,), generator=g))[:chunks].to(torch.int32)
    rk = torch.randn(chunks, hkv * d, generator=g)
    q = torch.randn(b, 2 * hkv, s, d, generator=g)
    mask = torch.ones(b, s, dtype=torch.bool)
    if kind == "left":
        mask = torch.arange(s)[None] >= torch.randint(0, s, (b,), generator=g)[:, None]
    elif kind == "holes":
        mask = torch.rand(b, s, generator=g) < 0.1
        mask[::2] = False
    wide = torch.zeros(chunks, hkv * d + pad, device=DEV)
    wide[:, :hkv * d] = rk.to(DEV)
    return q, mask, doc, rk, wide[:, :hkv * d]


def scores(q, mask, doc, rk, alpha):
    b, h, s, d = q.shape
    folded = q.double().view(b, h // 2, 2, s, d).sum(2).permute(0, 2, 1, 3).reshape(b, s, -1)
    z = (folded @ rk.double().t() * alpha).masked_fill(~mask[:, :, None], -float("inf")).amax(1)
    n = int(doc.max())
    out = torch.full((b, n + 1), torch.finfo(torch.float32).min, dtype=torch.float64)
    return out.scatter_reduce(1, doc.long().expand(b, -1), z, "amax")


@pytest.mark.parametrize("kind", ["full", "left", "holes"])
@pytest.mark.parametrize("b,s,hkv,d,chunks", [(1, 2, 2, 64, 1), (1, 16, 2, 64, 63), (1, 64, 8, 128, 65), (3, 70, 2, 64, 200), (4, 200, 2, 128, 1000),
                                              (1, 129, 9, 4, 64), (9, 16, 3, 16, 130), (2, 300, 2, 64, 129)])
def test_fp32_routing(b, s, hkv, d, chunks, kind):
    from msa_b200 import ops
    q, mask, doc, rk, dev = setting(b, s, hkv, d, chunks, kind)
    qf, bias, s_pad = ops.fold_queries(q.to(DEV), mask.to(DEV), 2)
    assert s_pad % 16 == 0
    keys, status = ops.route_scores(qf, bias, b, s_pad, dev, doc.to(DEV), int(doc.max()), 0.25)
    want = scores(q, mask, doc, rk, 0.25)
    got = ops.keys_to_scores(keys).cpu().double()
    assert status.tolist() == [0, 0, 0, 0]
    # K products of about 1.4 in fp32: each addition is off by 2^-24 of a partial sum below 8 sqrt(K); times alpha
    k = hkv * d
    assert torch.allclose(got, want, rtol=1e-6, atol=0.25 * k * 2.0 ** -24 * 8 * k ** 0.5)


def test_forms_of_the_general_kernel_and_ids_out_of_range():
    """Rows off the 16-byte boundary and one row per sequence go through the general kernel, with the same scores; chunk ids
    outside the table are counted and skipped by both."""
    from msa_b200 import ops
    q, mask, doc, rk, dev = setting(2, 40, 2, 64, 150, "left")
    shifted = setting(2, 40, 2, 64, 150, "left", pad=1)[4]
    qf, bias, s_pad = ops.fold_queries(q.to(DEV), mask.to(DEV), 2)
    want = scores(q, mask, doc, rk, 0.25)
    for bank in (dev, shifted):
        bad = doc.clone()
        bad[3], bad[149] = 0, int(doc.max()) + 1
        for ids, n_bad in ((doc, 0), (bad, 4)):                           # two sequences, two ids each; a tile counts its own
            keys, status = ops.route_scores(qf, bias, 2, s_pad, bank, ids.to(DEV), int(doc.max()), 0.25)
            assert status[2] >= n_bad and bool(status[2]) == bool(n_bad) and not status[[0, 1, 3]].any()
            if n_bad == 0:
                assert torch.allclose(ops.keys_to_scores(keys).cpu().double(), want, rtol=1e-6, atol=1e-4)
    one, ones = q[:, :, :1], torch.ones(2, 1, dtype=torch.bool)
    qf, bias, s_pad = ops.fold_queries(one.to(DEV), ones.to(DEV), 2)
    keys, _ = ops.route_scores(qf, bias, 2, s_pad, dev, doc.to(DEV), int(doc.max()), 0.25)
    assert s_pad == 1 and torch.allclose(ops.keys_to_scores(keys).cpu().double(), scores(one, ones, doc, rk, 0.25), rtol=1e-6, atol=1e-4)
