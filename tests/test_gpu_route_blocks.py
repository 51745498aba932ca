"""Routing over the 16-row blocks that hold valid tokens (CTA pairs) against the CUDA-core kernel over all rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def masks(kind, b, s, g):
    m = torch.ones(b, s, dtype=torch.bool)
    if kind == "left":                                    # questions padded on the left, as the engine's
        first = torch.randint(0, s, (b,), generator=g)
        m = torch.arange(s)[None] >= first[:, None]
    elif kind == "holes":
        m = torch.rand(b, s, generator=g) < 0.1
        m[::3] = False                                    # questions without a token
    elif kind == "none":
        m[:] = False
    return m


# (questions, tokens): one column tile and its remainders, 17 blocks, sequences cut over tiles, more than one list round
@pytest.mark.parametrize("kind", ["full", "left", "holes", "none"])
@pytest.mark.parametrize("b,s", [(1, 256), (17, 16), (5, 200), (3, 500), (33, 33), (130, 130)])
def test_live_blocks_match_the_cuda_core_kernel(b, s, kind):
    from msa_b200 import _cabi as A, ops
    g = torch.Generator().manual_seed(b * 1000 + s)
    hkv, d, groups = 2, 64, 2
    tiles = -(-2 * 148 // max(1, b * ops.route_s_pad(s) // 256))          # enough chunk tiles for the pair kernel
    lens = torch.randint(1, 40, (tiles * 128 // 20 + 8,), generator=g)
    doc = torch.repeat_interleave(torch.arange(1, lens.numel() + 1), lens).to(torch.int32)
    doc = doc[:tiles * 128 - 7].to(DEV)
    n_docs, c = int(doc.max()), doc.numel()
    rk = torch.randn(c, hkv * d, generator=g).to(torch.bfloat16).to(DEV)
    q = torch.randn(b, hkv * groups, s, d, generator=g).to(torch.bfloat16).to(DEV)
    mask = masks(kind, b, s, g).to(DEV)
    qf, bias, s_pad = ops.fold_queries(q, mask, groups)
    kw = dict(n_seq=b, s_pad=s_pad, rk=rk, chunk_doc=doc, n_docs=n_docs, alpha=0.25)
    got, status = ops.route_scores(qf, bias, **kw)
    want, _ = ops.route_scores(qf, bias, flags=A.ROUTE_FORCE_SIMT, **kw)
    assert status.tolist() == [0, 0, 0, 0]
    got, want = ops.keys_to_scores(got), ops.keys_to_scores(want)
    # fp32 sums of 128 products of size ~2 in another order: 128 * 2^-24 of the sum of their sizes at most, times alpha
    assert torch.allclose(got, want, rtol=0, atol=0.25 * 128 * 2 ** -24 * 128 * 2)
    if kind == "none":
        assert (got == torch.finfo(torch.bfloat16).min).all()
