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


def bank(b, s, g, hkv, d):
    """Documents over chunk tiles enough for the pair kernel: two 128-chunk tiles per SM and 256 rows."""
    from msa_b200 import _cabi as A, ops
    n_sm, s_pad = torch.cuda.get_device_properties(0).multi_processor_count, ops.route_s_pad(s)
    tiles = -(-2 * n_sm // -(-b * s_pad // 256))
    c = tiles * 128 - 7
    lens = torch.randint(1, 40, (c,), generator=g)
    doc = torch.repeat_interleave(torch.arange(1, c + 1), lens)[:c].to(torch.int32).to(DEV)
    assert A.lib().msa_route_live_rows(b, s_pad, c) == b * s_pad and A.lib().msa_route_live_rows(b, s_pad, (tiles - 1) * 128) == 0
    return doc, torch.randn(c, hkv * d, generator=g).to(torch.bfloat16).to(DEV)


# (questions, tokens): one column tile and its remainders, 17 blocks, sequences cut over tiles, more than one list round
@pytest.mark.parametrize("kind", ["full", "left", "holes", "none"])
@pytest.mark.parametrize("b,s", [(1, 256), (17, 16), (5, 200), (3, 500), (33, 33), (130, 130)])
def test_live_blocks_match_the_cuda_core_kernel(b, s, kind):
    from msa_b200 import _cabi as A, ops
    g = torch.Generator().manual_seed(b * 1000 + s)
    hkv, d, groups = 2, 64, 2
    doc, rk = bank(b, s, g, hkv, d)
    n_docs, c = int(doc.max()), doc.numel()
    q = torch.randn(b, hkv * groups, s, d, generator=g).to(torch.bfloat16).to(DEV)
    mask = masks(kind, b, s, g).to(DEV)
    qf, bias, s_pad = ops.fold_queries(q, mask, groups)
    kw = dict(n_seq=b, s_pad=s_pad, rk=rk, chunk_doc=doc, n_docs=n_docs, alpha=0.25)
    table, status = ops.route_scores(qf, bias, **kw)
    want, _ = ops.route_scores(qf, bias, flags=A.ROUTE_FORCE_SIMT, **kw)
    assert status.tolist() == [0, 0, 0, 0]
    got, want = ops.keys_to_scores(table), ops.keys_to_scores(want)
    # fp32 sums of 128 products of size ~2 in another order: 128 * 2^-24 of the sum of their sizes at most, times alpha
    assert torch.allclose(got, want, rtol=0, atol=0.25 * 128 * 2 ** -24 * 128 * 2)
    if kind == "none":
        assert (got == torch.finfo(torch.bfloat16).min).all()
    # the same call with scratch that can be looked at: the list, and the rows behind it (none where every block is listed)
    blocks = b * s_pad // 16
    live, packed = torch.full((blocks + 1,), -5, dtype=torch.int32, device=DEV), torch.full_like(qf, 7)
    keys, status = torch.empty_like(table), torch.zeros(4, dtype=torch.int32, device=DEV)
    A.check(A.lib().msa_route_scores_live(A.ptr(qf), A.ptr(bias), A.dtype_code(rk.dtype), b, s_pad, A.ptr(rk), rk.stride(0), c, hkv * d, A.ptr(doc),
                                          0.25, A.ptr(keys), keys.stride(0), n_docs, torch.finfo(rk.dtype).min, 0, A.ptr(status), A.ptr(live),
                                          A.ptr(packed), A.stream_ptr(qf.device)), "msa_route_scores_live")
    listed = torch.nonzero((bias.view(blocks, 16) > -float("inf")).any(1)).flatten()
    n = listed.numel()
    assert torch.equal(keys, table) and live[0] == n and live[1:n + 1].tolist() == listed.tolist() and (live[n + 1:] == -5).all()
    assert n == blocks if kind == "full" and s_pad - s < 16 else n < blocks or kind == "left"
    rows = packed.view(blocks, 16, -1)
    if n == blocks:
        assert (packed == 7).all()
    else:
        assert torch.equal(rows[:n], qf.view(blocks, 16, -1)[listed]) and (rows[n:] == 7).all()


def test_scratch_is_asked_for_where_it_is_used():
    from msa_b200 import _cabi as A
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    ask = A.lib().msa_route_live_rows
    assert ask(128, 1, 1 << 20) == 0 and ask(4, 64, 128 * (2 * n_sm - 1)) == 0 and ask(0, 64, 1 << 20) == 0 and ask(4, 64, 0) == 0
    assert ask(4, 64, 128 * (2 * n_sm - 1) + 1) == 256 and ask(48, 208, 128 * 2 * n_sm // 39 + 128) == 48 * 208
