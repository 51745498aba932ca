"""The winners of a single rank written by the selection itself, against selection and merge."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n_seq,n_cols,k", [(1, 5, 16), (3, 700, 16), (32, 24415, 16), (2, 9000, 64), (4, 6000, 100), (2, 3, 200), (5, 2049, 1)])
def test_selection_writes_the_winners(n_seq, n_cols, k):
    from msa_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n_cols + k)
    score = torch.randn(n_seq, n_cols, generator=g, device=DEV)
    score = torch.where(torch.rand(score.shape, generator=g, device=DEV) < 0.3, score.round(), score)          # ties
    score[:, n_cols // 3:] = torch.where(torch.rand(score[:, n_cols // 3:].shape, generator=g, device=DEV) < 0.9, torch.tensor(-3e38, device=DEV),
                                         score[:, n_cols // 3:])                                               # documents nobody scored
    bits = score.view(torch.int32)
    keys = torch.where(bits < 0, ~bits, bits | -2 ** 31).contiguous()
    ids = torch.randint(0, 10 ** 12, (n_cols,), generator=g, device=DEV)
    sc, li, gi = ops.topk_select(keys, k, ids)
    want = ops.topk_merge(sc.unsqueeze(0), li.unsqueeze(0), gi.unsqueeze(0), k)
    got = ops.topk_select(keys, k, ids, winners=True)
    assert all(a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("n_seq,docs,k", [(1, 4, 16), (7, 40, 16), (33, 900, 32)])
def test_routing_of_single_tokens_writes_the_winners(n_seq, docs, k):
    from msa_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(docs)
    chunk_doc = torch.repeat_interleave(torch.arange(1, docs + 1, device=DEV), torch.randint(1, 5, (docs,), generator=g, device=DEV)).int()
    rk = torch.randn(chunk_doc.numel(), 128, generator=g, device=DEV).to(torch.bfloat16)
    q, bias = torch.randn(n_seq, 128, generator=g, device=DEV).to(torch.bfloat16), torch.zeros(n_seq, device=DEV)
    args = (q, bias, n_seq, rk, chunk_doc, docs, 0.1, k, torch.arange(docs + 1, device=DEV) + 500)
    sc, li, gi = ops.route_score_select(*args)
    want = ops.topk_merge(sc.unsqueeze(0), li.unsqueeze(0), gi.unsqueeze(0), k)
    assert all(torch.equal(a, b) for a, b in zip(ops.route_score_select(*args, winners=True), want))
