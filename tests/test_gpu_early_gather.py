"""The gather that takes its total on the device: the same packed entries, whatever the host expected."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def service(n_docs, longest, dtype, top_k=4):
    from msa_b200.memory import AttentionGeometry, Document, ModelConfig
    from msa_b200.service import MSAService
    g = torch.Generator(device=DEV).manual_seed(n_docs)
    lens = torch.randint(1, longest + 1, (n_docs,), generator=torch.Generator().manual_seed(3)).tolist()
    geo = AttentionGeometry(num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, head_dim=64, dtype=dtype)
    svc = MSAService(0, None, ModelConfig(doc_top_k=top_k, pooling_kernel_size=64, router_layer_idx="0"), None, geo, world_size=1, rank=0)
    rnd = lambda: torch.randn(sum(lens), 2, 64, generator=g, device=DEV).to(dtype)
    svc.load_pooled([Document(doc_id=10 + i, num_chunks=n) for i, n in enumerate(lens)], {0: (rnd(), rnd(), rnd())})
    svc.publish_directory()
    svc.early_gather_from = 0                               # small calls too
    return svc, lens


def query(svc, batch, dtype):
    g = torch.Generator(device=DEV).manual_seed(batch)
    q = torch.nn.functional.normalize(torch.randn(batch, 4, 20, 64, generator=g, device=DEV), dim=-1).to(dtype)
    return svc.doc_query(q, torch.ones(batch, 20, dtype=torch.bool, device=DEV), 0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_docs,longest,batch", [(3, 1, 1), (40, 9, 5), (200, 17, 33)])
def test_the_same_entries(n_docs, longest, batch, dtype):
    svc, lens = service(n_docs, longest, dtype)
    early = query(svc, batch, dtype)
    svc.early_gather_bytes = 0
    late = query(svc, batch, dtype)
    assert all(torch.equal(a, b) for a, b in zip(early, late))
    assert early[0].is_contiguous() and early[1].is_contiguous() and early[0].shape[1] == int(early[3].sum())
    svc.early_gather_bytes = 1 << 30
    svc._longest = 1                                        # less room than the winners need
    assert all(torch.equal(a, b) for a, b in zip(query(svc, batch, dtype), late))


@pytest.mark.parametrize("early_from", [0, 5 << 20])
def test_results_hold_no_more_than_they_show(early_from):
    """One long document in the bank sizes the storage that the gather writes to, not what a caller keeps."""
    svc, lens = service(60, 40, torch.bfloat16)
    svc.early_gather_from = early_from
    k, v = query(svc, 7, torch.bfloat16)[:2]
    assert k.shape[1] < 7 * 4 * max(lens) and k.shape == v.shape
    for t in (k, v):
        assert t.untyped_storage().nbytes() == t.numel() * t.element_size() and t.storage_offset() == 0
