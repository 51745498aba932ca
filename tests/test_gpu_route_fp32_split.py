"""fp32 routing as sums of bf16 products: accuracy against chains of fp32 multiply-adds, and numbers that have no exact split."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def route(q, rk, doc, alpha=0.125):
    from msa_b200 import ops
    b, _, s, _ = q.shape
    qf, bias, s_pad = ops.fold_queries(q, torch.ones(b, s, dtype=torch.bool, device=DEV), 1)
    keys, status = ops.route_scores(qf, bias, b, s_pad, rk, doc, int(doc.max()), alpha)
    assert status.tolist() == [0, 0, 0, 0]
    return ops.keys_to_scores(keys)[:, 1:]


def want(q, rk, dtype, alpha=0.125):
    """Every chunk its own document: the best row of the question, rows whose score is not a number left out."""
    b, h, s, d = q.shape
    z = q.to(dtype).permute(0, 2, 1, 3).reshape(b, s, -1) @ rk.to(dtype).t()
    return z.masked_fill(z.isnan(), -torch.inf).amax(1) * alpha


@pytest.mark.parametrize("s,h,d,chunks", [(16, 8, 128, 300), (64, 8, 128, 1000), (65, 2, 64, 257), (200, 8, 128, 500), (17, 1, 4, 128), (48, 5, 4, 127)])
@pytest.mark.parametrize("mean", [0.0, 1.0])
def test_no_further_off_than_fp32_chains(s, h, d, chunks, mean):
    g = torch.Generator(device=DEV).manual_seed(s + chunks)
    q = torch.randn(2, h, s, d, generator=g, device=DEV) + mean           # with a mean every partial sum grows: truncation would add up
    rk = torch.randn(chunks, h * d, generator=g, device=DEV) + mean
    doc = torch.arange(1, chunks + 1, device=DEV, dtype=torch.int32)
    ref = want(q, rk, torch.float64)
    rows = q.permute(0, 2, 1, 3).reshape(2, s, 1, -1)
    chain = torch.zeros(2, s, chunks, device=DEV)
    for k in range(h * d):
        chain = torch.addcmul(chain, rows[..., k], rk[:, k].view(1, 1, -1))
    err = lambda x: float((x.double() - ref).norm() / ref.norm())
    # one chain of fp32 additions over all channels is what the result may be as far off as; 2^-24: its own rounding
    assert err(route(q, rk, doc)) <= err(chain.amax(1) * 0.125) + 2.0 ** -24


@pytest.mark.parametrize("where", ["key", "query"])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan"), 1e30, -1e36, 2.0 ** 60, 1e-35, 1e-40, 0.0])
def test_numbers_without_a_split(where, value):
    g = torch.Generator(device=DEV).manual_seed(5)
    q = torch.randn(1, 4, 40, 32, generator=g, device=DEV)
    rk = torch.randn(200, 128, generator=g, device=DEV)
    if where == "key":
        rk[131, 77] = value
    else:
        q[0, 2, 9, 3] = value
    doc = torch.arange(1, 201, device=DEV, dtype=torch.int32)
    ref, got = want(q, rk, torch.float64), route(q, rk, doc).double()
    ref = torch.where(ref.abs() > torch.finfo(torch.float32).max, ref.sign() * torch.inf, ref).clamp(min=torch.finfo(torch.float32).min)
    # 128 additions in 32 bits, each off by 2^-24 of a partial sum below the sum of absolute products
    finite = lambda t: t.abs().nan_to_num(0.0, 0.0, 0.0)
    size = want(finite(q), finite(rk), torch.float64)
    assert torch.equal(got.isinf(), ref.isinf()) and torch.equal(got[got.isinf()], ref[ref.isinf()])
    on = ~ref.isinf()
    assert bool(((got - ref).abs()[on] <= (128 * 2.0 ** -24 * size)[on]).all())


def test_all_small_numbers_keep_their_digits():
    g = torch.Generator(device=DEV).manual_seed(6)
    q = torch.randn(1, 4, 16, 32, generator=g, device=DEV) * 1e6
    rk = torch.randn(150, 128, generator=g, device=DEV) * 1e-36
    doc = torch.arange(1, 151, device=DEV, dtype=torch.int32)
    ref, got = want(q, rk, torch.float64), route(q, rk, doc).double()
    assert float((got - ref).norm() / ref.norm()) < 1e-5


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 1e30, 1e-40])
def test_such_numbers_leave_the_other_scores_alone(value):
    """Two questions in one tile of rows, two tiles of chunks: what has no split costs its own row or chunk another kind of sum, no other."""
    g = torch.Generator(device=DEV).manual_seed(7)
    q = torch.randn(2, 4, 20, 32, generator=g, device=DEV)
    rk = torch.randn(200, 128, generator=g, device=DEV)
    doc = torch.arange(1, 201, device=DEV, dtype=torch.int32)
    plain = route(q, rk, doc)
    odd = q.clone()
    odd[0, 2, 9, 3] = value
    assert torch.equal(route(odd, rk, doc)[1], plain[1])
    key = rk.clone()
    key[131, 77] = value
    others = torch.arange(200, device=DEV) != 131
    assert torch.equal(route(q, key, doc)[:, others], plain[:, others])


@pytest.mark.parametrize("kdim", [4, 124, 1024, 1100])
def test_every_row_and_chunk_without_a_split(kdim):
    g = torch.Generator(device=DEV).manual_seed(8)
    q = torch.randn(3, kdim // 4, 70, 4, generator=g, device=DEV)
    rk = torch.randn(150, kdim, generator=g, device=DEV)
    q[..., 0] = 1e-33
    rk[:, -1] *= 2.0 ** 61
    doc = torch.arange(1, 151, device=DEV, dtype=torch.int32)
    ref, got = want(q, rk, torch.float64), route(q, rk, doc).double()
    # chains of kdim multiply-adds, each off by 2^-24 of the sum of absolute products
    assert bool(((got - ref).abs() <= kdim * 2.0 ** -24 * want(q.abs(), rk.abs(), torch.float64)).all())


def test_more_rows_than_a_grid_has_tiles():
    from msa_b200 import ops
    rows = 65535 * 64 + 80
    g = torch.Generator(device=DEV).manual_seed(9)
    qf, rk = torch.randn(rows, 4, generator=g, device=DEV), torch.randn(3, 4, generator=g, device=DEV)
    qf[-1] = 50 * rk[1]                           # the best row of the second chunk is the last one
    keys, status = ops.route_scores(qf, torch.zeros(rows, device=DEV), 1, rows, rk, torch.arange(1, 4, device=DEV, dtype=torch.int32), 3, 1.0)
    got, ref = ops.keys_to_scores(keys)[0, 1:].double(), (qf.double() @ rk.double().t()).amax(0)
    assert status.tolist() == [0, 0, 0, 0] and bool(((got - ref).abs() <= 4 * 2.0 ** -24 * (qf.double().abs() @ rk.double().abs().t()).amax(0)).all())


@pytest.mark.parametrize("form", ["expanded", "overlapping"])
def test_keys_that_share_memory(form):
    """A bank of views: rows that a tensor map does not take."""
    g = torch.Generator(device=DEV).manual_seed(10)
    flat = torch.randn(128 + 4 * 40, generator=g, device=DEV)
    rk = flat[:128].expand(40, 128) if form == "expanded" else flat.as_strided((40, 128), (4, 1))
    q, doc = torch.randn(1, 4, 20, 32, generator=g, device=DEV), torch.arange(1, 41, device=DEV, dtype=torch.int32)
    bound = 128 * 2.0 ** -24 * want(q.abs(), rk.abs(), torch.float64)
    assert bool(((route(q, rk, doc).double() - want(q, rk, torch.float64)).abs() <= bound).all())
