"""Products of few rows (``lm_ops.rows_gemm``) at the edges of tiles, K blocks and warps, against fp64 torch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


def randn(*shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(BF16).to(DEV)


def product(x, w):
    """The exact product and a bound on fp32 summation in any order: 2^-24 per addition, of the sum of magnitudes."""
    x, w = x.double(), w.double()
    return x @ w.transpose(-1, -2), (x.abs() @ w.abs().transpose(-1, -2)) * (x.shape[-1] * 2.0 ** -23)


# one K block and a tail, slices of unequal length, 1 .. 16 warps, a tile that is hardly used, low and high tiles
SIZES = [(8, 8), (32, 72), (100, 136), (128, 2048), (129, 520), (2056, 1096), (6151, 320), (40000, 192)]


@pytest.mark.parametrize("n", [1, 2, 5, 7, 8])
@pytest.mark.parametrize("rows,k", SIZES)
def test_rows_gemm(n, rows, k):
    from msa_b200 import lm_ops as K
    x, w = randn(n, k + 24, seed=n)[:, 8:8 + k], randn(rows, k, seed=rows, scale=k ** -0.5)
    want, bound = product(x, w)
    assert K.few_rows(x, w)
    for dtype, step in ((torch.float32, 0.0), (BF16, 2.0 ** -8)):
        got = K.rows_gemm(x, w, torch.empty((n, rows), dtype=dtype, device=DEV), act=False)
        assert ((got.double() - want).abs() <= bound + step * want.abs()).all()
        assert torch.equal(got, K.matmul(x, w, dtype, weight=True))


@pytest.mark.parametrize("n", [1, 3, 8])
@pytest.mark.parametrize("ff,k", [(1, 64), (20, 200), (64, 128), (65, 2048), (6144, 1024), (9999, 72)])
def test_rows_gemm_silu(n, ff, k):
    from msa_b200 import lm_ops as K
    x, w = randn(n, k, seed=n), randn(2 * ff, k, seed=ff, scale=k ** -0.5)
    (g, bg), (u, bu) = product(x, w[:ff]), product(x, w[ff:])
    want = F.silu(g) * u
    out = torch.full((n, ff + 13), 7.0, dtype=BF16, device=DEV)
    got = K.rows_gemm(x, w, out[:, 5:5 + ff], act=True)
    # silu has slopes up to 1.1; its fp32 evaluation is off by a few 2^-24 of itself
    assert ((got.double() - want).abs() <= 1.1 * bg * u.abs() + bu * F.silu(g).abs() + 1.1 * bg * bu + 1.01 * 2.0 ** -8 * want.abs()).all()
    assert (out[:, :5] == 7).all() and (out[:, 5 + ff:] == 7).all()
    assert torch.equal(got, K.matmul_silu(x, w, ff))


@pytest.mark.parametrize("b,n,rows,k", [(2, 3, 40, 72), (4, 8, 2048, 2048), (5, 7, 200, 128)])
def test_rows_gemm_batched(b, n, rows, k):
    from msa_b200 import lm_ops as K
    x, w = randn(n, b, k, seed=b).transpose(0, 1), randn(b, rows, k, seed=rows, scale=k ** -0.5)
    want, bound = product(x, w)
    assert ((K.bmm(x, w).double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()


def test_other_forms_keep_the_general_product():
    """Rows off the 16-byte boundaries, other types, no rows and many rows take torch's product, with the same results."""
    from msa_b200 import lm_ops as K
    x, w = randn(8, 264, seed=1), randn(48, 264, seed=2)
    want, bound = product(x, w)
    for a, b in ((x, w), (x.t().contiguous().t(), w), (F.pad(x, (1, 2))[:, 1:-2], w), (x, F.pad(w, (1, 2))[:, 1:-2]), (x.float(), w.float())):
        assert K.few_rows(a, b) == (a is x and b is w)
        assert ((K.matmul(a, b, weight=True).double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()
    assert not K.few_rows(randn(K.ROWS_GEMM_MAX + 1, 264, seed=3), w) and K.matmul(x[:0], w, weight=True).shape == (0, 48)


def test_in_a_graph_behind_its_own_results():
    """A chain in which every product reads what the one before wrote, launched early, from a CUDA graph."""
    from msa_b200 import lm_ops as K
    ws = [randn(512, 512, seed=i, scale=512 ** -0.5) for i in range(12)]
    x = randn(8, 512, seed=99)

    def chain():
        y = x
        for w in ws:
            y = K.matmul(y, w, weight=True)
        return y
    want = chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain()
    for _ in range(20):
        graph.replay()
        assert torch.equal(got, want)
    y = x.double()
    for w in ws:
        y = y @ w.double().t()
    assert float((got.double() - y).norm() / y.norm()) < 12 * 2.0 ** -8
