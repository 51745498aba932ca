"""``lm_ops.rows_gemm`` where x comes two turns ahead: more than two turns of K per warp, and the sizes beside that line."""
import pytest
import torch

from tests.test_gpu_rows_gemm import BF16, DEV, product, randn

pytestmark = pytest.mark.gpu

# 16 rows of w by 16 warps: a turn is 2048 of K; 32 rows by 4 warps (from 64 rows of w per SM on): 256, by 8 warps 512
SIZES = [(40, 4096), (40, 4104), (17, 6152), (2048, 8192), (1000, 10280), (2500, 2056), (9473, 512), (9473, 520), (9500, 1544), (9472, 1032), (32768, 776)]


@pytest.mark.parametrize("n", [1, 4, 8])
@pytest.mark.parametrize("rows,k", SIZES)
def test_rows_ahead(n, rows, k):
    from msa_b200 import lm_ops as K
    x, w = randn(n, k + 16, seed=n)[:, 8:8 + k], randn(rows, k + 8, seed=rows, scale=k ** -0.5)[:, :k]
    want, bound = product(x, w)
    for dtype, step in ((torch.float32, 0.0), (BF16, 2.0 ** -8)):
        got = K.rows_gemm(x, w, torch.empty((n, rows), dtype=dtype, device=DEV), act=False)
        assert ((got.double() - want).abs() <= bound + step * want.abs()).all()
    some = slice(0, (n + 1) // 2)                       # a row's sums do not depend on the rows beside it
    less = K.rows_gemm(x[some], w, torch.empty((x[some].shape[0], rows), dtype=BF16, device=DEV), act=False)
    assert torch.equal(less, got[some])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_rows_ahead_keeps_to_its_row(bad):
    from msa_b200 import lm_ops as K
    x, w = randn(3, 8192, seed=1), randn(48, 8192, seed=2)
    x[1, 5000] = bad
    w[7, 8191] = bad
    got = K.rows_gemm(x, w, torch.empty((3, 48), dtype=torch.float32, device=DEV), act=False)
    ok = torch.ones(3, 48, dtype=torch.bool, device=DEV)
    ok[1], ok[:, 7] = False, False
    assert torch.equal(torch.isfinite(got), ok)


@pytest.mark.parametrize("b,n,rows,k", [(3, 8, 40, 4616), (5, 2, 2048, 1288)])
def test_rows_ahead_batched(b, n, rows, k):
    from msa_b200 import lm_ops as K
    x, w = randn(n, b, k, seed=b).transpose(0, 1), randn(b, rows, k, seed=rows, scale=k ** -0.5)
    want, bound = product(x, w)
    assert ((K.bmm(x, w).double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all()
