"""Residual step and gated activation of many rows (``lm_ops.residual_norm``, ``lm_ops.silu_mul``) at the edges of their
variants, against fp64 torch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16, F32 = torch.bfloat16, torch.float32


def randn(*shape, seed, dtype=F32):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g).to(dtype).to(DEV)


def near(got, want, scale, bf16):
    """fp32 sums of up to 12,000 squares and a few products: 2^-18 of the operands' size; a rounding to bf16 on top."""
    return bool(((got.double() - want).abs() <= 2.0 ** -18 * scale + (2.0 ** -8 * want.abs() if bf16 else 0.0)).all())


# few rows (one pass) up to 512, then a row in registers up to 4096 columns, then through shared memory; widths around the limits
@pytest.mark.parametrize("rows,width", [(513, 4), (513, 508), (600, 512), (513, 516), (700, 2048), (515, 2052), (514, 4096), (3, 4100), (2, 12000), (514, 2050), (3, 4101)])
@pytest.mark.parametrize("dtype", [BF16, F32], ids=["bf16", "f32"])
def test_residual_norm(rows, width, dtype):
    from msa_b200 import lm_ops as K
    base, y, add = randn(rows, width, seed=1), randn(rows, width, seed=2, dtype=dtype), randn(rows, width, seed=3)
    wb, w1, w2 = (1 + 0.1 * randn(width, seed=i) for i in (4, 5, 6))
    rms = lambda t, w: t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    for branch_norm in (True, False):
        x_out, cat = torch.empty_like(base), torch.zeros(rows, 2 * width, dtype=dtype, device=DEV)
        h, h2 = K.residual_norm(base, y, wb if branch_norm else None, w1, 1e-5, dtype, x_out=x_out, cat=cat, add=add, w_next2=w2)
        x = base.double() + (rms(y.double(), wb) if branch_norm else y.double()) + add.double()
        size = base.abs().double() + 2 * y.abs().double() + add.abs().double() + 1
        assert near(x_out, x, size, False) and near(cat[:, :width], x, size, dtype == BF16) and not cat[:, width:].any()
        assert near(h, rms(x, w1), 4 * size, dtype == BF16) and near(h2, rms(x, w2), 4 * size, dtype == BF16)


@pytest.mark.parametrize("width,top", [(516, 3), (2048, 4), (2050, 2)])
def test_residual_norm_of_a_mixture_and_of_chosen_rows(width, top):
    from msa_b200 import lm_ops as K
    n = 520
    y, inv = randn(n * top, width, seed=1, dtype=BF16), torch.randperm(n * top, generator=torch.Generator().manual_seed(2)).to(torch.int32).view(n, top).to(DEV)
    mix, base, w = randn(n, top, seed=3).softmax(-1), randn(n, width, seed=4), 1 + 0.1 * randn(width, seed=5)
    rms = lambda t: t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    branch = (y.double()[inv.long()] * mix.double()[..., None]).sum(1)
    h = K.residual_norm(base, y, None, w, 1e-5, BF16, inv=inv, mix=mix)
    assert near(h, rms(base.double() + branch), 8 * (base.abs().double() + branch.abs() + 1), True)
    rows = torch.randint(0, n, (600,), generator=torch.Generator().manual_seed(6)).to(torch.int32).to(DEV)
    h = K.residual_norm(base, None, None, w, 1e-5, F32, rows=rows)
    assert near(h, rms(base.double()[rows.long()]), 4 * base.abs().double()[rows.long()] + 1, False)


@pytest.mark.parametrize("rows,ff,offset", [(1, 8, 0), (3, 2048, 0), (2, 2056, 0), (591, 2048, 0), (592, 2048, 0), (300, 2056, 0), (65537, 8, 0), (65536, 20, 0), (5, 6144, 0), (3, 20, 0), (4, 13, 0), (3, 64, 4), (2, 64, 1)])
@pytest.mark.parametrize("dtype", [BF16, F32], ids=["bf16", "f32"])
def test_silu_mul(rows, ff, offset, dtype):
    from msa_b200 import lm_ops as K
    wide = randn(rows, 2 * ff + 8, seed=ff, dtype=dtype) * 4
    wide[0, offset], wide[0, offset + 1] = -100.0, 100.0
    gu = wide[:, offset:offset + 2 * ff]
    out = torch.full((rows, ff + 8), 7.0, dtype=dtype, device=DEV)
    want = F.silu(gu[:, :ff].double()) * gu[:, ff:].double()
    tiny = 2.0 ** -100          # where 1 + e^-z passes 2^126 (z < -87) the quotient may be 0: less than 2^-118 of the other factor
    assert near(K.silu_mul(gu, ff, out[:, offset:offset + ff]), want, want.abs() + tiny, dtype == BF16)
    assert (out[:, :offset] == 7).all() and (out[:, offset + ff:] == 7).all()


@pytest.mark.parametrize("rows,cols,pad", [(1, 1, 0), (3, 31, 0), (2, 4097, 3), (8, 32768, 0), (2, 32768, 1), (3, 151936, 0), (9, 151936, 0), (4, 131072, 0), (4, 131073, 0), (2, 36868, 4)])
def test_argmax(rows, cols, pad):
    from msa_b200 import lm_ops as K
    x = randn(rows, cols + pad, seed=cols)[:, :cols]
    assert torch.equal(K.argmax(x), x.argmax(-1).to(torch.int32))
    top = x.max() + 1
    x[:, cols // 3] = x[:, cols // 2] = x[:, cols - 1] = top              # equals: the lowest place
    assert K.argmax(x).tolist() == [cols // 3] * rows
    x[-1, cols // 2], x[-1, cols - 1] = float("nan"), float("nan")
    assert K.argmax(x).tolist() == [cols // 3] * (rows - 1) + [cols // 2]
    assert K.argmax(torch.full_like(x, -float("inf"))).tolist() == [0] * rows
