"""The norm over parts of a row: a warp per part for many of them, a block per part for few."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def operands(rows, parts, size, dtype, seed=0):
    """x and out inside wider rows, a guard of sevens around the output."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    width = parts * size
    x = torch.randn((rows, width + 12), generator=g, device=DEV) * torch.exp(torch.randn((rows, 1), generator=g, device=DEV))
    w = 1.0 + 0.3 * torch.randn(width, generator=g, device=DEV)
    return x[:, 4:4 + width], w, torch.full((rows, width + 16), 7.0, dtype=dtype, device=DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("size", [4, 128, 132, 256, 260, 512, 516, 1020, 1024, 1028])
@pytest.mark.parametrize("more", [-1, 0, 3])
def test_many_parts(size, dtype, more):
    from msa_b200 import lm_ops as K
    parts, eps = 2, 1e-3
    rows = 8 * torch.cuda.get_device_properties(0).multi_processor_count + more      # 16 parts per SM are the line; not always a multiple of 8
    x, w, whole = operands(rows, parts, size, dtype)
    out = whole[:, 8:8 + parts * size]
    K.part_norm(x, w, parts, eps, out)
    z = x.double().view(rows, parts, size)
    want = (z / (z.square().mean(-1, keepdim=True) + eps).sqrt()).reshape(rows, -1) * w.double()
    # a sum of squares of up to 20 roundings, halved by the root; root, quotient and two products; the rounding to the output (8 bits in bf16: 2^-8)
    bound = 16 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert bool(((out.double() - want).abs() <= bound * want.abs()).all())
    assert bool((whole[:, :8] == 7.0).all()) and bool((whole[:, 8 + parts * size:] == 7.0).all())
    few = torch.empty((9, parts * size), dtype=dtype, device=DEV)
    for first in (0, rows - 9):                   # the bits that the same rows have in a call of few
        K.part_norm(x[first:first + 9], w, parts, eps, few)
        assert torch.equal(few, out[first:first + 9])
