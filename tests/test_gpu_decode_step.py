"""Kernels of a decode step: states held in registers and shared memory, convolutions of one token, launches of few rows."""
import pytest
import torch

from tests import hybrid_util as U
from tests.test_gpu_hybrid import OneMixer, bf16_rows, exact_products, mixer_case, mixer_close, model  # noqa: F401

pytestmark = pytest.mark.gpu

# delta: 256 threads hold five rows each of the state, 40 rows of 128 columns, 80 of 64, 255 of 20; the rest is in shared memory.
# mamba2: 512 channels of a head, its B and its C are convolved at once; more than four taps take the general loop.
CASES = ([("delta", U.delta(2, 1, dim, vdim, taps)) for dim, vdim, taps in
          [(39, 128, 4), (40, 128, 2), (41, 128, 5), (80, 64, 1), (81, 64, 4), (128, 128, 3), (48, 20, 4), (256, 16, 4), (256, 24, 4), (16, 1100, 4)]]
         + [("mamba2", U.mamba2(4, vdim, state, 2, 2, taps)) for vdim, state, taps in
            [(64, 96, 4), (64, 97, 3), (64, 224, 4), (68, 223, 2), (4, 5, 1), (64, 128, 5)]])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("kind,spec", CASES, ids=lambda v: v if isinstance(v, str) else "-".join(str(x) for x in v.values()))
def test_token_by_token(kind, spec, dtype):
    """Tokens one at a time from the start, behind a portion, and after it again."""
    w, oracle = mixer_case(kind, spec, 64, 3)
    m, h = OneMixer(kind, spec, w, 64, dtype), bf16_rows(24, 64, 8)
    cache = m.cache(1, 32)
    cache.acquire("s")
    cuts, out, at = [1] * 7 + [6] + [1] * 11, [], 0
    for n in cuts:
        out.append(m.run(cache, [("s", h[at:at + n])])[0])
        at += n
    assert at == h.shape[0]
    mixer_close(torch.cat(out), oracle(h), dtype)


@pytest.mark.parametrize("rows", [1, 3, 8, 9])
@pytest.mark.parametrize("name", ["wide", "par-wide", "mixed", "par-mixed"])
def test_queued_steps_are_as_steps_that_wait(name, rows):
    """Up to 8 rows, kernels start while the one before them runs: the bits are those of steps with the device idle in between,
    and of a second run."""
    m = model(name, torch.bfloat16)
    g = torch.Generator().manual_seed(rows)
    toks = torch.randint(0, m.config.vocab, (6, rows), generator=g).tolist()
    seen = []
    for wait in (True, False, False):
        cache = m.new_cache(rows, 16)
        for i in range(rows):
            cache.acquire(i)
        out = []
        for t in toks:
            out.append(m.run([(i, [t[i]], [0]) for i in range(rows)], cache))
            if wait:
                torch.cuda.synchronize()
        seen.append(torch.stack(out))
    assert torch.isfinite(seen[0]).all() and torch.equal(seen[0], seen[1]) and torch.equal(seen[0], seen[2])
