"""The state-space recurrence walked chunk by chunk with the states in TMEM, against the recurrence token by token in 64 bits."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64


def case(heads, groups, state, vdim, lens, n_decode, seed=0, dev="cuda:0", step=-1.0):
    """Packed rows: ``n_decode`` single tokens (not this kernel's), then the portions; odd portions continue, even ones start anew."""
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device=dev)
    n_seq, rows, inner = n_decode + len(lens), sum(lens), heads * vdim
    cu = torch.tensor([0] + [1] * n_decode + list(lens), device=dev).cumsum(0).int()
    c = dict(heads=heads, groups=groups, n_state=state, vdim=vdim, n_seq=n_seq, n_decode=n_decode, n_tok=n_decode + rows, cu=cu,
             slot=torch.randperm(n_seq + 2, generator=g, device=dev)[:n_seq].int(),
             start=torch.tensor([3] * n_decode + [7 * (i % 2) for i in range(len(lens))], device=dev).int(),
             xbc=rnd(rows, inner + 2 * groups * state).to(BF16), dt=F.softplus(rnd(rows, heads) + step), a_log=rnd(heads), d_skip=rnd(heads),
             proj=rnd(n_decode + rows, inner + 8).to(BF16), state=rnd(n_seq + 2, heads, state, vdim))
    c["y"] = torch.full((n_decode + rows, inner), 7.0, device=dev)
    return c


def args_of(c):
    from msa_b200 import _cabi_lm as A
    p = A.ptr
    return A.SsdArgs(proj=p(c["proj"]), proj_stride=c["proj"].stride(0), conv_w=p(c["d_skip"]), conv_b=p(c["d_skip"]), dt_bias=p(c["d_skip"]),
                     a_log=p(c["a_log"]), d_skip=p(c["d_skip"]), conv_state=p(c["xbc"]), state=p(c["state"]), tok_seq=p(c["cu"]), slot=p(c["slot"]),
                     start=p(c["start"]), cu=p(c["cu"]), y=p(c["y"]), taps=4, dtype=A.dtype_code(BF16),
                     **{k: c[k] for k in ("n_tok", "n_seq", "n_decode", "heads", "vdim", "n_state", "groups")})


def walk(c):
    from msa_b200 import _cabi_lm as A
    p, args = A.ptr, args_of(c)
    status = torch.zeros(4, dtype=torch.int32, device=c["y"].device)
    A.call("msa_lm_ssd_walk", ctypes.byref(args), p(c["xbc"]), p(c["dt"]), p(status), A.stream_ptr(c["y"].device))
    assert status.tolist() == [0, 0, 0, 0]


def all_at_once(c):
    """The kernels over all chunks at once: (outputs, states), ``c`` as it was."""
    from msa_b200 import _cabi_lm as A
    p, dev = A.ptr, c["y"].device
    mine = dict(c, y=c["y"].clone(), state=c["state"].clone())
    lens = c["cu"].diff()[c["n_decode"]:]
    off = torch.cat([torch.zeros(1, device=dev), ((lens + 63) // 64).cumsum(0)]).int()
    n = int(off[-1])
    gcum = torch.empty((c["xbc"].shape[0], c["heads"]), dtype=F64, device=dev)
    work = torch.empty((n, c["heads"], c["n_state"], c["vdim"]), device=dev)
    A.call("msa_lm_ssd_chunk", ctypes.byref(args_of(mine)), p(c["xbc"]), p(c["dt"]), p(off), n, p(gcum), p(work), A.stream_ptr(dev))
    return mine["y"], mine["state"]


def recurrence(c, size):
    """(outputs of the portions' rows, states by portion); ``size``: of absolute values, what rounding errors are relative to."""
    f = (lambda t: t.to(F64).abs()) if size else (lambda t: t.to(F64))
    heads, groups, ns, vd, inner = c["heads"], c["groups"], c["n_state"], c["vdim"], c["heads"] * c["vdim"]
    x, b, k = f(c["xbc"]).split([inner, groups * ns, groups * ns], 1)
    b, k = (t.view(-1, groups, ns).repeat_interleave(heads // groups, 1) for t in (b, k))
    x, dt = x.view(-1, heads, vd), c["dt"].to(F64)
    decay = torch.exp(-torch.exp(c["a_log"].to(F64)) * dt)
    z = c["proj"][c["n_decode"]:, :inner].to(F64)
    y, states, cu = torch.empty_like(x), [], c["cu"].tolist()
    for s in range(c["n_decode"], c["n_seq"]):
        st = f(c["state"][int(c["slot"][s])]) if int(c["start"][s]) else torch.zeros((heads, ns, vd), dtype=F64, device=x.device)
        for t in range(cu[s] - c["n_decode"], cu[s + 1] - c["n_decode"]):
            st = decay[t][:, None, None] * st + dt[t][:, None, None] * b[t][:, :, None] * x[t][:, None]
            y[t] = (k[t][:, None] @ st)[:, 0] + f(c["d_skip"])[:, None] * x[t]
        states.append(st)
    return y.reshape(-1, inner) * f(F.silu(z)), states


@pytest.mark.parametrize("heads,groups,lens,n_decode", [
    (2, 1, [200, 64, 1], 0), (4, 2, [63, 65, 128], 3), (12, 2, [129, 16, 17], 1), (64, 8, [1, 300], 0), (2, 1, [640], 2)])
@pytest.mark.parametrize("step", [-1.0, 6.0])     # steps of about 0.3, and of 6, which leave nothing of what came before
def test_walk_is_the_recurrence(heads, groups, lens, n_decode, step):
    c = case(heads, groups, 128, 64, lens, n_decode, step=step)
    want, states = recurrence(c, False)
    size, sizes = recurrence(c, True)
    untouched = c["state"].clone()
    walk(c)
    # operands keep 16 bits or more (2^-17 each of state, scores and weighted values); sums over 64 tokens and 128 channels in 32 bits
    bound = 2.0 ** -14
    assert bool(((c["y"][n_decode:].to(F64) - want).abs() <= bound * size + 1e-30).all())
    assert bool((c["y"][:n_decode] == 7.0).all())
    mine = c["slot"][n_decode:].long()
    for i, slot in enumerate(mine.tolist()):
        assert bool(((c["state"][slot].to(F64) - states[i]).abs() <= bound * sizes[i] + 1e-30).all())
    other = torch.ones(untouched.shape[0], dtype=torch.bool, device=mine.device)
    other[mine] = False
    assert torch.equal(c["state"][other], untouched[other])


def test_walk_repeats_itself():
    """Many blocks and whole chunks, so that every role runs ahead of the others as far as it may: the same bits each time."""
    first = None
    for _ in range(5):
        c = case(32, 4, 128, 64, [700, 512, 333, 640], 0, seed=2)
        walk(c)
        if first is None:
            first = c["y"].clone(), c["state"].clone()
        assert torch.equal(c["y"], first[0]) and torch.equal(c["state"], first[1])


def test_walk_keeps_portions_apart():
    """What one portion holds, not-a-numbers too, stays out of the next one's rows and state."""
    c = case(4, 2, 128, 64, [40, 90], 0, seed=1)
    want, states = recurrence(c, False)
    size, sizes = recurrence(c, True)
    c["xbc"][40:] = float("nan")
    walk(c)
    assert bool(((c["y"][:40].to(F64) - want[:40]).abs() <= 2.0 ** -14 * size[:40] + 1e-30).all())
    slot = int(c["slot"][0])
    assert bool(((c["state"][slot].to(F64) - states[0]).abs() <= 2.0 ** -14 * sizes[0] + 1e-30).all())
    assert bool(c["state"][int(c["slot"][1])].isnan().all())


def same(x, y):
    """Equal numbers; not-a-numbers in the same places."""
    return torch.equal(x.nan_to_num(12345.0), y.nan_to_num(12345.0))


@pytest.mark.parametrize("heads,groups,lens,n_decode", [
    (2, 1, [1, 2, 15, 16, 17, 31, 33], 0), (4, 2, [47, 48, 49, 63, 64, 65], 3), (12, 2, [129, 190, 191, 192], 1), (64, 8, [1, 300, 4096], 0),
    (32, 4, [2048, 1500, 1911, 777], 2)])
@pytest.mark.parametrize("step,a_log", [(-1.0, 0.0), (6.0, 0.0), (-4.0, -9.0)])
def test_walk_gives_the_bits_of_all_chunks_at_once(heads, groups, lens, n_decode, step, a_log):
    """What else is in a step decides between the two, so a sequence's numbers may not depend on it."""
    c = case(heads, groups, 128, 64, lens, n_decode, seed=4, step=step)
    c["a_log"] += a_log
    y, state = all_at_once(c)
    walk(c)
    assert torch.equal(c["y"], y) and torch.equal(c["state"], state)


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("at", [5, 16, 40, 63, 64, 100, 127])
def test_walk_spreads_non_finite_values_no_further(at, value):
    """Neither to earlier tokens than those of its 16 rows, where masked weights multiply it, nor to other heads."""
    c = case(4, 2, 128, 64, [130], 0, seed=6)
    c["xbc"][at, 64:128] = value                  # values of head 1
    y, state = all_at_once(c)
    walk(c)
    assert same(c["y"], y) and same(c["state"], state)
    assert bool(c["y"][:at // 16 * 16].isfinite().all()) and not bool(c["y"][at, 64:128].isfinite().any())
    assert bool(c["y"][:, :64].isfinite().all()) and bool(c["y"][:, 128:].isfinite().all())


def test_walk_keeps_what_decays_slowly():
    """Steps that nothing is forgotten over, all writes of one sign, two portions in a row: the state against 64 bits.  Its operands keep
    2^-17; a chunk's sum of eight products loses up to 2^-23 each; the state is rounded to nearest once a chunk, its decay likewise."""
    c = case(4, 1, 128, 64, [4096, 1000], 0, seed=7, step=-4.0)
    c["a_log"].fill_(-9.0)
    c["xbc"] = c["xbc"].abs() + 0.5
    exact, chunks, slots = c["state"].to(F64), 0, c["slot"].tolist()
    for start in (0, 1):
        c["start"].fill_(start)
        for slot, want in zip(slots, recurrence(dict(c, state=exact), False)[1]):
            exact[slot] = want
        walk(c)
        chunks += 64
        off = ((c["state"].to(F64) - exact).abs() / exact.abs())[slots]
        assert float(off.max()) <= 2.0 ** -17 + 2.0 ** -20 + 2 * chunks * 2.0 ** -24 and float(off.mean()) <= 2.0 ** -19
