"""The fetch plan at the edges of its layout (lanes of a warp, samples of a round), against a sequential restatement."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def sequential(local, rank, base, n_rows, off, lens, kv_base, chunk_bytes, stride, resident):
    plan, n_sel, dropped, carry = [], [], 0, 0
    world = len(base)
    for b, (ls, rs) in enumerate(zip(local, rank)):
        k, keys = len(ls), []
        for lid, r in zip(ls, rs):
            if lid <= 0:
                continue
            if not 0 <= r < world or lid >= (base[r + 1] if r + 1 < world else n_rows) - base[r]:
                dropped += 1
                continue
            keys.append((r, lid))
        keys.sort()
        row = lambda r, lid: base[r] + lid
        slot = stride // k if resident is not None else 0
        if resident is not None and len(keys) == k and all(lens[row(*x)] == slot for x in keys):
            have = resident[b]
            code = [(r << 40) | lid for r, lid in keys]
            free = [s for s in range(k) if have[s] not in code]
            for x, c in zip(keys, code):
                if c in have:
                    plan.append([0, 0, 0, b])
                else:
                    s = free.pop(0)
                    have[s] = c
                    plan.append([kv_base[x[0]] + off[row(*x)] * chunk_bytes, slot, s * slot, b])
            n_sel.append(k * slot)
            continue
        if resident is not None:
            resident[b] = [-1] * k
        mine, mark = 0, len(plan)
        for x in keys:
            n = lens[row(*x)]
            if stride > 0:
                n = min(n, stride - mine)
            plan.append([kv_base[x[0]] + off[row(*x)] * chunk_bytes, n, mine if n > 0 else 0, b])
            mine += n
        plan += [[0, 0, 0, b]] * (k - len(keys))
        if stride == 0:
            for i in range(mark, len(plan)):
                if plan[i][1] > 0:
                    plan[i] = plan[i][:2] + [plan[i][2] + carry, b]
        carry += mine
        n_sel.append(mine)
    return plan, n_sel, dropped


@pytest.mark.parametrize("mode", ["packed", "room", "resident"])
@pytest.mark.parametrize("n_seq,k", [(1, 1), (1, 16), (33, 16), (5, 32), (40, 33), (7, 64), (1025, 4), (2049, 3)])
def test_plan_matches_the_sequential_one(n_seq, k, mode):
    from msa_b200 import ops
    g = torch.Generator().manual_seed(n_seq * 100 + k)
    counts = [120, 75, 200]                                   # documents of three shards, each behind a dummy row
    base = [0, 121, 197]
    n_rows = 398
    lens = (torch.full((n_rows,), 4) if mode == "resident" else torch.randint(0, 9, (n_rows,), generator=g)).to(torch.int32)
    off = torch.randint(0, 10_000, (n_rows,), generator=g)
    kv_base = [1 << 40, 2 << 40, 3 << 40]
    stride = {"packed": 0, "room": 3 * k, "resident": 4 * k}[mode]
    resident = torch.full((n_seq, k), -1, dtype=torch.int64, device=DEV) if mode == "resident" else None
    kept = [[-1] * k for _ in range(n_seq)] if mode == "resident" else None
    dev = lambda t, dt=torch.int64: torch.as_tensor(t, dtype=dt).to(DEV)
    for step in range(3):
        picks = [torch.randperm(sum(counts), generator=g)[:k].tolist() for _ in range(n_seq)]
        if step:                                              # half of the winners of the step before come again
            picks = [list(dict.fromkeys(old[:k // 2] + new))[:k] for old, new in zip(before, picks)]
        before = picks
        rank = [[0 if p < 120 else 1 if p < 195 else 2 for p in row] for row in picks]
        local = [[p + 1 - (0, 120, 195)[r] for p, r in zip(row, rk)] for row, rk in zip(picks, rank)]
        for b in range(0, n_seq, 3):                          # dummies, invalid winners, ids and ranks outside the directory
            if b % 2 and mode != "packed":
                continue
            local[b][-1] = [0, -1, 900, 5][b % 4]
            rank[b][-1] = [0, 0, 1, 7][b % 4]
        status, report = torch.zeros(4, dtype=torch.int32, device=DEV), torch.zeros(3, dtype=torch.int64).pin_memory()
        plan, n_sel, total = ops.gather_plan(dev(local), dev(rank, torch.int32), 3, dev(base), dev(off), dev(lens, torch.int32),
                                             dev(kv_base), 4096, sample_stride=stride, status=status, resident=resident,
                                             report=report if mode == "packed" else None)
        want, want_n, dropped = sequential(local, rank, base, n_rows, off.tolist(), lens.tolist(), kv_base, 4096, stride, kept)
        torch.cuda.synchronize()
        assert plan.tolist() == want and n_sel.tolist() == want_n
        assert total.item() == sum(want_n) and status.tolist() == [0, 0, dropped, 0]
        if mode == "packed":
            assert report[0] == sum(want_n) and report[1:].view(torch.int32).tolist() == [0, 0, dropped, 0]
        if resident is not None:
            assert resident.tolist() == kept
