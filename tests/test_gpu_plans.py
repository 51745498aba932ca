"""The two small planning kernels of the attention layer (``ops.segments``, ``ops.question_plan``) against plain Python, at the edges
of their tiles (8 tokens a thread, 8192 a tile) and of what they are given."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def table(doc, listed, by_id):
    """(tokens, offsets, longest, runs) of a [rows][len] block."""
    tok, off, runs, before = [], [], True, None
    row_len = len(doc[0]) if doc else 0
    for r, row in enumerate(doc):
        for c, d in enumerate(row):
            if not listed(r, c):
                continue
            key = (r, d if by_id else 0)
            if before is None or before[0] != key:
                off.append(len(tok))
            elif before[1] != c - 1:
                runs = False
            before = (key, c)
            tok.append(r * row_len + c)
    off.append(len(tok))
    return tok, off, max([b - a for a, b in zip(off, off[1:])], default=0), runs


@pytest.mark.parametrize("masked", [0.0, 0.02, 0.6, 1.0])
@pytest.mark.parametrize("rows,size", [(1, 1), (1, 3), (1, 4096), (1, 4097), (1, 8192), (1, 8193), (1, 20001), (3, 1365), (5, 4096), (40, 7), (9000, 1)])
def test_segments(rows, size, masked):
    from msa_b200 import ops
    g = torch.Generator().manual_seed(rows * size)
    doc = torch.cumsum((torch.rand(rows, size, generator=g) < 0.02).long(), 1)          # 0: belongs to nothing
    doc[:, :min(3, size - 1)] = -2
    doc = torch.where(torch.rand(rows, size, generator=g) < 0.005, -1, doc)
    doc[0, size // 2] += 2 ** 33 if size > 8 else 1                                       # ids of 64 bits
    mask = torch.rand(rows, size, generator=g) >= masked
    (tok, off, longest, runs), template, n_template = ops.segments(doc.to(DEV), mask.to(DEV))
    ids, m = doc.tolist(), mask.tolist()
    want = table(ids, lambda r, c: ids[r][c] > 0 and m[r][c], True)
    assert (tok.tolist(), off.tolist(), longest, runs) == want
    want = table(ids, lambda r, c: ids[r][c] == -2 and m[r][c], False)
    assert (template[0].tolist(), template[1].tolist(), template[2]) == want[:3] and template[3] is True
    assert n_template == sum(x == -2 for row in ids for x in row) and tok.dtype == off.dtype == torch.int32


@pytest.mark.parametrize("b,s", [(1, 1), (2, 31), (33, 64), (70, 100), (3, 1000)])
@pytest.mark.parametrize("kind", ["left", "full", "none", "holes"])
def test_question_plan(b, s, kind):
    from msa_b200 import ops
    g = torch.Generator().manual_seed(b + s)
    first = torch.randint(0, s, (b, 1), generator=g)
    valid = {"left": torch.arange(s)[None] >= first, "full": torch.ones(b, s, dtype=torch.bool), "none": torch.zeros(b, s, dtype=torch.bool),
             "holes": torch.rand(b, s, generator=g) < 0.5}[kind]
    n_sel, status = torch.randint(0, 500, (b,), generator=g), torch.tensor([7, 0, 0, 0], dtype=torch.int32, device=DEV)
    lengths, report = ops.question_plan(valid.to(DEV), n_sel.to(DEV), 5, status)
    want = n_sel + 5 + valid.sum(1)
    runs = all(x[-1] - x[0] + 1 == len(x) for x in (torch.nonzero(r).flatten().tolist() for r in valid) if x)
    assert lengths.dtype == torch.int64 and lengths.tolist() == want.tolist() and report.tolist() == [int(want.max()), int(runs), 7]
    assert ops.question_plan(valid.to(DEV), n_sel.to(DEV), 5)[1].tolist()[2] == 0
