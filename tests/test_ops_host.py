"""What the wrappers refuse before anything is launched, and the forms of a device, on fake CUDA tensors."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

pytestmark = pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")


class Library:
    def __init__(self):
        self.seen = []

    def __getattr__(self, name):
        return lambda *a: self.seen.append(name) or 0


@pytest.fixture
def library(monkeypatch):
    from msa_b200 import _cabi as A
    lib = Library()
    monkeypatch.setattr(A, "lib", lambda: lib)
    monkeypatch.setattr(A, "stream_ptr", lambda device=None: 0)
    monkeypatch.setattr(A, "ptr", lambda t: 0)
    return lib


def new(*shape, dtype=torch.int64, device="cuda:0"):
    return torch.empty(shape, dtype=dtype, device=device)


def test_question_plan_wants_a_length_for_every_row(library):
    from msa_b200 import _cabi as A, ops
    with FakeTensorMode():
        valid = new(3, 10, dtype=torch.bool)
        for n_sel in (new(2), new(1), new(3, 2), new(3, device="cuda:1")):
            with pytest.raises(A.MsaError):
                ops.question_plan(valid, n_sel, 5)
        for bad in (new(3, 10, dtype=torch.uint8), new(3, 10, dtype=torch.float32)):
            with pytest.raises(A.MsaError):
                ops.question_plan(bad, new(3), 5)
        with pytest.raises(A.MsaError):
            ops.question_plan(valid, new(3), 5, new(4, dtype=torch.int32, device="cuda:1"))
        assert not library.seen
        ops.question_plan(valid, new(3), 5)
        ops.question_plan(valid, new(6)[::2], 5, new(4, dtype=torch.int32))
        assert library.seen == ["msa_question_plan"] * 2


def test_segments_wants_a_mask(library):
    from msa_b200 import _cabi as A, ops
    with FakeTensorMode():
        for valid in (new(3, 10), new(3, 10, dtype=torch.bool, device="cuda:1")):
            with pytest.raises(A.MsaError):
                ops.segments(new(3, 10), valid)
        with pytest.raises(RuntimeError):
            ops.segments(new(3, 10), new(3, 9, dtype=torch.bool))
    assert not library.seen


def test_a_report_is_written_or_refused(library):
    """A resident plan writes no report; one that the kernel could not write whole is refused too."""
    from msa_b200 import _cabi as A, ops
    pinned = type("Pinned", (torch.Tensor,), {"is_pinned": lambda self: True})
    reports = [torch.zeros(3, dtype=torch.int64).as_subclass(pinned), torch.zeros(6, dtype=torch.int64)[::2].as_subclass(pinned),
               torch.zeros(3, dtype=torch.int32).as_subclass(pinned), torch.zeros(3, dtype=torch.int64)]
    with FakeTensorMode(allow_non_fake_inputs=True):
        plan = lambda report, **kw: ops.gather_plan(new(2, 4), None, 1, new(1), new(9), new(9, dtype=torch.int32), new(1), 64, report=report, **kw)
        with pytest.raises(A.MsaError):
            plan(reports[0], resident=new(2, 4), sample_stride=16)
        for report in reports[1:]:
            with pytest.raises(A.MsaError):
                plan(report)
        assert not library.seen
        plan(reports[0])
    assert library.seen == ["msa_gather_plan_report"]


def test_argmax_of_other_types(monkeypatch):
    from msa_b200 import lm_ops as K
    seen = []
    monkeypatch.setattr(K.A, "call", lambda name, *a: seen.append(name))
    monkeypatch.setattr(K.A, "stream_ptr", lambda device=None: 0)
    monkeypatch.setattr(K.A, "ptr", lambda t: 0)
    with FakeTensorMode():
        for x in (new(3, 40, dtype=torch.bfloat16), new(3, 40, dtype=torch.float64), new(40, 3, dtype=torch.float32).t(), new(2, 3, 40, dtype=torch.float32)):
            assert K.argmax(x).dtype == torch.int32 and K.argmax(x).shape == x.shape[:-1]
        assert not seen
        assert K.argmax(new(3, 41, dtype=torch.float32)[:, :40]).shape == (3,)
    assert seen == ["msa_lm_argmax"]


def test_forms_of_a_device(monkeypatch):
    from msa_b200 import _cabi as A
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 1000 + index)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 5)
    assert [A.stream_ptr(d) for d in (None, "cuda", torch.device("cuda"))] == [1005] * 3
    assert [A.stream_ptr(d) for d in (2, "cuda:2", torch.device("cuda:2"))] == [1002] * 3
    for d in ("cpu", torch.device("cpu")):
        with pytest.raises(ValueError):
            A.stream_ptr(d)


def test_rows_and_weights_of_unequal_sizes(library):
    from msa_b200 import _cabi as A, ops
    b16 = lambda *shape: new(*shape, dtype=torch.bfloat16)
    with FakeTensorMode():
        for x, y, w in (((4, 64), None, 32), ((4, 64), (4, 32), 64), ((4, 64), (2, 64), 64), ((4, 64), None, 128)):
            with pytest.raises(A.MsaError):
                ops.add_rmsnorm(b16(*x), None if y is None else b16(*y), b16(w), 1e-6)
        for q, k, qw, kw in ((250, 128, 128, 128), (256, 100, 128, 128), (256, 128, 64, 128), (256, 128, 128, 256)):
            with pytest.raises(A.MsaError):
                ops.heads_norm_rope(b16(4, q), b16(4, k), b16(qw), b16(kw), 1e-6, b16(4, 128), b16(4, 128))
        assert not library.seen
        ops.add_rmsnorm(b16(4, 64), b16(4, 64), b16(64), 1e-6)
        ops.heads_norm_rope(b16(4, 256), b16(4, 128), b16(128), b16(128), 1e-6, b16(2, 128), b16(2, 128))
    assert library.seen == ["msa_add_rmsnorm", "msa_heads_norm_rope"]


def test_pointers_off_the_pairs_are_refused():
    """Two bf16 values are read at a time; a pointer between them is an error of the call, not of the GPU."""
    from msa_b200 import _cabi as A
    lib, at = A.lib(), 1 << 20
    for shift in range(3):
        gate, up, out = (at + 2 * (shift == i) for i in range(3))
        assert lib.msa_silu_mul_parts(gate, 64, up, 64, 1, 64, out, 0) != 0 and b"4-byte aligned" in lib.msa_last_error()
    for shift in range(5):
        x, y, w, x_out, h = (at + 2 * (shift == i) for i in range(5))
        assert lib.msa_add_rmsnorm(x, y, w, 1e-6, 1, 64, x_out, h, 0) != 0 and b"4-byte aligned" in lib.msa_last_error()
