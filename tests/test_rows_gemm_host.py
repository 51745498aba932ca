"""Which products ``lm_ops`` hands to the few-row kernel, on fake CUDA tensors: sizes that do not fit one another are torch's to refuse and
never reach a launch."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

BF16 = torch.bfloat16


@pytest.fixture
def launches(monkeypatch):
    from msa_b200 import lm_ops as K
    seen = []
    monkeypatch.setattr(K.A, "call", lambda name, *a: seen.append(name))
    monkeypatch.setattr(K.A, "stream_ptr", lambda device=None: 0)
    monkeypatch.setattr(K.A, "ptr", lambda t: 0)
    with FakeTensorMode():
        yield seen


def new(*shape, dtype=BF16, device="cuda:0"):
    return torch.empty(shape, dtype=dtype, device=device)


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
@pytest.mark.parametrize("x,w", [((3, 64), (32, 72)), ((3, 72), (32, 64)), ((3, 64), (2, 32, 64)), ((2, 3, 64), (2, 32, 64)), ((3, 64), (0, 72))])
def test_matmul_of_unequal_sizes(launches, x, w):
    from msa_b200 import lm_ops as K
    for call in (lambda: K.matmul(new(*x), new(*w), weight=True), lambda: K.matmul_silu(new(*x), new(*w), 16)):
        with pytest.raises((RuntimeError, IndexError)):
            call()
    assert not launches


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
@pytest.mark.parametrize("x,w", [((2, 3, 64), (2, 32, 72)), ((2, 3, 64), (3, 32, 64)), ((3, 3, 64), (2, 32, 64)), ((3, 64), (2, 32, 64))])
def test_bmm_of_unequal_sizes(launches, x, w):
    from msa_b200 import lm_ops as K
    with pytest.raises((RuntimeError, IndexError)):
        K.bmm(new(*x), new(*w))
    assert not launches


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
def test_operands_on_two_devices(launches):
    from msa_b200 import lm_ops as K
    for w in (new(32, 64, device="cuda:1"), new(32, 64, device="cpu")):
        with pytest.raises(RuntimeError):
            K.matmul(new(3, 64), w, weight=True)
    assert not launches


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
def test_empty_products(launches):
    from msa_b200 import lm_ops as K
    assert K.matmul(new(3, 0), new(32, 0), weight=True).shape == (3, 32)
    assert K.matmul(new(3, 64), new(0, 64), weight=True).shape == (3, 0)
    assert K.bmm(new(0, 3, 64), new(0, 32, 64)).shape == (0, 3, 32)
    assert K.bmm(new(2, 3, 0), new(2, 32, 0)).shape == (2, 3, 32)
    assert not launches


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
def test_activation_of_other_widths_and_outputs(launches):
    """Fewer gate rows than half of ``w``, and outputs of another width, take product and activation one after the other, as
    they did; the launch itself refuses what it would write out of range."""
    from msa_b200 import lm_ops as K
    x, w = new(3, 64), new(64, 64)
    assert K.matmul_silu(x, w, 16).shape == (3, 16)
    K.matmul_silu(x, w, 32, new(3, 40))
    K.matmul_silu(x, w, 32, new(4, 32))
    assert launches == ["msa_lm_silu_mul"] * 3
    for out, act in ((new(3, 63), False), (new(2, 64), False), (new(3, 64), True), (new(64, 3).t(), False), (new(3, 64, device="cuda:1"), False)):
        with pytest.raises(K.A.MsaError):
            K.rows_gemm(x, w, out, act=act)
    with pytest.raises(K.A.MsaError):
        K.rows_gemm(x, new(63, 64), new(3, 31), act=True)
    with pytest.raises(K.A.MsaError):
        K.rows_gemm(new(9, 64), w, new(9, 64), act=False)
    assert launches == ["msa_lm_silu_mul"] * 3


@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
def test_what_fits_takes_the_kernel(launches):
    from msa_b200 import lm_ops as K
    assert K.matmul(new(3, 64), new(32, 64), torch.float32, weight=True).dtype == torch.float32
    assert K.matmul_silu(new(3, 64), new(64, 64), 32, new(3, 50)[:, 9:41]).shape == (3, 32)
    assert K.bmm(new(2, 3, 64), new(2, 32, 64)).shape == (2, 3, 32)
    assert launches == ["msa_lm_rows_gemm"] * 3
    K.matmul(new(3, 64), new(32, 64))
    K.matmul_silu(new(3, 64), new(64, 64), 32, weight=False)
    K.bmm(new(2, 3, 64), new(2, 32, 64), weight=False)
    assert launches == ["msa_lm_rows_gemm"] * 3 + ["msa_lm_silu_mul"]
