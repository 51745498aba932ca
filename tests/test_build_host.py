"""The native extension is the one for the torch and the Python that run."""
import os
import sysconfig

import pytest
import torch

from msa_b200 import _cabi as A
from msa_b200 import build


def test_another_torch_takes_another_build(monkeypatch):
    here = build.native_path()
    assert os.path.dirname(here) == os.path.dirname(os.path.abspath(build.__file__)) and torch.__version__ in here
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build.native_path() != here and build._stale("native")
    monkeypatch.setattr(A, "_native", None)
    monkeypatch.setattr(A, "lib", lambda: None)
    with pytest.raises(A.MsaError, match="python -m msa_b200.build"):
        A.native()


def test_another_python_takes_another_build(monkeypatch):
    here, real = build.native_path(), sysconfig.get_config_var
    monkeypatch.setattr(sysconfig, "get_config_var", lambda n: ".cpython-399-x86_64-linux-gnu.so" if n == "EXT_SUFFIX" else real(n))
    assert build.native_path() != here and build._stale("native")
