"""Which native module is loaded, and what serves the calls where there is none.  CPU only."""
import sys

import pytest
import torch
from gguf.constants import GGMLQuantizationType as QT

import gguf_jax_b200 as gj
from gguf_jax_b200 import _lib, build, synth
from gguf_jax_b200 import _matmul as mm


@pytest.fixture
def fresh(monkeypatch):
    """As at the first call of a process: no module loaded, the first-call function in place."""
    monkeypatch.setattr(_lib, "_native_module", None)

    def first_call(*args):
        try:
            return _lib.native().fast_matmul(*args)
        except RuntimeError:
            return None

    if mm._native_matmul.__module__ != mm.__name__:
        monkeypatch.setattr(mm, "_native_matmul", first_call)


def test_a_build_for_another_torch_or_python_has_another_name(built_lib, monkeypatch):
    path = build.build_native()
    assert path == _lib.native_path() and torch.__version__ in path and sys.implementation.cache_tag in path
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert _lib.native_path() != path


def test_without_the_module_the_python_path_serves_the_calls(built_lib, fresh, monkeypatch):
    monkeypatch.setattr(_lib, "native_path", lambda: "/nonexistent/_native.so")
    w, x = synth.make_weight(64, 256, QT.Q8_0, device="cpu"), torch.zeros((1, 256), dtype=torch.bfloat16)
    with pytest.warns(UserWarning, match="gguf_jax_b200.build"):
        native = _lib.native()
    assert native.fast_matmul(x, w.data, w.qtype, w.shape, False, 0) is None
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert native.capture_id(5) == 0
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    assert native.capture_id(5) != native.capture_id(5)
    with pytest.raises(ValueError, match="contraction"):
        gj.matmul(x[:, :128], w)
    with pytest.raises(TypeError):
        gj.matmul(x, w.data)


def test_arguments_are_checked_before_a_missing_library_is_reported(fresh, monkeypatch):
    def missing():
        raise RuntimeError("libggq_b200.so is missing")

    monkeypatch.setattr(_lib, "lib", missing)
    mm._fused.cache_clear()
    w, x = synth.make_weight(64, 256, QT.Q8_0, device="cpu"), torch.zeros((1, 256), dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="contraction"):
        gj.matmul(x[:, :128], w)
    with pytest.raises(RuntimeError, match="missing"):
        gj.matmul(x, w)
