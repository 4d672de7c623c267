"""When the C library and its torch binding are built, and that a binding of another torch is not loaded."""
import builtins

import pytest

from sharq_b200 import _build, _lib


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """Both outputs present and current, in a folder of their own; what build() builds is recorded."""
    built = []
    for name in ("LIB_PATH", "BIND_PATH", "BIND_TAG_PATH"):
        monkeypatch.setattr(_build, name, tmp_path / getattr(_build, name).name)
        getattr(_build, name).write_text("")
    _build.BIND_TAG_PATH.write_text(_build.binding_tag())
    monkeypatch.setattr(_build, "_build_library", lambda verbose: built.append("library"))
    monkeypatch.setattr(_build, "_build_binding", lambda: built.append("binding"))
    return built


def test_nothing_is_built_when_both_are_current(tree):
    assert _build.build() == _build.LIB_PATH and tree == []


def test_a_missing_output_is_built_alone(tree):
    _build.BIND_PATH.unlink()
    _build.build()
    assert tree == ["binding"]
    _build.BIND_PATH.write_text("")
    _build.LIB_PATH.unlink()
    _build.build()
    assert tree == ["binding", "library"]


@pytest.mark.parametrize("tag", [None, "", "torch 0.0.1"])
def test_a_binding_of_another_torch_is_built_again(tree, tag):
    if tag is None:
        _build.BIND_TAG_PATH.unlink()
    else:
        _build.BIND_TAG_PATH.write_text(tag)
    _build.build()
    assert tree == ["binding"]


def test_the_library_is_built_without_torch(tree, monkeypatch):
    real = builtins.__import__
    monkeypatch.setattr(builtins, "__import__", lambda name, *a, **kw: _no_torch(name, real, *a, **kw))
    _build.LIB_PATH.unlink()
    assert _build.build() == _build.LIB_PATH and tree == ["library"]


def _no_torch(name, real, *args, **kw):
    if name == "torch" or name.startswith("torch."):
        raise ImportError("no torch")
    return real(name, *args, **kw)


def test_a_binding_of_another_torch_is_not_loaded(tree, monkeypatch):
    monkeypatch.setattr(_lib, "_NATIVE", None)
    monkeypatch.setattr(_lib, "NATIVE_PATH", _build.BIND_PATH)
    _build.BIND_TAG_PATH.write_text("torch 0.0.1")
    with pytest.raises(ImportError, match="another torch"):
        _lib.native()
