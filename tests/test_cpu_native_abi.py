"""The extension module is bound to the torch and Python it was built with: another version rebuilds it, or refuses it."""
import pytest

from blockgtq_b200 import _lib, build


def test_another_torch_version_rebuilds(monkeypatch):
    _lib.lib()
    assert not build.needs_build()
    monkeypatch.setattr(build, "native_abi", lambda: "torch 0.0, other")
    assert build.needs_build()


def test_a_module_of_another_version_is_refused(monkeypatch):
    _lib.lib()
    monkeypatch.setattr(build, "native_abi", lambda: "torch 0.0, other")
    monkeypatch.setattr(build, "needs_build", lambda: False)
    monkeypatch.setattr(_lib, "_lib", None)
    with pytest.raises(RuntimeError, match="rebuild"):
        _lib.lib()
