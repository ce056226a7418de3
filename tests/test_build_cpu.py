"""The host module is tied to the torch and the interpreter that it was compiled against."""
import pytest

from acctransformer_b200 import _lib, build


def test_host_module_of_another_torch_is_rebuilt(monkeypatch):
    import torch
    build.build()
    assert not build.host_is_stale()
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert build.host_is_stale()


def test_host_module_of_another_torch_is_refused(monkeypatch):
    monkeypatch.setattr(_lib, "_host", None)
    assert _lib.host() is _lib.host()
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(build, "host_built_for", lambda: "torch 0.0.0")
    with pytest.raises(ImportError, match="was built for torch .* but this is torch 0.0.0"):
        _lib.host()


def test_library_is_built_without_torch(monkeypatch, capfd):
    import os
    import sys
    monkeypatch.setitem(sys.modules, "torch", None)      # `import torch` fails
    assert os.path.exists(build.build())
    assert "_torch_host is not built" in capfd.readouterr().err
