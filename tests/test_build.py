"""The build where torch is missing, and the guard that ties the extension to the torch it was built against."""
import importlib.util
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("lib_build", os.path.join(ROOT, "aihwkit-lightning_b200", "build.py"))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    for name in ("OUT", "HOST_OUT"):
        monkeypatch.setattr(module, name, str(tmp_path / os.path.basename(getattr(module, name))))
    return module


def test_c_library_without_torch(build, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)  # `import torch` raises ImportError
    open(build.OUT, "w").close()
    build.build_host()
    assert "extension" in capsys.readouterr().out and not os.path.exists(build.HOST_OUT)
    assert not build._stale()  # nothing is missing that could be built
    os.remove(build.OUT)
    assert build._stale()


def test_rebuilt_for_another_torch(build):
    open(build.OUT, "w").close()
    for version, stale in ((torch.__version__, False), ("1.0", True)):
        with open(build.HOST_OUT, "w") as fh:
            fh.write(f"...built for torch {version};...")
        assert build._stale() == stale


def test_extension_of_another_torch_is_refused(tmp_path):
    from aihwkit_lightning_b200 import _lib

    path = tmp_path / "_host_calls.so"
    for text in ("", "built for torch 1.0;"):
        path.write_text(text)
        with pytest.raises(RuntimeError, match="another torch"):
            _lib._check_torch(str(path))
    path.write_text(f"built for torch {torch.__version__};")
    _lib._check_torch(str(path))
    assert _lib.host()  # the one in the tree
