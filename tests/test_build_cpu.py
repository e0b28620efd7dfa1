"""What the build does where something is missing or has changed."""
import importlib.util
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def build(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("qfb_build_under_test", os.path.join(ROOT, "qfactory-ae_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    for name in ("LIB", "TORCH_LIB"):
        path = tmp_path / os.path.basename(getattr(mod, name))
        path.write_bytes(b"built")
        monkeypatch.setattr(mod, name, str(path))
    monkeypatch.setattr(mod, "TORCH_FOR", str(tmp_path / "_qfb_torch.for"))
    return mod


def test_the_library_does_not_need_torch(build, monkeypatch, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)   # import torch raises
    monkeypatch.setattr(build.importlib.metadata, "version", lambda name: (_ for _ in ()).throw(
        build.importlib.metadata.PackageNotFoundError(name)))
    os.remove(build.TORCH_LIB)
    assert build.build() == build.LIB and "torch is not installed" in capsys.readouterr().err


def test_the_module_is_rebuilt_for_another_torch_or_python(build, monkeypatch):
    assert build.torch_module_is_stale("2.0")          # nobody knows what it was built for
    with open(build.TORCH_FOR, "w") as f:
        f.write(build._built_for("2.0"))
    assert not build.torch_module_is_stale("2.0") and build.torch_module_is_stale("2.1")
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name: "cpython-399")
    assert build.torch_module_is_stale("2.0")
    os.remove(build.TORCH_LIB)
    assert build.torch_module_is_stale("2.0")
