"""The extension module of the binding's hot calls is optional: without it, or with one built for another torch, every call
goes the general way, and the library builds without torch and g++.  No CUDA device is needed here."""
import pytest
import torch


@pytest.fixture
def binding(engine, monkeypatch):
    from qwen35x_b200 import engine as e

    monkeypatch.setattr(e, "_native_module", None)
    monkeypatch.setattr(e, "_torch", lambda: torch)  # which asks for a CUDA device
    return e


def _declines(binding):
    with pytest.warns(RuntimeWarning, match="q35b_torch.so"):
        assert binding._native().gemv(0, None, None, 0) is NotImplemented
    assert binding._native().batch_run(0) is NotImplemented


def test_module_is_missing(binding, monkeypatch, tmp_path):
    monkeypatch.setattr(binding, "_NATIVE_PATH", tmp_path / "q35b_torch.so")
    _declines(binding)


def test_module_of_another_torch(binding, monkeypatch, tmp_path):
    (tmp_path / "stamp").write_text("torch-1.0 python-3.1")
    monkeypatch.setattr(binding, "_NATIVE_STAMP", tmp_path / "stamp")
    _declines(binding)


@pytest.mark.parametrize("without", ["torch", "g++"])
def test_library_builds_without(engine, monkeypatch, without):
    from qwen35x_b200 import build

    if without == "torch":
        monkeypatch.setattr(build.importlib.util, "find_spec", lambda name: None)
    else:
        monkeypatch.setattr(build.shutil, "which", lambda name: None)
    monkeypatch.setattr(build, "_stale", lambda out, deps: False)
    monkeypatch.setattr(build, "build_binding", lambda force=False: pytest.fail("needs torch and g++"))
    assert build.build() == build.LIB


def test_module_is_rebuilt_for_another_torch(engine, monkeypatch, tmp_path):
    from qwen35x_b200 import build
    from qwen35x_b200.engine import native_stamp

    (tmp_path / "stamp").write_text("torch-1.0 python-3.1")
    monkeypatch.setattr(build, "BINDING_STAMP", tmp_path / "stamp")
    monkeypatch.setattr(build, "_stale", lambda out, deps: False)
    ran = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, check: ran.append(cmd))
    build.build_binding()
    assert len(ran) == 1 and (tmp_path / "stamp").read_text() == native_stamp(torch)
    build.build_binding()
    assert len(ran) == 1
