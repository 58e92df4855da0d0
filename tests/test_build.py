"""What build.py needs for what, and what the operator module does without the native form of its call."""
import importlib.util
import os
import re
import subprocess
import sys

import pytest
import torch

from conftest import PKG, ROOT


@pytest.fixture
def build():
    spec = importlib.util.spec_from_file_location("rsfa_build", os.path.join(PKG, "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.fixture
def fresh(build, tmp_path, monkeypatch):
    """A build whose two outputs are up to date, in a folder of their own."""
    for name, want in (("OUT", build.source_hash(build.FLAGS)), ("OUT_BINDING", build.binding_hash(build.torch_home()))):
        out = tmp_path / (name + ".so")
        out.write_bytes(b"x")
        (tmp_path / (name + ".so.stamp")).write_text(want + "\n")
        monkeypatch.setattr(build, name, str(out))
    return build


def missing(*_):
    raise RuntimeError("nvcc not found")


def test_nothing_to_compile_needs_no_compiler(fresh, monkeypatch):
    monkeypatch.setattr(fresh, "find_nvcc", missing)
    monkeypatch.setattr(fresh.shutil, "which", lambda name: None)
    monkeypatch.setattr(fresh.subprocess, "run", missing)
    assert fresh.build() == fresh.OUT


@pytest.mark.parametrize("without", ["torch", "CUDA in torch", "g++"])
def test_the_library_is_built_where_the_extension_cannot_be(fresh, tmp_path, monkeypatch, capsys, without):
    os.remove(fresh.OUT_BINDING)
    if without == "torch":
        find = importlib.util.find_spec
        monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    elif without == "CUDA in torch":
        (tmp_path / "__init__.py").write_text("")
        spec = importlib.util.spec_from_file_location("torch", str(tmp_path / "__init__.py"))
        monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: spec)
    else:
        monkeypatch.setattr(fresh.shutil, "which", lambda name: None)
    built = []
    monkeypatch.setattr(fresh, "build_library", lambda *a: built.append(a) or fresh.OUT)
    assert fresh.build() == fresh.OUT and len(built) == 1
    assert not os.path.exists(fresh.OUT_BINDING) and "is not built" in capsys.readouterr().err


def test_the_library_comes_first(fresh, monkeypatch):
    order = []
    monkeypatch.setattr(fresh, "build_library", lambda *a: order.append("library") or fresh.OUT)
    monkeypatch.setattr(fresh, "build_binding", lambda *a: order.append("binding"))
    fresh.build()
    fresh.build(trace=True)
    assert order == ["library", "binding", "library"]


def test_the_extension_is_stale_when_the_c_interface_or_torch_changes(build, tmp_path, monkeypatch):
    home = build.torch_home()
    before = build.binding_hash(home)
    assert os.path.join(ROOT, "include", "rsfa.h") in [os.path.abspath(f) for f in build.BINDING_INPUTS]
    header = tmp_path / "rsfa.h"
    header.write_text("changed")
    monkeypatch.setattr(build, "BINDING_INPUTS", build.BINDING_INPUTS[:-1] + [str(header)])
    assert build.binding_hash(home) != before
    monkeypatch.undo()
    monkeypatch.setattr(build, "find_nvcc", missing)
    assert build.binding_hash(home) == before                     # where nvcc lies is no part of it
    (tmp_path / "version.py").write_text("__version__ = '0.1'\n")
    assert build.binding_hash(str(tmp_path)) != before and build.torch_version(str(tmp_path)) == "0.1"


def test_the_extension_takes_the_signature_from_the_header():
    text = open(os.path.join(PKG, "csrc", "torch_binding.cpp")).read()
    assert '#include "../../include/rsfa.h"' in text and re.search(r"using FwdFn = decltype\(&rsfa_fwd\)", text)


IMPORT = """
import sys, types, warnings
sys.path.insert(0, %r)
import torch
if %r == "missing":
    sys.modules["ascend_rsfa._rsfa_torch"] = None
else:
    m = types.ModuleType("ascend_rsfa._rsfa_torch")
    if %r == "older":
        m.torch_version = "1.0"
    m.bind = m.forward = lambda *a: 1 / 0
    sys.modules["ascend_rsfa._rsfa_torch"] = m
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    import ascend_rsfa.flash_attention_forward as fa
assert fa._rsfa_torch is None
assert any("native form" in str(w.message) for w in seen)
q = torch.zeros(1, 1, 64, 64, dtype=torch.float16)
try:
    fa.attention(q, q, q, False, 0.5, 64, 64)
except RuntimeError as e:
    assert "no CPU path" in str(e)
    print("python-route-ok", fa.get_tiling(1, 1, 2048, 128, False))
"""


@pytest.mark.parametrize("extension", ["missing", "older", "without a version"])
def test_the_operator_runs_without_the_extension(extension):
    """Not built, or built for another torch, whose tensors may be laid out differently: the ctypes route."""
    r = subprocess.run([sys.executable, "-c", IMPORT % (PKG, extension, extension)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "python-route-ok (128, 128)" in r.stdout, r.stdout + r.stderr


def test_the_extension_in_use_was_built_for_this_torch():
    import ascend_rsfa.flash_attention_forward as fa

    assert fa._rsfa_torch is not None and fa._rsfa_torch.torch_version == str(torch.__version__)
