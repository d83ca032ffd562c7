"""What a build compiles (no compiler runs here)."""
import os
import subprocess
import sys

import pytest
import torch

from nanochat_b200.csrc import build as b


@pytest.fixture
def built(monkeypatch, tmp_path):
    """Both libraries in place and newer than every source; returns the list of commands that a build runs."""
    commands = []

    def compile_(cmd, verbose):
        commands.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w"):
            return 0
    monkeypatch.setattr(b, "PKG", str(tmp_path))
    monkeypatch.setattr(b, "_compile", compile_)
    for name, path in (("OUT", tmp_path / "libnckv.so"), ("NATIVE", tmp_path / "_native.so")):
        path.touch()
        monkeypatch.setattr(b, name, str(path))
    monkeypatch.setattr(b, "NATIVE_FOR", b.NATIVE + ".for", raising=False)
    with open(b.NATIVE_FOR, "w") as f:
        f.write(b.native_wanted() if hasattr(b, "native_wanted") else "")
    return commands


def test_nothing_to_do(built):
    assert b.up_to_date() and b.build() == b.OUT and built == []


def test_the_binding_alone(built):
    os.utime(b.NATIVE, (0, 0))
    b.build()
    assert [cmd[cmd.index("-o") + 1].endswith("_native.so") for cmd in built] == [True] and b.up_to_date()


def test_the_kernels_alone(built):
    os.utime(b.OUT, (0, 0))
    b.build()
    assert len(built) == len(b.SOURCES) + 1 and not any(b.BINDING in cmd for cmd in built) and b.up_to_date()


def test_everything_on_demand(built):
    b.build(force=True)
    assert len(built) == len(b.SOURCES) + 2


def test_another_torch_asks_for_another_binding(built, monkeypatch):
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other")
    assert not b.up_to_date()
    b.build()
    assert len(built) == 1 and b.BINDING in built[0] and b.up_to_date()


def test_a_binding_for_another_torch_is_not_loaded():
    code = ("import torch; torch.__version__ += '.other'\n"
            "try:\n import nanochat_b200._lib\nexcept ImportError as e:\n assert 'built for' in str(e) and '--force' in str(e); raise SystemExit(7)")
    assert subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(b.PKG + "/"))).returncode == 7


def test_a_torch_without_cuda_needs_no_binding(built, monkeypatch):
    os.remove(b.NATIVE)
    monkeypatch.setattr(torch.version, "cuda", None)
    assert b.up_to_date()
    b.build(force=True)
    assert len(built) == len(b.SOURCES) + 1 and not any(b.BINDING in cmd for cmd in built)


def test_the_package_imports_under_a_torch_without_cuda():
    code = ("import sys, torch; torch.version.cuda = None; sys.modules['nanochat_b200._native'] = None\n"
            "from nanochat_b200 import _lib, ops, gpt\n"
            "try:\n ops.glue_relu_sq(torch.zeros(8, dtype=torch.bfloat16))\nexcept RuntimeError as e:\n assert 'CUDA' in str(e); raise SystemExit(7)")
    assert subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.dirname(b.PKG + "/"))).returncode == 7
