"""What the build does with and without torch, with the compiler replaced by a list of its command lines."""
import importlib.util
import os
import re
import subprocess

import pytest

from jjjetson_ops_b200 import _build


@pytest.fixture
def commands(monkeypatch, tmp_path):
    """A package folder whose library and binding modules are up to date, and what is compiled there."""
    ran = []

    def run(cmd):
        ran.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w"):
            pass

    monkeypatch.setattr(_build, "_run", run)
    monkeypatch.setattr(_build, "_build_library", lambda *a: None)
    monkeypatch.setattr(_build, "BINDINGS", {})
    for name, folder in (("PKG_DIR", tmp_path), ("PY_DIR", tmp_path / "python"), ("OBJ_DIR", tmp_path / "build")):
        monkeypatch.setattr(_build, name, str(folder))
    return ran


def test_without_torch_the_rest_is_built(commands, monkeypatch):
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert _build.build_all() == _build.LIB_PATH and commands == []


def test_another_torch_is_another_build(commands, monkeypatch):
    _build.build_all()
    assert len(commands) == 1 and os.path.basename(commands[0][commands[0].index("-o") + 1]).startswith("_torch_calls")
    _build.build_all()
    assert len(commands) == 1
    monkeypatch.setattr(_build.importlib.metadata, "version", lambda name: "0.0.0")
    _build.build_all()
    assert len(commands) == 2


def test_the_fp16_operand_gemm_keeps_nothing_in_local_memory(tmp_path):
    """As the compiler reports it: no instance has a stack frame (a look-up by matrix in a by-value parameter takes one) or spills."""
    done = subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-Xptxas", "-v", "-I", _build.INCLUDE_DIR, "-cubin", "-o", str(tmp_path / "x.cubin"),
                           os.path.join(_build.CSRC, "mmq_gemm_f16_sm100.cu")], capture_output=True, text=True, check=True)
    frames = re.findall(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", done.stdout + done.stderr)
    assert len(frames) == 12 and set(frames) == {("0", "0", "0")}  # one and several matrices, three forms, with and without time stamps
