"""The native host side is built for one torch and Python; the library and the calls do without it."""
import os
import warnings

import pytest

from pbs_attn_b200 import _cabi, build, prefill


def test_nvcc_found_on_the_path_only(monkeypatch, tmp_path):
    tool = tmp_path / "toolkit" / "bin" / "nvcc"
    tool.parent.mkdir(parents=True)
    tool.write_text("#!/bin/sh\n")
    tool.chmod(0o755)
    exists, which = os.path.exists, build.shutil.which
    monkeypatch.setenv("PATH", f"{tool.parent}{os.pathsep}{os.environ['PATH']}")
    monkeypatch.setattr(build.os.path, "exists", lambda p: p != "/usr/local/cuda/bin/nvcc" and exists(p))
    monkeypatch.setattr(build.shutil, "which", lambda c: None if c == "/usr/local/cuda/bin/nvcc" else which(c))
    monkeypatch.delenv("NVCC", raising=False)
    monkeypatch.chdir(tmp_path)
    assert build._nvcc() == str(tool)
    command = build._host_command(str(tmp_path / "x.so"))
    assert str(tmp_path / "toolkit" / "include") in command and "-L" + str(tmp_path / "toolkit" / "lib64") in command


def test_another_torch_has_another_file(monkeypatch):
    import torch
    here = build.host_path()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.host_path() != here


def test_without_it_calls_go_through_python(monkeypatch):
    monkeypatch.setattr(build, "host_path", lambda: "/nowhere/pbs_host.so")
    monkeypatch.setattr(_cabi, "_host", None)
    with pytest.warns(UserWarning, match="go through Python"):
        assert _cabi.load_host() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert _cabi.load_host() is None                   # said once
    plan = object.__new__(prefill.Plan)
    plan.lib, plan.shape, plan.scratch = _cabi.load(), _cabi.Shape(), _cabi.Scratch()
    plan._go_native()
    assert plan._native is None
    monkeypatch.setattr(prefill, "_PLANS", {"some": plan})
    assert prefill._common_call(None, None, None, 64, 128, 0.5, True) is None


def test_a_host_build_that_fails_stops_nothing(monkeypatch, capsys):
    def fail(cmd):
        raise RuntimeError("no headers")

    monkeypatch.setattr(build, "_stale", lambda *a: True)
    monkeypatch.setattr(build.os, "listdir", lambda d: [])
    build._build_host(fail, False)
    assert "no headers" in capsys.readouterr().err
