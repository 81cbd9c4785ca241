"""The native host side of the operators (_b200_host.so) saves time only: without one that fits, the same calls go through Python, and the libraries build."""
import types

import pytest

import tgis_b200  # noqa: F401
from tgis_b200 import _lib


@pytest.fixture
def build(monkeypatch):
    mod = _lib._build_module()
    monkeypatch.setattr(_lib, "_build_module", lambda: mod)
    monkeypatch.setattr(_lib, "_host", None)
    return mod


@pytest.mark.parametrize("how", ["absent", "for another torch", "not a library"])
def test_calls_go_through_python(build, monkeypatch, tmp_path, how):
    path = tmp_path / "_b200_host.so"
    if how != "absent":
        path.write_bytes(b"\x7fELF" + (build.host_tag() if how == "not a library" else build.host_tag().replace("torch ", "torch 1")).encode())
    monkeypatch.setattr(build, "HOST_LIB", str(path))
    monkeypatch.setattr(_lib, "HOST_PATH", str(path))
    with pytest.warns(UserWarning, match="is not used"):
        host = _lib.load_host(0, types.SimpleNamespace(), None, None)
    assert host.gemm_f16(1, 2, 3) is None and host.linear_bf16() is None


def test_libraries_build_without_it(build, monkeypatch, capsys):
    def fails(force=False):
        raise FileNotFoundError("Python.h")
    monkeypatch.setattr(build, "build_host", fails)
    assert build.build(target="seq") == build.SEQ_LIB
    assert "calls go through Python" in capsys.readouterr().err


def test_built_again_for_another_torch(build, monkeypatch, tmp_path):
    path = tmp_path / "_b200_host.so"
    path.write_bytes(b"b200_host for python 3.1, torch 0.0;")
    ran = []
    monkeypatch.setattr(build, "HOST_LIB", str(path))

    def run(cmd, **kw):
        ran.append(cmd)
        (tmp_path / cmd[cmd.index("-o") + 1]).write_bytes(b"new " + build.host_tag().encode())
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")
    monkeypatch.setattr(build.subprocess, "run", run)
    build.build_host()
    assert len(ran) == 1 and build.host_fits()
    build.build_host()
    assert len(ran) == 1
