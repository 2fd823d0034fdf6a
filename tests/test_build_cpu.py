"""The two built files: the C library needs no torch, and the host extension is rebuilt for another torch."""
import importlib.metadata
import importlib.util

import pytest


@pytest.fixture
def build(monkeypatch, tmp_path):
    from moe_routers_b200 import build as b

    monkeypatch.setattr(b, "HOST_PATH", str(tmp_path / "_host.so"))
    monkeypatch.setattr(b, "HOST_STAMP", str(tmp_path / "host_stamp.txt"))
    return b


def test_library_builds_where_torch_is_absent(build, monkeypatch):
    find_spec = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda n, *a: None if n == "torch" else find_spec(n, *a))
    assert build.build_library() == build.LIB_PATH


def test_host_extension_follows_the_installed_torch(build, monkeypatch):
    """Fresh only where it is newer than its source and was built for this torch: the compiler is called again
    once the version is another one, and not for the same one."""
    calls = []

    def compiler(cmd, **kwargs):
        calls.append(cmd)
        open(build.HOST_PATH, "w").close()
        return type("Done", (), {"returncode": 0, "stdout": ""})()

    monkeypatch.setattr(build.subprocess, "run", compiler)
    version = importlib.metadata.version
    build.build_host()
    build.build_host()
    assert len(calls) == 1
    monkeypatch.setattr(importlib.metadata, "version", lambda n: "99.0" if n == "torch" else version(n))
    build.build_host()
    build.build_host()
    assert len(calls) == 2

    import torch

    assert f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}" in calls[0]
