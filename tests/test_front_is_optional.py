"""The native front of calls on torch tensors is a convenience: without it, or with one for another torch, the library is built and the calls are served (no GPU)."""
import contextlib
import ctypes
import os
import subprocess

import pytest
import torch

from jitnn_b200 import DType, Gguf, Tensor, _lib, build, ops


@pytest.fixture()
def tree(tmp_path, monkeypatch):
    """A tree with one source whose compilers only note what they are asked for."""
    (tmp_path / "one.cu").write_text("")
    (tmp_path / "one.cuh").write_text("")
    (tmp_path / "front.cpp").write_text("")
    for name, value in {"HERE": tmp_path / "package", "CSRC": tmp_path, "OBJ": tmp_path / "build", "LIB": tmp_path / "lib.so", "FRONT_SRC": tmp_path / "front.cpp"}.items():
        monkeypatch.setattr(build, name, str(value))
    monkeypatch.setattr(_lib, "HERE", str(tmp_path))
    monkeypatch.setattr(build, "nvcc", lambda: "nvcc")
    built = []

    def run(cmd, **kwargs):
        out = cmd[cmd.index("-o") + 1]
        built.append(os.path.basename(out))
        if run.front_fails and build.FRONT_SRC in cmd:
            return subprocess.CompletedProcess(cmd, 1, "", "no headers")
        open(out, "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")

    run.front_fails = False
    monkeypatch.setattr(build.subprocess, "run", run)
    return built, run


def test_without_torch_the_library_is_built(tree, monkeypatch):
    def missing(name):
        raise _lib.importlib.metadata.PackageNotFoundError(name)

    monkeypatch.setattr(_lib.importlib.metadata, "version", missing)
    monkeypatch.setattr(build, "find_spec", lambda name: None)
    assert os.path.exists(build.build()) and tree[0] == ["one.o", "lib.so"]


def test_where_the_front_cannot_be_built_the_library_is(tree, capsys):
    tree[1].front_fails = True
    assert os.path.exists(build.build()) and "lib.so" in tree[0]
    assert "no headers" in capsys.readouterr().err


def test_another_torch_has_another_front(tree, monkeypatch):
    build.build()
    first = _lib.front_path()
    assert os.path.exists(first)
    monkeypatch.setattr(_lib.importlib.metadata, "version", lambda name: "99.0")
    assert _lib.front_path() != first and not os.path.exists(_lib.front_path())
    assert _lib.load_front(Tensor) is None  # the other's is not loaded
    build.build()
    assert os.path.exists(_lib.front_path()) and not os.path.exists(first)


@pytest.mark.parametrize("content", [None, b"not a shared object"])
def test_calls_go_on_without_it(content, tmp_path, monkeypatch):
    monkeypatch.setattr(_lib, "HERE", str(tmp_path))
    monkeypatch.setattr(ops, "_torch", None)
    monkeypatch.setattr(ops, "_front", None)
    if content is not None:
        with open(_lib.front_path(), "wb") as f:
            f.write(content)
    w = Tensor(ctypes.c_void_p(1), DType.Q4_K, (4, 256), 0)
    try:
        with pytest.warns(UserWarning) if content is not None else contextlib.nullcontext(), pytest.raises(ValueError, match="input on cpu"):
            Gguf.linear(torch.zeros(1, 256), w)  # (the general code's refusal: it has been reached)
        assert ops._front is None
    finally:
        w._h = None
