"""Building the host module of the calls: where it cannot be built, when it is built again."""

from __future__ import annotations

from pathlib import Path

import pytest

from edgerag_b200.ops import native


@pytest.mark.parametrize("error", [native.NativeBuildError("no C++ compiler"), FileNotFoundError("c++")])
def test_libraries_are_built_without_the_host_module(monkeypatch, capfd, error):
    """A machine that has nvcc alone runs through ctypes; the build of everything does not end there."""
    def no_host(*a, **k):
        raise error

    monkeypatch.setattr(native, "build_host", no_host)
    monkeypatch.setattr(native, "build", lambda library, elem, verbose=True: Path(f"lib{library}_{elem}.so"))
    built = native.build_all(verbose=False)
    assert len(built) > 10 and all(p.name.startswith("lib") for p in built)
    assert "ctypes" in capfd.readouterr().err


@pytest.fixture()
def folder(monkeypatch, tmp_path):
    """An empty folder for what is built, and a compiler that counts its runs and writes what it is asked for, or fails."""
    runs = []

    def command(out):
        runs.append(out)
        return ["sh", "-c", "exit 3" if (tmp_path / "broken").exists() else f"echo built > {out}"]

    monkeypatch.setattr(native, "PACKAGE_EXT", tmp_path)
    monkeypatch.setattr(native.tempfile, "gettempdir", lambda: str(tmp_path / "other"))
    monkeypatch.delenv("EDGERAG_B200_EXT_DIR", raising=False)
    monkeypatch.setattr(native, "_host_command", command)
    return tmp_path, runs


def test_other_flags_or_another_compiler_build_anew(folder, monkeypatch):
    _, runs = folder
    native.build_host(False), native.build_host(False)
    assert len(runs) == 1
    monkeypatch.setattr(native, "HOST_FLAGS", (*native.HOST_FLAGS, "-g"))
    native.build_host(False), native.build_host(False)
    assert len(runs) == 2
    monkeypatch.setenv("CXX", "another-c++")
    native.build_host(False), native.build_host(False)
    assert len(runs) == 3


def test_a_failed_compilation_is_remembered(folder):
    """A program's start does not ask a compiler again that failed on the same; the build of everything does."""
    at, runs = folder
    (at / "broken").touch()
    for _ in range(2):
        assert native.load_host() is None
    assert len(runs) == 1
    with pytest.raises(native.NativeBuildError):
        native.build_host(False)
    assert len(runs) == 2
    (at / "broken").unlink()
    assert native.load_host() is None and len(runs) == 2
    assert native.build_host(False).is_file() and native.build_host(False, retry=False).is_file() and len(runs) == 3
