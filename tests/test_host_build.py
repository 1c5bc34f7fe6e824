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
