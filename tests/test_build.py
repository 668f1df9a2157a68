"""The in-tree build and the loading of its two files (no GPU, nothing is compiled here)."""
import ctypes
import importlib.util
import os
import shutil

import pytest
import torch

from yasakani_b200 import _lib, build


@pytest.fixture(scope="module", autouse=True)
def built():
    build.build()


def test_library_alone_needs_no_torch(monkeypatch):
    monkeypatch.setattr(importlib.util, "find_spec", lambda name: None)
    monkeypatch.setattr(build, "build_host", lambda *a: pytest.fail("the extension needs torch"))
    assert build.build() == build.LIB


def test_stale_with_other_flags_or_sources(monkeypatch):
    assert not build._stale()
    with monkeypatch.context() as m:
        m.setattr(build, "NVCC_FLAGS", build.NVCC_FLAGS + ["-O2"])
        assert build._stale()
    with monkeypatch.context() as m:                                 # a source that went away
        left = build.sources()[1:]
        m.setattr(build, "sources", lambda: left)
        assert build._stale()


def test_extension_of_another_torch_or_header_is_another_file(monkeypatch, tmp_path):
    mine = build.host_path()
    assert os.path.exists(mine)
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.1")
        assert build.host_path() != mine
    header = tmp_path / "abi.h"
    header.write_bytes(open(build.ABI, "rb").read() + b"\n")
    monkeypatch.setattr(build, "ABI", str(header))
    assert build.host_path() != mine


def test_loading_never_rebuilds_a_library_in_use(monkeypatch):
    _lib.load()
    monkeypatch.setattr(build, "build", lambda *a, **k: pytest.fail("the library is loaded already"))
    monkeypatch.setattr(build, "build_lib", lambda *a, **k: pytest.fail("the library is loaded already"))
    made = []
    monkeypatch.setattr(build, "build_host", lambda: made.append(1) or build.host_path())
    assert callable(_lib._Host().decode) and made


def test_two_copies_of_the_library_are_refused(monkeypatch, tmp_path):
    """Status words, algorithm choice and error texts live in the library: the launchers must call the copy that ctypes calls."""
    copy = shutil.copy(build.LIB, tmp_path / "libyskn_kv4.so")
    monkeypatch.setattr(_lib, "_LIB", ctypes.CDLL(str(copy)))
    with pytest.raises(ImportError, match="another copy"):
        _lib._Host().decode
