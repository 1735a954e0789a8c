"""When the native side of the frequent calls is taken as it lies there: only with the torch, the sources and the library that
it was made for. Otherwise it is made again, or the calls go without it and say so."""
import ctypes
import subprocess

import pytest
import torch

from ccbench_b200 import _lib


@pytest.fixture
def load():
    _lib.build_calls()
    return _lib.calls.__wrapped__   # as in a process that has not asked yet


def _no_compiler(monkeypatch, asked):
    def build(force=False, verbose=False):
        asked.append(force)
        raise subprocess.CalledProcessError(1, "g++")

    monkeypatch.setattr(_lib, "build_calls", build)


def test_it_is_loaded_where_it_fits(load, monkeypatch, recwarn):
    _no_compiler(monkeypatch, asked := [])
    module = load()
    assert not asked and not recwarn.list
    assert module.built_for().startswith(f"torch {torch.__version__} ") and set(_lib._calls_marks()) == set(module.built_for().split("; "))


@pytest.mark.parametrize("what", ["version", "build", "sources"])
def test_another_torch_or_other_sources_are_not_loaded(load, monkeypatch, tmp_path, what):
    if what == "version":
        monkeypatch.setattr(torch, "__version__", "2.99.0")
    elif what == "build":
        monkeypatch.setattr(torch.version, "git_version", "0" * 40)
    else:
        source = tmp_path / "ccb_calls.cpp"
        source.write_bytes(_lib.CALLS_SOURCE.read_bytes() + b"\n")
        monkeypatch.setattr(_lib, "CALLS_SOURCE", source)
    _no_compiler(monkeypatch, asked := [])

    def loaded(*_):
        raise AssertionError("a module of another torch was loaded")

    monkeypatch.setattr(_lib.importlib.machinery.ExtensionFileLoader, "create_module", loaded)
    with pytest.warns(RuntimeWarning, match="slower way"):
        assert load() is None
    assert asked == [False]


def test_a_library_without_what_it_calls(load, monkeypatch):
    class Old:
        def __getattr__(self, name):
            if name == "ccb_sz_container_sums":
                raise AttributeError(name)
            return ctypes.CFUNCTYPE(None)(lambda: None)

    monkeypatch.setattr(_lib, "lib", Old)
    with pytest.warns(RuntimeWarning, match="ccb_sz_container_sums"):
        assert load() is None
