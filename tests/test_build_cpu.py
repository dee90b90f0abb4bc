"""``_host.so`` is bound to one PyTorch and Python: it is rebuilt when they change, and one that does not load says what to do."""
import sys

import pytest

import swamla_b200
from swamla_b200 import _cabi, build, functional


def test_host_library_is_rebuilt_for_another_pytorch(monkeypatch):
    build.build()
    calls = []
    monkeypatch.setattr(build, "_build_host", lambda: calls.append(1))
    build.build()
    assert not calls
    monkeypatch.setattr(build, "_host_versions", lambda: "torch 0.0, python 0.0")
    build.build()
    assert calls == [1]


def test_unloadable_host_library_says_how_to_build_it(monkeypatch):
    monkeypatch.setattr(functional, "_native", None)
    monkeypatch.delattr(swamla_b200, "_host", raising=False)
    monkeypatch.setitem(sys.modules, "swamla_b200._host", None)
    with pytest.raises(_cabi.LmoeError, match="swamla_b200.build"):
        functional._host()
