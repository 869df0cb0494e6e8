"""Environment switches: what os.environ says at the call, whatever its mapping keeps inside."""
import os

import pytest

from fused_cpp_b200 import _lib


class _TextTable(dict):
    """A mapping whose private table is keyed by text."""

    @property
    def _data(self):
        return dict(self)


@pytest.mark.parametrize("environ", [None, _TextTable, dict], ids=["os.environ", "text table", "no table"])
def test_switch_follows_the_environment(monkeypatch, environ):
    if environ is not None:
        monkeypatch.setattr(os, "environ", environ())
    switch = _lib.Switch("FUSED_CPP_MOE_TEST_SWITCH", "default")
    assert switch.get() == "default"
    monkeypatch.setitem(os.environ, switch.name, "grün")
    assert switch.get() == "grün"
    monkeypatch.delitem(os.environ, switch.name)
    assert switch.get() == "default"
