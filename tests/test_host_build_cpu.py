"""Loading of the native host path."""

import pytest

from velox_voice_b200 import _lib


def test_a_host_module_of_another_build_is_not_loaded(monkeypatch):
    """The module is compiled against one torch, one Python and one C ABI; when it does not belong to the present ones and
    cannot be rebuilt, loading it would call through a wrong layout."""
    _lib.host()  # the present module is there
    monkeypatch.setattr(_lib, "_host", None)
    monkeypatch.setattr(_lib._build, "host_is_current", lambda: False)

    def fails(*a, **k):
        raise RuntimeError("g++ failed")

    monkeypatch.setattr(_lib._build, "build_host", fails)
    with pytest.raises(RuntimeError, match="g\\+\\+ failed"):
        _lib.host()
