"""Looking for the native host side of the per-layer calls (no GPU): what does not load is passed by."""
import sys
import warnings

import pytest

from inquant import _native as N


@pytest.fixture
def unsought(monkeypatch):
    monkeypatch.setattr(N, "_host", None)
    monkeypatch.setattr(N, "_host_sought", False, raising=False)
    return monkeypatch


def test_the_built_module_is_found(unsought):
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        host = N.host()
    assert host is not None and host is N.host() and all(callable(getattr(host, n)) for n in ("append_token", "decode", "paged_decode"))


def test_a_module_that_does_not_load_is_passed_by_with_one_warning(unsought):
    unsought.setitem(sys.modules, "inquant._host", None)       # an import of it raises ImportError
    with pytest.warns(RuntimeWarning, match="does not load|built for"):
        assert N.host() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert N.host() is None
