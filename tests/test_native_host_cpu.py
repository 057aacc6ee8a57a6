"""Looking for the native host side of the per-layer calls (no GPU): what does not load is passed by."""
import sys
import types
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


@pytest.mark.parametrize("built_for", [None, "PyTorch 1.0.0, cpython-39, C++11 ABI 0"])
def test_a_module_for_another_pytorch_is_never_bound(unsought, built_for):
    """It may load all the same and misread tensors."""
    module = types.ModuleType("inquant._host")
    module.bind = lambda *_: pytest.fail("bound")
    if built_for:
        module.built_for = built_for
    unsought.setitem(sys.modules, "inquant._host", module)
    with pytest.warns(RuntimeWarning, match="built for"):
        assert N.host() is None


def test_the_module_is_built_anew_for_another_pytorch(unsought, tmp_path):
    import build
    commands = []
    unsought.setattr(build, "HERE", str(tmp_path))
    unsought.setattr(build, "HOST", str(tmp_path / "_host.so"))
    (tmp_path / "build").mkdir()

    def compiled(command, check):
        commands.append(command)
        (tmp_path / "_host.so").write_text("")
    unsought.setattr(build.subprocess, "run", compiled)
    unsought.setattr(build, "_stale", lambda target, _: not (tmp_path / "_host.so").exists())
    for version, runs in (("2.0", 1), ("2.0", 1), ("2.1", 2), ("2.1", 2)):
        unsought.setattr(N, "host_built_for", lambda: f"PyTorch {version}")
        build.build_host()
        assert len(commands) == runs and f'-DINQ_BUILT_FOR="PyTorch {version}"' in commands[-1]


@pytest.mark.parametrize("native", [True, False])
def test_lists_of_the_same_objects(unsought, native):
    if not native:
        unsought.setattr(N, "_host_sought", True)
    assert (N.host() is not None) == native
    a, b = object(), object()
    for x, y, same in (([], [], True), ([a], [], False), ([a, b], [a, b], True), ([a, b], [b, a], False), ([a, a], [a, b], False),
                       ([1000.5], [float("1000.5")], False)):       # equal, but another object
        assert N.same_objects(x, y) is same
