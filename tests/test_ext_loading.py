"""Which front end the package's per-call functions take: the extension when it is there and complete, else ctypes."""
import sys
import types
import warnings

import pytest

import h100_gdn_cuda_b200 as package
from h100_gdn_cuda_b200 import api, build


@pytest.fixture
def fresh(monkeypatch, tmp_path):
    """api with nothing decided yet; `place(module, built)` puts a module (None: one that does not import) in its place."""
    monkeypatch.setattr(api, "_ext", None)
    monkeypatch.delattr(package, "gdn_cuda", raising=False)

    def place(module, built):
        monkeypatch.setitem(sys.modules, package.__name__ + ".gdn_cuda", module)
        if module is not None:
            monkeypatch.setattr(package, "gdn_cuda", module, raising=False)
        out = tmp_path / "gdn_cuda.so"
        if built:
            out.write_bytes(b"")
        monkeypatch.setattr(build, "ext_path", lambda: str(out))
    return place


def _module(names):
    m = types.ModuleType("gdn_cuda")
    for n in names:
        setattr(m, n, lambda *a: n)
    return m


def test_complete_extension_is_used(fresh):
    m = _module(api._FAST)
    fresh(m, True)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert api._load_ext() is m


@pytest.mark.parametrize("names", [(), api._FAST[:-1]])
def test_older_extension_is_left_alone(fresh, names):
    fresh(_module(names), True)
    with pytest.warns(RuntimeWarning, match="older"):
        assert api._load_ext() is False


def test_extension_that_does_not_import(fresh):
    fresh(None, True)
    with pytest.warns(RuntimeWarning, match="build --ext"):
        assert api._load_ext() is False


def test_library_alone_is_silent(fresh):
    fresh(None, False)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert api._load_ext() is False
