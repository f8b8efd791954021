"""The native front end on CPU: when it is loaded, and what happens where it has not been built."""
import os
import shutil
import subprocess
import sys

import pytest
import torch

import helpers
from pypto_b200 import _lib

BUILT = ("libdsv32_b200.so", "_front.so")


@pytest.fixture(scope="module")
def built():
    if not all(os.path.exists(os.path.join(os.path.dirname(_lib.LIB_PATH), f)) for f in BUILT):
        from pypto_b200 import build
        build.build()
    return os.path.join(helpers.ROOT, "pypto_b200")


@pytest.fixture
def checkout(built, tmp_path):
    """The tree's files without anything built, and where the built files are."""
    shutil.copytree(built, tmp_path / "pypto_b200", ignore=shutil.ignore_patterns("*.so", "build", "__pycache__"))
    shutil.copytree(os.path.join(helpers.ROOT, "include"), tmp_path / "include")
    shutil.copy(os.path.join(helpers.ROOT, "__graft_entry__.py"), tmp_path)
    return tmp_path


def _python(code, cwd):
    env = {k: v for k, v in os.environ.items() if k not in ("PYTHONPATH", "DSV32_B200_LIB")}
    return subprocess.run([sys.executable, "-c", code], cwd=cwd, env=env, capture_output=True, text=True, timeout=300)


def test_first_build_of_a_clean_checkout_loads_in_the_same_process(checkout, built):
    # the compilers are replaced by a copy of what they made before; everything else is build()'s own way
    r = _python(f"""
import shutil
import __graft_entry__
from pypto_b200 import build
def made(**kw):
    for f in {BUILT!r}:
        shutil.copy({built!r} + "/" + f, "pypto_b200")
    return "pypto_b200/libdsv32_b200.so"
build.build = made
__graft_entry__.build()
from pypto_b200 import _lib
assert _lib.front.__name__ == "pypto_b200._front", _lib.front
""", checkout)
    assert r.returncode == 0, r.stderr


def test_package_and_oracle_leave_the_native_code_alone(built):
    r = _python("""
import pypto_b200
from pypto_b200 import decode_chain, sharding, synth
from oracle import dsv32_oracle
assert "_front.so" not in open("/proc/self/maps").read()
assert "libdsv32_b200.so" not in open("/proc/self/maps").read()
""", helpers.ROOT)
    assert r.returncode == 0, r.stderr


def test_missing_front_end_is_an_error_that_says_so(checkout, built):
    shutil.copy(os.path.join(built, "libdsv32_b200.so"), checkout / "pypto_b200")
    r = _python("from pypto_b200 import _lib; _lib.load()", checkout)
    assert r.returncode != 0
    assert "_front.so) cannot be imported" in r.stderr and "python -m pypto_b200.build" in r.stderr
    assert "circular import" not in r.stderr


class _Front:
    """Stands in for the native module."""
    ABI_VERSION, TORCH_VERSION = _lib.ABI_VERSION, torch.__version__.split("+")[0]

    def bind(self, *args):
        pass

    def set_status(self, *args):
        pass


@pytest.mark.parametrize("name,value", [("ABI_VERSION", _lib.ABI_VERSION - 1), ("TORCH_VERSION", "1.0.0")])
def test_front_end_of_another_build_is_refused(built, monkeypatch, name, value):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_import_front", type("Front", (_Front,), {name: value}))
    with pytest.raises(_lib.Dsv32Error, match=f"built for .* {value}"):
        _lib.load()


def test_front_end_says_what_it_was_built_for(built):
    _lib.load()
    assert (_lib.front.ABI_VERSION, _lib.front.TORCH_VERSION) == (_Front.ABI_VERSION, _Front.TORCH_VERSION)


def test_front_end_linked_against_another_torch_is_stale(built, monkeypatch, tmp_path):
    from pypto_b200 import build
    stamp = tmp_path / "front_torch"
    monkeypatch.setattr(build, "FRONT_TORCH", str(stamp))
    monkeypatch.setattr(build, "_newest_source_mtime", lambda: 0.0)
    assert build.is_stale()
    stamp.write_text("1.0.0")
    assert build.is_stale()
    stamp.write_text(torch.__version__)
    assert not build.is_stale()


def test_status_words_made_before_the_load_reach_the_front_end(built, monkeypatch):
    seen = []

    class Front(_Front):
        def set_status(self, *args):
            seen.append(args)

    for name, value in (("_lib", None), ("front", _lib._NotLoaded()), ("_status_words", {}), ("_import_front", Front)):
        monkeypatch.setattr(_lib, name, value)
    _lib.set_status(3, 0x1000)
    assert _lib.front.indexer(None) is None and not seen   # declined: the Python layer takes the call
    _lib.load()
    _lib.set_status(4, 0x2000)
    assert seen == [(3, 0x1000), (4, 0x2000)]
