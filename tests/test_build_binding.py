"""The binding of the hot call: built for this interpreter's ABI, and not needed where it cannot be built."""
import ctypes
import sysconfig

import pytest

from georefine_b200 import _native
from georefine_b200 import build as lib_build

BAD_ARGUMENT = 1


def test_named_for_the_interpreter():
    assert lib_build.FASTCALL.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


@pytest.mark.parametrize("broken", [None, "no compiler", "no headers"])
def test_the_call_is_there_with_and_without_a_compiler(monkeypatch, tmp_path, broken):
    _native.lib()
    monkeypatch.setattr(_native, "_FASTCALL", None)
    monkeypatch.setattr(lib_build, "FASTCALL", tmp_path / lib_build.FASTCALL.name)
    if broken == "no compiler":
        monkeypatch.setattr(lib_build.shutil, "which", lambda name: None)
    elif broken == "no headers":
        monkeypatch.setattr(lib_build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
        monkeypatch.setenv("CPATH", "")
    assert lib_build.build() == lib_build.OUT                      # the library itself needs neither
    assert lib_build.FASTCALL.exists() == (broken is None)
    call, entry = _native.gemm_partials()
    assert call(entry, *[0] * 16) == BAD_ARGUMENT                  # reached the library: null pointers are refused there
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        call(entry, 1.5, *[0] * 15)


def test_a_binding_older_than_its_source_is_built_again(monkeypatch, tmp_path):
    import os

    monkeypatch.setattr(lib_build, "FASTCALL", tmp_path / lib_build.FASTCALL.name)
    assert lib_build.build_fastcall()
    os.utime(lib_build.FASTCALL, (0, 0))
    assert lib_build.build_fastcall() and lib_build.FASTCALL.stat().st_mtime > 0
    assert [p.name for p in tmp_path.iterdir()] == [lib_build.FASTCALL.name]
