"""The binding's native half belongs to one interpreter: its file carries that
interpreter's ABI tag, so that another one neither loads it nor takes it for
fresh, and it compiles without what only newer headers have."""
import importlib.machinery
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest

from conftest import ROOT
from p3arsec_gb300 import abi, build


def test_the_file_is_named_for_this_interpreter():
    build.build()
    name = os.path.basename(build.PYCALL)
    assert name == "_pycall" + importlib.machinery.EXTENSION_SUFFIXES[0]
    assert sys.implementation.cache_tag in name
    assert os.path.exists(build.PYCALL)
    abi.load()
    assert abi._call.__file__ == build.PYCALL


def test_another_interpreters_file_is_not_loaded(tmp_path, monkeypatch):
    build.build()
    for name in ("_pycall.so", "_pycall.cpython-311.so"):
        shutil.copy(build.PYCALL, tmp_path / name)
    monkeypatch.setattr(build, "PYCALL", str(tmp_path / ("_pycall" + sysconfig.get_config_var("EXT_SUFFIX"))))
    with pytest.raises(RuntimeError, match="build it with this Python"):
        abi._load_pycall()


def test_it_compiles_for_an_older_interpreter(tmp_path):
    """As version 3.11, without the functions that 3.12 added."""
    (tmp_path / "old.cpp").write_text("""
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#undef PY_VERSION_HEX
#define PY_VERSION_HEX 0x030B0000
#pragma GCC poison PyUnstable_Long_IsCompact PyUnstable_Long_CompactValue
#include "bsg_pycall.cpp"
""")
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-Wall", "-I" + os.path.join(ROOT, "include"),
                        "-I" + build.CSRC, "-I" + sysconfig.get_paths()["include"], str(tmp_path / "old.cpp")],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
