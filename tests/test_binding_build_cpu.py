"""The binding's CPython module: built for the interpreter that asks for it, and
left out where there are no Python headers (the C and C++ user's build)."""
import os
import stat
import subprocess
import sys
import sysconfig

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cheddar-fhe_b200")


def commands(python):
    return subprocess.run(["make", "-n", "-B", "-C", PKG, "all", f"PYTHON={python}"], check=True, text=True,
                          stdout=subprocess.PIPE, stderr=subprocess.PIPE).stdout


def test_module_is_named_after_the_interpreter(pkg):
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert pkg.CALLS_PATH.endswith("cheddar_b200_calls" + suffix)
    assert os.path.basename(pkg.CALLS_PATH) in commands(sys.executable)


def test_build_without_python_headers(tmp_path):
    """An interpreter without headers, and none at all: the library and the host
    programs are built all the same."""
    bare = tmp_path / "python3"
    bare.write_text("#!/bin/sh\necho /nonexistent .suffix.so\n")
    bare.chmod(bare.stat().st_mode | stat.S_IXUSR)
    for python in (bare, tmp_path / "none"):
        out = commands(python)
        assert "py_calls.c" not in out and "libcheddar_b200.so" in out


def test_package_builds_for_its_own_interpreter(pkg, monkeypatch):
    seen = []
    monkeypatch.setattr(pkg.subprocess, "check_call", lambda cmd: seen.append(cmd))
    pkg.build()
    assert f"PYTHON={sys.executable}" in seen[0]
