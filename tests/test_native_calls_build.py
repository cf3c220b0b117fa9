"""The calls without ctypes are built for the interpreter that builds them, under its name, and only where it has headers; the
library is built all the same."""
import os
import subprocess
import sys
import sysconfig

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "semi_pd_b200", "csrc")


def _commands(python):
    out = subprocess.run(["make", "-n", "-B", "-C", CSRC, "PYTHON=" + python], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert "libspd.so" in out.stdout
    return [line.split() for line in out.stdout.splitlines() if line.strip().startswith("g++")]


def test_name_is_the_interpreters():
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    (words,) = _commands(sys.executable)
    assert words[words.index("-o") + 1] == "../_calls" + suffix and suffix != ".so"


def test_without_headers_the_library_alone(tmp_path):
    python = tmp_path / "python"
    python.write_text("#!/bin/sh\necho %s\n" % tmp_path)  # its headers' folder, and as suffix: no Python.h there
    python.chmod(0o755)
    assert _commands(str(python)) == []
    assert _commands(str(tmp_path / "missing")) == []
