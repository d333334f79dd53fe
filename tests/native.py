"""Compiles a host program against the engine's host-only headers (no CUDA) and runs it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "culsh_b200", "csrc")


def run_native(tmp_path, source, stdin="", timeout=60, flags=()):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "program.cpp", tmp_path / "program"
    src.write_text(source)
    subprocess.run([gxx, "-std=c++17", "-O1", "-g", "-pthread", "-I", CSRC, str(src), "-o", str(exe), *flags], check=True)
    res = subprocess.run([str(exe)], input=stdin, capture_output=True, text=True, timeout=timeout)
    assert res.returncode == 0, res.stdout + res.stderr
    return res.stdout
