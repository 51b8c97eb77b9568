"""A mesh whose move to host memory fails is read whole or not at all: the copy
and each of the three allocations failing, before another extraction and when
the context goes (host code with stubs, no GPU)."""
import os
import shutil
import subprocess

import pytest

from tgvreconclaude_gb300 import _native as N

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "mesh_moves.cpp")


def test_failed_moves_lose_nothing_silently(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "mesh_moves")
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-O1", "-I", N.INCLUDE, "-I", N.CSRC, SRC,
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
