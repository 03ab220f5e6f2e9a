"""Windows and chunks of a layer call, checked on the CPU with the library's own functions (tests/layer_windows_host.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_windows_and_chunks(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++ to build the host harness")
    exe = str(tmp_path / "layer_windows_host")
    build = subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-o", exe, os.path.join(ROOT, "tests", "layer_windows_host.cpp")],
                           capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr[-3000:]
    env = {k: v for k, v in os.environ.items() if k != "MOK_CHUNK_ROWS"}
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300, env=env)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout[-2000:]
