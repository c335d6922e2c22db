"""The host check in front of the composed block solver: tests/host/block_parts.cpp
against the library's own assembly (no GPU)."""
import os
import shutil
import subprocess

import pytest

from mke_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_systems_that_the_parts_do_not_make_up_are_refused(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "block_parts")
    r = subprocess.run(["g++", *build.HOST, "-I", build.SRC, os.path.join(HERE, "host", "block_parts.cpp"),
                        *[os.path.join(build.SRC, f) for f in ("phg_mesh.cpp", "phg_assemble.cpp", "phg_mgplan.cpp")],
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "block parts checked" in r.stdout, r.stdout + r.stderr
