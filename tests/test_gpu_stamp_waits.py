"""The give-up path of the stamped cells' waits: tests/device/stamp_waits.cu is
compiled against the library's device headers and run; it exits 0 when every
block left within the wait limit, with the timeout status raised."""
import os
import subprocess

import pytest

from mke_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def compiled(tmp_path):
    exe = str(tmp_path / "stamp_waits")
    r = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-I", build.SRC,
                        os.path.join(HERE, "device", "stamp_waits.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.gpu
def test_waits_end_and_free_the_barrier(tmp_path):
    r = subprocess.run([compiled(tmp_path)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "waits ended" in r.stdout, r.stdout + r.stderr
