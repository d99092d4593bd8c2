"""Host memory that runs out while the tiles are built is reported as MEL_ERR_OOM, from the calling thread as
from the builder's other threads, and ends neither (tests/emul/tile_oom.cpp fails one allocation
after the other)."""
import os
import subprocess

import pytest

from conftest import ROOT


# 20 bodies of 100 points of 10 supports: one thread; 60 of 400 of 20 (480,000 entries): three
@pytest.mark.parametrize("size", [(20, 100, 10), (60, 400, 20)])
def test_allocation_failures_are_reported(tmp_path, size):
    exe = str(tmp_path / "tile_oom")
    csrc = os.path.join(ROOT, "melody2d_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + csrc, "-I" + os.path.join(ROOT, "include"),
                    "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "emul", "tile_oom.cpp"),
                    os.path.join(csrc, "mel_tiles.cpp"), "-o", exe], check=True)
    p = subprocess.run([exe, *map(str, size)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr[-500:])
    plan, fill, fine = map(int, p.stdout.split())
    assert plan > 10 and fill > 10 and fine > 0
