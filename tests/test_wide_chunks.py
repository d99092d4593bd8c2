"""Chunk sizes of bodies above 4,096 nodes, checked on the CPU: the images take as many entries as their form
allows and leave room for two thread blocks on a multiprocessor; with less room they get smaller."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

ROOM = 116736 - 1024             # half a B200 multiprocessor's 233,472 bytes less what a block reserves


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emul") / "libwideemul.so")
    csrc = os.path.join(ROOT, "melody2d_b200", "csrc")
    emul_dir = os.path.join(ROOT, "tests", "emul")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + csrc, "-I" + os.path.join(ROOT, "include"),
                    "-I/usr/local/cuda/include", os.path.join(emul_dir, "wide_emul.cpp"), os.path.join(emul_dir, "error_stub.cpp"),
                    os.path.join(csrc, "mel_chunks.cpp"), "-o", out], check=True)
    L = C.CDLL(out)
    L.emul_wide_chunks.argtypes = [C.c_void_p, C.c_longlong, C.c_int, C.c_void_p]
    return L


@pytest.fixture(scope="module")
def flat():
    from melody2d_b200 import generator as g
    return g.flatten(g.biaxial_scene(seed=3, n_discs=2, n_border=160, n_interior=4200, workers=1))


def chunks(emul, flat, room, mixed):
    from melody2d_b200.abi import Desc
    st = np.zeros(4, dtype=np.int64)
    assert emul.emul_wide_chunks(C.byref(Desc(flat).desc), room, mixed, st.ctypes.data) == 0
    assert st[1] == len(flat["gp_weight"])
    return st


@pytest.mark.parametrize("mixed,points,ceiling", [(0, 110, 224), (1, 194, 224)])
def test_points_of_a_chunk(emul, flat, mixed, points, ceiling):
    """Mixed images of 3,584 entries hold some 200 points of 17 supports for 224 threads (of 2,048 entries,
    117); FP64 ones of 2,048 entries some 115."""
    st = chunks(emul, flat, ROOM, mixed)
    assert st[3] <= ceiling and st[1] / st[0] >= points
    assert 128 + 2 * st[2] <= ROOM


@pytest.mark.parametrize("mixed", [0, 1])
def test_less_room(emul, flat, mixed):
    full = chunks(emul, flat, ROOM, mixed)
    half = chunks(emul, flat, ROOM // 2, mixed)
    assert 128 + 2 * half[2] <= ROOM // 2 and half[0] > full[0]
