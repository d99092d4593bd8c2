"""Tiles (the body kernel's Gauss-point input, mel_tiles.h) checked on the CPU: a model of the
kernel's pass (tests/emul/tile_emul.cpp) follows every record with its bounds checked, finds no
shared-memory wavefront that meets a bank twice, and reproduces the oracle's internal forces bit
for bit from the FP64 tiles, and a direct scatter within rounding from the FP32 ones."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, flat_of, squeezed_lattice


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("emul") / "libtileemul.so")
    csrc = os.path.join(ROOT, "melody2d_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-I" + csrc,
                    "-I" + os.path.join(ROOT, "include"), "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "emul", "tile_emul.cpp"), os.path.join(csrc, "mel_tiles.cpp"), "-o", out],
                   check=True)
    L = C.CDLL(out)
    L.emul_tiles.argtypes = [C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 4
    L.emul_error.restype = C.c_char_p
    return L


def run(emul, flat, cap, mixed, up):
    from melody2d_b200.abi import Desc
    desc = Desc(flat)
    f, direct, stats = np.zeros_like(up), np.zeros_like(up), np.zeros(4, dtype=np.int64)
    rc = emul.emul_tiles(C.byref(desc.desc), cap, mixed, up.ctypes.data, f.ctypes.data, direct.ctypes.data, stats.ctypes.data)
    assert rc == 0, (rc, emul.emul_error())
    return f, direct, stats


@pytest.mark.parametrize("cap", [2048, 2176, 3840, 8192])
def test_fp64_tiles_match_oracle(emul, oracle_built, cap):
    from oracle.pyoracle import Oracle
    flat = flat_of(squeezed_lattice(3, 3))
    o = Oracle(flat)
    o.step(30)
    up = np.ascontiguousarray(o.node_state()[:, 6:8]).copy()
    o.step(1)
    f, _, stats = run(emul, flat, cap, 0, up)
    assert 0 < stats[3] <= cap
    np.testing.assert_array_equal(f, o.forces()["internal"])
    assert np.abs(f).max() > 0


@pytest.mark.parametrize("cap", [4096, 8192])
def test_mixed_tiles_match_a_direct_scatter(emul, cap):
    flat = flat_of(squeezed_lattice(3, 3))
    up = np.random.default_rng(5).standard_normal((len(flat["node_x0"]) // 2, 2)) * 1e-5
    f, direct, stats = run(emul, flat, cap, 1, up)
    assert 0 < stats[3] <= cap
    # sums of at most a few hundred FP64 terms in another order
    np.testing.assert_allclose(f, direct, rtol=0, atol=1e-12 * np.abs(direct).max())


def thinned(flat, seed, counts):
    """`flat` with every Gauss point's support list cut to, or repeated up to, a drawn length: points with
    as few as one support and as many as the 255 a point may have, as the tile's groups, rows and word
    padding see them.  A longer list names other nodes of the body, each once."""
    rng = np.random.default_rng(seed)
    f = dict(flat)
    ptr, idx, gp = flat["gp_sup_ptr"], flat["gp_sup_idx"], flat["body_gp_ptr"]
    nptr = flat["body_node_ptr"]
    out_ptr, out_idx, dx, dy = [0], [], [], []
    for b in range(len(flat["body_type"])):
        n = nptr[b + 1] - nptr[b]
        for g in range(gp[b], gp[b + 1]):
            c = min(int(rng.choice(counts)), n)
            out_idx.append(np.sort(rng.choice(n, c, replace=False)))
            dx.append(rng.standard_normal(c)); dy.append(rng.standard_normal(c))
            out_ptr.append(out_ptr[-1] + c)
    f["gp_sup_ptr"] = np.array(out_ptr, dtype=np.int32)
    f["gp_sup_idx"] = np.concatenate(out_idx).astype(np.int32)
    f["gp_dNdx"], f["gp_dNdy"] = np.concatenate(dx), np.concatenate(dy)
    f["gp_N"] = np.zeros_like(f["gp_dNdx"])
    return f


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("counts", [[1], [1, 2, 3, 4, 5], [15, 16, 17], [7, 20, 33], [1, 16, 140], [255]])
def test_support_counts_at_the_edges(emul, mixed, counts):
    flat = thinned(flat_of(squeezed_lattice(3, 3)), 3, counts)
    up = np.random.default_rng(6).standard_normal((len(flat["node_x0"]) // 2, 2)) * 1e-5
    f, direct, stats = run(emul, flat, 4096, mixed, up)
    assert stats[1] == len(flat["gp_sup_idx"]) and 0 < stats[3] <= 4096
    if mixed:
        np.testing.assert_allclose(f, direct, rtol=0, atol=1e-12 * np.abs(direct).max())
