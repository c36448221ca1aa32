"""Tile arithmetic of the CTA-pair kernel, compiled for the host: the tiles of a group cover its rows once, every box
holds the half tile it is taken for, and the boxes encoded for a group of known size are those its tiles use -- at most
two, since a forward with a shared expert encodes them on every call."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("pair") / "libpairprobe.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(ROOT, "tests", "pair_tiles_probe.cpp"), "-o", str(so)])
    return C.CDLL(str(so))


def test_tiles_and_boxes(lib):
    a = [(C.c_int * 64)() for _ in range(4)]
    for rows in list(range(1, 3000)) + [4095, 4096, 4097, 8191, 8192, 8193, 16383]:
        n = lib.pair_probe_walk(rows, *a)
        row0, size, box, half = (list(x[:n]) for x in a)
        assert n == -(-rows // 256)
        assert row0[0] == 0 and all(row0[i] + size[i] == row0[i + 1] for i in range(n - 1)) and row0[-1] + size[-1] == rows
        assert all(1 <= s <= 256 for s in size)
        assert all(0 <= b < 8 and half[i] <= 16 * (b + 1) < half[i] + 16 for i, b in enumerate(box))
        mask = lib.pair_probe_mask(rows)
        assert mask == sum(1 << b for b in set(box))
        assert bin(mask).count("1") <= 2
    assert lib.pair_probe_mask(0) == 0
