"""How the CTA-pair kernel deals its tiles when one more group, whose tiles may be longer, rides along (csrc/pair_tiles.cuh,
compiled for the host): every tile once, each pair's routed tiles in ascending order, no pair far above the average."""
import ctypes as C
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("deal") / "libdeal.so"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(ROOT, "tests", "pair_tiles_probe.cpp"), "-o", str(so)])
    return C.CDLL(str(so))


def deal(lib, pairs, extra, routed, extra_kb, kb):
    got_extra, got_routed, load = [], [], [0] * pairs
    weight = max(1, (extra_kb + kb // 2) // kb)
    t = C.c_int()
    for p in range(pairs):
        last, i = -1, 0
        while True:
            if lib.pair_probe_deal(pairs, extra, extra_kb, kb, p, i, C.byref(t)):
                got_extra.append(t.value)
                load[p] += weight
                i += 1
                continue
            assert t.value > last
            last = t.value
            if t.value >= routed:
                break
            got_routed.append(t.value)
            load[p] += 1
            i += 1
    return got_extra, got_routed, load


@pytest.mark.parametrize("pairs", [1, 2, 66, 74])
def test_every_tile_once_and_in_order(lib, pairs):
    kbs = ((32, 32, 1), (8, 32, 1), (44, 22, 2), (88, 22, 4), (200, 22, 9))
    for extra, routed, (ekb, kb, weight) in itertools.product((0, 1, 8, 44, 73, 74, 75, 148, 200), (0, 5, 73, 480, 660), kbs):
        e, r, load = deal(lib, pairs, extra, routed, ekb, kb)
        assert sorted(e) == list(range(extra)) and sorted(r) == list(range(routed))
        if routed >= weight * pairs:  # enough short tiles to even the long ones out
            assert max(load) <= sum(load) / pairs + weight + 1


def test_shapes_of_the_shared_expert(lib):
    # 60 experts x 8 feature tiles of 22 k-blocks beside 8 of 88; 64 x 8 beside 8 of 44; gate/up, all of 32
    assert max(deal(lib, 74, 8, 480, 88, 22)[2]) == 7 and max(deal(lib, 74, 8, 512, 44, 22)[2]) == 8
    assert max(deal(lib, 74, 22, 704, 32, 32)[2]) == 10
