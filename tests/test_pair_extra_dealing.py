"""How the CTA-pair kernel deals its tiles when one more group, whose tiles may be longer, rides along
(csrc/grouped_gemm_2cta.cu, `seek`): every tile once, each pair's routed tiles in ascending order, no pair far above the
average."""
import itertools

import pytest


def deal(pairs, extra, routed, weight):
    full, rest = divmod(extra, pairs)
    others, late = pairs - rest, weight * (pairs - rest)
    got_extra, got_routed, load = [], [], [0] * pairs
    for p in range(pairs):
        last, i = -1, 0
        while True:
            tile, m = p + i * pairs, i - full
            if m < 0 or (m == 0 and p < rest):
                got_extra.append(tile)
                load[p] += weight
                i += 1
                continue
            if p < rest:
                t = late + (m - 1) * pairs + p
            elif m < weight:
                t = m * others + p - rest
            else:
                t = late + (m - weight) * pairs + p
            assert t > last
            last = t
            if t >= routed:
                break
            got_routed.append(t)
            load[p] += 1
            i += 1
    return got_extra, got_routed, load


@pytest.mark.parametrize("pairs", [1, 2, 66, 74])
def test_every_tile_once_and_in_order(pairs):
    for extra, routed, weight in itertools.product((0, 1, 8, 44, 73, 74, 75, 148, 200), (0, 5, 73, 480, 660), (1, 2, 4, 9)):
        e, r, load = deal(pairs, extra, routed, weight)
        assert sorted(e) == list(range(extra)) and sorted(r) == list(range(routed))
        if routed >= weight * pairs:  # enough short tiles to even the long ones out
            assert max(load) <= sum(load) / pairs + weight + 1


def test_shapes_of_the_shared_expert():
    # 60 experts x 8 feature tiles of 22 k-blocks beside 8 of 88; 64 x 8 beside 8 of 44; gate/up, all of 32
    assert max(deal(74, 8, 480, 4)[2]) == 7 and max(deal(74, 8, 512, 2)[2]) == 8 and max(deal(74, 22, 704, 1)[2]) == 10
