"""The rules for the form of a conv launch (host code): how many CTAs share a tile, so that every cluster of the launch is resident
at once, and how wide the tiles of the others are."""
import ctypes

import pytest

from lokinfer_b200 import _lib

SMS = 148
CLUSTERS = (0, 0, 74, 45, 33, 26, 22, 15, 15)  # what cudaOccupancyMaxActiveClusters answers on a B200


def split(ci, co, lo, sms=SMS, clusters=CLUSTERS):
    table = (ctypes.c_int32 * 9)(*clusters)
    return _lib.lib().lkc_conv1d_tc_split(ci, co, lo, sms, table)


@pytest.mark.parametrize("c", [16, 32, 48, 112, 128, 256, 512, 1104, 4096])
@pytest.mark.parametrize("sms", [SMS, SMS * 26 // 100, SMS * 70 // 100, 1, 7])
def test_every_split_launch_is_resident_at_once(c, sms):
    blocks, chunks = -(-c // 128), c // 16
    for lo in [*range(1, 1400, 41), *range(1023, 9700, 129), 9472, 9473, 20000]:
        for clusters in (CLUSTERS, (0,) * 9, (0, 0, 60, 40, 30, 20, 20, 8, 1)):
            n, tiles = split(c, c, lo, sms, clusters), -(-lo // 128) * blocks
            assert n == 0 or 2 <= n <= min(8, chunks)
            if n:
                assert tiles <= clusters[n] and tiles * n <= sms
                assert -(-chunks // n) < -(-chunks // (n - 1))  # no CTA that shortens no run
            else:  # nothing would fit
                for m in range(2, min(8, chunks, sms // tiles) + 1):
                    ctas = -(-chunks // -(-chunks // m))
                    assert tiles > clusters[ctas]


def test_lengths_around_the_limits():
    assert split(128, 128, 15 * 128) == 8 and split(128, 128, 15 * 128 + 1) == 4  # 16 tiles: 15 clusters of eight fit
    assert split(128, 128, 48 * 128) == 2  # 45 clusters of three fit
    assert split(256, 256, 896) == 8 and split(256, 256, 897) == 6
    assert split(128, 128, 9472) == 2 and split(128, 128, 9473) == 0
    assert split(16, 16, 1) == 0 and split(100, 16, 1) == 0 and split(128, 128, 0) == 0


def test_columns_of_a_split_tile():
    cols = _lib.lib().lkc_conv1d_tc_split_cols
    assert [cols(n) for n in (1, 32, 63, 64)] == [64] * 4 and [cols(n) for n in (65, 128, 129, 9472)] == [128] * 4
    assert cols(0) == cols(-1) == 0


def tile_cols(co, lo, percent=100, sms=SMS):
    return _lib.lib().lkc_conv1d_tc_tile_cols(co, lo, sms, percent)


@pytest.mark.parametrize("co", [22, 128, 256, 512])
@pytest.mark.parametrize("percent", [26, 50, 99, 100])
@pytest.mark.parametrize("sms", [SMS, 20])
def test_tile_widths(co, percent, sms):
    """Alone: no width takes fewer SM-columns in whole rounds (48 columns of cost beside a tile's own), the widest of equals. Beside
    other launches: the narrowest that fits one round of the share, else whole tiles. Widths are multiples of the 32 columns that
    the narrow tiles' statistics cover, so no pair spans two tiles."""
    blocks, widths = -(-co // 128), (256, 224, 192, 160)
    for lo in [*range(1, 3000, 97), *range(3001, 130000, 1009), 9472, 9473, 19201, 23680, 23681, 124801]:
        w = tile_cols(co, lo, percent, sms)
        tiles = {v: -(-lo // v) * blocks for v in widths}
        cost = {v: -(-tiles[v] // sms) * (v + 48) for v in widths}
        if percent == 100:
            assert w == min(widths, key=lambda v: (cost[v], -v))
        else:
            fits = [v for v in widths[1:] if tiles[v] <= sms * percent // 100]
            assert w == (min(fits) if fits else 256)
    assert tile_cols(0, 100) == tile_cols(128, 0) == tile_cols(128, 100, 0) == tile_cols(128, 100, 100, 0) == 0


def test_tile_widths_of_known_lengths():
    assert tile_cols(128, 19201) == 160 and tile_cols(256, 12001) == 192  # 121 and 126 tiles on 148 SMs
    assert tile_cols(128, 124801, 50) == 256 and tile_cols(128, 9601, 50) == 160  # 976 tiles of any width; 61 on 74 SMs


def branch_sms(t, stage, branch, sms=SMS, clusters=CLUSTERS):
    return _lib.lib().lkc_generator_branch_sms(t, stage, branch, sms, (ctypes.c_int32 * 9)(*clusters))


@pytest.mark.parametrize("stage,branch,base,wider", [(0, 0, 26, 40), (0, 1, 36, 40), (0, 2, 60, 60), (1, 0, 26, 26), (1, 1, 36, 36),
                                                     (1, 2, 50, 50)])
def test_generator_branches_take_more_sms_only_where_their_tiles_would_be_whole(stage, branch, base, wider):
    c = (256, 128)[stage]
    for t in [*range(1, 300), 747, 2080]:
        whole = split(c, c, (10 * t, 60 * t + 1)[stage], SMS * base // 100) == 0
        assert branch_sms(t, stage, branch) == (wider if whole else base)


def test_generator_branches_of_known_lengths():
    # k = 3 of stage 0: 18 tiles at T = 115, two CTAs each on 38 SMs; 20 at T = 116, two CTAs each on 59 SMs only
    assert [branch_sms(t, 0, 0) for t in (24, 80, 100, 115, 116, 160)] == [26, 26, 26, 26, 40, 40]
    assert [branch_sms(t, 0, 1) for t in (24, 100, 121, 166, 167, 320)] == [36, 36, 36, 36, 40, 40]
    assert [branch_sms(t, 0, 0, clusters=(0,) * 9) for t in (24, 160)] == [40, 40]  # a device that holds no clusters
    assert branch_sms(0, 0, 0) == branch_sms(10, 2, 0) == branch_sms(10, -1, 0) == branch_sms(10, 0, 3) == branch_sms(10, 0, 0, 0) == 0
