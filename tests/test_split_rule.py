"""The rules for the form of a conv launch (host code): how many CTAs share a tile, so that every cluster of the launch is resident
at once, how wide the tiles of the others are, which of them go to CTA pairs, and which convs go in two launches."""
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


def pair_cols(ci, co, lo, k, d=1, act=1, fine=False, behind=False, percent=100, clusters=CLUSTERS):
    table = (ctypes.c_int32 * 9)(*clusters)
    return _lib.lib().lkc_conv1d_tc_pair_cols(ci, co, lo, k, d, d * (k - 1) // 2, act, fine, behind, percent, SMS, table)


@pytest.mark.parametrize("ci", [16, 112, 128, 256, 512, 1104, 4096])
@pytest.mark.parametrize("clusters", [CLUSTERS, (0, 0, 60, 40, 30, 20, 20, 8, 1), (0,) * 9])
def test_what_goes_to_pairs(ci, clusters):
    for co in (128, 250, 256, 384, 512, 1024):
        for lo in [*range(1, 30000, 997), 9472, 9473, 124801]:
            for k in (1, 3, 7, 11):
                for fine in (False, True):
                    w, few = (pair_cols(ci, co, lo, k, fine=fine, percent=p, clusters=clusters) for p in (100, 60))
                    width = 160 if fine else 128
                    rounds = -(-(-(-lo // width) * (co // 256)) // clusters[2]) if clusters[2] and co % 256 == 0 else 0
                    assert w in (0, width) and few in (0, width)
                    if rounds == 0 or split(ci, co, lo, SMS, clusters):
                        assert w == 0
                    if rounds == 0 or split(ci, co, lo, SMS * 60 // 100, clusters):
                        assert few == 0
                    elif ci < 4096:  # beside other launches: one round (4096 channels: K = 11 finds no room)
                        assert (few != 0) == (rounds == 1)
                    assert not (w and ci < 128 and rounds > 3)


def test_pairs_are_left_where_their_rounds_cost_more():
    # a resblock of 256 channels: one round of 148 tiles of 160 columns as 74 pairs; 126 to 148 tiles of 192 to 256 columns; two rounds
    for k in (3, 7, 11):
        assert [pair_cols(256, 256, lo, k, fine=True, behind=True) for lo in (4737, 11840, 20800)] == [160] * 3
    for k in (7, 11):
        assert [pair_cols(256, 256, lo, k, fine=True, behind=b) for lo in (11841, 12000, 15000, 18000) for b in (0, 1)] == [0] * 8
    assert [pair_cols(256, 256, 14000, 3, fine=True, behind=b) for b in (0, 1)] == [0, 160]
    # statistics per 128 columns: the other form's tiles are 256 wide
    assert [pair_cols(256, 256, lo, k) for lo in (4864, 9472, 19200) for k in (3, 7, 11)] == [128] * 9
    assert [pair_cols(256, 256, 9600, 7), pair_cols(512, 512, 4800, 7), pair_cols(512, 512, 4800, 3)] == [0, 0, 128]
    # few channels, no Snake
    assert [pair_cols(16, 256, 9600, 1), pair_cols(64, 256, 9600, 3), pair_cols(64, 256, 9472, 3)] == [0, 0, 128]
    assert [pair_cols(64, 256, lo, 3) for lo in (20800, 60000)] == [128, 0]
    assert [pair_cols(256, 256, 12000, 3, act=a) for a in (0, 1, 2)] == [0, 128, 0]
    # 60 pairs at a time
    few = (0, 0, 60, 40, 30, 20, 20, 8, 1)
    assert [pair_cols(256, 256, lo, 7, fine=True, clusters=few) for lo in (9472, 9600, 9601)] == [160, 160, 0]
    lib, t = _lib.lib(), (ctypes.c_int32 * 9)(*CLUSTERS)
    good = [256, 256, 9472, 3, 1, 1, 1, 0, 0, 100, SMS]
    assert lib.lkc_conv1d_tc_pair_cols(*good, t) == 128 and lib.lkc_conv1d_tc_pair_cols(*good, None) == 0
    for i, v in ((0, 100), (1, 0), (2, 0), (3, 0), (4, 0), (4, 26), (4, 1 << 20), (5, -1), (6, 3), (9, 0), (9, 101), (10, 0)):
        assert lib.lkc_conv1d_tc_pair_cols(*good[:i], v, *good[i + 1:], t) == 0


def full_rounds(ci, co, lo, k, clusters=CLUSTERS):
    return _lib.lib().lkc_conv1d_tc_full_rounds(ci, co, lo, k, SMS, (ctypes.c_int32 * 9)(*clusters))


@pytest.mark.parametrize("clusters", [CLUSTERS, (0, 0, 60, 40, 30, 20, 20, 8, 1), (0,) * 9])
def test_two_launches_are_whole_rounds_and_a_split_rest(clusters):
    taken = 0
    for c in (16, 128, 250, 256, 384, 512, 640, 1024):
        ci, blocks = -(-c // 16) * 16, -(-c // 128)
        for lo in [*range(1, 45000, 331), 9473, 18945, 37889, 124801]:
            for k in (1, 3, 7, 11):
                cols = full_rounds(ci, c, lo, k, clusters)
                if not cols:
                    continue
                taken += 1
                assert 0 < cols < lo and cols % 256 == 0 and cols // 256 * blocks <= -(-lo // 256) * blocks // SMS * SMS
                assert split(ci, c, lo, SMS, clusters) == 0 and split(ci, c, cols, SMS, clusters) == 0
                assert split(ci, c, lo - cols, SMS, clusters) >= 2
    assert (taken > 0) == (clusters[2] > 0)


def test_two_launches_of_known_lengths():
    assert [full_rounds(512, 512, lo, 7) for lo in (9472, 9473, 9500, 19200)] == [0, 9472, 9472, 18944]
    assert [full_rounds(256, 256, lo, 11) for lo in (18944, 18945, 19201, 20800)] == [0, 18944, 18944, 18944]
    assert [full_rounds(128, 128, lo, k) for lo, k in ((37889, 11), (37889, 3), (9473, 11))] == [37888, 0, 0]
    assert full_rounds(512, 512, 19200, 3) == 0 and full_rounds(256, 256, 9473, 11) == 0  # 76 of 148 tiles
    assert [full_rounds(*bad) for bad in ((100, 256, 19201, 11), (256, 0, 19201, 11), (256, 256, 0, 11), (256, 256, 19201, 65))] == [0] * 4
