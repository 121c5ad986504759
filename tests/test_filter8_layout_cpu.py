"""Shared-memory layout of the 8-lane collaborative filter (csrc/zb3d_filter.cuh), restated and
checked on the CPU: each position of a group has a place of its own inside the group's
buffer, every 16-byte access of a warp (4 groups of 8 lanes) is free of bank conflicts in both
layouts, and what a lane reads after a change of layout is what the other lanes stored."""
import numpy as np

PATCH, GROUP, OFF = 68, 552, 18


def col_off(x, half):
    return x * 8 + ((half ^ (x >> 2)) << 2)


def addr(g, p, x, half):
    return g * GROUP + p * PATCH + col_off(x, half)


def quads_distinct(addrs):  # 8 lanes of a 16-byte access: 8 different bank quads
    return len({(a // 4) % 8 for a in addrs}) == 8 and all(a % 4 == 0 for a in addrs)


def test_positions_are_distinct_and_inside():
    seen = {addr(0, p, x, half) + i for p in range(8) for x in range(8) for half in range(2) for i in range(4)}
    assert len(seen) == 512 and min(seen) >= 0 and max(seen) < GROUP


def test_accesses_are_conflict_free():
    for g in range(4):  # a quarter warp is one group
        for half in range(2):
            for p in range(8):  # layout X: lane x, patch p
                assert quads_distinct([addr(g, p, lane, half) for lane in range(8)])
            for x in range(8):  # layout P: lane p, column x
                assert quads_distinct([addr(g, lane, x, half) for lane in range(8)])
    # 8-byte patch offsets, one per group and access: different banks
    assert len({(2 * OFF * g) % 32 for g in range(4)}) == 4


def test_changes_of_layout_deliver_every_value():
    rng = np.random.default_rng(1)
    v = rng.integers(0, 1 << 30, (4, 8, 8, 8))  # group, patch, row, column
    buf = np.zeros(4 * GROUP, np.int64)
    for g in range(4):
        for lane in range(8):  # X: the lane's column of every patch, rows 4 half .. 4 half + 3
            for p in range(8):
                for half in range(2):
                    a = addr(g, p, lane, half)
                    buf[a:a + 4] = v[g, p, 4 * half:4 * half + 4, lane]
    for g in range(4):
        for lane in range(8):  # P: the lane's patch, every column, rows as pairs
            for x in range(8):
                got = np.concatenate([buf[addr(g, lane, x, half):addr(g, lane, x, half) + 4] for half in range(2)])
                assert np.array_equal(got, v[g, lane, :, x])
