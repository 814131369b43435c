# SPDX-License-Identifier: Apache-2.0
"""The level arrays hold every level that a call, or one shard of it, writes:
level l takes 2^l nodes of 2 * pcap slots, pcap = ceil(ceil(n / 2^l) / 2)
rounded up to even, and the last node's slots must lie inside the arrays.
Host arithmetic only."""
import numpy as np
import pytest

from helpers import b200_format


def slots_of(n, level):
    cap = -(-n // (1 << level))
    pairs = (-(-cap // 2) + 1) // 2 * 2
    return (2 * pairs) << level


def check(b200, n, kw, shards):
    fmt = b200_format(b200, kw)
    _, tile_level = b200.describe(n, fmt)
    if shards > 1 << tile_level:
        return 0
    for shard in {0, shards - 1}:
        levels, slots = b200.probe_scratch(n, fmt, shard, shards)
        assert levels == sorted(set(levels)) and (not levels or levels[-1] >= tile_level)
        for level in levels:
            assert slots_of(n, level) <= slots, (n, kw, shards, level)
    return len(levels)


@pytest.mark.parametrize("shards", [1, 2, 4, 8, 64])
def test_level_arrays_hold_every_level(b200, shards):
    rng = np.random.default_rng(shards)
    sizes = [4097, 8192, 8193, 16385, 100_003, (1 << 18) - 1, 1 << 18, (1 << 20) + 5, (1 << 22) + 1,
             2045 << 12, (1 << 23) + 4097, 100_000_007, 1 << 30, 1 << 31]
    sizes += [int(2 ** e) for e in rng.uniform(11, 31, 400)]
    handed = [check(b200, n, kw, shards) for n in sizes
              for kw in (dict(), dict(middle_group_log2=1, middle_placement=1))]
    assert max(handed) >= 3


def test_scratch_probe_rejects_bad_shards(b200):
    for shard, shards in ((0, 3), (2, 2), (0, 1 << 20)):
        with pytest.raises(ValueError):
            b200.probe_scratch(100_003, None, shard, shards)
