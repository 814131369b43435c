# SPDX-License-Identifier: Apache-2.0
"""Permutations that keep neighbours together: their constraint graphs join
pair-nodes next to each other, so that union-find hangs every pair-node under
its predecessor and a node's chains get as long as the node.  Each is a valid
input and has to give the oracle's bytes, on every path that uses union-find:
nodes above the walk limit of 2^23 entries, and the second pass of any size
after a walk gave up."""
import ctypes

import numpy as np
import pytest

from helpers import b200_format, oracle_format

pytestmark = pytest.mark.gpu


def structured(kind, n):
    rng = np.random.default_rng(n)
    i = np.arange(n, dtype=np.int64)
    if kind == "pairs":  # neighbours (2k + 1, 2k + 2) stay together, in any order
        order = rng.permutation((n - 1) // 2)
        p = np.empty(n, dtype=np.int64)
        p[1 + 2 * order] = 2 * np.arange(order.size)
        p[2 + 2 * order] = 2 * np.arange(order.size) + 1
        rest = [0] if n & 1 else [0, n - 1]
        p[rest] = np.arange(2 * order.size, n)
    elif kind == "blocks":  # blocks of odd length, shuffled as a whole
        size = 100_001 if n > 1 << 23 else 4_001
        order = rng.permutation(-(-n // size))
        p = np.concatenate([np.arange(b * size, min(n, (b + 1) * size)) for b in order])
    elif kind == "rotation":
        p = (i + n // 2 + 1) % n
    elif kind == "odd_rotation":
        p = (i + 12345) % n
    elif kind == "reverse":
        p = n - 1 - i
    else:  # the even places first, then the odd ones
        assert kind == "riffle"
        p = np.where(i % 2 == 0, i // 2, (n + 1) // 2 + i // 2)
    return p.astype(np.uint32)


KINDS = ("pairs", "blocks", "rotation", "odd_rotation", "reverse", "riffle")


def check(gpu, oracle, kind, n, **kw):
    perm = structured(kind, n)
    assert gpu.compress(perm, gpu.CompressOptions(format=b200_format(gpu, kw))) == \
        oracle.compress(perm, oracle_format(kw))


@pytest.mark.parametrize("n", [(1 << 23) + 1, (1 << 23) + 2])
@pytest.mark.parametrize("kind", KINDS)
def test_smallest_union_nodes(gpu, oracle, kind, n):
    check(gpu, oracle, kind, n, middle_placement=n & 1)


@pytest.mark.slow
@pytest.mark.parametrize("kind,n", [("pairs", (1 << 25) + 2), ("odd_rotation", (1 << 25) + 3),
                                    ("blocks", (1 << 25) + 3)])
def test_unions_by_windows(gpu, oracle, kind, n):
    """Nodes above 2^25 entries, whose unions go by windows, over two levels
    of union-find."""
    check(gpu, oracle, kind, n)


@pytest.mark.parametrize("n", [8193, 16387, 40_000, (1 << 17) + 1, (1 << 18) - 2, (1 << 20) + 1])
@pytest.mark.parametrize("mode", [True, "fallback"])
def test_union_find_on_every_level(gpu, oracle, n, mode):
    gpu.set_union_find_only(mode)
    try:
        for m, kind in enumerate(KINDS):
            check(gpu, oracle, kind, n, middle_group_log2=1 + m % 5)
    finally:
        gpu.set_union_find_only(False)


def test_batch_allocation_free_and_shards(gpu, oracle):
    """The other forms with union-find on every level: a batch's members that
    meet a long chain are encoded again by themselves, beside one that does
    not; a shard sees its own part of the levels."""
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    fmt = gpu.FormatOptions()
    cfmt = gpu.to_c_format(fmt)
    gpu.set_union_find_only(True)
    try:
        items, keep = [], []
        for n, kind in ((100_003, "pairs"), (70_000, "riffle"), (131_073, None), (200_000, "reverse")):
            perm = structured(kind, n) if kind else \
                gpu.fill_permutation(gpu.PermutationKind.uniform, n, n, np.uint32)
            want = oracle.compress(perm, oracle_format({}))
            src = torch.from_numpy(perm.view(np.int32)).cuda()
            blob = torch.zeros((len(want) + 3) // 4 * 4, dtype=torch.uint8, device="cuda")
            keep.append((src, blob, want))
            items.append((src.data_ptr(), n, 4, fmt, blob.data_ptr(), len(want)))
        torch.cuda.synchronize()
        gpu.compress_batch_device(items)
        for _, blob, want in keep:
            assert blob.cpu().numpy()[:len(want)].tobytes() == want
        err = ctypes.create_string_buffer(256)
        for src, blob, want in keep:
            blob.zero_()
            rc = gpu.library().bpb200_compress_device_noalloc(
                ctypes.c_void_p(src.data_ptr()), ctypes.c_uint64(src.numel()), ctypes.c_uint32(4),
                ctypes.byref(cfmt), ctypes.c_void_p(blob.data_ptr()), ctypes.c_uint64(len(want)),
                ctypes.c_void_p(stream), err, ctypes.c_size_t(256))
            assert rc == 0, err.value.decode()
            assert blob.cpu().numpy()[:len(want)].tobytes() == want
        src, blob, want = keep[0]
        total = np.zeros(len(want), dtype=np.uint32)
        for shard in range(2):
            gpu.compress_device_shard(src.data_ptr(), src.numel(), 4, blob.data_ptr(), len(want),
                                      shard, 2, fmt, stream)
            total += blob.cpu().numpy()[:len(want)]
        assert total.max() <= 255 and total.astype(np.uint8).tobytes() == want
    finally:
        gpu.set_union_find_only(False)


def test_calls_at_once(gpu, oracle):
    """Several host threads' calls at once, on streams of their own: the
    launches of one wait for their own blocks only."""
    from concurrent.futures import ThreadPoolExecutor
    n = (1 << 23) + 5
    perms = [structured(kind, n) for kind in ("pairs", "riffle", "reverse", "rotation")]
    with ThreadPoolExecutor(4) as pool:
        wants = list(pool.map(lambda p: oracle.compress(p, oracle_format({})), perms))
        for _ in range(5):
            assert list(pool.map(gpu.compress, perms)) == wants
