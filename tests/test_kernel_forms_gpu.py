# SPDX-License-Identifier: Apache-2.0
"""Byte parity with the oracle at the edges of the kernels' forms (tile and
node sizes, group sizes, word boundaries); the bar is byte equality."""
import numpy as np
import pytest

from helpers import b200_format, oracle_format

pytestmark = pytest.mark.gpu


def check(gpu, oracle, n, seed, kind=None, dtype=np.uint32, **kw):
    perm = gpu.fill_permutation(kind if kind is not None else gpu.PermutationKind.uniform, seed,
                                n, dtype)
    got = gpu.compress(perm, gpu.CompressOptions(format=b200_format(gpu, kw)))
    assert got == oracle.compress(perm, oracle_format(kw))


@pytest.mark.parametrize("n", [1, 2, 3, 19, 20, 21, 22, 31, 32, 33, 39, 40, 41, 63, 64, 65,
                               32 * 128 - 1, 32 * 128 + 1])
@pytest.mark.parametrize("placement", [0, 1, 2])
def test_middle_group_ranks(gpu, oracle, n, placement):
    """Groups of 1..32 entries: the 64-bit and the 128-bit Horner steps meet
    at 20 entries; ranks start at every bit offset of a word."""
    for m in (4, 5):
        check(gpu, oracle, n, 7 * n + m, middle_group_log2=m, middle_placement=placement)


@pytest.mark.parametrize("n", [34, 63, 64, 65, 66, 127, 128, 129, 130, 131, 255, 257, 258, 259,
                               1023, 1025, 2049, 4097, 8191, 8192])
def test_tile_nodes(gpu, oracle, n):
    """Odd and even nodes around the one-thread colouring's limits (32 and 64
    pair-nodes) and around the ruler walks' buckets, random and structured."""
    kinds = gpu.PermutationKind
    for m in (1, 2, 5):
        for kind in (kinds.uniform, kinds.single_cycle, kinds.identity, kinds.reverse):
            check(gpu, oracle, n, n + m, kind, np.uint64 if m == 2 else np.uint32,
                  middle_group_log2=m)


@pytest.mark.parametrize("n", [8193, 8194, 16385, 16386, 16387, 32771, (1 << 17) + 6, (1 << 18) - 1,
                               1 << 18, (1 << 18) + 2, (1 << 18) + 3, (1 << 20) + 1])
@pytest.mark.parametrize("jump", [10, 14])
def test_walk_lists(gpu, oracle, n, jump):
    """Global levels coloured by walks, with nodes ranked straight from their
    rulers and after one to three contractions; random and structured."""
    kinds = gpu.PermutationKind
    gpu.set_tuning({"jump_block_log2": jump, "tile_max_log2": 13})
    try:
        for i, kind in enumerate((kinds.uniform, kinds.single_cycle, kinds.identity,
                                  kinds.reverse)):
            check(gpu, oracle, n, n + i, kind, np.uint64 if i & 1 else np.uint32)
    finally:
        gpu.set_tuning(None)


@pytest.mark.parametrize("n,m,placement", [(33, 5, 0), (4097, 1, 1), (70001, 4, 2), (65536, 5, 0)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_lookup_words(gpu, oracle, n, m, placement, shift):
    """Lookups of every entry in a blob at any byte alignment: ranks are read
    as aligned words, the first and last of which reach over its ends."""
    import torch
    kw = dict(middle_group_log2=m, middle_placement=placement)
    perm = gpu.fill_permutation(gpu.PermutationKind.uniform, n + m, n, np.uint64)
    blob = oracle.compress(perm, oracle_format(kw))
    room = torch.zeros(len(blob) + shift, dtype=torch.uint8, device="cuda")
    room[shift:] = torch.frombuffer(bytearray(blob), dtype=torch.uint8).cuda()
    out = torch.empty(n, dtype=torch.int64, device="cuda")
    want = torch.from_numpy(perm.astype(np.int64))
    for inverse in (False, True):
        gpu.lookup_device(room.data_ptr() + shift, len(blob), n, b200_format(gpu, kw),
                          out.data_ptr(), n, inverse=inverse)
        assert torch.equal(out.cpu(), torch.argsort(want) if inverse else want)


@pytest.mark.parametrize("n", [4097, 8193, 16383, 16385, 24577, 32767, 32768, 32769, 65535, 65537,
                               131073])
@pytest.mark.parametrize("m", [1, 4, 5])
def test_stages(gpu, oracle, n, m):
    """Nodes around the stage limit (2^15 entries) and launches of few tiles,
    which hand their subtrees over to more CTAs; the batched form runs the
    same stages from job lists."""
    import torch
    kinds = gpu.PermutationKind
    items, keep = [], []
    for i, kind in enumerate((kinds.uniform, kinds.single_cycle, kinds.reverse)):
        kw = dict(middle_group_log2=m, middle_placement=i)
        dtype = np.uint64 if i == 1 else np.uint32
        check(gpu, oracle, n, n + i, kind, dtype, **kw)
        perm = gpu.fill_permutation(kind, n + i, n, dtype)
        want = oracle.compress(perm, oracle_format(kw))
        src = torch.from_numpy(perm.view(np.int64 if i == 1 else np.int32)).cuda()
        blob = torch.zeros((len(want) + 3) // 4 * 4, dtype=torch.uint8, device="cuda")
        keep.append((src, blob, want))
        items.append((src.data_ptr(), n, perm.dtype.itemsize, b200_format(gpu, kw),
                      blob.data_ptr(), len(want)))
    torch.cuda.synchronize()
    gpu.compress_batch_device(items)
    for _, blob, want in keep:
        assert blob.cpu().numpy()[:len(want)].tobytes() == want


def test_stage_rejects_repeats(gpu):
    """A stage reads the caller's values itself: out of range and repeated
    values are reported, and the next call is right again."""
    for n in (12289, 30000):
        perm = gpu.fill_permutation(gpu.PermutationKind.uniform, n, n, np.uint32)
        good = gpu.compress(perm)
        for bad in (n, int(perm[1])):
            wrong = perm.copy()
            wrong[0] = bad
            with pytest.raises(ValueError):
                gpu.compress(wrong)
            assert gpu.compress(perm) == good


@pytest.mark.slow
@pytest.mark.parametrize("n,kind", [((1 << 25) + 3, 1), ((1 << 25) + 2, 0)])
def test_union_windows(gpu, oracle, n, kind):
    """The smallest nodes whose unions go by windows: the upper window holds
    one or two pair-nodes, the odd tail among them.  (The 100,000,007 and 2^30
    entry digests cover several windows.)"""
    kinds = gpu.PermutationKind
    check(gpu, oracle, n, n, (kinds.uniform, kinds.single_cycle)[kind])


@pytest.mark.parametrize("n", [(1 << 23) + 1, 3 * (1 << 22) + 4093])
def test_bucket_pass(gpu, oracle, n):
    """The smallest partitioned inverses: a last window of one slot, a last
    chunk that is not whole, inputs on and off 16-byte boundaries."""
    import torch
    perm = gpu.fill_permutation(gpu.PermutationKind.uniform, n, n, np.uint32)
    want = oracle.compress(perm, oracle_format({}))
    stream = torch.cuda.current_stream().cuda_stream
    blob = torch.empty((len(want) + 3) // 4 * 4, dtype=torch.uint8, device="cuda")
    for dtype, as_torch in ((np.uint32, np.int32), (np.uint64, np.int64)):
        for shift in (0, 1):
            src = np.zeros(n + 1, dtype=dtype)
            src[shift:shift + n] = perm
            d = torch.from_numpy(src.view(as_torch)).cuda()
            blob.zero_()
            gpu.compress_device(d.data_ptr() + shift * src.itemsize, n, src.itemsize,
                                blob.data_ptr(), len(want), b200_format(gpu, {}), stream)
            assert blob.cpu().numpy()[:len(want)].tobytes() == want, (dtype, shift)
