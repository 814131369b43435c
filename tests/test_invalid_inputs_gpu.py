# SPDX-License-Identifier: Apache-2.0
"""Inputs that are not permutations end with invalid_argument after one pass,
wherever the fault shows, and leave the next call right."""
import numpy as np
import pytest

from test_long_chains_gpu import structured

pytestmark = pytest.mark.gpu


def broken(perm):
    """Copies of perm with a repeat or a value out of range."""
    n = perm.size
    last, first, mid = (int(np.flatnonzero(perm == v)[0]) for v in (n - 1, 0, n // 2))
    for at, value in ((last, 0), (first, n - 1), (mid, 3), (mid, n), (last, 0xFFFFFFFF)):
        bad = perm.copy()
        bad[at] = value
        yield bad


@pytest.mark.parametrize("n", [8193, 16385, 40_001, 100_003, (1 << 18) - 1, (1 << 20) + 1,
                               (1 << 23) + 1])
def test_one_pass(gpu, n):
    perm = gpu.fill_permutation(gpu.PermutationKind.uniform, n, n, np.uint32)
    good = gpu.compress(perm)
    launches = gpu.last_profile()[2]
    for bad in broken(perm):
        with pytest.raises(ValueError, match="every value"):
            gpu.compress(bad)
        assert gpu.last_profile()[2] == launches
    assert gpu.compress(perm) == good


@pytest.mark.parametrize("n,mode", [(16_387, True), (100_003, True), (100_003, "fallback"),
                                    ((1 << 23) + 1, False)])
def test_levels_with_long_chains(gpu, n, mode):
    gpu.set_union_find_only(mode)
    try:
        for kind in ("pairs", "riffle"):
            perm = structured(kind, n)
            good = gpu.compress(perm)
            for bad in broken(perm):
                with pytest.raises(ValueError, match="every value"):
                    gpu.compress(bad)
            assert gpu.compress(perm) == good
    finally:
        gpu.set_union_find_only(False)


def test_batch_members_once(gpu):
    import torch
    fmt = gpu.FormatOptions()
    items, keep = [], []
    for n, break_it in ((40_001, False), (100_003, True), (150_000, True)):
        perm = gpu.fill_permutation(gpu.PermutationKind.uniform, n, n, np.uint32)
        size = gpu.encoded_size(n, fmt)
        for p in (perm, next(broken(perm)) if break_it else perm):
            src = torch.from_numpy(p.view(np.int32)).cuda()
            blob = torch.zeros((size + 3) // 4 * 4, dtype=torch.uint8, device="cuda")
            keep.append((src, blob))
            items.append((src.data_ptr(), n, 4, fmt, blob.data_ptr(), size))
    torch.cuda.synchronize()
    _, alone = gpu.compress_batch_device(items[::2], raise_errors=False)
    statuses, launches = gpu.compress_batch_device(items[1::2], raise_errors=False)
    assert statuses == [0, 1, 1] and launches == alone
