"""Radix sort of pairs at the sizes where it changes its kernel: one-launch sort
up to 65,536 keys with 256 threads a block up to 32,768 and 512 above, tiles of
2,048 keys up to 2^19, 4,096 up to 2^22 and 6,144 above; and a smaller sort in
the scratch of a larger one.  Keys with few different digits and random ones:
the order is the stable order of the digits sorted."""
import numpy as np
import pytest
import torch

from astraea_gb300 import engine

pytestmark = pytest.mark.gpu


def check(n, end_bit, mask, seed):
    rng = np.random.default_rng(seed)
    keys = rng.integers(0, 2 ** 63, n, dtype=np.uint64) & np.uint64(mask)
    vals = np.arange(n, dtype=np.int32)
    ks, vs = engine.radix_sort_pairs(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda(), end_bit)
    bits = (end_bit + 7) // 8 * 8
    part = keys if bits == 64 else keys & np.uint64(2 ** bits - 1)
    order = np.argsort(part, kind="stable")
    assert np.array_equal(vs.cpu().numpy(), vals[order])
    assert np.array_equal(ks.cpu().numpy().view(np.uint64), keys[order])


@pytest.mark.parametrize("n", [31, 32, 32_767, 32_768, 32_769, 57_344, 65_535, 65_536, 65_537, 1 << 19, (1 << 19) + 1,
                               1 << 22, (1 << 22) + 1, 5_000_003])
@pytest.mark.parametrize("end_bit,mask", [(40, 0x8300000000050103), (63, 2 ** 64 - 1)])
def test_pairs_around_the_kernels_limits(n, end_bit, mask):
    check(n, end_bit, mask, n + end_bit)


@pytest.mark.parametrize("n", [100, 65_536, 70_001, 1 << 19])
def test_small_sort_in_large_scratch(n):
    check(4_300_001, 16, 2 ** 64 - 1, 1)
    check(n, 63, 2 ** 64 - 1, n)
