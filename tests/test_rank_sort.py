"""The counting sort of up to 8,192 pairs (rank_sort_kernel in mb2_sort.cu), its
index arithmetic run on the host: 32 elements a block, keys in quads padded with
the largest key, eight warps that take every eighth quad; quads before the
block's own count keys up to and including an element's, quads after it smaller
ones, the block's own by key and position, with the padding left out. The ranks
must be a stable argsort's for every size, whole quads and blocks or not. The
device kernel itself is checked against a host stable sort in the GPU tests."""
import numpy as np
import pytest


def ranks(keys):
    n = len(keys)
    quads = (n + 3) // 4
    sk = np.full(4 * quads, 0xFFFFFFFF, np.uint32)
    sk[:n] = keys
    out = np.zeros(n, np.int64)
    for first in range(0, n, 32):
        q0, q1 = first // 4, min(first // 4 + 8, quads)
        i = np.arange(first, min(first + 32, n))
        key = sk[i]
        total = np.zeros(len(i), np.int64)
        for warp in range(8):
            before = (np.arange(warp, q0, 8)[:, None] * 4 + np.arange(4)).ravel()
            after = (np.arange(q1 + warp, quads, 8)[:, None] * 4 + np.arange(4)).ravel()
            own = (np.arange(q0 + warp, q1, 8)[:, None] * 4 + np.arange(4)).ravel()
            own = own[own < n]
            total += (sk[before][None] <= key[:, None]).sum(1) + (sk[after][None] < key[:, None]).sum(1)
            total += ((sk[own][None] < key[:, None]) |
                      ((sk[own][None] == key[:, None]) & (own[None] < i[:, None]))).sum(1)
        out[i] = total
    return out


@pytest.mark.parametrize("n", [2, 3, 5, 31, 32, 33, 63, 64, 65, 1000, 2047, 2048, 4097])
@pytest.mark.parametrize("distinct", [3, 1 << 32])
def test_ranks_are_a_stable_sorts(n, distinct):
    rng = np.random.default_rng(n * 7 + distinct % 97)
    keys = rng.integers(0, distinct, n, dtype=np.uint64).astype(np.uint32)
    if distinct > 3:
        keys[::3] = 0xFFFFFFFF   # as the padding
    order = np.empty(n, np.int64)
    order[ranks(keys)] = np.arange(n)
    assert np.array_equal(order, np.argsort(keys, kind="stable"))
