"""The sort at the sizes where its launch changes (the counting sort's last size,
the small and the large tiles' first and last, whole tiles and one element
more), with many equal keys and with all 32 bits in use, against a stable host
sort: integers, so equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 8191, 8192, 8193, 9216, 9217, 262144, 262145, 266240, 266241,
                               1000003])
@pytest.mark.parametrize("bits", [3, 9, 32])
def test_sort_is_the_stable_sort(ctx_factory, n, bits):
    rng = np.random.default_rng(n + bits)
    keys_np = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if bits == 32 and n > 2:
        keys_np[n // 2:n // 2 + n // 8] = 0xFFFFFFFF   # as the padding of a last tile
    vals_np = rng.permutation(n).astype(np.int32)
    keys = torch.from_numpy(keys_np.view(np.int32).copy()).cuda()
    vals = torch.from_numpy(vals_np.copy()).cuda()
    ctx = ctx_factory(n)
    ctx.radix_sort_pairs(keys, vals)
    torch.cuda.synchronize()
    order = np.argsort(keys_np, kind="stable")
    assert np.array_equal(keys.cpu().numpy().view(np.uint32), keys_np[order])
    assert np.array_equal(vals.cpu().numpy(), vals_np[order])


@pytest.mark.parametrize("n", [1, 2, 8192, 8193, 262144, 262145])
def test_morton_sort_leaves_the_inverse(ctx_factory, n):
    rng = np.random.default_rng(n)
    pos = torch.from_numpy(rng.uniform(0.0, 50.0, (n, 4)).astype(np.float32)).cuda()
    pos[n // 3:n // 2] = pos[0]   # one key many times: the sort is stable
    keys, s2o, inv, sp = (t.cpu().numpy() for t in ctx_factory(n).sort_morton(
        pos, [0.0, 0.0, 0.0], [50.0, 50.0, 50.0]))
    keys = keys.view(np.uint32)
    assert np.array_equal(np.sort(s2o), np.arange(n))
    assert np.array_equal(inv[s2o], np.arange(n))
    assert np.array_equal(sp, pos.cpu().numpy()[s2o])
    assert np.all((keys[1:] > keys[:-1]) | ((keys[1:] == keys[:-1]) & (s2o[1:] > s2o[:-1])))


@pytest.mark.parametrize("polls", [0, 1, 3])
@pytest.mark.parametrize("n", [8193, 9217, 262145, 300001])
@pytest.mark.parametrize("bits", [3, 32])
def test_sort_without_the_earlier_tiles_counts(ctx_factory, n, bits, polls):
    """Tiles that are not told the counts before them in time count them
    themselves: none waits (0 polls), or some do and some do not."""
    rng = np.random.default_rng(n + bits)
    keys_np = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys = torch.from_numpy(keys_np.view(np.int32).copy()).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    inv = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    ctx_factory(n).selftest_sort_polls(keys, vals, polls, inv)
    order = np.argsort(keys_np, kind="stable")
    assert np.array_equal(keys.cpu().numpy().view(np.uint32), keys_np[order])
    assert np.array_equal(vals.cpu().numpy(), order)
    assert np.array_equal(inv.cpu().numpy()[order], np.arange(n))
