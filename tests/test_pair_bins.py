"""The table bins of fast_pair_kernel (mb2_forces.cu), restated in numpy float32:
the bin coordinate added to 2^23 plus the row's first bin and rounded down must
hold, in the sum's low bits, the reference's bin, for every distance that the
kernel does not send to the reference's clamps, and never leave the table."""
import numpy as np
import pytest

f = np.float32


# end: the last bin never holds a force, so a reach ends at its start at most
@pytest.mark.parametrize("first", [0, 200, 400 * 15, 32000])
@pytest.mark.parametrize("start,step_inv,last,end", [
    (0.0, 10.0, 199, 4.5), (0.0, 13.333333, 399, 29.925), (0.05, 10.0, 99, 9.95),
    (3.0, 25.0, 300, 15.0), (-1.0, 8.0, 120, 14.0),
    (-541.27612, 6.8795, 3829, 0.349)])
def test_sum_rounded_down_holds_the_references_bin(first, start, step_inv, last, end):
    rng = np.random.default_rng(7)
    start, step_inv = f(start), f(step_inv)
    # all over the range, next to every bin edge, and the smallest distances
    edges = float(start) + np.arange(0, last + 2) / float(step_inv)
    near = edges[:, None] * (1.0 + rng.uniform(-1, 1, (1, 64)) * 10.0 ** rng.uniform(-8, -2, (1, 64)))
    d = np.concatenate([rng.uniform(0, end, 200000), near.ravel(), 10.0 ** rng.uniform(-5, -1, 20000),
                        [1e-6, 1.1e-5, 0.25 / float(step_inv), end]]).astype(f)
    reach = end + 1e-6 * (end + max(0.0, -float(start)))       # fast_args: loose
    close = max(1e-5, float(start) * (1 + 1e-6))                # fast_args: close2
    d = d[(d <= f(reach * (1 + 1e-6))) & (d >= f(close * (1 + 1e-6)))]
    w = ((d - start).astype(f) * step_inv).astype(f)
    # float32 addition rounded down: exact in double, then down to the grid of
    # 2^23 .. 2^24, the whole numbers
    magic = 8388608.0 + first
    total = np.floor(w.astype(np.float64) + magic)
    assert total.min() >= 8388608.0 and total.max() < 2.0 ** 24
    home = total.astype(f).view(np.uint32).astype(np.int64) - 0x4B000000 - first
    want = np.clip(np.floor(w).astype(np.int64), 0, last)
    assert home.min() >= 0 and home.max() <= last
    assert np.array_equal(home, want)
