"""Positions outside the box on a step that builds its list: beads a whole box
edge away, and a few A past an edge, as in a restart from unwrapped
coordinates. The list holds a pair in whatever image its beads are stored, and
the step's forces must be those of the listed pairs' nearest images, as the
reference's per-pair minimum image gives them (the oracle, over the list the
step built). Two float sums of the same pair values in another order: ulps of
the sum of magnitudes."""
import numpy as np
import pytest
import torch

from conftest import box_of, force_errors, tableset
from mars_md_b200 import workloads as W
from mars_md_b200.engine import setup_workload, step_params

pytestmark = pytest.mark.gpu


def _shifted(w, kind):
    rng = np.random.default_rng(11)
    L = w.box_size[0]
    pos = w.pos.copy()
    pick = rng.random(w.n) < 0.3
    axis = rng.integers(0, 3, w.n)
    for a in range(3):
        m = pick & (axis == a)
        x = pos[m, a]
        if kind == "edge":      # the image beyond the nearer face
            x = np.where(x > 0.5 * L, x + np.float32(L), x - np.float32(L))
        else:                   # stored past the other face: x up to 9 A keeps its place, L higher
            x = np.where(x < 9.0, x + np.float32(L), np.where(x > L - 9.0, x - np.float32(L), x))
        pos[m, a] = x
    return pos


@pytest.mark.parametrize("n", [20011, 140001])
@pytest.mark.parametrize("kind", ["edge", "past"])
def test_step_that_builds_outside_the_box(ctx_factory, oracle, n, kind):
    w = W.plain_bd(n=n, box=float((n / 0.002) ** (1 / 3)))
    w.pos = _shifted(w, kind)
    ctx = ctx_factory(w.n)
    dev = setup_workload(ctx, w)
    ctx.step(dev["pos"], dev["fe"], dev["type"], None, 1, step_params(w))
    fe = dev["fe"].cpu().numpy()
    pairs = ctx.export_pairs().cpu().numpy()
    # the list: every pair of beads inside the box that the oracle lists
    inside = np.all((w.pos[:, :3] >= 0.0) & (w.pos[:, :3] <= np.float32(w.box_size[0])), axis=1)
    want, _, _ = oracle.build_pairlist(w.pos, box_of(w), w.list_radius)
    keep = inside[want].all(axis=1)
    have = np.sort(pairs.astype(np.int64), axis=1)
    have = have[inside[have].all(axis=1)]
    have = have[np.lexsort((have[:, 1], have[:, 0]))]
    assert np.array_equal(have, want[keep].astype(np.int64))
    # and the forces of all listed pairs
    tags = oracle.resolve_tags(pairs, w.type_ids, w.term_matrix, w.num_types)
    _, f64, fabs = oracle.pair_forces(pairs, w.pos, tags, tableset(w), box_of(w),
                                      np.float32(w.cutoff) ** 2)
    mixed = (inside[pairs[:, 0]] != inside[pairs[:, 1]]).sum()
    assert mixed > 1000            # pairs across images are there to be lost
    scaled, plain = force_errors(fe, f64, fabs)
    assert scaled <= 1e-5, (scaled, plain)


def test_batch_builds_outside_the_box(oracle):
    """The same through a batch, in which a system's own displacement word says
    whether its rows' far entries are read."""
    from mars_md_b200.engine import setup_batch
    ws = [W.plain_bd(seed=s, n=n, box=float((n / 0.002) ** (1 / 3)))
          for s, n in ((1, 3001), (2, 1203))]
    ws[0].pos = _shifted(ws[0], "edge")
    b, dev = setup_batch(ws)
    try:
        b.step(dev["pos"], dev["fe"], dev["type"], 1, step_params(ws[0]))
        fe = dev["fe"].cpu().numpy()
        pairs = b.export_pairs().cpu().numpy().astype(np.int64)
        for s, w in enumerate(ws):
            lo, hi = b.offsets[s], b.offsets[s + 1]
            mine = pairs[(pairs[:, 0] >= lo) & (pairs[:, 0] < hi)] - lo
            tags = oracle.resolve_tags(mine.astype(np.int32), w.type_ids, w.term_matrix, w.num_types)
            _, f64, fabs = oracle.pair_forces(mine.astype(np.int32), w.pos, tags, tableset(w),
                                              box_of(w), np.float32(w.cutoff) ** 2)
            scaled, plain = force_errors(fe[lo:hi], f64, fabs)
            assert scaled <= 1e-5, (s, scaled, plain)
    finally:
        b.close()
