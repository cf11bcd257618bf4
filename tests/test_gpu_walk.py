"""The pairlist walk where its branches change, against the oracle's pair set
(whole numbers: equal): rows per warp (1, 2, 4, 8) and a last warp that is not
full, boxes in which the image nearest a run's box need not be a row's, all
beads in one cell, open axes, exclusions, and beads a little outside the
box."""
import numpy as np
import pytest
import torch

import pyoracle
from mars_md_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _compare(ctx, oracle, pos, size, periodic, rc, excl_np=None, origin=(0.0, 0.0, 0.0)):
    ctx.set_box(origin, size, periodic)
    if excl_np is not None:
        keep = tuple(torch.from_numpy(a).cuda() for a in excl_np[:2])
        ctx.set_exclusions(keep[0], keep[1], excl_np[2])
    d = torch.from_numpy(pos).cuda()
    t = torch.zeros(len(pos), dtype=torch.int32, device="cuda")
    box = pyoracle.Box.make(origin, size, periodic)
    want, count, _ = oracle.build_pairlist(pos, box, rc, excl=excl_np)
    for cutoff in (0.0, 0.8 * rc):
        assert ctx.build_pairlist(d, t, rc, cutoff) == count
        p = np.sort(ctx.export_pairs().cpu().numpy().astype(np.int64), axis=1)
        p = p[np.lexsort((p[:, 1], p[:, 0]))]
        assert np.array_equal(p, want.astype(np.int64))
    return count


def _pos(xyz):
    p = np.zeros((len(xyz), 4), np.float32)
    p[:, :3] = xyz
    return p


@pytest.mark.parametrize("n,size,rc", [
    (1, 100.0, 25.0), (2, 60.0, 25.0), (31, 55.0, 25.0), (700, 56.0, 25.0), (4097, 101.0, 25.0),
    (16387, 190.0, 20.0), (40001, 260.0, 15.0), (65541, 330.0, 15.0), (3000, 40.0, 19.0)])
def test_pair_set_over_sizes_and_tight_boxes(ctx_factory, oracle, n, size, rc):
    rng = np.random.default_rng(n)
    pos = _pos(rng.uniform(0.0, size, size=(n, 3)))
    _compare(ctx_factory(n), oracle, pos, (size, size * 1.01, size * 0.99), (1, 1, 1), rc)


@pytest.mark.parametrize("periodic", [(1, 1, 0), (0, 0, 0), (0, 1, 1)])
def test_pair_set_with_open_axes(ctx_factory, oracle, periodic):
    rng = np.random.default_rng(5)
    pos = _pos(rng.uniform(-30.0, 200.0, size=(5003, 3)))
    for a in range(3):
        if periodic[a]:
            pos[:, a] = np.mod(pos[:, a], 150.0)
    _compare(ctx_factory(5003), oracle, pos, (150.0, 150.0, 150.0), periodic, 21.0)


def test_pair_set_of_one_crowded_cell(ctx_factory, oracle):
    rng = np.random.default_rng(6)
    pos = _pos(np.concatenate([rng.normal(50.0, 0.3, size=(300, 3)),
                               rng.uniform(0.0, 100.0, size=(2000, 3))]))
    assert _compare(ctx_factory(2300), oracle, pos, (100.0,) * 3, (1, 1, 1), 12.0) > 300 * 299 // 2


def test_pair_set_with_beads_just_outside_the_box(ctx_factory, oracle):
    # (a bead farther out than its cell's neighbours reach keeps only the pairs
    # that the stencil of its clamped cell finds, as in the reference)
    rng = np.random.default_rng(8)
    size, n = 120.0, 6007
    xyz = rng.uniform(-0.5, size + 0.5, size=(n, 3))
    _compare(ctx_factory(n), oracle, _pos(xyz), (size,) * 3, (1, 1, 1), 20.0)


@pytest.mark.parametrize("chains", [3, 70])
def test_pair_set_with_exclusions(ctx_factory, oracle, chains):
    w = W.polymers(n_chains=chains, beads=1001, box=600.0 * (chains / 64) ** (1 / 3), with_grid=False)
    off, nb, k = oracle.exclusion_csr(w.exclusions)
    _compare(ctx_factory(w.n), oracle, w.pos, w.box_size, (1, 1, 1), 15.0, excl_np=(off, nb, k))
