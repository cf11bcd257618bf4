"""The general pair kernel (analytical terms, tables of different bin widths, an
open axis with uniform tables) at the sizes where the kernel of the uniform
tables tracks displacements and this one does not: forces after some steps on
one list against the oracle's over the same list, as the 262,144-bead test of
the uniform tables holds them. And the step that builds with positions outside
the box, as test_gpu_outside_box has it for those tables."""
import numpy as np
import pytest
import torch

import pyoracle
from conftest import box_of, force_errors, tableset
from mars_md_b200 import workloads as W
from mars_md_b200.engine import setup_workload, step_params

pytestmark = pytest.mark.gpu

CHARGE = np.array([1.0, -1.0, 1.0, -1.0], np.float32)
RADIUS = np.array([2.0, 2.2, 2.4, 2.6], np.float32)
EPS = np.array([0.1, 0.12, 0.14, 0.16], np.float32)


def _workload(kind):
    w = W.large_plain(n=140003)
    # beads that keep apart: a jittered lattice of that density
    rng = np.random.default_rng(3)
    k = int(np.ceil(w.n ** (1 / 3)))
    box = float((k ** 3 / 0.002) ** (1 / 3))
    site = np.sort(rng.permutation(k ** 3)[:w.n])
    xyz = np.stack([site // (k * k), site // k % k, site % k], axis=1) * (box / k)
    w.pos[:, :3] = np.mod(xyz + rng.uniform(-1.8, 1.8, size=(w.n, 3)), box).astype(np.float32)
    w.box_size = (box,) * 3
    if kind == "mixed":
        w.pair_tables[9] = W.dh_softcore_table(-1.0, -1.0, bins=300)
    elif kind == "terms":
        w.term_matrix = w.term_matrix | np.uint32(2 | 16)   # Debye-Hueckel, softcore
    elif kind == "open":
        w.periodic = (1, 1, 0)
    return w


def _setup(ctx_factory, w, kind):
    ctx = ctx_factory(w.n)
    dev = setup_workload(ctx, w)
    if kind == "terms":
        ctx.set_pair_terms(CHARGE, RADIUS, EPS)
    return ctx, dev


def _compare(ctx, oracle, w, kind, pos, fe, every):
    sample = np.arange(0, w.n, every)
    mask = torch.zeros(w.n, dtype=torch.bool, device="cuda")
    mask[torch.from_numpy(sample).cuda()] = True
    pairs = ctx.export_pairs()
    sub = pairs[mask[pairs[:, 0].long()] | mask[pairs[:, 1].long()]].cpu().numpy()
    tags = oracle.resolve_tags(sub, w.type_ids, w.term_matrix, w.num_types)
    rc2 = np.float32(w.cutoff) ** 2
    if kind == "terms":
        _, f64, fabs = oracle.pair_forces_terms(sub, pos, w.type_ids, tags, tableset(w),
                                                pyoracle.PairTermSet(CHARGE, RADIUS, EPS), box_of(w), rc2)
    else:
        _, f64, fabs = oracle.pair_forces(sub, pos, tags, tableset(w), box_of(w), rc2)
    scaled, plain = force_errors(fe[sample], f64[sample], fabs[sample])
    assert np.abs(f64[sample]).max() > 0.0
    assert scaled <= 1e-5, (scaled, plain)


@pytest.mark.parametrize("kind", ["mixed", "terms", "open"])
def test_forces_after_steps(ctx_factory, oracle, kind):
    w = _workload(kind)
    ctx, dev = _setup(ctx_factory, w, kind)
    prm = step_params(w)
    prm.rebuild_period = 1000
    for s in range(1, 7):
        ctx.step(dev["pos"], dev["fe"], dev["type"], None, s, prm)
    fe = torch.zeros_like(dev["fe"])
    ctx.pair_forces(dev["pos"], dev["type"], fe, w.cutoff, get_energy=False)
    pos = dev["pos"].cpu().numpy()
    moved = np.abs(pos[:, :3] - w.pos[:, :3])
    moved = np.minimum(moved, w.box_size[0] - moved)
    assert 0.5 < np.sqrt((moved ** 2).sum(1).max()) < 5.0
    _compare(ctx, oracle, w, kind, pos, fe.cpu().numpy(), 16)


@pytest.mark.parametrize("kind", ["mixed", "terms"])
def test_step_that_builds_outside_the_box(ctx_factory, oracle, kind):
    w = _workload(kind)
    L = np.float32(w.box_size[0])
    pick = (np.random.default_rng(5).random(w.n) < 0.3) & (w.pos[:, 0] > 0.5 * L)
    # beyond one face only: three images apart and more, the packed image arithmetic
    # rounds k l and the sum once where the reference rounds both (k l is exact to 2 l)
    w.pos[pick, 0] += L
    ctx, dev = _setup(ctx_factory, w, kind)
    ctx.step(dev["pos"], dev["fe"], dev["type"], None, 1, step_params(w))
    _compare(ctx, oracle, w, kind, w.pos, dev["fe"].cpu().numpy(), 16)
