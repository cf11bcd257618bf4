"""The pair kernel for uniform tables against the oracle, pair by pair: isolated
pairs of beads along x at distances next to bin edges, to the tables' start and
to the last bin that holds a force, and down to where the reference skips a
pair, for tables that start at, above and below zero (far below too: the bin
coordinate's rounding grows with the start), with each type pair's bins side by
side and through offsets (many types). A bead has one pair, so every force and
energy is the reference's float itself: equal."""
import numpy as np
import pytest
import torch

import pyoracle
from mars_md_b200 import workloads as W

pytestmark = pytest.mark.gpu
f = np.float32


def _tables(start, step, size, last_force, count, seed):
    rng = np.random.default_rng(seed)
    x = (start + np.arange(size) * step).astype(f)
    out = []
    for _ in range(count):
        u = np.cumsum(rng.uniform(-2.0, 2.0, size)).astype(f)
        u[last_force + 1:] = 0.0
        u[last_force] = f(1.5)     # the last bin that holds a force
        out.append(W.table_from_xy(x, u, "pair"))
    return out


def _distances(t, last_force, cutoff, rng):
    s, inv = float(f(t.start)), float(f(t.step_inv))
    end = s + (last_force + 1) / inv
    # (not 1e-6 itself, where the reference neither skips the pair nor gives it a
    # direction: its unit vector is zero up to and including 1e-6)
    d = [np.array([1e-7, 9e-7, 1.1e-6, 9e-6, 1e-5, 1.1e-5, 1e-4, 1e-2]), rng.uniform(0.0, cutoff, 400)]
    edges = s + np.arange(len(t.values) + 1) / inv
    edges = edges[(edges > 0.0) & (edges < cutoff)]
    edges = edges[rng.permutation(len(edges))[:40]]
    for e, reach in [(e, 4) for e in edges] + [(end, 250), (abs(s), 4), (cutoff, 4)]:
        if 0.0 < e <= cutoff:
            d.append(f(e) + np.arange(-reach, 2 * reach + 1) * np.spacing(f(e)))
    return np.concatenate(d).astype(f)


@pytest.mark.parametrize("energy", [False, True])
@pytest.mark.parametrize("start,step,size,last_force,types", [
    (0.0, 0.1, 200, 44, 1), (0.0, 0.075, 400, 398, 4), (0.05, 0.1, 100, 60, 2), (3.0, 0.04, 301, 250, 1),
    (-1.0, 0.125, 121, 100, 3), (0.0, 0.05, 300, 120, 12),
    # starts far below the end: where the coordinate's rounding is the coarsest
    # against the bin's own
    (-541.2761446184406, 0.14535900023070578, 3830, 3726, 1),
    (-287.41124961970047, 0.35411184951900926, 860, 812, 1)])
def test_pairs_next_to_bin_edges(ctx_factory, oracle, start, step, size, last_force, types, energy):
    cutoff, radius = 15.0, 18.0
    count = min(types * (types + 1) // 2, 10)
    tabs = _tables(start, step, size, last_force, count, types + size)
    rng = np.random.default_rng(size)
    d = _distances(tabs[0], last_force, cutoff, rng)
    k = len(d)
    side = int(np.ceil(np.sqrt(k)))
    pos = np.zeros((2 * k, 4), np.float32)
    pos[:, 1] = np.repeat(25.0 * (np.arange(k) // side), 2)
    pos[:, 2] = np.repeat(25.0 * (np.arange(k) % side), 2)
    pos[1::2, 0] = d
    ids = rng.integers(0, types, 2 * k).astype(np.int32)
    index = {p: q for q, p in enumerate((a, b) for a in range(types) for b in range(a, types))}
    tags = W._term_matrix(types, lambda a, b: index[(a, b)] % count)
    size3 = (60.0, 25.0 * side, 25.0 * side)
    ctx = ctx_factory(2 * k)
    ctx.set_box((0.0,) * 3, size3, (1, 1, 1))
    ctx.set_pair_tables(types, tags, [(t.values, t.start, t.step_inv) for t in tabs])
    dp, dt = torch.from_numpy(pos).cuda(), torch.from_numpy(ids).cuda()
    fe = torch.zeros_like(dp)
    assert ctx.build_pairlist(dp, dt, radius) == k
    ctx.pair_forces(dp, dt, fe, cutoff, get_energy=energy)
    got = fe.cpu().numpy()
    pairs = np.arange(2 * k, dtype=np.int32).reshape(k, 2)
    want, _, _ = oracle.pair_forces(
        pairs, pos, oracle.resolve_tags(pairs, ids, tags, types),
        pyoracle.TableSet([(t.values, t.start, t.step_inv) for t in tabs]),
        pyoracle.Box.make((0.0,) * 3, size3), f(cutoff) ** 2, get_energy=energy)
    wrong = np.flatnonzero(~np.all(got[1::2] == want[1::2], axis=1))
    assert np.abs(want[:, 0]).max() > 0.0
    assert wrong.size == 0, (wrong.size, d[wrong][:4], got[1::2][wrong][:4], want[1::2][wrong][:4])
    assert np.array_equal(got, want)
