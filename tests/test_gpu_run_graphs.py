"""Context.run at the lengths where its replays change (whole intervals between
rebuild checks as one graph, the rest step by step, starts within an interval),
BD and Langevin, against one step call per step. As test_gpu_run holds them:
the two differ by the order of the float sums, which now and then puts a pair
on the other side of a table-bin edge."""
import numpy as np
import pytest
import torch

from mars_md_b200 import workloads as W
from mars_md_b200.engine import setup_workload, step_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("langevin", [False, True])
@pytest.mark.parametrize("first,lengths", [(1, [1, 19, 20, 45]), (7, [13, 1, 20]), (2, [19, 19])])
def test_run_matches_steps(ctx_factory, langevin, first, lengths):
    w = W.plain_bd(n=2500, box=170.0)
    got = []
    for by_run in (True, False):
        ctx = ctx_factory(w.n)
        dev = setup_workload(ctx, w)
        prm = step_params(w)
        if langevin:
            ctx.set_langevin_types([150.0], [[2e4] * 3])
            g = torch.Generator(device="cuda").manual_seed(3)
            dev["mom"] = torch.randn((w.n, 4), device="cuda", generator=g) * 19.0
            prm.integrator, prm.mom4, prm.deferred_kick_pending = 1, dev["mom"].data_ptr(), 1
        s = first
        for k in lengths:
            if by_run:
                ctx.run(dev["pos"], dev["fe"], dev["type"], None, s, k, prm)
            else:
                for q in range(k):
                    ctx.step(dev["pos"], dev["fe"], dev["type"], None, s + q, prm)
            s += k
        got.append((dev["pos"].cpu().numpy()[:, :3],
                    dev["mom"].cpu().numpy() if langevin else None))
    d = np.abs(got[0][0] - got[1][0])
    d = np.minimum(d, w.box_size[0] - d).max(axis=1)
    assert (d <= 1e-4).mean() >= 0.99 and d.max() <= 0.1, float(d.max())
    if langevin:
        m = np.abs(got[0][1] - got[1][1]).max(axis=1)
        assert (m <= 1e-3).mean() >= 0.99


@pytest.mark.parametrize("period,steps", [(34, 70), (65, 140), (100, 130), (2, 9)])
def test_run_over_intervals_of_other_lengths(ctx_factory, period, steps):
    """Rebuild checks further apart than the longest graph (32 steps), whose
    intervals are one graph and single steps or several graphs, and every other
    step."""
    w = W.plain_bd(n=2500, box=170.0)
    got = []
    for by_run in (True, False):
        ctx = ctx_factory(w.n)
        dev = setup_workload(ctx, w)
        prm = step_params(w)
        prm.rebuild_period = period
        if by_run:
            ctx.run(dev["pos"], dev["fe"], dev["type"], None, 1, steps, prm)
        else:
            for s in range(1, steps + 1):
                ctx.step(dev["pos"], dev["fe"], dev["type"], None, s, prm)
        got.append(dev["pos"].cpu().numpy()[:, :3])
    d = np.abs(got[0] - got[1])
    d = np.minimum(d, w.box_size[0] - d).max(axis=1)
    assert (d <= 1e-4).mean() >= 0.99 and d.max() <= 0.1, float(d.max())


@pytest.mark.parametrize("langevin", [False, True])
def test_run_with_other_buffers_every_call(ctx_factory, langevin):
    """Buffers met once are stepped without a graph, buffers that come back with
    one: every call here has another ForceEnergy than the call before, then two
    have the same."""
    w = W.polymers(n_chains=3, beads=257, box=300.0, with_grid=False)
    # (checks every five steps, so that few steps pass all the cases: over many the
    # order of the float sums would part the two, as above)
    lengths, which = [5, 5, 2, 3, 5, 5, 5], [0, 1, 0, 1, 0, 0, 0]
    got = []
    for by_run in (True, False):
        ctx = ctx_factory(w.n)
        dev = setup_workload(ctx, w)
        fes = [dev["fe"], torch.zeros_like(dev["fe"])]
        prm = step_params(w, bonds=dev["bonds"], bond_idx=dev["bond_idx"], angles=dev["angles"],
                          angle_idx=dev["angle_idx"])
        prm.rebuild_period = 5
        if langevin:
            t = len(w.diffusion)
            ctx.set_langevin_types([150.0] * t, [[2e4] * 3] * t)
            g = torch.Generator(device="cuda").manual_seed(3)
            dev["mom"] = torch.randn((w.n, 4), device="cuda", generator=g) * 19.0
            prm.integrator, prm.mom4, prm.deferred_kick_pending = 1, dev["mom"].data_ptr(), 1
        s = 1
        for k, b in zip(lengths, which):
            if by_run:
                ctx.run(dev["pos"], fes[b], dev["type"], None, s, k, prm)
            else:
                for q in range(k):
                    ctx.step(dev["pos"], fes[b], dev["type"], None, s + q, prm)
            s += k
        got.append((dev["pos"].cpu().numpy()[:, :3], [f.cpu().numpy()[:, :3] for f in fes]))
    d = np.abs(got[0][0] - got[1][0])
    d = np.minimum(d, w.box_size[0] - d).max(axis=1)
    assert (d <= 1e-4).mean() >= 0.99 and d.max() <= 0.1, float(d.max())
    for a, b in zip(got[0][1], got[1][1]):
        f = np.abs(a - b).max(axis=1)
        assert (f <= 1e-2 * np.maximum(1.0, np.abs(b).max(axis=1))).mean() >= 0.99


@pytest.mark.parametrize("beads,chains,langevin,grid", [(33, 1, False, False), (257, 3, True, False),
                                                        (1024, 17, False, True)])
def test_steps_in_one_graph_hand_over(ctx_factory, beads, chains, langevin, grid):
    """Steps 2-20 as one graph, where each leaves the next its packed positions,
    cleared sums (bonded ones too) and displacement track (17,408 beads keep it;
    the tables end well short of the cutoff), a third of the particles attached to
    rigid bodies: against step by step, ForceEnergy included."""
    w = W.polymers(n_chains=chains, beads=beads, box=300.0, with_grid=grid)
    flags = torch.zeros(w.n, dtype=torch.int32, device="cuda")
    flags[::3] = 4
    flags[:40] = 4   # a whole warp, and a part of one
    got = []
    for by_run in (True, False):
        ctx = ctx_factory(w.n)
        dev = setup_workload(ctx, w)
        prm = step_params(w, bonds=dev["bonds"], bond_idx=dev["bond_idx"], angles=dev["angles"],
                          angle_idx=dev["angle_idx"])
        if langevin:
            t = len(w.diffusion)
            ctx.set_langevin_types([150.0] * t, [[2e4] * 3] * t)
            g = torch.Generator(device="cuda").manual_seed(3)
            dev["mom"] = torch.randn((w.n, 4), device="cuda", generator=g) * 19.0
            prm.integrator, prm.mom4, prm.deferred_kick_pending = 1, dev["mom"].data_ptr(), 1
        if by_run:
            ctx.run(dev["pos"], dev["fe"], dev["type"], flags, 1, 20, prm)
        else:
            for s in range(1, 21):
                ctx.step(dev["pos"], dev["fe"], dev["type"], flags, s, prm)
        got.append((dev["pos"].cpu().numpy()[:, :3], dev["fe"].cpu().numpy()[:, :3]))
    held = flags.cpu().numpy() == 4
    assert np.array_equal(got[0][0][held], got[1][0][held])
    assert np.array_equal(got[0][0][held], w.pos[held, :3])
    d = np.abs(got[0][0] - got[1][0])
    d = np.minimum(d, w.box_size[0] - d).max(axis=1)
    # as above: another order of the sums moves a bead by ulps, or a bin's step of force
    assert (d <= 1e-4).mean() >= 0.99 and d.max() <= 0.1, float(d.max())
    f = np.abs(got[0][1] - got[1][1]).max(axis=1)
    assert (f <= 1e-2 * np.maximum(1.0, np.abs(got[1][1]).max(axis=1))).mean() >= 0.99
