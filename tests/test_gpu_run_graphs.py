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
