"""Rows split near / far where the tables end short of the cutoff: forces from a
split list, whose far entries the pair kernel leaves out while the
displacements since the build allow it, against forces from a list without a
split (built from the same positions, so the same pairs), after displacements
on both sides of that limit. Two float sums of the same pair values in another
order differ by at most a few ulps of the sum of magnitudes."""
import numpy as np
import pytest
import torch

from mars_md_b200 import workloads as W
from mars_md_b200.engine import setup_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16385, 20011, 140001])
@pytest.mark.parametrize("moved", [0.0, 1.5, 3.2, 6.0])
def test_forces_do_not_depend_on_the_split(ctx_factory, n, moved):
    w = W.plain_bd(n=n, box=float((n / 0.002) ** (1 / 3)))
    rng = np.random.default_rng(n)
    step = rng.normal(size=(n, 3))
    step *= moved / np.linalg.norm(step, axis=1, keepdims=True)   # every bead by `moved`
    later = w.pos.copy()
    later[:, :3] = np.mod(w.pos[:, :3] + step, w.box_size[0]).astype(np.float32)
    out = []
    for cutoff in (w.cutoff, 0.0):
        ctx = ctx_factory(n)
        dev = setup_workload(ctx, w)
        ctx.build_pairlist(dev["pos"], dev["type"], w.list_radius, cutoff)
        pos = torch.from_numpy(later).cuda()
        fe = torch.zeros_like(pos)
        ctx.pair_forces(pos, dev["type"], fe, w.cutoff, get_energy=False)
        fe2 = torch.zeros_like(pos)
        ctx.pair_forces(pos, dev["type"], fe2, w.cutoff, get_energy=True)
        out.append((fe.cpu().numpy(), fe2.cpu().numpy(), ctx.num_pairs()))
    assert out[0][2] == out[1][2]
    for k in (0, 1):
        a, b = out[0][k].astype(np.float64), out[1][k].astype(np.float64)
        # at most some 20 contacts a bead, the largest of 300 kcal/mol/A: ulps of that
        assert np.abs(a - b).max() <= 20 * 2.0 ** -22 * max(np.abs(b).max(), 1.0)
