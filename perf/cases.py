"""The work that a user of this framework has it do, as cases that can be timed
and compared: Brownian and Langevin dynamics of one system, single force
evaluations, batches of replicas, a differentiable window and the Morton sort,
each through the framework's public entry points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes the inputs and the handles a program keeps, ``run`` is one
pass, and ``exact`` says in float64 (plain torch) what a first pass returns.

Sizes: the benchmark configurations of ``mars_md_b200.workloads`` (4,096 beads;
64 chains of 1,024 beads with a 256^3 grid; 2,097,152 beads of four types; 512
replicas of 500 to 20,000 beads; a window over 16 chains of 1,024 beads) and
odd sizes between and below them.
"""
import math

import numpy as np
import torch

from mars_md_b200 import workloads as W
from mars_md_b200.adjoint import BDWindowLoss, Window
from mars_md_b200.engine import (Batch, Context, exclusion_csr, setup_batch, setup_workload,
                                 step_params)

DEV = "cuda:0"
WCA_DENSITY = 4096 / 200.0 ** 3   # the plain 4,096-bead configuration's
DH_DENSITY = 0.002                # the 2,097,152-bead configuration's
COULOMB = 332.0636                # kcal A / (mol e^2)


def listed():
    return [
        # One step of a small system at a time: a program that looks at every
        # step (its own output, a coupled code) pays the call's latency.
        {"name": "step_1000", "op": "step", "kind": "wca", "n": 1000},
        # The plain configuration, run in blocks between two outputs.
        {"name": "run_4096", "op": "run", "kind": "wca", "n": 4096, "steps": 100},
        # A small bonded system under Langevin dynamics, odd chain length.
        {"name": "langevin_12x1001", "op": "run", "kind": "polymers", "chains": 12,
         "beads": 1001, "grid": False, "langevin": True, "steps": 40},
        # Bead-spring polymers in a grid potential, the polymer configuration.
        {"name": "polymers_64x1024", "op": "run", "kind": "polymers", "chains": 64,
         "beads": 1024, "grid": True, "langevin": False, "steps": 40},
        # A medium and the largest plain system: one rebuild period a pass.
        {"name": "run_300007", "op": "run", "kind": "dh", "n": 300007, "steps": 20},
        {"name": "run_2097152", "op": "run", "kind": "dh", "n": 2097152, "steps": 20},
        # A single evaluation on new positions: list, forces and energies
        # (analysis of a trajectory's frames; the reference's functors called
        # one by one).
        {"name": "energy_131071", "op": "forces", "kind": "dh", "n": 131071},
        # The same with analytical pair terms beside the tables.
        {"name": "terms_20011", "op": "forces", "kind": "terms", "n": 20011},
        # Batched replicas, each checked for a rebuild at every step (the
        # cadence that the autotuner picks for them).
        {"name": "batch_512", "op": "batch", "systems": 512, "nmin": 500, "nmax": 20000,
         "steps": 20},
        # Gradients of a window (forward and backward), a checkpoint every 10
        # steps: one period of the window configuration, after which table-bin
        # crossings of single pairs would outweigh what is compared.
        {"name": "window_16x1024", "op": "window", "chains": 16, "beads": 1024, "steps": 20},
        # Morton keys, stable sort and both permutations of a large system.
        {"name": "sort_1000003", "op": "sort", "n": 1000003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["step", "run", "run", "polymers", "dh", "dh", "forces", "terms", "batch",
                     "window", "sort"])
    if op == "step":
        return {"op": "step", "kind": "wca", "n": _log_int(rng, 500, 16000)}
    if op == "run":
        return {"op": "run", "kind": "wca", "n": _log_int(rng, 1000, 200000),
                "steps": rng.randint(21, 100)}
    if op == "polymers":
        return {"op": "run", "kind": "polymers", "chains": rng.randint(3, 64),
                "beads": _log_int(rng, 100, 1024), "grid": rng.random() < 0.5, "langevin": False,
                "steps": rng.randint(21, 60)} if rng.random() < 0.6 else {
                    "op": "run", "kind": "polymers", "chains": rng.randint(3, 32),
                    "beads": _log_int(rng, 100, 1024), "grid": False, "langevin": True,
                    "steps": rng.randint(21, 60)}
    if op == "dh":
        return {"op": "run", "kind": "dh", "n": _log_int(rng, 8000, 1500000), "steps": 20}
    if op == "forces":
        return {"op": "forces", "kind": "dh", "n": _log_int(rng, 4000, 600000)}
    if op == "terms":
        return {"op": "forces", "kind": "terms", "n": _log_int(rng, 3000, 60000)}
    if op == "batch":
        return {"op": "batch", "systems": _log_int(rng, 12, 300), "nmin": 500,
                "nmax": rng.randint(2000, 20000), "steps": rng.randint(10, 20)}
    if op == "window":
        return {"op": "window", "chains": rng.randint(4, 16), "beads": _log_int(rng, 128, 1024),
                "steps": rng.randint(8, 24)}
    return {"op": "sort", "n": _log_int(rng, 1000, 2000000)}


def _lattice_jitter(n, seed):
    """Beads that keep apart, as an equilibrated system's do: a cubic lattice at
    the large configuration's density, each bead moved by up to 1.8 A an axis."""
    rng = np.random.default_rng(seed)
    k = int(math.ceil(n ** (1.0 / 3.0)))
    box = float((k ** 3 / DH_DENSITY) ** (1.0 / 3.0))
    site = np.sort(rng.permutation(k ** 3)[:n])
    xyz = np.stack([site // (k * k), site // k % k, site % k], axis=1) * (box / k)
    return np.mod(xyz + rng.uniform(-1.8, 1.8, size=(n, 3)), box), box


def _folded(chains, beads, box, seed):
    """Chains as they lie once they have relaxed, with bonds near 5 A and no two
    beads inside each other's core: each folded back and forth in a block of its
    own (rows and layers 10 A apart), about as dense as the coils of the polymer
    configuration, every bead moved by the thermal width of a bond."""
    rng = np.random.default_rng(seed)
    g = int(math.ceil(chains ** (1 / 3) - 1e-9))
    cell = box / g
    m, rows = max(2, int((cell - 15.0) / 5.0)), max(1, int((cell - 15.0) / 10.0))
    at, dx, dy, path = np.zeros(3), 5.0, 5.0, []

    def step(axis, by):
        at[axis] += by
        path.append(at.copy())

    path.append(at.copy())
    while len(path) < beads:
        for r in range(rows):
            for _ in range(m - 1):
                step(0, dx)
            dx = -dx
            if r < rows - 1:
                step(1, dy)
                step(1, dy)
        dy = -dy
        step(2, 5.0)
        step(2, 5.0)
    path = np.array(path[:beads])
    slack = np.maximum(cell - 8.0 - path.max(axis=0), 0.0)
    cells = rng.permutation(g ** 3)[:chains]
    corner = np.stack([cells // (g * g), cells // g % g, cells % g], axis=1) * cell
    xyz = path[None] + (corner + rng.uniform(0.0, 1.0, size=(chains, 3)) * slack)[:, None, :]
    xyz = xyz.reshape(-1, 3) + rng.normal(0.0, 0.24, size=(chains * beads, 3))
    return np.mod(xyz, box).astype(np.float32)


def _workload(c, seed):
    kind = c["kind"]
    if kind == "wca":
        return W.plain_bd(seed=seed, n=c["n"], box=float((c["n"] / WCA_DENSITY) ** (1 / 3)))
    if kind == "dh":
        return W.large_plain(seed=seed, n=c["n"])
    if kind == "polymers":
        box = 600.0 * (c["chains"] * c["beads"] / 65536.0) ** (1 / 3)
        w = W.polymers(seed=seed, n_chains=c["chains"], beads=c["beads"], box=box,
                       with_grid=c["grid"])
        w.pos[:, :3] = _folded(c["chains"], c["beads"], box, seed)
        w.angle_tables = ANGLES
        return w
    # terms: a Debye-Hueckel and a softcore term beside the table of each pair
    w = W.large_plain(seed=seed, n=c["n"])
    xyz, box = _lattice_jitter(c["n"], seed)
    w.pos[:, :3] = xyz
    w.box_size = (box, box, box)
    w.term_matrix = (w.term_matrix | np.uint32((1 << 1) | (1 << 4))).astype(np.uint32)
    return w


# The configurations' angle potential with a row past 180 degrees: angle tables
# wrap, and with 181 rows an angle that rounds to pi would read the bin between
# 180 and 0 degrees.
ANGLES = [W.harmonic_angle_table(rows=182)]
TERM_CHARGE = np.array([1.0, -1.0, 0.5, -0.5], np.float32)
TERM_RADIUS = np.array([4.0, 4.5, 5.0, 5.5], np.float32)
TERM_EPS = np.array([0.1, 0.2, 0.3, 0.4], np.float32)
MASS = np.array([150.0, 180.0], np.float32)        # Da
DAMPING = np.full((2, 3), 2.0e4, np.float32)       # 1/ns


def _window_workload(c, seed):
    w = W.adjoint(seed=seed, n_chains=c["chains"], beads=c["beads"])
    w.pos[:, :3] = _folded(c["chains"], c["beads"], w.box_size[0], seed)
    w.angle_tables = ANGLES
    return w


def _replicas(c, seed):
    # the sizes are the case's, the positions the seed's
    rng = np.random.default_rng(c["systems"])
    sizes = np.exp(rng.uniform(math.log(c["nmin"]), math.log(c["nmax"]), size=c["systems"]))
    return [W.plain_bd(seed=seed + 1 + k, n=int(n), box=float((n / DH_DENSITY) ** (1 / 3)))
            for k, n in enumerate(np.round(sizes))]


def _sort_input(c, seed):
    rng = np.random.default_rng(seed)
    box = float((c["n"] / DH_DENSITY) ** (1 / 3))
    pos = np.zeros((c["n"], 4), np.float32)
    pos[:, :3] = rng.uniform(0.0, box, size=(c["n"], 3)).astype(np.float32)
    return pos, box


def _momenta(n, kT, types, seed):
    """Maxwell-Boltzmann momenta (Da A/ns)."""
    rng = np.random.default_rng(seed + 7)
    # kT in kcal/mol; 1 kcal/mol = 4.1868e8 Da A^2/ns^2
    s = np.sqrt(MASS[types].astype(np.float64) * kT * 4.1868e8)
    mom = np.zeros((n, 4), np.float32)
    mom[:, :3] = rng.normal(size=(n, 3)) * s[:, None] * 1e-4   # the library's momentum unit
    return mom


def prepare(case, seed):
    op = case["op"]
    if op == "sort":
        pos, box = _sort_input(case, seed)
        return {"op": op, "ctx": Context(case["n"]), "pos": torch.from_numpy(pos).to(DEV),
                "lo": (0.0, 0.0, 0.0), "hi": (box, box, box)}
    if op == "batch":
        ws = _replicas(case, seed)
        b, dev = setup_batch(ws)
        b.set_rebuild_period(1)
        length = np.repeat([w.box_size[0] for w in ws], [w.n for w in ws]).astype(np.float32)
        return {"op": op, "batch": b, "dev": dev, "prm": step_params(ws[0], seed=seed),
                "box": torch.from_numpy(length[:, None]).to(DEV), "step": 1,
                "steps": case["steps"]}
    if op == "window":
        w = _window_workload(case, seed)
        win = Window(w, case["steps"], 10, seed=seed)
        pv, bv = win.pair_values(), win.bond_values()
        return {"op": op, "win": win, "pv": pv, "bv": bv, "pos": torch.from_numpy(w.pos).to(DEV),
                "target": torch.from_numpy(_target(win.rdf.bins)).to(DEV)}
    w = _workload(case, seed)
    ctx = Context(w.n)
    dev = setup_workload(ctx, w)
    s = {"op": op, "ctx": ctx, "dev": dev, "w": w}
    if case["kind"] == "terms":
        ctx.set_pair_terms(TERM_CHARGE, TERM_RADIUS, TERM_EPS)
    if op == "forces":
        return s
    if w.exclusions is not None:
        _, off, nb, npart = exclusion_csr(w.exclusions)
        s["excl"] = (torch.from_numpy(off).to(DEV), torch.from_numpy(nb).to(DEV))
        ctx.set_exclusions(*s["excl"], npart)
    s["prm"] = step_params(w, bonds=dev.get("bonds"), bond_idx=dev.get("bond_idx"),
                           angles=dev.get("angles"), angle_idx=dev.get("angle_idx"))
    if case.get("langevin"):
        ctx.set_langevin_types(MASS, DAMPING)
        s["mom"] = torch.from_numpy(_momenta(w.n, w.kT, w.type_ids, seed)).to(DEV)
        s["prm"].integrator = 1
        s["prm"].mom4 = s["mom"].data_ptr()
        s["prm"].deferred_kick_pending = 1
    s["step"] = 1
    s["steps"] = case.get("steps", 1)
    return s


def _moved(after, before, box):
    """How far each bead went, across the periodic boundary: what a program that
    follows diffusion reads from two frames (wrapped positions of a bead at the
    boundary differ by a whole box for a rounding)."""
    d = (after - before)[:, :3]
    return d - box * torch.round(d / box)


def run(s):
    op = s["op"]
    if op == "step":
        s["ctx"].step(s["dev"]["pos"], s["dev"]["fe"], s["dev"]["type"], None, s["step"], s["prm"])
        s["step"] += 1
        return s["dev"]["pos"], s["dev"]["fe"]
    if op == "run":
        before = s["dev"]["pos"].clone()
        s["ctx"].run(s["dev"]["pos"], s["dev"]["fe"], s["dev"]["type"], None, s["step"],
                     s["steps"], s["prm"])
        s["step"] += s["steps"]
        out = {"moved": _moved(s["dev"]["pos"], before, float(s["w"].box_size[0]))}
        if "mom" in s:
            out["mom"] = s["mom"]
        return out
    if op == "forces":
        ctx, dev, w = s["ctx"], s["dev"], s["w"]
        pairs = ctx.build_pairlist(dev["pos"], dev["type"], w.list_radius, w.cutoff)
        dev["fe"].zero_()
        ctx.reset_energies()
        ctx.pair_forces(dev["pos"], dev["type"], dev["fe"], w.cutoff, get_energy=True)
        return {"pairs": pairs, "fe": dev["fe"], "energies": ctx.energies()[:2]}
    if op == "batch":
        before = s["dev"]["pos"].clone()
        s["batch"].run(s["dev"]["pos"], s["dev"]["fe"], s["dev"]["type"], s["step"], s["steps"],
                       s["prm"])
        s["step"] += s["steps"]
        return {"moved": _moved(s["dev"]["pos"], before, s["box"])}
    if op == "window":
        pv = s["pv"].detach().requires_grad_(True)
        bv = s["bv"].detach().requires_grad_(True)
        pos = s["pos"].detach().requires_grad_(True)
        loss = BDWindowLoss.apply(pv, bv, pos, s["win"], s["target"])
        loss.backward()
        return {"loss": loss.detach(), "pair": pv.grad, "bond": bv.grad, "pos": pos.grad}
    keys, s2o, inv, sp = s["ctx"].sort_morton(s["pos"], s["lo"], s["hi"])
    return keys, s2o, inv, sp


def _beads(case):
    if case["op"] == "batch":
        span = math.log(case["nmax"] / case["nmin"])
        return case["systems"] * (case["nmax"] - case["nmin"]) / max(span, 1e-9)
    return case["n"] if "n" in case else case["chains"] * case["beads"]


def work(case):
    """Bytes: positions, types and (where kept) momenta in, positions and forces
    out, once a pass. Flops: about 30 a pair within the cutoff, each step (a
    difference, its square, a root, a table value, a force on both), and twice
    that again for the reverse step of a window."""
    n, op = _beads(case), case["op"]
    if op == "sort":
        return {"bytes": n * (16 + 16 + 3 * 4), "flops": 30.0 * n}
    density, rc = {"dh": (DH_DENSITY, 30.0), "terms": (DH_DENSITY, 30.0),
                   "wca": (WCA_DENSITY, 20.0)}.get(
                       case.get("kind"), (DH_DENSITY if op == "batch" else 65536 / 600.0 ** 3, 20.0))
    pairs = n * density * 4.0 / 3.0 * math.pi * rc ** 3 / 2.0
    steps = case.get("steps", 1)
    flops = 30.0 * pairs * steps * (3 if op == "window" else 1)
    nbytes = n * (16 + 4 + 16 + 16) + (n * 32 if case.get("langevin") else 0)
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """Measured: the same inputs with the pair sums in another order (other lanes
    per row), and against ``exact``. Tabulated forces are constant within a bin,
    so a last-bit difference of two positions now and then moves one pair to the
    neighbouring bin: a displacement then differs by D dt / kT times the step in
    the force, up to 0.03 A at a bond or a contact and 0.004 A in the smooth
    four-type tables, of about 1.5 A that a bead moves in a pass."""
    op = case["op"]
    if op == "sort":
        return "exact"
    if op == "forces":   # the sums alone: 1e-7; rounding of the minimum image: 1e-6
        return {"rel": 1e-5, "max": 4e-4, "differ": 0.0}
    if op == "window":
        return {"rel": 2e-3, "max": 0.2}
    if op == "step":
        return {"rel": 1e-5, "max": 1e-2}
    if case.get("kind") == "dh":   # seen: 1.2e-5, 4e-3
        return {"rel": 5e-5, "max": 2e-2}
    return {"rel": 1e-3, "max": 0.2}   # contacts, bonds: seen 2.4e-4, 3e-2


# -- the same in float64 -----------------------------------------------------------------------


def _target(bins):
    """A target profile: a soft onset at the bead diameter."""
    r = (np.arange(bins) + 0.5) * 0.25
    return 1.0 / (1.0 + np.exp(-(r - 5.0) / 0.5))


class _System:
    """One periodic cubic system in float64: pairs within the cutoff from a list
    of candidates, renewed every 10 steps (10 steps move no pair by the 7 A it
    has in hand), forces as the tables and terms say."""

    MARGIN = 7.0

    def __init__(self, w, excluded=True):
        self.w, self.n, self.box = w, w.n, float(np.float32(w.box_size[0]))
        self.types = torch.from_numpy(w.type_ids.astype(np.int64)).to(DEV)
        T = w.num_types
        tab = (w.term_matrix.astype(np.int64) >> 8).reshape(T, T)
        self.table_of = torch.from_numpy(tab).to(DEV)
        self.values = [torch.from_numpy(t.values.astype(np.float64)).to(DEV)
                       for t in w.pair_tables]
        size = max(len(v) for v in self.values)
        self.u = torch.stack([torch.cat([v, v[-1:].expand(size - len(v))]) for v in self.values])
        t0 = w.pair_tables[0]
        self.start, self.inv, self.size = float(t0.start), float(t0.step_inv), size
        self.excl = None
        if excluded and w.exclusions is not None and len(w.exclusions):
            e = np.sort(np.asarray(w.exclusions, np.int64), axis=1)
            self.excl = torch.from_numpy(e[:, 0] * self.n + e[:, 1]).to(DEV).unique()
        self.cand = None

    def wrap(self, d):
        return d - self.box * torch.round(d / self.box)

    def within(self, x, radius):
        """(i, j), i < j, within the radius and not excluded; x sorted along its
        first axis so that a block of rows only meets a window of columns."""
        order = torch.argsort(x[:, 0])
        s = x[order]
        sx = s[:, 0].contiguous()
        out, rows = [], max(1, min(4096, 120_000_000 // max(self.n, 1)))
        for a in range(0, self.n, rows):
            b = min(a + rows, self.n)
            lo, hi = float(sx[a]) - radius, float(sx[b - 1]) + radius
            q = torch.tensor([lo, hi, lo + self.box, hi - self.box], device=DEV, dtype=x.dtype)
            k = torch.searchsorted(sx, q)
            l0, h0, l1, h1 = (int(v) for v in k)
            cols = [torch.arange(l0, h0, device=DEV)]
            if hi - lo < self.box:
                if lo < 0:
                    cols.append(torch.arange(max(l1, h0), self.n, device=DEV))
                if hi > self.box:
                    cols.append(torch.arange(0, min(h1, l0), device=DEV))
            else:
                cols = [torch.arange(self.n, device=DEV)]
            cols = torch.cat(cols)
            d2 = torch.zeros((b - a, len(cols)), device=DEV, dtype=x.dtype)
            for ax in range(3):
                d2 += self.wrap(s[a:b, ax, None] - s[cols, ax][None, :]).square_()
            r, c = torch.nonzero(d2 <= radius * radius, as_tuple=True)
            i, j = order[r + a], order[cols[c]]
            m = i < j
            out.append(torch.stack([i[m], j[m]]))
        p = torch.cat(out, dim=1)
        if self.excl is not None and p.shape[1]:
            key = p[0] * self.n + p[1]
            at = torch.searchsorted(self.excl, key).clamp(max=len(self.excl) - 1)
            p = p[:, self.excl[at] != key]
        return p

    def pairs(self, x, step=0):
        if self.cand is None or step % 10 == 0:
            self.cand = self.within(x.detach(), self.w.cutoff + self.MARGIN)
        i, j = self.cand
        with torch.no_grad():
            d = self.wrap(x.detach()[j] - x.detach()[i])
            r2 = d.square().sum(1)
            m = (r2 <= float(self.w.cutoff) ** 2) & (r2 >= 1e-12)
        return i[m], j[m]

    def pair_force(self, x, i, j, u=None, terms=False):
        """-dU/dr, U, the vector i -> j and its length for each pair."""
        u = self.u if u is None else u
        d = self.wrap(x[j] - x[i])
        r = d.square().sum(1).sqrt()
        tab = self.table_of[self.types[i], self.types[j]]
        w = (r.detach() - self.start) * self.inv
        h = torch.floor(w).long().clamp(0, self.size - 1)
        h1 = (h + 1).clamp(max=self.size - 1)
        du = u[tab, h1] - u[tab, h]
        f, e = -du * self.inv, u[tab, h] + du * (w - h)
        if terms:
            q = torch.from_numpy(TERM_CHARGE.astype(np.float64)).to(DEV)[self.types]
            rad = torch.from_numpy(TERM_RADIUS.astype(np.float64)).to(DEV)[self.types]
            eps = torch.from_numpy(TERM_EPS.astype(np.float64)).to(DEV)[self.types]
            dh = q[i] * q[j] * COULOMB / 80.0 * torch.exp(-r / 10.0) / r
            f, e = f + dh * (1.0 / r + 0.1), e + dh
            s6 = (0.5 * (rad[i] + rad[j]) / r) ** 6
            ee = torch.sqrt(eps[i] * eps[j])
            f = f + 12.0 * ee * (s6 * s6 - s6) / r
            e = e + torch.where(s6 > 1.0, ee * (s6 * s6 - 2.0 * s6 + 1.0), torch.zeros_like(s6))
        return f, e, d, r

    def bonded(self, x, bond_u=None):
        """Forces of the tabulated bonds and angles."""
        w, out = self.w, torch.zeros_like(x)
        if w.bonds is not None and len(w.bonds):
            t = w.bond_tables[0]
            u = torch.from_numpy(t.values.astype(np.float64)).to(DEV) if bond_u is None else bond_u
            b = torch.from_numpy(w.bonds.astype(np.int64)).to(DEV)
            d = self.wrap(x[b[:, 1]] - x[b[:, 0]])
            r = d.square().sum(1).sqrt()
            h = torch.floor((r.detach() - float(t.start)) * float(t.step_inv)).long()
            h = h.clamp(0, len(u) - 1)
            f = -(u[(h + 1).clamp(max=len(u) - 1)] - u[h]) * float(t.step_inv)
            g = d / r[:, None] * f[:, None]
            out = out.index_add(0, b[:, 1], g).index_add(0, b[:, 0], -g)
        if w.angles is not None and len(w.angles):
            t = w.angle_tables[0]
            u = torch.from_numpy(t.values.astype(np.float64)).to(DEV)
            a = torch.from_numpy(w.angles.astype(np.int64)).to(DEV)
            p = self.wrap(x[a[:, 0]] - x[a[:, 1]])
            q = self.wrap(x[a[:, 2]] - x[a[:, 1]])
            rp, rq = p.square().sum(1).sqrt()[:, None], q.square().sum(1).sqrt()[:, None]
            cos = ((p * q).sum(1, keepdim=True) / (rp * rq)).clamp(-1.0, 1.0)
            sin = torch.linalg.cross(p, q).square().sum(1, keepdim=True).sqrt() / (rp * rq)
            theta = torch.atan2(sin, cos).squeeze(1).detach()
            sin = sin.clamp(min=1e-3)   # as the force's definition bounds it
            m = len(u)
            h = torch.floor((theta - float(t.start)) * float(t.step_inv)).long() % m
            f = (-(u[(h + 1) % m] - u[h]) * float(t.step_inv))[:, None]   # -dU/dtheta
            fp = -f * (q / rq - cos * p / rp) / (rp * sin)
            fq = -f * (p / rp - cos * q / rq) / (rq * sin)
            out = out.index_add(0, a[:, 0], fp).index_add(0, a[:, 2], fq)
            out = out.index_add(0, a[:, 1], -fp - fq)
        return out

    def grid(self, x):
        """Force and energy of the grid potential (trilinear, 0 outside)."""
        spec = self.w.grids[0]
        g = torch.from_numpy(spec["data"].astype(np.float64)).to(DEV)
        origin = [float(np.float32(o)) for o in spec["origin"]]
        q = x - torch.tensor(origin, device=DEV, dtype=x.dtype)
        i0 = torch.floor(q).long()
        t = q - i0
        force, energy = torch.zeros_like(x), torch.zeros(len(x), device=DEV, dtype=x.dtype)
        for corner in range(8):
            c = [(corner >> k) & 1 for k in range(3)]
            idx = [i0[:, k] + c[k] for k in range(3)]
            inside = torch.ones(len(x), dtype=torch.bool, device=DEV)
            for k in range(3):
                inside &= (idx[k] >= 0) & (idx[k] < g.shape[k])
            v = torch.where(inside, g[tuple(torch.where(inside, idx[k], 0) for k in range(3))], 0.0)
            wt = [t[:, k] if c[k] else 1.0 - t[:, k] for k in range(3)]
            energy += v * wt[0] * wt[1] * wt[2]
            for k in range(3):
                o = [wt[m] for m in range(3) if m != k]
                force[:, k] -= v * (1.0 if c[k] else -1.0) * o[0] * o[1]
        return force, energy

    def forces(self, x, step=0, pair_u=None, bond_u=None):
        i, j = self.pairs(x, step)
        f, _, d, r = self.pair_force(x, i, j, pair_u)
        g = d * (f / r)[:, None]
        out = self.bonded(x, bond_u)
        return out.index_add(0, j, g).index_add(0, i, -g)


def _u32(v):
    return v & 0xFFFFFFFF


def _noise(n, seed, step, stream=0x5324120):
    """Three standard normals a particle: Philox 4x32-10 (Salmon et al., SC'11)
    keyed on the mixed seed, counter (particle, stream, step, 0), Box-Muller."""
    key = (seed * 0x9E3779B97F4A7C15 ^ step * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
    k0, k1 = key >> 32, key & 0xFFFFFFFF
    c = [torch.arange(n, dtype=torch.int64, device=DEV),
         torch.full((n,), stream, dtype=torch.int64, device=DEV),
         torch.full((n,), step, dtype=torch.int64, device=DEV),
         torch.zeros(n, dtype=torch.int64, device=DEV)]

    def product(a, v):
        lo, hi = a * (v & 0xFFFF), a * (v >> 16)   # each below 2^48
        mid = (lo >> 16) + (hi & 0xFFFF)
        return _u32(lo & 0xFFFF | (mid & 0xFFFF) << 16), _u32((hi >> 16) + (mid >> 16))

    for r in range(10):
        a, b = (k0 + r * 0x9E3779B9) & 0xFFFFFFFF, (k1 + r * 0xBB67AE85) & 0xFFFFFFFF
        lo0, hi0 = product(0xD2511F53, c[0])
        lo1, hi1 = product(0xCD9E8D57, c[2])
        c = [hi1 ^ c[1] ^ a, lo1, hi0 ^ c[3] ^ b, lo0]
    u = [v.double() * 2.0 ** -32 + 2.0 ** -33 for v in c]
    r1, r2 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    return torch.stack([r1 * torch.cos(2 * math.pi * u[1]), r1 * torch.sin(2 * math.pi * u[1]),
                        r2 * torch.cos(2 * math.pi * u[3])], dim=1)


def _advance(sys_, x, force, seed, step):
    w = sys_.w
    kT, dt = float(np.float32(w.kT)), float(np.float32(w.dt))
    d = torch.from_numpy(w.diffusion.astype(np.float64)).to(DEV)[sys_.types]
    x = x + d / kT * force * dt + torch.sqrt(2.0 * d * dt) * _noise(sys_.n, seed, step)
    return x - sys_.box * torch.floor(x.detach() / sys_.box)


def _pos4(x):
    return torch.cat([x, torch.zeros((len(x), 1), device=DEV, dtype=x.dtype)], dim=1)


def _exact_window(case, seed):
    w = _window_workload(case, seed)
    s = _System(w)
    pu = s.u[0].clone().requires_grad_(True)
    t = w.bond_tables[0]
    bu = torch.from_numpy(t.values.astype(np.float64)).to(DEV).requires_grad_(True)
    x0 = torch.from_numpy(w.pos[:, :3].astype(np.float64)).to(DEV).requires_grad_(True)
    x = x0
    for k in range(case["steps"]):
        x = _advance(s, x, s.forces(x, k, pu[None], bu), seed, k + 1)
    # the Gaussian-smoothed histogram of pair distances and its squared error
    bins, dr, sigma, r_max = 100, 0.25, 0.25, 25.0
    i, j = s.within(x.detach(), r_max)
    r = s.wrap(x[j] - x[i]).square().sum(1).sqrt()
    centre = (torch.arange(bins, device=DEV, dtype=x.dtype) + 0.5) * dr
    hist = torch.zeros(bins, device=DEV, dtype=x.dtype)
    b0 = torch.floor(r.detach() / dr).long()
    for o in range(-6, 7):
        b = b0 + o
        ok = (b >= 0) & (b < bins)
        z = (r[ok] - centre[b[ok]]) / sigma
        v = torch.exp(-0.5 * z * z) * (z.detach().abs() <= 5.0)
        hist = hist.index_add(0, b[ok], v)
    vol = s.box ** 3
    norm = vol / (s.n * (s.n - 1) / 2.0 * 4.0 * math.pi * centre * centre * dr)
    loss = ((hist * norm - torch.from_numpy(_target(bins)).to(DEV)) ** 2).sum()
    loss.backward()
    return {"loss": loss.detach(), "pair": pu.grad, "bond": bu.grad, "pos": _pos4(x0.grad)}


def exact(case, seed):
    op = case["op"]
    if op == "sort":
        return None
    n = _beads(case)
    if op == "window":
        return _exact_window(case, seed)
    if op == "batch":
        if n > 400000:
            return None
        out = []
        for k, w in enumerate(_replicas(case, seed)):
            s = _System(w)
            x = torch.from_numpy(w.pos[:, :3].astype(np.float64)).to(DEV)
            for q in range(case["steps"]):
                x = _advance(s, x, s.forces(x, q), seed + k, q + 1)
            out.append(s.wrap(x - torch.from_numpy(w.pos[:, :3].astype(np.float64)).to(DEV)))
        return {"moved": torch.cat(out)}
    if n > 310000 or case.get("langevin"):
        return None   # Langevin: its unit conversions are the framework's own
    w = _workload(case, seed)
    s = _System(w)
    x = torch.from_numpy(w.pos[:, :3].astype(np.float64)).to(DEV)
    if op == "forces":
        count = s.within(x, float(w.list_radius)).shape[1]
        i, j = s.pairs(x)
        f, e, d, r = s.pair_force(x, i, j, terms=case["kind"] == "terms")
        g = d * (f / r)[:, None]
        fe = torch.zeros((s.n, 4), device=DEV, dtype=x.dtype)
        half = torch.cat([g, 0.5 * e[:, None]], dim=1)
        back = torch.cat([-g, 0.5 * e[:, None]], dim=1)
        fe = fe.index_add(0, j, half).index_add(0, i, back)
        return {"pairs": count, "fe": fe,
                "energies": torch.stack([e.sum(), (f * r).sum()]).cpu().numpy()}
    for k in range(case.get("steps", 1)):
        force = s.forces(x, k)
        fe = _pos4(force)
        if w.grids:
            more, fe[:, 3] = s.grid(x)
            force = force + more
        x = _advance(s, x, force, w.seed, k + 1)
    if op == "step":
        return _pos4(x), fe
    return {"moved": s.wrap(x - torch.from_numpy(w.pos[:, :3].astype(np.float64)).to(DEV))}
