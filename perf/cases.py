"""Performance cases: what a program that uses this package has it compute.

Every case goes through the public entry points (potentials, md, batch,
adjoint). The systems are water boxes with a chain ligand at 1 g/cm^3
(testsystems), the shapes of the tests and of bench.py: a few hundred atoms up
to about 100,000, at 1.2 nm cutoff.

Kinds of case (the "kind" key):

- "execute":      one host call, numpy in and out (`execute`): the smallest
                  calls, where launches and copies count;
- "frames":       device tensors, one call per coordinate frame, as an engine
                  of its own integrator ("moving": consecutive MD steps) or a
                  rescoring of stored frames (independent ones) makes them;
- "windows":      one frame at all lambda windows of a schedule, one call;
- "host_batch":   `execute_selective_batch` over stored frames and lambdas;
- "md":           `Context.multiple_steps` with bonds, angles and (optional)
                  Monte Carlo barostat;
- "group":        the interpolated ligand-environment interaction group;
- "replicas":     `ReplicaBatch` evaluations of several systems x windows;
- "replicas_md":  `ReplicaBatch` Langevin steps of the same;
- "grad":         loss over frames through the differentiable forces, and its
                  gradient (forward and adjoint kernels).
"""

import numpy as np
import torch

from timemachine_b200 import md as mdmod
from timemachine_b200 import potentials as P
from timemachine_b200 import testsystems
from timemachine_b200.adjoint import nonbonded_forces
from timemachine_b200.batch import ReplicaBatch

BOLTZ = 0.008314462618  # kJ/mol/K
TEMPERATURE = 300.0
# FP32 operations of one pair within the cutoff, and of its Lennard-Jones part
# (one water pair in nine); directions of the adjoint counted as twice that
FLOPS_PER_PAIR = 69.0
PAIRS_PER_ATOM = 362.0  # half of 4/3 pi 1.2^3 nm^3 at 100 atoms per nm^3


def listed():
    return [
        # one energy call of a solvated fragment, numpy in and out: launch and copy latency
        dict(name="execute_900", kind="execute", n=912, precision=32),
        # forces of consecutive MD steps of a small box (bench and parity tests: 3,000-atom water box)
        dict(name="frames_forces_3k", kind="frames", n=3000, frames=16, moving=True, outputs="forces", precision=32),
        # all outputs of stored frames of a large solvated complex: a new neighbour list for each
        dict(name="frames_all_98k", kind="frames", n=98000, frames=2, moving=False, outputs="all", precision=32),
        # one frame at the 12 windows of a schedule (the benchmark's shape), both precisions
        dict(name="windows_f32_23k", kind="windows", n=22840, windows=12, precision=32),
        dict(name="windows_f64_23k", kind="windows", n=22840, windows=12, precision=64),
        # reweighting: stored frames x lambdas through the host batch call
        dict(name="host_batch_5k", kind="host_batch", n=5003, frames=4, windows=6, precision=32),
        # Langevin MD with barostat at the benchmark's size, and of a small box without
        dict(name="md_23k", kind="md", n=22840, steps=50, barostat=True),
        dict(name="md_2500", kind="md", n=2503, steps=100, barostat=False),
        # ligand in its environment with interpolated parameters
        dict(name="group_23k", kind="group", n=22840, windows=1),
        # many systems x windows together: one evaluation, and MD steps
        dict(name="replicas_eval", kind="replicas", n=4000, systems=6, windows=4),
        dict(name="replicas_md", kind="replicas_md", n=4000, systems=6, windows=4, steps=20),
        # force-matching loss and gradient over frames of a 5,000-atom box
        dict(name="grad_5k", kind="grad", n=5000, frames=4),
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(
        ["execute", "frames", "frames", "windows", "windows", "host_batch", "md", "group", "replicas", "replicas_md", "grad"]
    )
    if kind == "execute":
        return dict(kind=kind, n=_log(rng, 150, 6000), precision=rng.choice([32, 64]))
    if kind == "frames":
        moving = rng.random() < 0.5
        n = _log(rng, 1000, 90000)
        return dict(
            kind=kind, n=n, frames=rng.randint(2, 16) if n < 12000 else 2, moving=moving,
            outputs=rng.choice(["forces", "energy", "all"]), precision=rng.choice([32, 32, 64]) if n < 30000 else 32,
        )
    if kind == "windows":
        return dict(kind=kind, n=_log(rng, 1000, 30000), windows=rng.randint(2, 16), precision=rng.choice([32, 32, 64]))
    if kind == "host_batch":
        return dict(kind=kind, n=_log(rng, 600, 10000), frames=rng.randint(2, 5), windows=rng.randint(2, 8), precision=32)
    if kind == "md":
        return dict(kind=kind, n=_log(rng, 1500, 30000), steps=rng.randint(20, 60), barostat=rng.random() < 0.5)
    if kind == "group":
        return dict(kind=kind, n=_log(rng, 1000, 40000), windows=rng.choice([1, 1, 8]))
    if kind in ("replicas", "replicas_md"):
        c = dict(kind=kind, n=_log(rng, 1500, 6000), systems=rng.randint(2, 6), windows=rng.randint(1, 4))
        if kind == "replicas_md":
            c["steps"] = rng.randint(5, 20)
        return c
    return dict(kind=kind, n=_log(rng, 1000, 8000), frames=rng.randint(1, 4))


# -- inputs --------------------------------------------------------------------


def _f32(a):
    """Values that FP32 holds, as coordinates and parameters of stored systems are."""
    return np.asarray(a, dtype=np.float32).astype(np.float64)


def _system(n, seed, hmr=False, n_ligand=None):
    n_ligand = min(40, max(4, n // 40)) if n_ligand is None else n_ligand
    s = testsystems.system_of_size(n, seed=seed, n_ligand=n_ligand, min_edge=2.9, hmr=hmr)
    s.x = _f32(s.x)
    s.params = _f32(s.params)
    return s


def _nonbonded(s, precision):
    nb = P.Nonbonded(s.exclusion_idxs, s.scales, s.lambda_plane_idxs, s.lambda_offset_idxs, s.beta, s.cutoff)
    return nb.unbound_impl(np.float32 if precision == 32 else np.float64)


def _velocities(s, rng):
    return rng.normal(size=(s.N, 3)) * np.sqrt(BOLTZ * TEMPERATURE / s.masses)[:, None]


def _frames(s, rng, count, moving):
    if moving:  # consecutive steps of 2.5 fs
        v = _velocities(s, rng)
        return np.stack([_f32(s.x + 0.0025 * k * v) for k in range(count)])
    # stored frames: the atoms of each lie elsewhere in the periodic box
    return np.stack(
        [_f32(s.x + rng.normal(scale=0.01, size=s.x.shape) + rng.uniform(0, 1, size=3) * np.diag(s.box)) for _ in range(count)])


def _end_states(s, rng):
    """Parameters of both ends of an alchemical change of the ligand."""
    p1 = s.params.copy()
    p1[s.ligand_idxs] *= 1 + 0.1 * rng.normal(size=(s.ligand_idxs.size, 3))
    return _f32(np.concatenate([s.params, p1]))


def _inputs(case, seed):
    """What prepare() and exact() both start from, on the host."""
    kind, n = case["kind"], case["n"]
    rng = np.random.default_rng(1000 + seed)
    if kind in ("replicas", "replicas_md"):
        systems = [_system(int(n * (0.5 + k)), seed + 17 * k, hmr=True) for k in range(case["systems"])]
        lams = np.linspace(0.0, 1.0, case["windows"]) if case["windows"] > 1 else np.array([0.4])
        return dict(systems=systems, lams=lams, v=[_velocities(s, rng) for s in systems])
    s = _system(n, seed, hmr=kind == "md")
    d = dict(s=s, rng=rng)
    if kind == "execute":
        d["lam"] = 0.1 + 0.8 * rng.random()
    elif kind == "frames":
        d["x"] = _frames(s, rng, case["frames"], case["moving"])
        d["lam"] = 0.35
    elif kind == "windows":
        d["lams"] = np.linspace(0.0, 1.0, case["windows"])
    elif kind == "host_batch":
        d["x"] = _frames(s, rng, case["frames"], False)
        d["lams"] = np.linspace(0.0, 1.0, case["windows"])
    elif kind == "group":
        d["p"] = _end_states(s, rng)
        d["lams"] = np.linspace(0.0, 1.0, case["windows"]) if case["windows"] > 1 else np.array([0.3])
    elif kind == "grad":
        d["x"] = [_f32(s.x + rng.normal(scale=0.01, size=s.x.shape)) for _ in range(case["frames"])]
        d["target"] = [rng.normal(scale=500.0, size=s.x.shape) for _ in range(case["frames"])]
        d["lam"] = 0.5
    return d


class _Outputs:
    """One int64 buffer for the accumulated outputs of K evaluations, and its decoding."""

    def __init__(self, K, N, n_params, which):
        sizes = {"dx": 3 * N if which != "energy" else 0, "dp": n_params if which == "all" else 0,
                 "dl": N if which == "all" else 0, "u": N if which != "forces" else 0}
        self.buf = torch.zeros(K * sum(sizes.values()), dtype=torch.int64, device="cuda")
        self.parts, o = {}, 0
        for name, size in sizes.items():
            self.parts[name] = self.buf[o : o + K * size].view(K, size) if size else None
            o += K * size
        self.unit = torch.tensor(2.0**-36, dtype=torch.float64, device="cuda")
        self.unit_dp = torch.tensor([2.0**-36, 2.0**-37, 2.0**-38], dtype=torch.float64, device="cuda")
        self.K, self.N = K, N

    def __getitem__(self, name):
        return self.parts[name]

    def row(self, name, k):
        return None if self.parts[name] is None else self.parts[name][k]

    def decoded(self):
        out = {}
        if self["dx"] is not None:
            out["du_dx"] = (self["dx"] * self.unit).view(self.K, self.N, 3)
        if self["dp"] is not None:
            out["du_dp"] = self["dp"].view(self.K, -1, 3) * self.unit_dp
        for name in ("dl", "u"):  # per-atom buffers: only their sums are defined
            if self[name] is not None:
                out["du_dl" if name == "dl" else "u"] = self[name].sum(dim=1) * self.unit
        return out


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind in ("replicas", "replicas_md"):
        b = ReplicaBatch()
        md = dict(temperature=TEMPERATURE, dt=0.0015, friction=1.0)
        st["ids"] = [
            b.add(s, float(lam), v=v, md=md, seed=seed + 100 * k + w)
            for k, (s, v) in enumerate(zip(d["systems"], d["v"])) for w, lam in enumerate(d["lams"])
        ]
        st["batch"] = b
        return st
    s = d["s"]
    if kind == "md":
        bps = [
            P.HarmonicBond(s.bond_idxs).bind(s.bond_params).bound_impl(np.float32),
            P.HarmonicAngle(s.angle_idxs).bind(s.angle_params).bound_impl(np.float32),
            P.BoundPotential(_nonbonded(s, 32), s.params),
        ]
        # a state away from the lattice start, then the run itself at 2.5 fs
        eq = mdmod.Context(
            s.x, _velocities(s, d["rng"]), s.box, mdmod.LangevinIntegrator(TEMPERATURE, 0.0005, 10.0, s.masses, seed), bps)
        eq.multiple_steps(np.full(100, 0.5))
        baro = None
        if case["barostat"]:
            order = np.argsort(s.group_of, kind="stable")
            groups = np.split(order, np.flatnonzero(np.diff(s.group_of[order])) + 1)
            baro = mdmod.MonteCarloBarostat(s.N, 1.0, TEMPERATURE, groups, 25, seed + 1)
        intg = mdmod.LangevinIntegrator(TEMPERATURE, 0.0025, 1.0, s.masses, seed + 7)
        st["ctx"] = mdmod.Context(eq.get_x_t(), eq.get_v_t(), eq.get_box(), intg, bps, baro)
        st["lam"] = np.full(case["steps"], 0.5)
        return st
    if kind == "execute":
        st.update(impl=_nonbonded(s, case["precision"]), x=s.x, p=s.params, box=s.box, lam=d["lam"])
    elif kind == "host_batch":
        F = case["frames"]
        st.update(impl=_nonbonded(s, case["precision"]), x=d["x"], p=s.params[None], boxes=np.stack([s.box] * F), lams=d["lams"])
    elif kind == "frames":
        st.update(impl=_nonbonded(s, case["precision"]), x=_dev(d["x"]), p=_dev(s.params).reshape(-1), box=_dev(s.box), lam=d["lam"],
                  out=_Outputs(case["frames"], s.N, 3 * s.N, case["outputs"]))
    elif kind == "windows":
        st.update(impl=_nonbonded(s, case["precision"]), x=_dev(s.x), p=_dev(s.params).reshape(-1), box=_dev(s.box), lams=d["lams"],
                  out=_Outputs(case["windows"], s.N, 3 * s.N, "all"))
    elif kind == "group":
        g = P.NonbondedInteractionGroupInterpolated(s.ligand_idxs, s.lambda_plane_idxs, s.lambda_offset_idxs, s.beta, s.cutoff)
        st.update(impl=g.unbound_impl(np.float32), x=_dev(s.x), p=_dev(d["p"]).reshape(-1), box=_dev(s.box), lams=d["lams"],
                  out=_Outputs(case["windows"], s.N, 6 * s.N, "all"))
    elif kind == "grad":
        st.update(impl=_nonbonded(s, 32), x=[_dev(x) for x in d["x"]], target=[_dev(t) for t in d["target"]], box=_dev(s.box),
                  p=_dev(s.params), off=_dev(s.lambda_offset_idxs.astype(np.float64)), lam=d["lam"])
    return st


# -- one pass ------------------------------------------------------------------


def run(st):
    kind = st["kind"]
    if kind == "execute":
        return st["impl"].execute(st["x"], st["p"], st["box"], st["lam"])
    if kind == "host_batch":
        return st["impl"].execute_selective_batch(st["x"], st["p"], st["boxes"], st["lams"], True, True, True, True)
    if kind == "frames":
        o = st["out"]
        o.buf.zero_()
        for k in range(o.K):
            st["impl"].execute_device(st["x"][k], st["p"], st["box"], st["lam"], o.row("dx", k), o.row("dp", k), o.row("dl", k), o.row("u", k))
        return o.decoded()
    if kind in ("windows", "group"):
        o = st["out"]
        o.buf.zero_()
        st["impl"].execute_windows_device(st["x"], st["p"], st["box"], st["lams"], o["dx"], o["dp"], o["dl"], o["u"])
        return o.decoded()
    if kind == "md":
        c = st["ctx"]
        c.multiple_steps(st["lam"])
        return c.get_x_t(), c.get_v_t(), c.get_box()
    if kind == "replicas":
        b = st["batch"]
        b.evaluate()
        res = [b.result(r) for r in st["ids"]]
        return [np.concatenate([r[c] for r in res]) for c in (0, 1)] + [np.array([r[c] for r in res]) for c in (2, 3)]
    if kind == "replicas_md":
        b = st["batch"]
        b.md(st["case"]["steps"])
        return np.concatenate([b.get_x(r) for r in st["ids"]]), np.concatenate([b.get_v(r) for r in st["ids"]])
    p = st["p"].clone().requires_grad_(True)
    off = st["off"].clone().requires_grad_(True)
    loss = 0.0
    for x, t in zip(st["x"], st["target"]):
        f, dl = nonbonded_forces(st["impl"], p, off, x, st["box"], st["lam"])
        loss = loss + ((f - t) ** 2).mean() + 0.1 * dl**2
    loss.backward()
    return loss.detach(), p.grad, off.grad


# -- what a pass cannot do without ----------------------------------------------


def work(case):
    kind, n = case["kind"], float(case["n"])
    pair = FLOPS_PER_PAIR * PAIRS_PER_ATOM
    out = 8 * 8.0  # bytes of the eight int64 outputs of an atom
    if kind == "execute":
        return {"bytes": n * (6 * 8 + out), "flops": n * pair}
    if kind == "frames":
        size = {"forces": 24.0, "energy": 8.0, "all": out}[case["outputs"]]
        return {"bytes": case["frames"] * n * (24 + size) + 24 * n, "flops": case["frames"] * n * pair}
    if kind in ("windows", "host_batch"):
        # pairs without a ligand atom are the same in every window
        f = case.get("frames", 1)
        lig = min(40.0, max(4.0, n // 40))
        return {"bytes": f * n * (24 + case["windows"] * out) + 24 * n, "flops": f * (n + 2 * lig * (case["windows"] - 1)) * pair}
    if kind == "md":
        return {"bytes": case["steps"] * n * 15 * 8.0, "flops": case["steps"] * n * pair}
    if kind == "group":
        lig = min(40.0, max(4.0, n // 40))
        return {"bytes": n * (24 + 48 + case["windows"] * (24 + 48 + 16)), "flops": case["windows"] * 2 * lig * pair}
    if kind in ("replicas", "replicas_md"):
        atoms = case["windows"] * sum(n * (0.5 + k) for k in range(case["systems"]))
        if kind == "replicas":
            return {"bytes": atoms * (48 + out), "flops": atoms * pair}
        return {"bytes": case["steps"] * atoms * 15 * 8.0, "flops": case["steps"] * atoms * pair}
    # forward and adjoint of every frame
    return {"bytes": case["frames"] * n * (2 * 48 + 32 + 32), "flops": case["frames"] * 3 * n * pair}


def tolerance(case):
    kind = case["kind"]
    if kind in ("md", "replicas_md"):
        # FP32 forces: a last-bit change of them, after some tens of steps
        return {"rel": 1e-5, "max": 1e-3}
    if case.get("precision") == 64:
        # FP64 terms, each rounded to 2^-36
        return {"rel": 1e-9, "max": 1e-7}
    # FP32 terms (sums are exact); energies and du_dl cancel by a factor of some tens
    return {"rel": 1e-5, "max": 1e-3}


# -- the same in 64 bits ---------------------------------------------------------


def _pairs(x, box, cutoff, rows=None):
    """i < j within the cutoff (3D minimum image); with rows: one of the two in rows."""
    N = x.shape[0]
    L = torch.diagonal(box)
    index = torch.arange(N, device=x.device)
    found = []
    step = max(1, int(2e8) // N)
    for a in range(0, N, step):
        r = torch.zeros(1, dtype=torch.float64, device=x.device)
        for c in range(3):
            t = x[a : a + step, c, None] - x[None, :, c]
            t = t - L[c] * torch.floor(t / L[c] + 0.5)
            r = r + t * t
        keep = (r < (cutoff * (1 + 1e-9)) ** 2) & (index[a : a + step, None] < index[None, :])
        if rows is not None:
            keep &= rows[a : a + step, None] != rows[None, :]
        i, j = torch.nonzero(keep, as_tuple=True)
        found.append(torch.stack([i + a, j]))
    return torch.cat(found, dim=1)


def _masks(pairs, N, s):
    keep = torch.ones(2, pairs.shape[1], dtype=torch.float64, device=pairs.device)
    e = np.sort(s.exclusion_idxs.reshape(-1, 2).astype(np.int64), axis=1)
    key = e[:, 0] * N + e[:, 1]
    order = np.argsort(key)
    key = torch.as_tensor(key[order], device=pairs.device)
    scale = torch.as_tensor(s.scales[order], device=pairs.device)
    at = torch.searchsorted(key, pairs[0] * N + pairs[1]).clamp(max=key.numel() - 1)
    hit = key[at] == pairs[0] * N + pairs[1]
    return torch.where(hit, 1 - scale[at].T, keep)


def _energy(x, p, off, lam, plane, box, beta, cutoff, pairs, masks):
    i, j = pairs
    L = torch.diagonal(box)
    r = x[i] - x[j]
    r = r - L * torch.floor(r.detach() / L + 0.5)
    w = cutoff * (plane + off * lam)
    d2 = (r * r).sum(-1) + (w[i] - w[j]) ** 2
    d = torch.sqrt(torch.where(d2 < cutoff**2, d2, torch.ones_like(d2)))
    inside = (d2 < cutoff**2).to(torch.float64)
    eps = p[i, 2] * p[j, 2]
    lj = (eps != 0).to(torch.float64)  # no Lennard-Jones term, and no derivative of one, without both epsilons
    s6 = ((p[i, 1] + p[j, 1]) / d) ** 6
    es = p[i, 0] * p[j, 0] * torch.special.erfc(beta * d) / d
    return (inside * (masks[0] * es + masks[1] * lj * 4 * eps * (s6 - 1) * s6)).sum()


def _exact_terms(s, x, params, lam, group=False):
    """(du_dx, du_dp, du_dl, u) of one frame at one lambda."""
    tx, box = _dev(x).requires_grad_(True), _dev(s.box)
    tp = _dev(params).requires_grad_(True)
    tl = torch.tensor(float(lam), dtype=torch.float64, device="cuda", requires_grad=True)
    plane, off = _dev(s.lambda_plane_idxs), _dev(s.lambda_offset_idxs)
    N = s.N
    rows = None
    if group:
        rows = torch.zeros(N, dtype=torch.bool, device="cuda")
        rows[torch.as_tensor(s.ligand_idxs.astype(np.int64), device="cuda")] = True
    pairs = _pairs(tx.detach(), box, s.cutoff, rows)
    masks = torch.ones(2, pairs.shape[1], dtype=torch.float64, device="cuda") if group else _masks(pairs, N, s)
    p = tp if tp.shape[0] == N else (1 - tl) * tp[:N] + tl * tp[N:]
    u = _energy(tx, p, off, tl, plane, box, s.beta, s.cutoff, pairs, masks)
    gx, gp, gl = torch.autograd.grad(u, [tx, tp, tl])
    return gx, gp, gl, u.detach()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("md", "replicas_md"):
        return None  # a trajectory has no 64-bit counterpart: it starts from this package's own equilibration
    d = _inputs(case, seed)
    if kind == "replicas":
        res = [_exact_terms(s, s.x, s.params, lam) for s in d["systems"] for lam in d["lams"]]
        return [torch.cat([r[c] for r in res]).cpu().numpy() for c in (0, 1)] + [
            torch.stack([r[c] for r in res]).cpu().numpy() for c in (2, 3)]
    s = d["s"]
    if kind == "execute":
        gx, gp, gl, u = _exact_terms(s, s.x, s.params, d["lam"])
        return gx.cpu().numpy(), gp.cpu().numpy(), float(gl), float(u)
    if kind == "host_batch":
        res = [_exact_terms(s, x, s.params, lam) for x in d["x"] for lam in d["lams"]]
        lead = (case["frames"], 1, case["windows"])
        return tuple(torch.stack([r[c] for r in res]).reshape(lead + tuple(res[0][c].shape)).cpu().numpy() for c in range(4))
    if kind == "grad":
        tp, off = _dev(s.params).requires_grad_(True), _dev(s.lambda_offset_idxs.astype(np.float64)).requires_grad_(True)
        plane, box = _dev(s.lambda_plane_idxs), _dev(s.box)
        total, grads = 0.0, [torch.zeros_like(tp), torch.zeros_like(off)]
        for x, t in zip(d["x"], d["target"]):
            tx = _dev(x).requires_grad_(True)
            tl = torch.tensor(d["lam"], dtype=torch.float64, device="cuda", requires_grad=True)
            pairs = _pairs(tx.detach(), box, s.cutoff)
            u = _energy(tx, tp, off, tl, plane, box, s.beta, s.cutoff, pairs, _masks(pairs, s.N, s))
            f, dl = torch.autograd.grad(u, [tx, tl], create_graph=True)
            loss = ((f - _dev(t)) ** 2).mean() + 0.1 * dl**2
            total = total + loss.detach()
            for g, part in zip(grads, torch.autograd.grad(loss, [tp, off])):
                g += part
        return total, grads[0], grads[1]
    if kind == "frames":
        res = [_exact_terms(s, x, s.params, d["lam"]) for x in d["x"]]
    elif kind == "windows":
        res = [_exact_terms(s, s.x, s.params, lam) for lam in d["lams"]]
    else:
        res = [_exact_terms(s, s.x, d["p"], lam, group=True) for lam in d["lams"]]
    out = {name: torch.stack([r[c] for r in res]) for c, name in enumerate(("du_dx", "du_dp", "du_dl", "u"))}
    which = case.get("outputs", "all")
    if which == "forces":
        return {"du_dx": out["du_dx"]}
    return {"u": out["u"]} if which == "energy" else out
