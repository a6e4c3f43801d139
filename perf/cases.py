"""The workloads by which the speed of this framework is judged: simulation boxes stepped through
the public API (`mdpd.Batch`, `mdpd.Lammps`), from one 2,000-particle box to a 4M-particle liquid
and 256 uneven boxes together.

A case is a dict: `kind` (which program it stands for), the particle count or box edges, `steps`
(time steps of one pass) and the physics that a deck would set. `prepare` makes the particles on
the GPU from the seed (a jittered lattice of the liquid's density, Maxwell velocities), creates
the boxes and sets them up; `run` is one pass: the steps and what the program reads back after
them; `exact` steps the same particles in 64 bits with plain torch, where that is quick.

Reduced units: cutoff 1, mass 1, kT 1, dt 0.01, skin 0.3; mDPD liquid at density 6.05, classic DPD
fluid at density 3.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("usermeso-2.0-mdpd_b200"))
import mdpd  # noqa: E402

RHO, RHO_DPD, RHO_WALL = 6.05, 3.0, 8.0
DT, SKIN, RC, GAMMA = 0.01, 0.3, 1.0, 4.5
SIGMA_DPD, A_DPD = 3.0, 25.0
PITCH, RADIUS, LAYER = 20.0, 7.0, 2.5  # pore cylinders: spacing, radius, wall layer


def listed():
    return [
        # the classic DPD fluid of the smallest deck (10 x 10 x 10, density 3): latency alone
        dict(name="dpd-cube-3k", kind="dpd", n=3000, steps=100),
        # the smallest box of a parameter study
        dict(name="liquid-2k", kind="liquid", n=2000, A=-40.0, B=25.0, rd=0.75, exact_rng=False, steps=50),
        # a validation run with the bit-exact 64-bit random transform
        dict(name="liquid-20k-exact-rng", kind="liquid", n=20011, A=-35.0, B=25.0, rd=0.75, exact_rng=True, steps=20),
        # an ordinary single box
        dict(name="liquid-42k", kind="liquid", n=42013, A=-40.0, B=25.0, rd=0.8, exact_rng=False, steps=20),
        # the liquid-vapour slab of the surface-tension deck, 60 x 30 x 30: most bins are empty
        dict(name="slab-109k", kind="slab", lx=60.0, ly=30.0, lz=30.0, half=10.0, steps=20),
        # a run with a thermo line at every step (energy and virial each step)
        dict(name="thermo-200k", kind="thermo", n=200003, steps=20),
        # the largest single box
        dict(name="liquid-4M", kind="liquid", n=4000000, A=-40.0, B=25.0, rd=0.75, exact_rng=False, steps=20),
        # the parameter study: 256 uneven boxes, 2k to 200k particles, stepped together
        dict(name="batch-256", kind="batch", boxes=256, lo=2000, hi=200000, pick=1, steps=20),
        # classic DPD at scale
        dict(name="dpd-1M", kind="dpd", n=1000003, steps=10),
        # flow through an array of frozen cylinders, driven by a body force, from a deck
        dict(name="pore-120x80", kind="pore", lx=120.0, ly=80.0, lz=4.0, steps=20),
        # two atom types, from a deck; each `run` sets up, steps and prints thermo
        dict(name="deck-two-types-60k", kind="deck", n=60007, steps=20),
        # short jobs: boxes from host arrays, setup, steps, state back, boxes released
        dict(name="turnover-16", kind="turnover", boxes=16, lo=5000, hi=50000, pick=2, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(n):
    return 50 if n < 10000 else 20 if n < 300000 else 10


def draw(rng: random.Random):
    kind = rng.choice(["liquid", "liquid", "liquid", "dpd", "dpd", "slab", "thermo", "batch", "batch", "pore", "deck",
                       "turnover"])
    if kind == "liquid":
        n = _log(rng, 2000, 3500000)
        return dict(kind=kind, n=n, A=round(rng.uniform(-50, -30), 3), B=round(rng.uniform(20, 30), 3),
                    rd=round(rng.uniform(0.7, 0.8), 4), exact_rng=rng.random() < 0.25, steps=_steps(n))
    if kind == "dpd":
        n = _log(rng, 3000, 2000000)
        return dict(kind=kind, n=n, steps=_steps(n))
    if kind == "slab":
        lx, ly, lz = (round(rng.uniform(a, b), 2) for a, b in ((20, 90), (10, 45), (10, 45)))
        half = round(lx * rng.uniform(0.12, 0.3), 2)
        return dict(kind=kind, lx=lx, ly=ly, lz=lz, half=half, steps=20)
    if kind == "thermo":
        n = _log(rng, 2000, 1000000)
        return dict(kind=kind, n=n, steps=_steps(n))
    if kind == "batch":
        lo = _log(rng, 2000, 20000)
        hi = min(200000, lo * rng.randint(2, 40))
        most = 8000000 // hi
        return dict(kind=kind, boxes=max(2, min(256, rng.randint(2, 256), most)), lo=lo, hi=hi,
                    pick=rng.randrange(1 << 20), steps=20)
    if kind == "pore":
        return dict(kind=kind, lx=PITCH * rng.randint(2, 10), ly=PITCH * rng.randint(1, 6),
                    lz=round(rng.uniform(4.0, 8.0), 2), steps=20)
    if kind == "deck":
        return dict(kind=kind, n=_log(rng, 4000, 300000), steps=20)
    lo = _log(rng, 2000, 20000)
    return dict(kind=kind, boxes=rng.randint(2, 24), lo=lo, hi=min(100000, lo * rng.randint(2, 10)),
                pick=rng.randrange(1 << 20), steps=20)


# --- inputs ---------------------------------------------------------------------------------------


def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + k)


def _lattice(n, lo, hi, gen):
    """n sites of the coarsest near-cubic lattice that has them, taken in random order, each moved
    by up to 0.3 of the spacing"""
    lo, hi = np.asarray(lo, float), np.asarray(hi, float)
    a = (np.prod(hi - lo) / n) ** (1.0 / 3.0)
    m = np.maximum(1, np.round((hi - lo) / a).astype(int))
    while int(np.prod(m)) < n:
        m[np.argmax((hi - lo) / m)] += 1
    site = torch.randperm(int(np.prod(m)), generator=gen, device="cuda")[:n]
    ijk = torch.stack([site % int(m[0]), site // int(m[0]) % int(m[1]), site // int(m[0] * m[1])], 1).double()
    jit = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * 0.6 - 0.3
    step = torch.tensor((hi - lo) / m, device="cuda")
    return torch.tensor(lo, device="cuda") + (ijk + 0.5 + jit) * step


def _maxwell(n, gen):
    v = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    return v - v.mean(0)


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=True)


def _boxes(case, seed):
    """the boxes of a case: dicts of lo, hi, x, v (device tensors) and mdpd.box_spec keywords"""
    kind = case["kind"]
    if kind in ("liquid", "thermo", "dpd"):
        n = case["n"]
        rho = RHO_DPD if kind == "dpd" else RHO
        g = _gen(seed)
        L = (n / rho) ** (1.0 / 3.0)
        kw = dict(style=1, A=A_DPD, sigma=SIGMA_DPD, rho_est=0.0) if kind == "dpd" else dict(
            A=case.get("A", -40.0), B=case.get("B", 25.0), cut_r=case.get("rd", 0.75), cut_rho=case.get("rd", 0.75),
            exact_rng=int(case.get("exact_rng", False)))
        return [dict(lo=(0.0,) * 3, hi=(L,) * 3, x=_lattice(n, (0,) * 3, (L,) * 3, g), v=_maxwell(n, g),
                     kw=dict(kw, seed=1000 + int(seed) % 100003))]
    if kind == "slab":
        half = np.array([case["lx"], case["ly"], case["lz"]]) / 2
        n = _slab_n(case)
        g = _gen(seed)
        inner = np.array([case["half"], half[1], half[2]])
        return [dict(lo=tuple(-half), hi=tuple(half), x=_lattice(n, -inner, inner, g), v=_maxwell(n, g),
                     kw=dict(seed=1000 + int(seed) % 100003))]
    out = []  # batch, turnover: sizes and coefficients belong to the case, particles to the seed
    for k, (n, A, B, rd) in enumerate(_sizes(case)):
        g = _gen(seed, k)
        L = (n / RHO) ** (1.0 / 3.0)
        out.append(dict(lo=(0.0,) * 3, hi=(L,) * 3, x=_lattice(n, (0,) * 3, (L,) * 3, g), v=_maxwell(n, g),
                        kw=dict(A=A, B=B, cut_r=rd, cut_rho=rd, seed=1000 + k + int(seed) % 100003)))
    return out


def _slab_n(case):
    return int(RHO * 2 * case["half"] * case["ly"] * case["lz"])


def _sizes(case):
    r = random.Random(case["pick"])
    return [(_log(r, case["lo"], case["hi"]), r.uniform(-50, -30), r.uniform(20, 30), r.uniform(0.7, 0.8))
            for _ in range(case["boxes"])]


def _spec(b, x, v):
    lo, hi = np.array(b["lo"]), np.array(b["hi"])
    return mdpd.box_spec(len(x), hi - lo, lo=lo, x=x, v=v, gamma=GAMMA, dt=DT, skin=SKIN, **b["kw"])


def _pore_particles(case, seed):
    """fluid around and wall particles inside the surfaces of cylinders along z, one per
    PITCH x PITCH tile, every second row shifted by half a tile"""
    L = np.array([case["lx"], case["ly"], case["lz"]])
    g = _gen(seed)

    def to_surface(p):
        row = torch.floor(p[:, 1] / PITCH)
        cx = p[:, 0] - 0.5 * PITCH * torch.remainder(row, 2)
        dx = torch.remainder(cx, PITCH) - 0.5 * PITCH
        dy = torch.remainder(p[:, 1], PITCH) - 0.5 * PITCH
        return torch.hypot(dx, dy) - RADIUS

    def sites(rho):
        m = np.maximum(1, np.round(L * rho ** (1.0 / 3.0)).astype(int))
        ax = [(torch.arange(int(k), device="cuda", dtype=torch.float64) + 0.5) * (l / k) for k, l in zip(m, L)]
        return torch.stack([c.reshape(-1) for c in torch.meshgrid(*ax, indexing="ij")], 1), torch.tensor(L / m).cuda()

    def moved(p, step, keep):
        p = p[keep]
        p = p[torch.randperm(len(p), generator=g, device="cuda")]
        return p + (torch.rand(p.shape, generator=g, device="cuda", dtype=torch.float64) * 0.6 - 0.3) * step

    pf, sf = sites(RHO)
    pw, sw = sites(RHO_WALL)
    df, dw = to_surface(pf), to_surface(pw)
    return moved(pf, sf, df >= 0.3), moved(pw, sw, (dw < 0) & (dw >= -LAYER))


def _deck(types, lo, hi, counts, seed, pair, fixes):
    lam = mdpd.Lammps()
    lam.commands("units lj\nboundary p p p\nneighbor %g bin\nneigh_modify every 1 delay 0 check yes\n"
                 "atom_style mdpd/atomic/meso 8" % SKIN)
    lam.command("region box block %r %r %r %r %r %r units box" % (lo[0], hi[0], lo[1], hi[1], lo[2], hi[2]))
    lam.command("create_box %d box" % types)
    for t, c in enumerate(counts):
        lam.command("create_atoms %d random %d %d box" % (t + 1, c, 11 + t))
    lam.commands("\n".join("mass %d 1" % (t + 1) for t in range(types)))
    lam.commands(pair % dict(seed=1000 + seed % 100003))
    lam.commands(fixes)
    lam.commands("timestep %g\nrun_style mvv/meso" % DT)
    return lam


def prepare(case, seed):
    """boxes on the device, set up and ready to step, and the pinned arrays that the state comes
    back to; for turnover the pinned arrays that jobs arrive in"""
    kind = case["kind"]
    s = dict(kind=kind, steps=case["steps"])
    if kind == "pore":
        pf, pw = _pore_particles(case, seed)
        nf, nw = len(pf), len(pw)
        s["lam"] = lam = _deck(
            2, (0.0, 0.0, 0.0), (case["lx"], case["ly"], case["lz"]), (nf, nw), seed,
            "group fluid type 1\ngroup solid type 2\npair_style mdpd/meso 1.0 1.0 %(seed)d fluid solid\n"
            "pair_coeff 1 1 -40 25 4.5 1.0 0.75\npair_coeff 1 2 -40 25 4.5 1.0 0.75\n"
            "pair_coeff 2 2 -40 25 4.5 1.0 0.75",
            "fix BC all aboundary/rho/meso cut_rho 0.75 phi_c 0.5 cut_phi 1.0 rho_wall 8.0 wall solid mobile fluid\n"
            "fix NVE fluid nve/meso\nfix F fluid addforce/meso 0.02 0.0 0.0")
        v = torch.cat([_maxwell(nf, _gen(seed, 1)), torch.zeros((nw, 3), dtype=torch.float64, device="cuda")])
        lam.set_state(torch.cat([pf, pw]).cpu().numpy(), v.cpu().numpy())
        lam.setup()
        return s
    if kind == "deck":
        n = case["n"]
        L = (n / RHO) ** (1.0 / 3.0)
        g = _gen(seed)
        s["lam"] = lam = _deck(
            2, (0.0,) * 3, (L,) * 3, (n - n // 3, n // 3), seed,
            "pair_style mdpd/meso 1.0 1.0 %(seed)d\npair_coeff 1 1 -40 25 4.5 1.0 0.75\n"
            "pair_coeff 1 2 -35 25 4.5 1.0 0.75\npair_coeff 2 2 -45 25 4.5 1.0 0.75",
            "fix RHO all aboundary/rho/meso cut_rho 0.75\nfix NVE all nve/meso\nthermo 10")
        lam.set_state(_lattice(n, (0,) * 3, (L,) * 3, g).cpu().numpy(), _maxwell(n, g).cpu().numpy())
        lam.setup()
        return s
    bx = _boxes(case, seed)
    n = [len(b["x"]) for b in bx]
    ends = np.cumsum([0] + n)
    xin, vin = _pinned(int(ends[-1])), _pinned(int(ends[-1]))
    for k, b in enumerate(bx):
        xin[ends[k]:ends[k + 1]].copy_(b["x"])
        vin[ends[k]:ends[k + 1]].copy_(b["v"])
    torch.cuda.synchronize()

    def views(t):
        a = t.numpy()
        return [a[ends[k]:ends[k + 1]] for k in range(len(n))]

    s["boxes"] = [{k: b[k] for k in ("lo", "hi", "kw")} for b in bx]
    s["xin"], s["vin"] = views(xin), views(vin)
    s["x"], s["v"] = _pinned(int(ends[-1])), _pinned(int(ends[-1]))
    s["xs"], s["vs"] = views(s["x"]), views(s["v"])
    if kind == "turnover":
        return s
    s["batch"] = mdpd.Batch([_spec(b, x, v) for b, x, v in zip(s["boxes"], s["xin"], s["vin"])])
    s["batch"].setup()
    return s


def run(s):
    kind = s["kind"]
    if kind == "pore":  # steps, then every particle's state and wall fraction, in the library's order
        s["lam"].step(s["steps"])
        return {k: s["lam"].field(k) for k in ("tag", "x", "v", "force", "phi")}
    if kind == "deck":  # LAMMPS' run command: setup, steps, thermo lines
        s["lam"].run(s["steps"])
        t = s["lam"].thermo()
        return {"thermo": [t.temp, t.press, t.pe], **{k: s["lam"].field(k) for k in ("tag", "x", "v", "force")}}
    if kind == "turnover":
        b = mdpd.Batch([_spec(b, x, v) for b, x, v in zip(s["boxes"], s["xin"], s["vin"])])
        b.setup()
        b.step(s["steps"])
        b.states(s["xs"], s["vs"])
        b.close()
        return {"x": s["x"], "v": s["v"]}
    b = s["batch"]
    if kind == "thermo":
        rows, _ = b.run_thermo(s["steps"])
        return {"thermo": np.array([[t.temp, t.press, t.pe, t.ke, *t.ptensor] for row in rows for t in row])}
    b.step(s["steps"])
    b.states(s["xs"], s["vs"])
    return {"x": s["x"], "v": s["v"]}


# --- what a pass cannot do without ----------------------------------------------------------------


def _particles(case):
    kind = case["kind"]
    if kind == "slab":
        return _slab_n(case)
    if kind == "pore":
        tile = PITCH * PITCH
        fluid = RHO * (tile - math.pi * (RADIUS + 0.3) ** 2)
        wall = RHO_WALL * math.pi * (RADIUS ** 2 - (RADIUS - LAYER) ** 2)
        return int((fluid + wall) / tile * case["lx"] * case["ly"] * case["lz"])
    if kind in ("batch", "turnover"):
        return sum(z[0] for z in _sizes(case))
    return case["n"]


def work(case):
    """bytes: each step reads and writes every particle's position, velocity (64 bits) and force
    (32 bits); the pass writes what it returns once. flops: each pair inside the cutoff once a
    step (about 60 for its force, 40 for its random number) and, in mDPD, each pair inside r_d
    once for the density (about 10)"""
    n, steps = _particles(case), case["steps"]
    dpd = case["kind"] == "dpd"
    pairs = (RHO_DPD if dpd else RHO) * 2.0 / 3.0 * math.pi * RC ** 3
    near = 0.0 if dpd else RHO * 2.0 / 3.0 * math.pi * case.get("rd", 0.75) ** 3
    return {"bytes": float(n) * (steps * 2 * (24 + 24 + 12) + 48), "flops": float(n) * steps * (100.0 * pairs + 10.0 * near)}


# --- the same pass in 64 bits -------------------------------------------------------------------------


M32 = 0xFFFFFFFF


def _tea(v0, v1, rounds):
    s = 0
    for _ in range(rounds):
        s = (s + 0x9E3779B9) & M32
        v0 = (v0 + ((((v1 << 4) + 0xA341316C) ^ (v1 + s) ^ ((v1 >> 5) + 0xC8013EA4)) & M32)) & M32
        v1 = (v1 + ((((v0 << 4) + 0xAD90777D) ^ (v0 + s) ^ ((v0 >> 5) + 0x7E95761E)) & M32)) & M32
    return v0, v1


def _signature(n, seed, step, dev):
    """the per-step word of tags 1..n: 32 TEA rounds of the tag's reversed bits and the step's seed"""
    a, b = _tea(torch.tensor([seed], device=dev), torch.tensor([step], device=dev), 64)
    tag = torch.arange(1, n + 1, device=dev)
    rev = torch.zeros_like(tag)
    for k in range(32):
        rev |= ((tag >> k) & 1) << (31 - k)
    a, b = _tea(rev, (a ^ b).expand(n), 32)
    return a ^ b


def _gaussian(si, sj):
    """the pair's random number: cosine polynomial of one word, radius from the other"""
    a, b = _tea(torch.maximum(si, sj), torch.minimum(si, sj), 4)
    x = 2.0 * ((a & 0x7FFFFFFF).double() * 2.0 ** -31) - 1.0
    x2 = x * x
    s = torch.full_like(x, 3.41817283473266926e-6)
    for c in (-1.60217135750921262e-4, 4.68162024021793872e-3, -7.96925872866600517e-2, 6.45964092644060746e-1,
              -1.57079632662144460):
        s = s * x2 + c
    f = torch.where((a >> 31) > 0, s * x, -s * x)
    return (torch.sqrt(-2.0 * torch.log(b.clamp(min=1).double() * 2.0 ** -32)) * f).clamp(-4.0, 4.0)


def _pairs(x, lo, L, cut):
    """every pair closer than cut, once, as index tensors (cells of at least cut, half stencil)"""
    m = torch.clamp((L / cut).long(), min=1)
    c = torch.minimum(((x - lo) / (L / m)).long(), m - 1)
    cell = c[:, 0] + m[0] * (c[:, 1] + m[1] * c[:, 2])
    order = torch.argsort(cell)
    ncell = int(m.prod())
    count = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    pi, pj = [], []
    for o in range(14):  # the centre cell and 13 of its 26 neighbours
        d = torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=x.device)
        q = torch.remainder(c + d, m)
        other = q[:, 0] + m[0] * (q[:, 1] + m[1] * q[:, 2])
        k = count[other]
        i = torch.repeat_interleave(torch.arange(len(x), device=x.device), k)
        at = torch.arange(len(i), device=x.device) - torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
        j = order[torch.repeat_interleave(start[other], k) + at]
        dr = x[i] - x[j]
        dr -= L * torch.round(dr / L)
        keep = (dr * dr).sum(1) < cut * cut
        if o == 13:
            keep &= i < j
        pi.append(i[keep])
        pj.append(j[keep])
    return torch.cat(pi), torch.cat(pj)


def _stepped(b, steps):
    """x, v of an mDPD box after `steps` steps of modified velocity Verlet from its setup, in 64 bits"""
    kw = dict(dict(A=-40.0, B=25.0, cut_r=0.75, cut_rho=0.75), **b["kw"])
    x, v = b["x"].clone(), b["v"].clone()
    lo, hi = torch.tensor(b["lo"], device=x.device).double(), torch.tensor(b["hi"], device=x.device).double()
    L, n, rd, h = hi - lo, len(x), kw["cut_r"], kw["cut_rho"]
    sigma, wd = math.sqrt(2.0 * GAMMA), 15.0 / (2.0 * math.pi * h ** 5)

    def wrap():
        nonlocal x, xh, i, j
        x = torch.where(x < lo, x + L, x)
        x = torch.where(x >= hi, torch.maximum(x - L, lo), x)
        xh = x.clone()
        i, j = _pairs(x, lo, L, RC + SKIN)

    def force(step):
        dr = x[i] - x[j]
        dr -= L * torch.round(dr / L)
        r = torch.sqrt((dr * dr).sum(1))
        w = wd * torch.clamp(h - r, min=0) ** 2
        rho = torch.zeros(n, device=x.device, dtype=torch.float64).index_add_(0, i, w).index_add_(0, j, w)
        k = r < RC
        a, c, dr, r = i[k], j[k], dr[k], r[k]
        e = dr / r[:, None]
        wc = 1.0 - r / RC
        sig = _signature(n, kw["seed"], step, x.device)
        f = (kw["A"] * wc + kw["B"] * (rho[a] + rho[c]) * torch.clamp(1.0 - r / rd, min=0)
             - GAMMA * wc * wc * (e * (v[a] - v[c])).sum(1) + sigma * wc * _gaussian(sig[a], sig[c]) / math.sqrt(DT))
        f = f[:, None] * e
        return torch.zeros_like(x).index_add_(0, a, f).index_add_(0, c, -f)

    xh = i = j = None
    wrap()
    f = force(0)
    for step in range(1, steps + 1):
        v = v + 0.5 * DT * f
        x = x + DT * v
        if float(((x - xh) ** 2).sum(1).max()) > 0.25 * SKIN * SKIN:
            wrap()
        f = force(step)
        v = v + 0.5 * DT * f
    return x, v


def exact(case, seed):
    """None for classic DPD (its random words are hashed from the rounded 32-bit velocities, so a
    64-bit run draws others), for decks (their arrays come in the library's own order), for thermo
    (its sums follow the whole trajectory) and where the pass is too long in plain torch"""
    if case["kind"] not in ("liquid", "slab", "batch", "turnover") or _particles(case) * case["steps"] > 8000000:
        return None
    got = [_stepped(b, case["steps"]) for b in _boxes(case, seed)]
    return {"x": torch.cat([g[0] for g in got]), "v": torch.cat([g[1] for g in got])}
