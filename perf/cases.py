"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one block of the energy-representation method, as ERmod's driver runs it:
``engclear``, one or more frames with their solute placements, and the accumulated
distributions read back.  The modes are the solution system (the solute sits in the frame,
one placement per frame) and the reference solvent (hundreds to thousands of test-particle
insertions per frame), each in the mixed and the plain FP64 arithmetic, through the host
API, the device API with placements generated on the device, or one CUDA graph over several
systems.  Sizes follow the repository's own workloads (``ermod_gb300/synth.py``): 300 to
60,000 waters, solutes of 6 to 40 sites, PME grids at about 1 A spacing.

``exact`` restates the method in plain FP64 torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DENSITY = 0.0334                      # waters per cubic Angstrom
SCALE = 18.22261721                   # charge unit: sqrt(kcal/mol A)
KT = 300.0 * 8.314510e-3 / 4.184      # kcal/mol
BETA = 0.34                           # Ewald screening, 1/A
# the default energy coordinate (1,396 bins); strongly bound waters take a lower first edge
# (gen_input's --minenergy)
HIST = dict(ecdmin=-20.0, ecfmns=-0.20, ecdcen=0.0, eccore=20.0, ecdmax=1.0e11, eclbin=5.0e-2, ecfbin=2.0e-3,
            ec0bin=2.0e-4, finfac=10.0, pecore=200)


def _case(name, **kw):
    c = dict(name=name, mode="refs", api="host", precision="mixed", nwater=4000, nsite=6, k1=48, k2=48, k3=48,
             order=4, frames=1, ins=1, batch=0, ljswitch=0, estype=2, cltype=2, wgtslf=1, corrcal=1, selfcal=0,
             ecdmin=-20.0, flexible=False, adjoint=False, uvengy=False, systems=1, aspect=1.0)
    c.update(kw)
    return c


def listed():
    return [
        # A droplet around its solute, without periodicity (bare Coulomb): the smallest call,
        # one frame of a few hundred molecules with every molecule's energy read back.
        _case("droplet", mode="droplet", nwater=300, estype=1, cltype=0, wgtslf=0, corrcal=0, uvengy=True,
              k1=32, k2=32, k3=32),
        # One frame of a solution run in a small box: what a trajectory repeats ten thousand
        # times, so that latency and launches count.
        _case("soln_1k", mode="soln", nwater=1000, k1=32, k2=32, k3=32, wgtslf=0, corrcal=0, uvengy=True),
        # The same frame in plain FP64, the arithmetic of the method's own program: what a user
        # runs who checks results, or wants no FP32 in them.
        _case("soln_1k_fp64", mode="soln", precision="fp64", nwater=1000, k1=32, k2=32, k3=32, wgtslf=0, corrcal=0,
              uvengy=True),
        # Force-field fitting: the bin-resolved derivatives for every charge, epsilon and sigma of
        # a 16-site solute, beside the distributions.
        _case("soln_8k_adjoint", mode="soln", nwater=8000, nsite=16, k1=64, k2=64, k3=64, wgtslf=0, corrcal=0,
              adjoint=True),
        # Several systems of uneven size replayed as one CUDA graph (a screening campaign), with
        # new coordinates and insertions written into the graph's buffers before each of the
        # block's five launches.
        _case("graph_4_systems", api="graph", systems=4, nwater=2000, nsite=8, k1=40, k2=40, k3=40, ins=400, batch=64,
              ecdmin=-60.0, frames=5),
        # A small reference-solvent run: two frames of 2,000 insertions with the pair correlations.
        _case("refs_4k", nwater=4000, ins=2000, frames=2),
        # The same in plain FP64.
        _case("refs_4k_fp64", precision="fp64", nwater=4000, ins=200),
        # The large reference-solvent run of the benchmark: 33,000 waters on a 96^3 grid, a 12-site
        # solute, in the benchmark's batches of 256.
        _case("refs_33k", nwater=33000, nsite=12, k1=96, k2=96, k3=96, ins=2048, batch=256),
        # The same in plain FP64, a sample of its insertions.
        _case("refs_33k_fp64", precision="fp64", nwater=33000, nsite=12, k1=96, k2=96, k3=96, ins=32),
        # The largest box and a big charged solute: 30 sites, 128^3, and the 4,996-bin coordinate
        # that strongly bound waters need.
        _case("refs_58k_wide", nwater=58000, nsite=30, k1=128, k2=128, k3=128, ins=400, ecdmin=-200.0, frames=2),
        # A drug-sized solute in a small box: 36 sites, where the solute's sites and the pair
        # correlations cost more than the grid.
        _case("refs_2k_wide", nwater=2000, nsite=36, k1=40, k2=40, k3=40, ins=1000, ecdmin=-200.0, frames=4),
        # A flexible solute with its structure weights in an orthorhombic box: order 6, a grid
        # without a compiled size, GROMACS force switching, NVT, the self-energy distribution, and placements
        # generated on the device (the whole step stays there).
        _case("flex_device_order6", api="device", nwater=7501, nsite=12, k1=54, k2=54, k3=80, order=6, ins=700,
              ljswitch=3, estype=1, selfcal=1, flexible=True, aspect=1.5),
    ]


_GRID = (32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 90, 96, 100, 108, 120, 128)


def draw(rng):
    mode = rng.choice(["soln", "soln", "refs", "refs", "refs", "refs", "droplet"])
    lo, hi = {"droplet": (150, 700), "soln": (600, 20000), "refs": (1500, 58000)}[mode]
    nw = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    ns = 6 if mode == "droplet" else rng.choice([6, rng.randint(7, 16), rng.randint(7, 40)])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    aspect = rng.choice([1.0, 1.0, 1.0, round(rng.uniform(1.1, 1.6), 2)])
    c = _case("", mode=mode, nwater=nw, nsite=ns, precision=precision, aspect=aspect if mode == "refs" else 1.0)
    del c["name"]
    box = _box(c)
    for a in range(3):  # about 1 A, at most 1.2 A
        want = box[a] / rng.uniform(0.95, 1.2)
        fits = [k for k in _GRID if k >= want]
        c["k%d" % (a + 1)] = fits[0] if fits else _GRID[-1]
    if c["aspect"] == 1.0:
        c["k2"] = c["k3"] = c["k1"]
    c["order"] = rng.choice([4, 4, 4, 6, 8])
    c["ljswitch"] = rng.choice([0, 0, 1, 2, 3])
    c["estype"] = rng.choice([1, 2])
    if ns not in ((6, 12) if mode == "refs" else (6, 16)):  # the other solutes may bind a water below -20 kcal/mol
        c["ecdmin"] = -60.0
    if mode == "droplet":
        c.update(estype=1, cltype=0, wgtslf=0, corrcal=0, uvengy=True, order=4)
    elif mode == "soln":
        c.update(wgtslf=rng.choice([0, 1]), corrcal=0, uvengy=rng.random() < 0.5, frames=rng.choice([1, 1, 3]),
                 adjoint=precision == "mixed" and rng.random() < 0.3)
    else:
        points = c["k1"] * c["k2"] * c["k3"] * (1.0 if c["order"] == 4 else 3.0)
        most = min(2.0e9 / points, 6.0e7 / nw, 2000.0) if precision == "mixed" else min(2.5e7 / points, 1.0e6 / nw, 200.0)
        c["ins"] = max(1, int(math.exp(rng.uniform(math.log(min(32.0, most)), math.log(most)))))
        c["wgtslf"] = rng.choice([1, 1, 0])
        c["flexible"] = rng.random() < 0.25
        c["selfcal"] = rng.choice([0, 0, 1])
        c["api"] = rng.choice(["host", "host", "device"])
        c["batch"] = rng.choice([0, 0, 64, 128, 256]) if precision == "mixed" else 0
    return c


# ---- inputs -------------------------------------------------------------------------------
def _solute(c):
    """The solute is a run's fixed molecule: the methanol-like one (6 sites), those of the
    33,000-water and the adjoint workloads (12, 16), and one for each other number of sites."""
    from ermod_gb300 import synth
    n = c["nsite"]
    return synth.methanol_like() if n == 6 else synth.random_solute(np.random.default_rng(({12: 3, 16: 5}.get(n, n), 11)), n)


def _cavity(c, sol):
    """Solution mode: no water centre closer to the box centre (the reference stops on a water
    beyond the coordinate's soft region)."""
    if c["mode"] == "refs":
        return 0.0
    return 4.5 if c["nsite"] == 6 else float(np.linalg.norm(sol["xyz"] - sol["xyz"].mean(0), axis=1).max()) + 3.3


def _box(c):
    vol = (c["nwater"] + (0 if c["mode"] == "refs" else 4.19 * 7.0 ** 3 * DENSITY)) / DENSITY
    if c["mode"] == "droplet":
        vol *= 2.2
    a = (vol / c["aspect"]) ** (1.0 / 3.0)
    return (a, a, a * c["aspect"])


class _Inputs:
    """Frames and placements of one system, from the seed."""

    def __init__(self, c, seed):
        from ermod_gb300 import insertion, synth
        rng = np.random.default_rng((int(seed), 17))
        self.sol = sol = _solute(c)
        self.box = np.array(_box(c))
        self.cell = np.diag(self.box) if c["mode"] != "droplet" else np.zeros((3, 3))
        n = c["nwater"]
        cav = _cavity(c, sol)
        m = 1
        while True:  # lattice of water centres, nearest the box centre first for a droplet
            dims = [max(1, int(math.ceil(m * b / self.box.min()))) for b in self.box]
            if dims[0] * dims[1] * dims[2] >= n:
                pts = np.stack(np.meshgrid(*[(np.arange(d) + 0.5) / d - 0.5 for d in dims], indexing="ij"), -1)
                pts = pts.reshape(-1, 3) * self.box
                r = np.linalg.norm(pts, axis=1)
                pts, r = pts[r > cav], r[r > cav]
                if c["mode"] == "droplet":
                    far = r < self.box.min() / 2
                    pts, r = pts[far], r[far]
                if len(pts) >= n:
                    break
            m += 1
        keep = np.argsort(r, kind="stable")[:n] if c["mode"] == "droplet" else np.sort(rng.choice(len(pts), n, replace=False))
        pts = pts[keep]
        body = synth.water_body()
        body = body - insertion.center_of_mass(body, synth.WATER_MASS)
        sxyz = sol["xyz"] - insertion.center_of_mass(sol["xyz"], sol["mass"])
        self.frames, self.placed, self.sws = [], [], []
        for _ in range(c["frames"]):
            q = insertion.random_quaternions(rng, n)
            wat = insertion.quat_rotate(q, np.broadcast_to(body, (n, 3, 3)))
            wat = wat + (pts + rng.uniform(-0.3, 0.3, (n, 3)))[:, None, :]
            pos = np.concatenate([wat.reshape(-1, 3), sxyz], axis=0)
            self.frames.append(np.ascontiguousarray(pos if c["mode"] == "droplet" else pos + self.box / 2))
        if c["flexible"]:  # the structure file of a flexible solute and its weights
            k = min(c["ins"], 64)
            self.conf = sol["xyz"] + rng.normal(0.0, 0.05, (k,) + sol["xyz"].shape)
            self.conf_w = rng.uniform(0.5, 1.5, k)
        if c["mode"] == "refs" and c["api"] != "device":
            for _ in range(c["frames"]):
                pl = insertion.random_placements(rng, sol["xyz"], sol["mass"], self.cell, c["ins"])
                if c["flexible"]:  # each placement's own structure
                    pl = pl + rng.normal(0.0, 0.05, pl.shape)
                self.placed.append(np.ascontiguousarray(pl))
                self.sws.append(rng.uniform(0.5, 1.5, c["ins"]) if c["flexible"] else None)
        self.key = int(rng.integers(1, 1 << 40))  # the device generator's seed


def _slttype(c):
    return 1 if c["mode"] != "refs" else (3 if c["flexible"] else 2)


def _engine(c, x):
    from ermod_gb300 import setconf, synth
    from ermod_gb300.engproc import EnergyRepresentation
    sol = x.sol
    params = dict(slttype=_slttype(c), estype=c["estype"], ljswitch=c["ljswitch"], splodr=c["order"], ms1max=c["k1"],
                  ms2max=c["k2"], ms3max=c["k3"], wgtslf=c["wgtslf"], corrcal=c["corrcal"], selfcal=c["selfcal"],
                  force_calculation=0, elecut=12.0, lwljcut=10.0, upljcut=12.0, screen=BETA, temp=KT,
                  block_threshold=4.0, cltype=c["cltype"], boxshp=0 if c["mode"] == "droplet" else 1)
    species = [dict(count=c["nwater"], sluvid=0, charge=synth.WATER_CHARGE, eps=synth.WATER_EPS, len=synth.WATER_SIG),
               dict(count=1, sluvid=_slttype(c), charge=sol["charge"], eps=sol["eps"], len=sol["sig"])]
    topo = setconf.setparam_topology(species, slttype=_slttype(c))
    bins = setconf.enginit_bins(topo["numslv"], dict(HIST, ecdmin=c["ecdmin"]))
    e = EnergyRepresentation(params, topo, bins, precision=c["precision"], batch=c["batch"])
    if c["adjoint"]:
        e.adjoint_enable()
    if c["flexible"] and c["api"] == "device":
        e.set_solute_library(x.conf, x.conf_w)
    return e, int(topo["nummol"])


def _systems(c):
    """The systems of a graph case: sizes, solutes and grids grow from one to the next."""
    out = []
    for i in range(c["systems"]):
        s = dict(c, nwater=int(c["nwater"] * 1.6 ** i), nsite=c["nsite"] + 5 * i, ins=c["ins"] + 60 * i)
        k = [k for k in _GRID if k >= _box(s)[0]][0]
        out.append(dict(s, k1=k, k2=k, k3=k))
    return out if c["systems"] > 1 else [c]


def prepare(case, seed):
    c = case
    if c["api"] == "graph":
        from ermod_gb300.multisystem import SystemGraph
        xs = [_Inputs(s, seed + 1000 * i) for i, s in enumerate(_systems(c))]
        es, mols = zip(*[_engine(s, x) for s, x in zip(_systems(c), xs)])
        for e, x, mol in zip(es, xs, mols):  # a graph needs one ordinary step of each system
            e.engconst(x.frames[0], x.cell, np.full(len(x.placed[0]), mol, np.int32), x.placed[0])
        g = SystemGraph(es, [(x.frames[0], x.cell) for x in xs], [x.placed[0] for x in xs], mols)
        return dict(case=c, engines=es, inputs=xs, graph=g)
    x = _Inputs(c, seed)
    e, mol = _engine(c, x)
    s = dict(case=c, engine=e, inputs=x, tags=np.full(c["ins"], mol, np.int32))
    if c["api"] == "device":
        s["pos"] = [torch.from_numpy(f).cuda() for f in x.frames]
        s["tag_d"] = torch.full((c["ins"],), mol, dtype=torch.int32, device="cuda")
    return s


def run(state):
    c = state["case"]
    if c["api"] == "graph":
        for e in state["engines"]:
            e.engclear()
        g = state["graph"]
        for t in range(c["frames"]):
            for i, x in enumerate(state["inputs"]):
                g.set_frame(i, x.frames[t])
                g.set_placements(i, x.placed[t])
            g.launch()
            g.sync()
        return [e.accum() for e in state["engines"]]
    e, x = state["engine"], state["inputs"]
    e.engclear()
    out = {}
    if c["api"] == "device":
        for i, pos in enumerate(state["pos"]):
            e.frame_device(pos.data_ptr(), x.cell)
            sol, sws = e.generate_placements(c["ins"], None if c["flexible"] else x.sol["xyz"], x.sol["mass"],
                                             seed=x.key, offset=i * c["ins"], weights=c["flexible"])
            e.placements_device(c["ins"], state["tag_d"].data_ptr(), sol.data_ptr(),
                                sws.data_ptr() if c["flexible"] else 0)
            e.sync()
        out["placed"] = sol
    else:
        for i, pos in enumerate(x.frames):
            r = e.engconst(pos, x.cell, state["tags"], x.placed[i] if c["mode"] == "refs" else None,
                           stat_weight_solute=x.sws[i] if c["flexible"] else None,
                           want_uvengy=c["uvengy"], want_flceng=c["uvengy"])
        if c["uvengy"]:
            out.update(r)
    out["accum"] = e.accum()
    if c["adjoint"]:
        out["adjoint"] = e.adjoint_get()
    return out


def _work_one(c):
    n = 3 * c["nwater"]
    e = 1396 + int(20.0 * (-20.0 - c["ecdmin"]))
    places = c["frames"] * c["ins"]
    grid = 0 if c["cltype"] == 0 else c["k1"] * c["k2"] * c["k3"]
    v = float(np.prod(_box(c)))
    near = 3 * min(c["nwater"], (4.19 * 14.0 ** 3 / v) * c["nwater"]) if c["mode"] != "droplet" else n
    byt = 24.0 * n * c["frames"] + 24.0 * c["nsite"] * places + 8.0 * e + (8.0 * e * e if c["corrcal"] else 0)
    if c["uvengy"]:
        byt += 8.0 * c["nwater"] * c["ins"]
    # per placement: the transform of its half spectrum, the solvent's gather, the pairs in reach
    one = 2.5 * grid * math.log2(max(grid, 2)) + (2.0 * n * c["order"] ** 3 if grid else 0) + 30.0 * near * c["nsite"]
    if c["adjoint"]:
        one *= 1 + c["nsite"]
        byt += 8.0 * e * 3 * c["nsite"]
    if c["corrcal"]:
        one += 2.0 * 150 ** 2 / 2  # the occupied pairs of bins
    return byt, one * places


def work(case):
    got = [_work_one(s) for s in _systems(case)]
    return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}


# ---- the method in plain FP64 torch ---------------------------------------------------------
def _edges(h):
    """enginit's coordinate (engproc.F90:163-218): edges, the soft count."""
    tmvl = h["finfac"] * h["ecfbin"]
    emin, fmns, mns0 = h["ecdmin"] - tmvl, h["ecfmns"] - tmvl, h["ecdcen"] - tmvl
    pls0, fpls = 2 * h["ecdcen"] - mns0, 2 * h["ecdcen"] - fmns
    reg = [emin, fmns, mns0, pls0, fpls, h["eccore"] + fpls - h["ecdcen"], h["ecdmax"]]
    step = [h["eclbin"], h["ecfbin"], h["ec0bin"], h["ecfbin"], h["eclbin"]]
    out = []
    for i in range(5):
        m = int(math.floor((reg[i + 1] - reg[i]) / step[i] + 0.5))
        per = (reg[i + 1] - reg[i]) / m
        out += [reg[i] + per * k for k in range(m)]
    soft = len(out)
    m = h["pecore"]
    per = math.log(reg[6] / reg[5]) / (m - 1)
    out += [reg[5] * math.exp(per * k) for k in range(m - 1)] + [reg[6]]
    return np.array(out), soft


def _spline(t, order):
    """B-spline weights M_order(t + j), j = 0 .. order - 1, on the last axis."""
    w = [t, 1.0 - t] + [torch.zeros_like(t)] * (order - 2)
    for n in range(3, order + 1):
        new = list(w)
        for j in range(n):
            a = w[j] if j <= n - 2 else 0.0
            b = w[j - 1] if j >= 1 else 0.0
            new[j] = ((t + j) * a + (n - t - j) * b) / (n - 1)
        w = new
    return torch.stack(w, -1)


def _lj(r2, eps, sg2, sw, lw=10.0, up=12.0):
    """(repulsive, attractive) parts: LJ = 4 eps (a - b); zero beyond up (realcal.F90:686-770)."""
    i6 = (sg2 / r2) ** 3
    s6 = sg2 ** 3
    if sw in (0, 1):
        if sw == 0:
            f = (2 * r2 + up ** 2 - 3 * lw ** 2) * (r2 - up ** 2) ** 2 / (up ** 2 - lw ** 2) ** 3
        else:
            t = (torch.sqrt(r2) - lw) / (up - lw)
            f = 1 - 10 * t ** 3 + 15 * t ** 4 - 6 * t ** 5
        f = torch.where(r2 <= lw ** 2, torch.ones_like(r2), f)
        a, b = i6 * i6 * f, i6 * f
    elif sw == 2:
        lw3, up3 = lw ** 3, up ** 3
        near = r2 <= lw ** 2
        fa = up3 ** 2 / (up3 ** 2 - lw3 ** 2) * (i6 - s6 / up3 ** 2) ** 2
        fb = up3 / (up3 - lw3) * (torch.sqrt(i6) - torch.sqrt(s6) / up3) ** 2
        a = torch.where(near, i6 * i6 - s6 * s6 / (lw3 ** 2 * up3 ** 2), fa)
        b = torch.where(near, i6 - s6 / (lw3 * up3), fb)
    else:
        def gmx(p):
            d = up - lw
            ga = -p * ((p + 4) * up - (p + 1) * lw) / (up ** (p + 2) * d ** 2) / 3
            gb = p * ((p + 3) * up - (p + 1) * lw) / (up ** (p + 2) * d ** 3) / 4
            return ga, gb, 1 / up ** p - ga * d ** 3 - gb * d ** 4
        t = torch.clamp(torch.sqrt(r2) - lw, min=0.0)
        parts = [g[0] * t ** 3 + g[1] * t ** 4 + g[2] for g in (gmx(12), gmx(6))]
        a, b = i6 * i6 - s6 * s6 * parts[0], i6 - s6 * parts[1]
    on = (r2 <= up ** 2) & (eps > 0)
    z = torch.zeros_like(r2)
    return torch.where(on, a, z), torch.where(on, b, z)


class _Exact:
    """One frame of one system."""

    def __init__(self, c, x, pos):
        f = dict(dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")
        self.c, self.f, n = c, f, c["nwater"]
        t = lambda a: torch.as_tensor(np.asarray(a, float), **f)  # noqa: E731
        self.per = c["mode"] != "droplet"
        self.pme = c["cltype"] != 0
        self.L, self.pos = t(x.box), t(pos[:3 * n])
        self.q = t(SCALE * np.tile([-0.834, 0.417, 0.417], n))
        self.eps_v, self.sig_v = t(np.tile([0.1521, 0.0, 0.0], n)), t(np.tile([3.1507, 0.0, 0.0], n))
        self.qu, self.eps_u, self.sig_u = t(SCALE * x.sol["charge"]), t(x.sol["eps"]), t(x.sol["sig"])
        self.V = float(np.prod(x.box)) if self.per else (2.0 ** math.ceil(math.log2(max(128.0, 8 * max(16.0, np.abs(pos).max()))))) ** 3
        if not self.pme:
            return
        self.K, P = [c["k1"], c["k2"], c["k3"]], c["order"]
        idx, wts = self.stencil(self.pos)
        self.idx, self.wts = idx, wts
        ms = [torch.fft.fftfreq(k, 1.0 / k, **f) for k in self.K]
        m2 = sum(torch.square(ms[a] / self.L[a]).reshape([-1 if b == a else 1 for b in range(3)]) for a in range(3))
        m2[0, 0, 0] = 1.0
        g = torch.exp(-math.pi ** 2 * m2 / BETA ** 2) / m2 / math.pi / self.V
        node = _spline(torch.zeros(1, **f), P)[0]  # M_P(0 .. P - 1)
        for a in range(3):
            ph = 2j * math.pi * torch.arange(self.K[a], **f)[:, None] * torch.arange(P - 1, **f) / self.K[a]
            b2 = (torch.exp(ph) * node[1:P]).sum(-1).abs() ** 2
            g = g / b2.reshape([-1 if b == a else 1 for b in range(3)])
        g[0, 0, 0] = 0.0
        self.green = g[..., :self.K[2] // 2 + 1]

    def stencil(self, x):
        """Flat grid points and weights, (..., order^3), of coordinates (..., 3)."""
        P, K = self.c["order"], self.K
        u = x / self.L
        u = u - torch.floor(u)
        idx = wts = None
        for a in range(3):
            f = u[..., a] * K[a]
            g = torch.floor(f)
            w = _spline(f - g, P)
            i = (g.long()[..., None] - torch.arange(P, device=x.device)) % K[a]
            idx = i if idx is None else (idx[..., :, None] * K[a] + i[..., None, :]).flatten(-2)
            wts = w if wts is None else (wts[..., :, None] * w[..., None, :]).flatten(-2)
        return idx, wts

    def potential(self, xu, qu):
        """(n, grid) potentials and the reciprocal self energies of charges qu at xu (n, ns, 3)."""
        n, K = xu.shape[0], self.K
        idx, wts = self.stencil(xu)
        grid = torch.zeros((n, K[0] * K[1] * K[2]), **self.f)
        grid.scatter_add_(1, idx.reshape(n, -1), (wts * qu[..., None]).reshape(n, -1))
        sp = torch.fft.rfftn(grid.reshape(n, *K), dim=(1, 2, 3)) * self.green
        phi = torch.fft.irfftn(sp, s=K, dim=(1, 2, 3), norm="forward").reshape(n, -1)
        return phi, 0.5 * (grid * phi).sum(1)

    def at_sites(self, phi):
        out = torch.zeros((phi.shape[0], self.idx.shape[0]), **self.f)
        for j in range(self.idx.shape[1]):
            out += self.wts[:, j] * phi[:, self.idx[:, j]]
        return out * self.q

    def pairs(self, xu, s):
        """r^2 (n, sites) from solute site s of each placement, minimum image."""
        d = self.pos[None] - xu[:, s, None]
        if self.per:
            d = d - self.L * torch.round(d / self.L)
        return (d * d).sum(-1)

    def site_terms(self, r2, s):
        eps = torch.sqrt(self.eps_u[s] * self.eps_v)
        sg2 = (0.5 * (self.sig_u[s] + self.sig_v)) ** 2
        a, b = _lj(r2, eps, sg2, self.c["ljswitch"])
        r = torch.sqrt(r2)
        if self.pme:
            el = torch.where(r2 <= 144.0, self.q * (1.0 - torch.erf(BETA * r)) / r, torch.zeros_like(r))
        else:
            el = self.q / r
        return eps, sg2, a, b, el

    def energies(self, xu):
        """(u (n, nwater), u0 (n)) of placements xu (n, ns, 3)."""
        n, ns, nw = xu.shape[0], xu.shape[1], self.c["nwater"]
        u = torch.zeros((n, 3 * nw), **self.f)
        u0 = torch.zeros(n, **self.f)
        Q = float(self.qu.sum())
        if self.pme:
            phi, self_rec = self.potential(xu, self.qu.expand(n, ns))
            u += self.at_sites(phi)
            d = xu[:, :, None] - xu[:, None]
            d = d - self.L * torch.round(d / self.L)
            r = torch.sqrt((d * d).sum(-1)) + torch.eye(ns, **self.f)
            e = self.qu[:, None] * self.qu * torch.erf(BETA * r) / r
            u0 = self_rec - torch.triu(e, 1).sum((1, 2)) - float((self.qu ** 2).sum()) * BETA / math.sqrt(math.pi)
            u0 = u0 - math.pi * Q * Q / BETA ** 2 / self.V / 2
        for s in range(ns):
            eps, _, a, b, el = self.site_terms(self.pairs(xu, s), s)
            u += 4 * eps * (a - b) + self.qu[s] * el
        u = u.reshape(n, nw, 3).sum(-1)
        if self.pme:
            u = u - math.pi * Q * float(self.q[:3].sum()) / BETA ** 2 / self.V
        return u, u0

    def gradients(self, xu):
        """(3 ns, nwater): derivatives for each site's charge, epsilon and sigma; one placement."""
        nw, out = self.c["nwater"], []
        one = torch.ones(1, 1, **self.f)
        for s in range(xu.shape[1]):
            eps, sg2, a, b, el = (v[0] if v.dim() == 2 else v for v in self.site_terms(self.pairs(xu, s), s))
            phi, _ = self.potential(xu[:, s:s + 1], one)
            out.append(el + self.at_sites(phi)[0])
            out.append(4 * eps * (a - b) / (2 * self.eps_u[s]) if self.eps_u[s] > 0 else torch.zeros_like(el))
            out.append(4 * eps * (6 * a - 3 * b) / sg2 * torch.sqrt(sg2))
        g = torch.stack(out).reshape(len(out), nw, 3).sum(-1)
        g[0::3] -= math.pi * float(self.q[:3].sum()) / BETA ** 2 / self.V
        return g


def _philox(ctr, key):
    m = 0xFFFFFFFF
    c0, c1, c2, c3 = ctr
    k0, k1 = key
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c0, 0xCD9E8D57 * c2
        c0, c1, c2, c3 = ((p1 >> 32) ^ c1 ^ k0) & m, p1 & m, ((p0 >> 32) ^ c3 ^ k1) & m, p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c0, c1, c2, c3


def _generated(c, x, frame):
    """The device generator's placements (uniform position and rotation, Philox4x32-10)."""
    out, w = [], []
    mass = x.sol["mass"]
    for p in range(c["ins"]):
        g = frame * c["ins"] + p
        xyz = x.conf[g % len(x.conf)] if c["flexible"] else x.sol["xyz"]
        w.append(x.conf_w[g % len(x.conf_w)] if c["flexible"] else 1.0)

        def uniforms():
            d = 0
            while True:
                b = _philox((d, 0, g, 0), (x.key & 0xFFFFFFFF, x.key >> 32))
                d += 1
                for i in (0, 2):
                    yield ((b[i] >> 5) * 67108864.0 + (b[i + 1] >> 6)) / 9007199254740992.0
        u = uniforms()
        com = x.cell @ np.array([next(u) for _ in range(3)])
        while True:
            q = np.array([2.0 * next(u) - 1.0 for _ in range(4)])
            if q @ q < 1.0:
                break
        q = q / math.sqrt(q @ q)
        v = xyz - (mass[:, None] * xyz).sum(0) / mass.sum()
        t = 2.0 * np.cross(q[1:], v)
        out.append(v + q[0] * t + np.cross(q[1:], t) + com)
    return np.array(out), np.array(w)


def _exact_one(c, x):
    edges, soft = _edges(dict(HIST, ecdmin=c["ecdmin"]))
    E, nw, soln = len(edges), c["nwater"], c["mode"] != "refs"
    first = None
    edens = ecorr = eself = None
    norm = smpl = avslf = slnuv = 0.0
    umin, umax, smin, smax = [], [], [], []
    out = {}
    for i, pos in enumerate(x.frames):
        X = _Exact(c, x, pos)
        f = X.f
        if edens is None:
            edens, eself = torch.zeros(E, **f), torch.zeros(soft, **f)
            ecorr = torch.zeros((E, E), **f) if c["corrcal"] else None
            grad, gw = torch.zeros((3 * c["nsite"], E), **f), torch.zeros(E, **f)
            ed = torch.as_tensor(edges, **f)
        if soln:
            xu, sw = pos[None, 3 * nw:], np.ones(1)
        elif c["api"] == "device":
            xu, sw = _generated(c, x, i)
            out["placed"] = xu
        else:
            xu, sw = x.placed[i], x.sws[i] if c["flexible"] else np.ones(c["ins"])
        xu, sw = torch.as_tensor(xu, **f), torch.as_tensor(np.asarray(sw), **f)
        step = max(1, int(2.0e7 / max(3 * nw, X.V if X.pme else 1)))
        for p0 in range(0, len(xu), step):
            xs = xu[p0:p0 + step]
            u, u0 = X.energies(xs)
            if first is None:
                first = float(u0[0])
            ws = torch.exp((u0 - first) / KT * (1 if soln else -1)) if c["wgtslf"] else torch.ones_like(u0)
            tw = sw[p0:p0 + step] * (X.V if c["estype"] == 2 else 1.0)
            ws = ws * tw
            b = torch.searchsorted(ed, u.contiguous(), right=False) - 1
            n = len(xs)
            h = torch.bincount((b + E * torch.arange(n, device=b.device)[:, None]).reshape(-1), minlength=n * E)
            h = h.reshape(n, E).double()
            edens += ws @ h
            if ecorr is not None:
                ecorr += (h * ws[:, None]).T @ h
            if c["selfcal"]:
                sb = torch.searchsorted(ed[:soft].contiguous(), u0, right=False) - 1
                eself.scatter_add_(0, sb, ws)
            norm, smpl, avslf = norm + float(ws.sum()), smpl + n, avslf + float(tw.sum())
            if soln:
                slnuv += float((u.sum(1) * ws).sum())
            for to, v in ((umin, u.min()), (smin, u0.min()), (umax, u.max()), (smax, u0.max())):
                to.append(float(v))
            if c["adjoint"]:
                gr = X.gradients(xs)
                for k in range(len(gr)):
                    grad[k].scatter_add_(0, b[0], gr[k] * ws[0])
                gw += ws[0] * h[0]
            if c["uvengy"]:  # the solute itself is the last physical molecule, without an energy
                out["uvengy"] = torch.cat([u0[:, None], u, torch.zeros((n, 1), **f)], 1).cpu().numpy()
                out["flceng"] = u.sum(1, keepdim=True).cpu().numpy()
    cpu = lambda t: None if t is None else t.cpu().numpy()  # noqa: E731
    out["accum"] = dict(edens=cpu(edens), ecorr=cpu(ecorr), ecorr_count=None, eself=cpu(eself), slnuv=np.array([slnuv]),
                        minuv=np.array([min(smin), min(umin)]), maxuv=np.array([max(smax), max(umax)]), engnorm=norm,
                        engsmpl=smpl, avslf=avslf, voffset=first if c["wgtslf"] else -1.0e50,
                        voffset_initialized=bool(c["wgtslf"]))
    if c["adjoint"]:
        out["adjoint"] = (cpu(grad), cpu(gw))
    return out


def exact(case, seed):
    got = [_exact_one(s, _Inputs(s, seed + 1000 * i)) for i, s in enumerate(_systems(case))]
    return [g["accum"] for g in got] if case["api"] == "graph" else got[0]
