"""Performance cases of casim_b200: the calls its users make, at the sizes they make them.

Three kinds of work, each through the public entry points:

  sites  ReleaseSiteBatch, one scenario of a batch of release sites as RunSimulations runs
         it: start (reset, opening of the first RyR, Update), `steps` time steps, then the
         outputs: every RyR's state and mouth concentrations, and the whole fields and pools
         of one watched site, as a trajectory output records them.
  qs     QuasiStationarySites, one run of all scenarios of a quasi-stationary release site
         (Gillespie gating) and the release-event analysis of its traces.
  net    Surrogate, the network that predicts mouth Ca: a forward pass, a stretch of
         training steps, and surrogate-driven gating of a batch.

A case's inputs (geometry, RyR positions, seeds, jSR loads, network inputs and weights) are
made from the seed alone. exact() computes the same outputs with torch in 64 bits.
"""
import math
import os
import tempfile

import numpy as np
import torch

from casim_b200 import QuasiStationarySites, ReleaseSiteBatch, configs
from casim_b200 import surrogate as sg

# 64-bit runs of more node-steps or draws than this take over about 20 seconds
MOST_NODE_STEPS = 6e9
MOST_DRAWS = 40000


def listed():
    return [
        # one site in FP64: the reference's own use (NumBatch 1), a chain of short steps
        sites_case("one_site", "2d", n=1, ny=64, nx=64, ryr=20, precision="fp64", steps=200),
        # the 100-site batch of 2D clefts (64 x 64, 20 RyRs, pool cytosol)
        sites_case("sites_2d", "2d", n=100, ny=64, nx=64, ryr=20, precision="fp32", steps=1000),
        # 1024 2D clefts of 50 RyRs with a jSR load of their own each
        sites_case("sites_2d_jsr", "2d_jsr", n=1024, ny=64, nx=64, ryr=50, precision="fp32", steps=300),
        # 2D clefts gated by the 60-state RyR model (two ions), FP64
        sites_case("sites_60state", "2d_60state", n=100, ny=64, nx=64, ryr=20, precision="fp64", steps=200),
        # the large workload: uneven 3D dyads with a 25^3 reaction-diffusion cytosol
        sites_case("dyads", "3d", n=2048, ny=40, nx=120, ryr=100, precision="fp32", steps=50),
        # the same in FP64
        sites_case("dyads_fp64", "3d", n=384, ny=40, nx=120, ryr=100, precision="fp64", steps=50),
        # dyads with Mg and tetrameric MWC gating: the large sweep
        sites_case("dyads_mg", "3d_mg", n=512, ny=40, nx=120, ryr=150, precision="fp32", steps=50),
        # quasi-stationary sites: many scenarios of a 20-RyR site, fewer of a 48-RyR site
        {"name": "qs_20", "kind": "qs", "ryr": 20, "scenarios": 131072, "max_ms": 50.0},
        {"name": "qs_48", "kind": "qs", "ryr": 48, "scenarios": 4096, "max_ms": 20.0},
        # the surrogate: a batch of predictions, training steps on mini-batches, a gating run
        {"name": "net_forward", "kind": "forward", "rows": 16384, "ryr": 20},
        {"name": "net_train", "kind": "train", "rows": 4096, "ryr": 20, "steps": 4},
        {"name": "net_gating", "kind": "gating", "n": 2048, "ryr": 20, "steps": 400},
    ]


def sites_case(name, what, n, ny, nx, ryr, precision, steps):
    """`what` 2d*: n sites of ny x nx nodes with `ryr` RyRs each; 3d*: n square sites of ny to nx
    nodes a side with 10 to `ryr` RyRs. Without a name: a drawn case."""
    c = {"kind": "sites", "what": what, "n": n, "ny": ny, "nx": nx, "ryr": ryr, "precision": precision, "steps": steps}
    return {"name": name, **c} if name else c


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("2d", "2d_jsr", "2d_60state", "3d", "3d", "3d_pool", "3d_mg", "qs", "qs", "forward", "train", "gating"))
    if kind == "qs":
        ryr = rng.randint(4, 64)
        return {"kind": "qs", "ryr": ryr, "scenarios": log_int(64, 131072 if ryr <= 20 else 4096), "max_ms": rng.uniform(5.0, 20.0)}
    if kind == "forward":
        return {"kind": "forward", "rows": 128 * log_int(1, 256), "ryr": rng.randint(5, 40)}
    if kind == "train":
        return {"kind": "train", "rows": 128 * log_int(2, 64), "ryr": rng.randint(5, 40), "steps": rng.randint(2, 6)}
    if kind == "gating":
        return {"kind": "gating", "n": log_int(1, 2048), "ryr": rng.randint(5, 40), "steps": 20 * rng.randint(5, 25)}
    precision = rng.choice(("fp32", "fp32", "fp64"))
    if kind.startswith("2d"):
        n = log_int(1, 1024 if kind == "2d_jsr" else 200)
        return sites_case(None, kind, n, rng.randint(36, 96), rng.randint(36, 96), rng.randint(5, 50), precision,
                          rng.randint(50, 300))
    lo = rng.randint(40, 90)
    return sites_case(None, kind, log_int(4, 512), lo, rng.randint(lo + 1, 120), rng.randint(12, 100), precision, rng.randint(20, 50))


# ------------------------------------------------------------------ inputs


def site_inputs(c, seed):
    """(params, sites) of a sites or gating case."""
    what, n, ny, nx, ryr = c["what"], c["n"], c["ny"], c["nx"], c["ryr"]
    rng = np.random.default_rng(seed)
    if what.startswith("2d"):
        p = configs._clean(configs.base_params(dim=2, nx=nx, ny=ny))
        if what == "2d_60state":
            p = configs.with_single_site_mwc(p)
        xs, ys = [], []
        for _ in range(n):
            x, y = configs.lattice(ryr, (nx - 1) * 5.0, (ny - 1) * 5.0, rng)
            xs += x
            ys += y
        seeds = rng.integers(1, 4294944443, size=(n, 6))
        jsr = None
        if what == "2d_jsr":
            jsr = rng.uniform(500.0, 1500.0, size=(n, 1))
        return p, configs.sites_table([nx] * n, [ny] * n, [1] * n, [ryr] * n, xs, ys, seeds, jsr_init=jsr,
                                      first=rng.integers(0, ryr, size=n))
    # the sizes of the shipped configs; positions (within the lattice's jitter), seeds and first RyRs of this seed
    if what == "3d_mg":
        with tempfile.TemporaryDirectory() as d:  # the rate tables of the other half are not used
            p, s = configs.config5(n_sites=2 * n, side=(ny, nx), ryr=(10, ryr), table_dir=d)[0]
    else:
        p, s = configs.config2(n_sites=n, side=(ny, nx), ryr=(10, ryr), cytosol="Pool" if what == "3d_pool" else "RD3D")
    s["ch_x"] = s["ch_x"] + rng.uniform(-1.0, 1.0, size=s["ch_x"].size)
    s["ch_y"] = s["ch_y"] + rng.uniform(-1.0, 1.0, size=s["ch_y"].size)
    s["seeds"] = rng.integers(1, 4294944443, size=(n, 6)).astype(np.uint32)
    s["first_channel"] = rng.integers(0, s["n_ch"]).astype(np.int32)
    return p, s


def net_inputs(c, seed):
    """Network inputs laid out as the batch's features (open flag and position of each RyR,
    jSR Ca, buffer totals) and mouth-Ca targets, `steps` mini-batches of them."""
    g = torch.Generator().manual_seed(seed)
    ryr, rows, k = c["ryr"], c["rows"], c.get("steps", 1)
    x = torch.rand((k, rows, 3 * ryr + 3), generator=g) * 2 - 1
    x[:, :, 0:3 * ryr:3] = (torch.rand((k, rows, ryr), generator=g) < 0.3).float()
    x[:, :, 3 * ryr] = 0.1 + 1.4 * torch.rand((k, rows), generator=g)
    x[:, :, 3 * ryr + 1:] = 1.0
    t = torch.randn((k, rows, ryr), generator=g) * 0.5 + x[:, :, 0:3 * ryr:3]
    return x, t


def net_shapes(ryr):
    """(dout, din) of the network's layers as the library pads them, and the sizes in use."""
    n_in, width, depth = 3 * ryr + 3, sg.WIDTH, sg.DEPTH
    dims = [(n_in + 63) // 64 * 64] + [width] * depth + [(ryr + 127) // 128 * 128]
    used = [n_in] + [width] * depth + [ryr]
    return [(dims[i + 1], dims[i], used[i + 1], used[i]) for i in range(depth + 1)]


def net_params(ryr, seed):
    """He-uniform weights and small biases, padded rows and columns zero."""
    g = torch.Generator().manual_seed(seed + 1)
    flat = []
    for dout, din, nout, nin in net_shapes(ryr):
        w, b = torch.zeros((dout, din)), torch.zeros(dout)
        w[:nout, :nin] = (torch.rand((nout, nin), generator=g) * 2 - 1) * math.sqrt(6.0 / nin)
        b[:nout] = (torch.rand(nout, generator=g) * 2 - 1) * 0.1
        flat += [w.reshape(-1), b]
    return torch.cat(flat).numpy()


def max_events(c):
    """Stored events per scenario, enough for every scenario of these sites."""
    return 1024 if c["ryr"] <= 32 else 4096


LR = 1e-4  # a rate from the falling part of the training schedule


def prepare(c, seed):
    kind = c["kind"]
    if kind == "sites":
        p, s = site_inputs(c, seed)
        return {"c": c, "sites": s, "sim": ReleaseSiteBatch(p, s, precision=c["precision"])}
    if kind == "qs":
        p, coords = configs.quasi_stationary(c["ryr"], seed=seed, max_time=c["max_ms"])
        rng = np.random.default_rng(seed)
        with tempfile.TemporaryDirectory() as d:
            np.savetxt(os.path.join(d, "coords.txt"), coords, fmt="%.17g")
            q = QuasiStationarySites(p, c["scenarios"], base_dir=d, max_events=max_events(c),
                                     seeds=rng.integers(1, 4294944443, size=(c["scenarios"], 6)))
        return {"c": c, "q": q, "first": rng.integers(0, c["ryr"], size=c["scenarios"]).astype(np.int32)}
    net = sg.Surrogate(3 * c["ryr"] + 3, c["ryr"])
    net.set_params(net_params(c["ryr"], seed))
    if kind == "gating":
        p, s = site_inputs({**c, "what": "2d", "ny": 64, "nx": 64}, seed)
        sim = ReleaseSiteBatch(p, s, precision="fp32")
        return {"c": c, "sites": s, "sim": sim, "net": net, "gating": sg.SurrogateGating(net, sim, max_ch=c["ryr"])}
    x, t = net_inputs(c, seed)
    return {"c": c, "net": net, "x": x.cuda(), "t": t.cuda()}


# ------------------------------------------------------------------ one pass


def run(state):
    c = state["c"]
    if c["kind"] == "sites":
        sim = state["sim"]
        sim.start(state["sites"]["first_channel"])
        sim.step(c["steps"])
        out = np.float32 if c["precision"] == "fp32" else np.float64  # the precision the fields are held in
        w, ni, npair = c["n"] // 2, sim.info.n_ions, sim.info.n_pairs
        res = {"states": sim.all_states(), "mouth": [sim.all_mouth(k).astype(out) for k in range(ni + npair)],
               "field": [sim.field(w, k).astype(out) for k in range(ni + npair)], "jsr": sim.jsr(w).astype(out),
               "release": sim.release(w)}
        if sim.info.cyto_nodes:
            res["cytosol"] = [sim.cyto_field(w, k).astype(out) for k in range(sim.info.n_cyto_species)]
        else:
            res["cytosol"] = [sim.cyto(w).astype(out)]
        res["release"] = np.array([res["release"]]).astype(out)
        return res
    if c["kind"] == "qs":
        q = state["q"]
        q.run(state["first"])
        per, classes = q.analysis(nadir=3)
        return {"metrics": per, "classes": classes, "increments": q.increments(), **padded(q.max_events, *q.events(0))}
    if c["kind"] == "forward":
        return state["net"].forward(state["x"][0])
    if c["kind"] == "train":
        net = state["net"]
        loss = [net.train_step(state["x"][k], state["t"][k], LR) for k in range(c["steps"])]
        return {"loss": np.array(loss, np.float32), "params": net.get_params()}
    sim = state["sim"]
    sim.start(state["sites"]["first_channel"])
    state["gating"].step(c["steps"])
    return {"states": sim.all_states(), "mouth": sim.all_mouth(0).astype(np.float32)}


def padded(n, t, ch, st):
    """The trace of the watched scenario in arrays of n events, zeros after the last."""
    out = {"times": np.zeros(n), "channels": np.zeros(n, np.int32), "states": np.zeros(n, np.int32)}
    for a, v in zip(out.values(), (t, ch, st)):
        a[:len(v)] = v
    return out


def work(c):
    """Each input once and each output once (a batch's fields live on the device: written once
    by the scenario), and the arithmetic of the steps."""
    kind = c["kind"]
    if kind in ("sites", "gating"):
        w = 8 if c.get("precision") == "fp64" else 4
        if kind == "gating":
            net = 2 * sum(o * i for o, i, _, _ in net_shapes(c["ryr"]))
            return {"bytes": c["n"] * (c["ryr"] * 8 + 200), "flops": c["n"] * (c["steps"] / 20 * net + c["steps"] * c["ryr"] * 5)}
        three, rd3d = c["what"].startswith("3d"), c["what"] in ("3d", "3d_mg")
        ions = 2 if c["what"] in ("3d_mg", "2d_60state") else 1
        lo, hi = (c["ny"], c["nx"]) if three else (0, 0)
        cleft = 3 * (((lo + hi) / 2) ** 2 + (hi - lo) ** 2 / 12) if three else c["ny"] * c["nx"]
        # per node and step: a 5- or 7-point Laplacian of each diffusing species, two reactions, the update
        per = 15 * (ions + 1) + 20 if three else 11 * (ions + 1) + 20
        cyto = 15625 if rd3d else 0
        ryr = (10 + c["ryr"]) / 2 if three else c["ryr"]
        nodes = c["n"] * ((ions + 2) * cleft + (ions + 2) * cyto)
        return {"bytes": w * nodes + c["n"] * ryr * (4 + w * (ions + 2)),
                "flops": c["n"] * c["steps"] * (per * cleft + (per + 20) * cyto)}
    if kind == "qs":
        # events in the mean, each with the mouth Ca, the rate and the share of every RyR
        events = 1.2 * c["ryr"]
        return {"bytes": c["scenarios"] * (24 + 4 + 40 + 12 * events), "flops": c["scenarios"] * events * (c["ryr"] ** 2 / 4 + 30 * c["ryr"])}
    n_par = sum(o * i + o for o, i, _, _ in net_shapes(c["ryr"]))
    k = c.get("steps", 1)
    io = 4 * c["rows"] * (3 * c["ryr"] + 3 + c["ryr"]) * k
    if kind == "forward":
        return {"bytes": io + 2 * n_par, "flops": 2 * n_par * c["rows"]}
    return {"bytes": io + 24 * n_par * k, "flops": 6 * n_par * c["rows"] * k}


# ------------------------------------------------------------------ the same in 64 bits


def exact(c, seed):
    kind = c["kind"]
    if kind == "sites":
        p, s = site_inputs(c, seed)
        nodes = float(np.sum(s["nx"].astype(np.int64) * s["ny"] * s["nz"])) + (15625.0 * c["n"] if c["what"] in ("3d", "3d_mg") else 0)
        if nodes * c["steps"] > MOST_NODE_STEPS or (c["steps"] + 1) * c["ryr"] > MOST_DRAWS:
            return None
        return exact_sites(p, s, c["steps"], c["n"] // 2)
    if kind == "qs":
        return exact_qs(c, seed)
    if kind == "gating":
        return None  # the network runs in BF16: another trajectory in 64 bits
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, t = net_inputs(c, seed)
    x, t = x.to(dev).double(), t.to(dev).double()
    layers, flat, off = [], torch.from_numpy(net_params(c["ryr"], seed)).to(dev).double(), 0
    for dout, din, nout, nin in net_shapes(c["ryr"]):
        w = flat[off:off + dout * din].reshape(dout, din).clone()
        b = flat[off + dout * din:off + dout * din + dout].clone()
        off += dout * din + dout
        layers.append((w, b, nin))

    def forward(ws, xk):
        h = xk
        for l, (w, b) in enumerate(ws):
            h = h @ w[:, :layers[l][2]].T + b
            if l + 1 < len(ws):
                h = torch.nn.functional.gelu(h)
        return h[:, :c["ryr"]]

    ws = [(w, b) for w, b, _ in layers]
    if kind == "forward":
        return forward(ws, x[0])
    par = [v.requires_grad_() for wb in ws for v in wb]
    m, v2 = [torch.zeros_like(q) for q in par], [torch.zeros_like(q) for q in par]
    losses = []
    for k in range(c["steps"]):
        loss = ((forward(ws, x[k]) - t[k]) ** 2).mean()
        grads = torch.autograd.grad(loss, par)
        losses.append(float(loss))
        with torch.no_grad():
            for q, g, mk, vk in zip(par, grads, m, v2):
                mk.mul_(0.9).add_(0.1 * g)
                vk.mul_(0.999).add_(0.001 * g * g)
                q -= LR * (mk / (1 - 0.9 ** (k + 1))) / ((vk / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"loss": np.array(losses), "params": torch.cat([q.detach().reshape(-1) for q in par]).cpu().numpy()}


M1, M2 = 4294967087, 4294944443


class Stream:
    """MRG32k3a streams (L'Ecuyer 1999), one per row, with RngStream's 53-bit uniforms."""

    def __init__(self, seeds, dev):
        s = torch.from_numpy(np.asarray(seeds).astype(np.int64)).to(dev)
        self.a, self.b = [s[:, k].clone() for k in range(3)], [s[:, k].clone() for k in range(3, 6)]

    def _half(self):
        p = (1403580 * self.a[1] - 810728 * self.a[0]) % M1
        q = (527612 * self.b[2] - 1370589 * self.b[0]) % M2
        self.a, self.b = self.a[1:] + [p], self.b[1:] + [q]
        d = p.double() - q.double()
        return torch.where(p > q, d, d + M1) * (1.0 / (M1 + 1.0))

    def next(self):
        u = self._half()
        u = u + self._half() * 5.9604644775390625e-8
        return torch.where(u < 1.0, u, u - 1.0)


class Model:
    """The species, kinetics and pools of a Parameters dict of configs.base_params."""

    def __init__(self, p):
        d, cy = p["Dyad"], p["Cytosol"]
        self.rd3d, self.dim3 = cy["Type"] == "RD3D", d["Type"] == "3D"
        self.dx, self.dz, self.dt = d["dx"], d["dz"], p["dt, ns"] * 1e-6
        self.ions = sorted(d["Ions"])
        ni = self.ni = len(self.ions)
        self.cb = [d["Ions"][k]["Concentration"] for k in self.ions]
        self.ca, self.mg = self.ions.index("Calcium"), self.ions.index("Magnesium") if "Magnesium" in self.ions else None
        bufs = [(n, b["Total Concentration"], b["Ions"]["Calcium"]) for n, b in sorted(d["Buffers"].items())]
        self.D = [d["Ions"][k]["D"] for k in self.ions] + [k["D"] for _, _, k in bufs]
        self.pairs = [(ni + i, tot, k["kon"], k["koff"]) for i, (_, tot, k) in enumerate(bufs)]
        ca0 = self.cb[self.ca]
        bound = lambda tot, k: tot * k["kon"] * ca0 / (k["kon"] * ca0 + k["koff"])  # noqa: E731
        self.init = self.cb + [bound(tot, k) for _, tot, k in bufs]
        # cytosol: the dyad buffers (RD3D: the mobile ones), then its own
        mine = [(i, tot, k) for i, (_, tot, k) in enumerate(bufs) if not self.rd3d or k["D"] > 0]
        mine += [(None, b["Total Concentration"], b["Ions"]["Calcium"]) for _, b in sorted(cy["Buffers"].items())]
        self.c_init = self.cb + [bound(tot, k) for _, tot, k in mine]
        self.c_D = [d["Ions"][k]["D"] for k in self.ions] + [k["D"] for _, _, k in mine]
        self.c_pairs = [(ni + i, tot, k["kon"], k["koff"]) for i, (_, tot, k) in enumerate(mine)]
        self.c_of = {ni + j: ni + i for i, (j, _, _) in enumerate(mine) if j is not None}  # dyad pair -> cytosol pair
        self.c_of.update({j: j for j in range(ni)})
        self.leak = cy.get("Leak mult", 0.0)
        self.serca = cy["SERCA"]["Calcium"]
        self.mc, self.hc = cy.get("Nodes", 0), cy.get("dx", 1.0)
        ch = d["Channels"]["RyR"]
        self.law, self.par = ch["Model"], ch["Parameters"]
        self.g = [ch["Conductance"].get(k, 0.0) for k in self.ions]
        j = p["jSR"]
        self.CQ, self.V_jsr = j["Total CQ (uM)"], j["V jSR (nm3)"]
        self.jsr = [j["Ions"][k] for k in self.ions]
        self.nsr = [p["nSR"]["Ions"][k]["Concentration (uM)"] for k in self.ions]
        self.face = d["dz"] if self.dim3 else d["z"]  # both edges: dx * height / dx
        self.V_elem = (0.5 * d["dx"] * d["dx"] * d["dz"]) if self.dim3 else d["dx"] * d["dx"] * d["z"]
        self.grad = 3.0 / (4 * math.pi * d["Radius"] ** 3)

    def react(self, u, pairs):
        """Rates of change of [.., species, ..] stacked on dim 1 from binding, Calcium with every pair."""
        e = torch.zeros_like(u)
        for f, tot, kon, koff in pairs:
            r = koff * u[:, f] - kon * u[:, self.ca] * (tot - u[:, f])
            e[:, f] -= r
            e[:, self.ca] += r
        return e

    def pump(self, ca):
        b2, k2 = self.cb[self.ca] ** 2, self.serca["Kup"] ** 2
        return self.serca["Jmax"] * (ca * ca / (ca * ca + k2) - b2 / (b2 + k2))

    def rate(self, state, ca, mg):
        p = self.par
        if self.law == "SheepCannell":
            k = torch.where(state, p["kclose0"] * (ca * 1e-3) ** p["ncaclose"],
                            torch.clamp(p["kopen0"] * (ca * 1e-3) ** p["ncaopen"], max=p["kopenmax"]))
            return k * 1e-3
        inac = p["KMgI"] ** 2 / (p["KMgI"] ** 2 + mg * mg)
        a = (ca + p["KCa"] * p["fCa"] * (1 + mg / (p["fMg"] * p["KMg"]))) ** 4
        b = p["KO0"] * (p["fCa"] * (ca + p["KCa"] * (1 + mg / p["KMg"]))) ** 4
        po = inac * a / (a + b)
        return torch.where(state, torch.full_like(ca, p["kclose"]), p["kclose"] * po / (1 - po))


class SixtyStates:
    """The 60-state single-site MWC RyR model: every transition rate is a constant times 1, Ca,
    Mg or Mg^2. State = occupancy (i Ca, j Mg of four sites) + 15 * block (closed, closed and
    Mg-inhibited, open and Mg-inhibited, open)."""

    def __init__(self, p, ca0, mg0, dev):
        idx = {(i, j): 15 - (6 - j) * (5 - j) // 2 + i for i in range(5) for j in range(5 - i)}
        n_to, to, co, kind = [0] * 60, np.zeros((60, 6), np.int64), np.zeros((60, 6)), np.zeros((60, 6), np.int64)

        def add(s, d, c, k):  # k: 0 constant, 1 Ca, 2 Mg, 3 Mg^2
            to[s, n_to[s]], co[s, n_to[s]], kind[s, n_to[s]] = d, c, k
            n_to[s] += 1

        koff_ca, koff_mg = p["KCa"] * p["konCa"], p["KMg"] * p["konMg"]
        koc, koff_i = p["KO0"] * p["kco"], p["KMgI"] ** 2 * p["konmgI"]
        aC, aM, aI = p["alphaCa"], p["alphaMg"], p["alphaMgI"]
        for (i, j), s in idx.items():
            for b in range(4):
                x, free = s + 15 * b, 4 - i - j
                if free > 0:
                    f = {0: 1.0, 1: 1.0, 3: p["fCa"] ** aC, 2: (p["fCa4I"] if i == 3 else p["fICa"]) ** aC}[b]
                    add(x, idx[i + 1, j] + 15 * b, free * p["konCa"] / f, 1)
                if i > 0:
                    f = {0: 1.0, 1: p["gCa"], 3: p["fCa"] ** (1 - aC), 2: (p["fCa4I"] if i == 4 else p["fICa"]) ** (1 - aC) * p["gCa"]}[b]
                    add(x, idx[i - 1, j] + 15 * b, i * koff_ca * f, 0)
                if free > 0:
                    f = {0: 1.0, 1: p["gMg"] ** aI, 3: p["fMg"] ** aM, 2: p["fIMg"] ** aM * p["gMg"] ** aI}[b]
                    add(x, idx[i, j + 1] + 15 * b, free * p["konMg"] / f, 2)
                if j > 0:
                    f = {0: 1.0, 1: p["gMg"] ** (1 - aI), 3: p["fMg"] ** (1 - aM), 2: p["fIMg"] ** (1 - aM) * p["gMg"] ** (1 - aI)}[b]
                    add(x, idx[i, j - 1] + 15 * b, j * koff_mg * f, 0)
            ff = p["fCa"] ** i * p["fMg"] ** j
            fi = p["fICa"] ** 3 * p["fCa4I"] if i == 4 else p["fICa"] ** i * p["fIMg"] ** j
            r = p["fICa"] / p["fCa"] * p["gCa"]
            back = koff_i * r ** 3 * p["fCa4I"] / p["fCa"] if i == 4 else koff_i * r ** i
            add(s, s + 15, p["konmgI"] / p["gMg"] ** j, 3)
            add(s + 15, s, koff_i * p["gCa"] ** i, 0)
            add(s + 45, s + 30, p["konmgI"] / (p["fIMg"] / p["fMg"] * p["gMg"]) ** j, 3)
            add(s + 30, s + 45, back, 0)
            add(s, s + 45, p["kco"] / ff ** p["alphakco"], 0)
            add(s + 45, s, koc * ff ** (1 - p["alphakco"]), 0)
            add(s + 15, s + 30, p["kco"] / fi ** p["alphakcoI"], 0)
            add(s + 30, s + 15, koc * fi ** (1 - p["alphakcoI"]), 0)
        q = np.zeros((60, 60))
        for s in range(60):
            for k in range(n_to[s]):
                q[s, to[s, k]] = co[s, k] * (1.0, ca0, mg0, mg0 ** 2)[kind[s, k]]
            q[s, s] = -q[s].sum()
        p0 = np.linalg.solve(q @ q.T + 1.0, np.ones(60))
        self.start = [np.cumsum(p0[:45]) / p0[:45].sum(), np.cumsum(p0[45:]) / p0[45:].sum()]
        self.to, self.co, self.kind = (torch.from_numpy(v).to(dev) for v in (to, co, kind))

    def first(self, macro, u):
        cum = torch.from_numpy(self.start[macro]).to(u.device)
        return torch.searchsorted(cum, u.contiguous()).clamp(max=cum.numel() - 1) + 45 * macro

    def row(self, s, ca, mg):
        scale = torch.stack([torch.ones_like(ca), ca, mg, mg * mg], -1)
        return self.co[s] * scale.gather(-1, self.kind[s])


def exact_sites(p, sites, steps, watched):
    """One scenario of the batch in 64 bits: sites of one grid size together."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = Model(p)
    nch = torch.from_numpy(sites["n_ch"].astype(np.int64)).to(dev)
    off = np.concatenate([[0], np.cumsum(sites["n_ch"])])
    n_draws = (steps + 1) * int(sites["n_ch"].max()) + 64 + steps * int(sites["n_ch"].max()) // 16
    stream = Stream(sites["seeds"], dev)
    draws = torch.stack([stream.next() for _ in range(n_draws)], 1)
    states = np.zeros(off[-1], np.int32)
    mouth = np.zeros((len(m.init), off[-1]))
    seen = {}
    size = np.stack([sites["nx"], sites["ny"]], 1)
    for nx, ny in np.unique(size, axis=0):
        at = np.nonzero((size == (nx, ny)).all(1))[0]
        jsr0 = [[q["Concentration"] for q in m.jsr]] * len(at) if sites["jsr_init"] is None else sites["jsr_init"][at]
        xs = [sites["ch_x"][off[k]:off[k + 1]] for k in at]
        ys = [sites["ch_y"][off[k]:off[k + 1]] for k in at]
        got = exact_group(m, int(nx), int(ny), xs, ys, nch[at], draws[at], torch.tensor(np.asarray(jsr0), dtype=torch.float64, device=dev),
                          torch.from_numpy(sites["first_channel"][at].astype(np.int64)).to(dev), steps, dev)
        for r, k in enumerate(at):
            states[off[k]:off[k + 1]] = got["states"][r, :sites["n_ch"][k]]
            mouth[:, off[k]:off[k + 1]] = got["mouth"][r][:, :sites["n_ch"][k]]
            if k == watched:
                seen = {"field": [f[r] for f in got["field"]], "jsr": got["jsr"][r], "release": got["release"][r:r + 1],
                        "cytosol": [f[r] for f in got["cytosol"]] if m.rd3d else [got["cytosol"][r]]}
    return {"states": states, "mouth": list(mouth), **seen}


def exact_group(m, nx, ny, xs, ys, nch, draws, jsr0, first, steps, dev):
    S, F, ni, nz = len(xs), len(m.init), m.ni, 3 if m.dim3 else 1
    C = int(nch.max())
    f64 = {"dtype": torch.float64, "device": dev}
    chx, chy = torch.zeros((S, C), dtype=torch.int64), torch.zeros((S, C), dtype=torch.int64)
    for r in range(S):
        chx[r, :len(xs[r])] = torch.from_numpy(((np.asarray(xs[r]) + 0.5 * m.dx) / m.dx).astype(np.int64))
        chy[r, :len(ys[r])] = torch.from_numpy(((np.asarray(ys[r]) + 0.5 * m.dx) / m.dx).astype(np.int64))
    chx, chy = chx.to(dev), chy.to(dev)
    rows, chans = torch.arange(S, device=dev)[:, None], torch.arange(C, device=dev)[None, :]
    here = chans < nch[:, None]
    u = torch.tensor(m.init, **f64).reshape(1, F, 1, 1, 1).expand(S, F, nz, ny, nx).clone()
    cur = torch.zeros((S, ni, nz, ny, nx), **f64)
    D = torch.tensor(m.D, **f64)
    # rim nodes of a layer and the layer-0 cytosol node under each
    edge = torch.ones((ny, nx), dtype=torch.bool)
    edge[1:-1, 1:-1] = False
    ry, rx = (v.to(dev) for v in torch.nonzero(edge, as_tuple=True))
    n_cy = len(m.c_init)
    if m.rd3d:
        mc = m.mc
        cyt = torch.tensor(m.c_init, **f64).reshape(1, n_cy, 1, 1, 1).expand(S, n_cy, mc, mc, mc).clone()
        before = cyt

        def under(y, x):
            ci = torch.floor((x - 0.5 * (nx - 1)) * m.dx / m.hc + 0.5 * (mc - 1) + 0.5).long().clamp(1, mc - 2)
            cj = torch.floor((y - 0.5 * (ny - 1)) * m.dx / m.hc + 0.5 * (mc - 1) + 0.5).long().clamp(1, mc - 2)
            return cj * mc + ci

        c_D = torch.tensor(m.c_D, **f64).reshape(1, -1, 1, 1, 1)
        deposit = torch.zeros((S, n_cy, mc * mc), **f64)
    else:
        pool = torch.tensor(m.c_init, **f64).repeat(S, 1)
        c_tau = m.leak * torch.tensor(m.c_D, **f64)
    efflux = torch.zeros((S, F), **f64)
    jsr, jsr_new, IjSR = jsr0.clone(), jsr0.clone(), torch.zeros((S, ni), **f64)
    nsr = jsr0.clone()
    release = torch.zeros(S, **f64)
    jp = [(q["Binding sites of CQ"], q["K CQ (uM)"], q["T refill (ms)"]) for q in m.jsr]
    used = nch + 1  # the opening: a draw for every RyR, one more for the first one
    is_open = torch.zeros((S, C), dtype=torch.bool, device=dev)
    is_open[rows[:, 0], first] = True
    sixty = SixtyStates(m.par, m.cb[m.ca], m.cb[m.mg], dev) if m.law == "SingleSiteMWC" else None
    if sixty:
        micro = torch.where(here, sixty.first(0, draws[:, :C]), 0)
        micro[rows[:, 0], first] = sixty.first(1, draws.gather(1, nch[:, None]))[:, 0]

    def update():
        nonlocal cur, IjSR, nsr, jsr, efflux, deposit
        mouth = u[rows, :, 0, chy, chx].transpose(1, 2)  # [S, F, C]; no RyR lies on the rim
        for f in range(F):
            c = m.c_of.get(f)
            if m.rd3d:
                v = before[:, c, 0].reshape(S, -1)[:, under(ry, rx)] if c is not None else m.init[f]
            else:
                v = pool[:, c:c + 1]
            for z in range(nz):
                u[:, f, z, ry, rx] = v if torch.is_tensor(v) else torch.full((S, len(ry)), v, **f64)
        if m.rd3d:
            deposit = torch.zeros((S, n_cy, mc * mc), **f64)
        efflux = torch.zeros((S, F), **f64)
        yi, xi = torch.arange(1, ny - 1, device=dev), torch.arange(nx, device=dev)
        for z in range(1 if nz == 1 else nz - 1):
            w = u[:, :, z]
            for g, y, x in ((2 * w[:, :, 1:-1, 1] - 1.5 * w[:, :, 1:-1, 0] - 0.5 * w[:, :, 1:-1, 2], yi, 0 * yi),
                            (2 * w[:, :, 1:-1, -2] - 1.5 * w[:, :, 1:-1, -1] - 0.5 * w[:, :, 1:-1, -3], yi, 0 * yi + nx - 1),
                            (2 * w[:, :, 1] - 1.5 * w[:, :, 0] - 0.5 * w[:, :, 2], 0 * xi, xi),
                            (2 * w[:, :, -2] - 1.5 * w[:, :, -1] - 0.5 * w[:, :, -3], 0 * xi + ny - 1, xi)):
                term = g * (D * m.face)[None, :, None]
                if m.rd3d:
                    for f, c in m.c_of.items():
                        deposit[:, c].index_add_(1, under(y, x), term[:, f] / m.hc ** 3)
                else:
                    efflux = efflux + m.grad * term.sum(-1)
        at_ch = u[rows, :, 0, chy, chx].transpose(1, 2)
        total = torch.zeros((S, ni), **f64)
        cur = torch.zeros_like(cur)
        for j in range(ni):
            flux = torch.where(is_open & here, m.g[j] * (jsr_new[:, j:j + 1] - at_ch[:, j]), 0.0)
            total[:, j] = flux.sum(1)
            cur[:, j, 0].reshape(S, -1).scatter_add_(1, chy * nx + chx, flux)
        IjSR = total * m.V_elem
        nsr = torch.tensor(m.nsr, **f64).repeat(S, 1)
        jsr = jsr_new.clone()
        return mouth

    mouth = update()
    for _ in range(steps):
        if not m.rd3d:
            e = m.react(pool, m.c_pairs)
            for f, c in m.c_of.items():
                e[:, c] += efflux[:, f]
            e[:, m.ca] -= m.pump(pool[:, m.ca])
            pool = pool + m.dt * (e - c_tau * (pool - torch.tensor(m.c_init, **f64)))
        beta = 1 + sum(n * K * m.CQ / (K + jsr[:, j]) ** 2 for j, (n, K, _) in enumerate(jp))
        tau = torch.tensor([t for _, _, t in jp], **f64)
        jsr_new = jsr + m.dt / beta[:, None] * ((nsr - jsr) / tau - IjSR / m.V_jsr)
        release = release + IjSR[:, m.ca] * m.dt
        # gating in RyR order: a draw for each RyR, one more after each transition
        ca, mg = mouth[:, m.ca], mouth[:, m.mg] if m.mg is not None else torch.zeros_like(mouth[:, 0])
        if sixty:
            out = sixty.row(micro, ca, mg)
            prob = out.sum(-1) * m.dt
        else:
            prob = m.rate(is_open, ca, mg) * m.dt
        extra = torch.zeros((S, C), dtype=torch.int64, device=dev)
        start = torch.zeros((S, 1), dtype=torch.int64, device=dev)
        moved = torch.zeros(S, dtype=torch.int64, device=dev)
        while True:
            pos = used[:, None] + chans + extra
            hit = (draws.gather(1, pos) < prob) & here & (chans >= start)
            if not bool(hit.any()):
                break
            some = hit.any(1)
            f = hit.long().argmax(1)
            r = rows[:, 0][some]
            if sixty:
                u2 = draws[r, pos[r, f[some]] + 1]
                cum = torch.cumsum(out[r, f[some]], -1) / out[r, f[some]].sum(-1, keepdim=True)
                micro[r, f[some]] = sixty.to[micro[r, f[some]]].gather(1, (cum >= u2[:, None]).long().argmax(1, keepdim=True))[:, 0]
            else:
                is_open[r, f[some]] ^= True
            extra = extra + (some[:, None] & (chans > f[:, None])).long()
            start = torch.where(some[:, None], f[:, None] + 1, C)
            moved = moved + some.long()
        used = used + nch + moved
        if sixty:
            is_open = micro >= 45
        if m.rd3d:
            before = cyt
            lo = torch.cat([cyt[:, :, 1:2], cyt[:, :, :-2]], 2)[:, :, :, 1:-1, 1:-1]  # plane 0 mirrors
            mid, up = cyt[:, :, :-1, 1:-1, 1:-1], cyt[:, :, 1:, 1:-1, 1:-1]
            e = c_D / m.hc ** 2 * (lo + up + cyt[:, :, :-1, 1:-1, 2:] + cyt[:, :, :-1, 1:-1, :-2] + cyt[:, :, :-1, 2:, 1:-1] +
                                   cyt[:, :, :-1, :-2, 1:-1] - 6 * mid) + m.react(mid, m.c_pairs)
            e[:, m.ca] -= m.pump(mid[:, m.ca])
            e[:, :, 0] += deposit.reshape(S, n_cy, mc, mc)[:, :, 1:-1, 1:-1]
            cyt = cyt.clone()
            cyt[:, :, :-1, 1:-1, 1:-1] = mid + m.dt * e
        mid = u[:, :, :, 1:-1, 1:-1]
        lap = (u[..., 1:-1, 2:] + u[..., 1:-1, :-2] + u[..., 2:, 1:-1] + u[..., :-2, 1:-1] - 4 * mid) / m.dx ** 2
        if nz > 1:
            lap = lap + (torch.cat([mid[:, :, 1:2], mid[:, :, :-1]], 2) + torch.cat([mid[:, :, 1:], mid[:, :, -2:-1]], 2) - 2 * mid) / m.dz ** 2
        e = D.reshape(1, F, 1, 1, 1) * lap + m.react(mid, m.pairs)
        e[:, :ni] += cur[..., 1:-1, 1:-1]
        u = u.clone()
        u[:, :, :, 1:-1, 1:-1] = mid + m.dt * e
        mouth = update()
    host = lambda v: v.cpu().numpy()  # noqa: E731
    return {"states": host(is_open & here), "mouth": host(mouth), "jsr": host(jsr_new), "release": host(release),
            "field": [host(u[:, f].permute(0, 3, 2, 1).reshape(S, -1)) for f in range(F)],
            "cytosol": [host(cyt[:, f].reshape(S, -1)) for f in range(n_cy)] if m.rd3d else host(pool)}


def exact_qs(c, seed):
    """Gillespie's method on every scenario at once, in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = {"dtype": torch.float64, "device": dev}
    p, coords = configs.quasi_stationary(c["ryr"], seed=seed, max_time=c["max_ms"])
    par = p["Calcium Release Site"]["Parameters"]
    ch, cleft = par["Channels"]["RyR"], par["Dyadic Cleft"]
    bg, dca, mg = cleft["Ions"]["Calcium"]["Concentration"], cleft["Ions"]["Calcium"]["D"], cleft["Ions"]["Magnesium"]["Concentration"]
    # linearised buffered diffusion around a point source (Naraghi and Neher 1997)
    bufs = [b for _, b in sorted(cleft["Buffers"].items())]
    n = len(bufs)
    A, Dm = np.zeros((n + 1, n + 1)), np.diag([b["D"] for b in bufs] + [dca])
    for i, b in enumerate(bufs):
        K, rate = b["koff"] / b["kon"], b["koff"] + b["kon"] * bg
        kappa = b["Total Concentration"] * K / (K + bg) ** 2
        A[i, i], A[i, n], A[n, i] = -rate, kappa * rate, rate
        A[n, n] -= kappa * rate
    mu, E = (v.real for v in np.linalg.eig(-np.linalg.inv(Dm) @ A))
    src = np.zeros(n + 1)
    src[n] = ch["Current"] / (4 * np.pi * 96485.33e-6 * dca)
    amp = np.linalg.solve(E, src) * E[n] * 1e-4
    r = np.sqrt(((coords[:, None] - coords[None]) ** 2).sum(-1))
    far = np.where(r > 1e-6, r, 1.0)
    added = np.where(r > 1e-6, (amp * np.exp(-far[..., None] * np.sqrt(np.abs(mu)) * 1e-8)).sum(-1) / far, par["Open Concentration"])
    A = torch.tensor(added, **f64)
    rng = np.random.default_rng(seed)
    S, C = c["scenarios"], c["ryr"]
    stream = Stream(rng.integers(1, 4294944443, size=(S, 6)), dev)
    first = torch.from_numpy(rng.integers(0, C, size=S)).to(dev)
    for _ in range(C + 1):
        stream.next()
    law = Model.__new__(Model)
    law.law, law.par = "TwoStateMWC", ch["Parameters"]
    on = torch.zeros((S, C), dtype=torch.bool, device=dev)
    on[torch.arange(S, device=dev), first] = True
    ids = torch.arange(S, device=dev)
    t = torch.zeros(S, **f64)
    res = torch.zeros((S, 5), **f64)
    res[:, 0] = 1
    trace, live0 = ([], [], []), True
    while ids.numel():
        ca = on.double() @ A + bg
        rates = law.rate(on, ca, torch.full_like(ca, mg))
        total = rates.sum(1, keepdim=True)
        count = on.sum(1).double()
        wait = -torch.log(stream.next()) / total[:, 0]
        u = stream.next()
        cum = torch.cumsum(rates / total, 1)
        pick = (cum >= u[:, None]).long().argmax(1)
        stream.next()
        res[ids, 3] += count * wait
        t = t + wait
        k = torch.arange(ids.numel(), device=dev)
        on[k, pick] ^= True
        count = on.sum(1).double()
        more = count > res[ids, 0]
        res[ids, 0] = torch.where(more, count, res[ids, 0])
        res[ids, 1] = torch.where(more, t, res[ids, 1])
        res[ids, 2] = t
        if live0:
            trace[0].append(float(t[0]))
            trace[1].append(int(pick[0]))
            trace[2].append(int(on[0, pick[0]]))
        go = (count >= 1) & (t < c["max_ms"])
        live0 = live0 and bool(go[0])
        if not bool(go.all()):
            ids, on, t = ids[go], on[go], t[go]
            stream.a, stream.b = [v[go] for v in stream.a], [v[go] for v in stream.b]
    res[:, 4] = res[:, 3] / res[:, 2]
    a = res[:, 0]
    classes = np.array([int((a == 1).sum()), int(((a > 1) & (a <= 3)).sum()), int((a > 3).sum())], np.int32)
    return {"metrics": res, "classes": classes, "increments": added, **padded(max_events(c), *trace)}
