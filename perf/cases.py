"""Performance cases: the work a user of this framework has it do, through its
public entry points, over the sizes, precisions and options it is used with.

Kinds of case
- "step":    a resident simulation takes a state from the host, advances it
             `steps` leapfrog steps and hands the next state back (what runs
             between two output frames).  REF physics (the drop-in profile,
             FP64) or WCSPH (FP64 or FP32 pair arithmetic), plain or as a
             CUDA graph, tanks, dam breaks, wave flumes with a moving piston
             and a sponge, batches of shaken tanks, the 40-nearest cap.
- "rates":   one rate evaluation on a caller's state, as a host solver that
             keeps its own time loop calls it (derivatives()).
- "search":  the neighbour search on its own (SearchNeighbors()).
- "predict": the learned surrogate's network on one graph.
- "train":   the loss and gradient of that network on one graph.

A case's flow is stirred: a smooth divergence-free velocity field, particles
moved off the lattice and a density ripple, all drawn from the seed, so that
neighbour counts and their changes are those of moving water and not of a
lattice at rest.
"""
import math
import os

import numpy as np
import torch

from uph_b200 import batch as B
from uph_b200 import deck as D
from uph_b200 import surrogate as SG
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH, empty_state
from uph_b200.sim import STEP_INPUT_FIELDS, STEP_OUTPUT_FIELDS, Simulation, search_neighbors

RATE_INPUT_FIELDS = ["Position", "Velocity", "localVelocity", "density", "localDensity", "DynamicPressure",
                     "localPressure", "mass", "itype", "spongeFactor"]
RATE_OUTPUT_FIELDS = ["ddensitydt", "dpdt", "dvdt", "ddensitydt_approx", "dpdt_approx", "dvdt_approx",
                      "densityFluctuation", "pressureFluctuation", "velocityFluctuation"]
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(SG.__file__)), "weights", "flume_mpnn.npz")


# ---- the cases ------------------------------------------------------------------
def _step(name, flow, n, physics, steps, precision="fp64", speed=0.02, graph=False, cap=0, near=0, tanks=0, draw=0):
    return {"name": name, "kind": "step", "flow": flow, "n": n, "physics": physics, "precision": precision,
            "steps": steps, "speed": speed, "graph": graph, "cap": cap, "near": near, "tanks": tanks, "draw": draw}


def listed():
    return [
        # the smallest tank anybody runs, 5,000 particles, in the drop-in's physics: launches and latency
        _step("dambreak_5k_ref", "dam", 5000, "ref", 100),
        # the same tank in the textbook physics, a whole frame as one CUDA graph
        _step("dambreak_5k_wcsph_graph", "dam", 5000, "wcsph", 200, graph=True),
        # a wave flume of an odd, middling size: moving piston, sponge layer
        _step("flume_61k_ref", "flume", 61003, "ref", 100),
        # the headline tank: 500,000 particles of nearly still water, drop-in physics
        _step("tank_500k_ref", "tank", 500000, "ref", 100, speed=0.002),
        # water in violent motion, FP64 textbook physics: the cell list is rebuilt every few steps
        _step("dambreak_300k_wcsph", "dam", 300000, "wcsph", 100, speed=0.1),
        # the large dam break with FP32 pair arithmetic
        _step("dambreak_2m_fp32", "dam", 2000000, "wcsph", 40, precision="fp32", speed=0.05),
        # a batch of uneven dam-break and sloshing tanks, FP32, one graph replay of 100 steps
        _step("batch_48_tanks_fp32", "batch", 0, "wcsph", 100, precision="fp32", graph=True, tanks=48, draw=1),
        # the reference's own decks: a wide kernel (nearNeighbor 91) under the 40-nearest cap
        _step("dambreak_40k_capped", "dam", 40000, "ref", 20, cap=40, near=91),
        # a host solver that keeps its own time loop asks for the rates of its state
        {"name": "rates_200k", "kind": "rates", "flow": "dam", "n": 200000, "cap": 0, "near": 0, "speed": 0.05},
        # the pair list of a cloud of points in no order, 20 of them within the radius, by the 40-nearest search
        {"name": "search_100k", "kind": "search", "n": 100000, "radius": 2.53, "neighbors": 40},
        # the surrogate's network on the 10 m flume's graph
        {"name": "network_200k", "kind": "predict", "n": 200000},
        # one training step's gradient on a frame of the training flumes
        {"name": "gradient_80k", "kind": "train", "n": 80000},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "rates", "search", "predict", "train"])
    if kind == "step":
        flow = rng.choice(["tank", "dam", "dam", "flume", "batch"])
        physics = rng.choice(["ref", "wcsph"])
        precision = rng.choice(["fp64", "fp32"]) if physics == "wcsph" else "fp64"
        speed = round(math.exp(rng.uniform(math.log(0.002), math.log(0.1))), 5)
        graph = rng.random() < 0.4
        if flow == "batch":
            tanks = rng.randint(4, 64)
            c = _step("", flow, 0, "wcsph", rng.randint(40, 100), rng.choice(["fp64", "fp32"]), 0.02, graph, 0, 0, tanks,
                      rng.randint(0, 999))
        elif physics == "ref" and flow == "dam" and rng.random() < 0.3:
            c = _step("", flow, _size(rng, 3000, 100000), "ref", rng.randint(10, 30), "fp64", speed, graph, 40,
                      rng.choice([37, 61, 91]))
        else:
            n = _size(rng, 3000, 1000000)
            steps = max(20, min(rng.randint(50, 200), int(5e7 / n)))
            c = _step("", flow, n, physics, steps, precision, speed, graph)
        del c["name"]
        return c
    if kind == "rates":
        cap = rng.choice([0, 0, 40])
        return {"kind": kind, "flow": rng.choice(["tank", "dam"]), "n": _size(rng, 3000, 100000 if cap else 500000),
                "cap": cap, "near": 91 if cap else 0, "speed": round(rng.uniform(0.002, 0.1), 5)}
    if kind == "search":
        return {"kind": kind, "n": _size(rng, 3000, 300000), "radius": rng.choice([1.7, 2.53, 3.38]),
                "neighbors": 40}
    return {"kind": kind, "n": _size(rng, 5000, 200000 if kind == "predict" else 100000)}


# ---- inputs ---------------------------------------------------------------------
def _deck(case):
    """The case's deck and, where walls shake, their table (x0, half stroke, omega)."""
    n, flow = case.get("n"), case["flow"]
    eta = math.sqrt(case["near"] / (4.0 * math.pi)) if case.get("near") else 1.3
    if flow == "tank":
        d = D.hydrostatic_tank(width=2.0, depth=1.0, dx=math.sqrt(2.0 / n), layers=3, eta=eta)
    elif flow == "dam":
        d = D.dam_break(tank=(4.0, 3.0), column=(1.0, 2.0), dx=math.sqrt(2.0 / n), layers=2, eta=eta, hydrostatic=True)
    elif flow == "flume":
        d = D.wave_flume(10.0, 0.5, math.sqrt(5.0 / n), piston_layers=3, hydrostatic_walls=True)
    else:
        b = B.build_batch(B.draw_tanks(seed=case["draw"], count=case["tanks"]))
        b.deck.wall_table = (b.wall_x0, b.wall_hs, b.wall_om)
        return b.deck
    return d


def _stir(deck, state, seed, speed):
    """Moves the fluid of `state` in place: velocities up to about `speed` times the speed of sound, positions off the
    lattice by up to a tenth of the spacing, a density ripple with the pressure that belongs to it."""
    rng = np.random.default_rng(seed)
    nf, p = deck.n_fluid, D.derive_params(deck.params, deck.eta_override)
    pos = state["Position"][:nf]
    lo, hi = pos.min(axis=0), pos.max(axis=0)
    s = math.pi * (pos - lo) / (hi - lo)
    vel = np.zeros((nf, 2))
    for _ in range(3):
        kx, ky = rng.integers(1, 4, 2)
        a = rng.uniform(-1.0, 1.0) / 2.0
        # stream function sin(kx x) sin(ky y): no flow through the block's faces
        vel[:, 0] += a * np.sin(kx * s[:, 0]) * np.cos(ky * s[:, 1])
        vel[:, 1] -= a * (kx * (hi[1] - lo[1])) / (ky * (hi[0] - lo[0])) * np.cos(kx * s[:, 0]) * np.sin(ky * s[:, 1])
    vel *= speed * p["speed_of_sound"] / max(1e-12, float(np.abs(vel).max()))
    state["Velocity"][:nf] = vel
    state["localVelocity"][:nf] = vel
    pos += rng.uniform(-0.1, 0.1, (nf, 2)) * p["dx"]
    ripple = 1e-4 * rng.standard_normal(nf) * p["density0"]
    state["density"][:nf] += ripple
    state["localDensity"][:nf] = state["density"][:nf]
    state["DynamicPressure"][:nf] += p["speed_of_sound"] ** 2 * ripple
    state["localPressure"][:nf] = state["DynamicPressure"][:nf]
    return state


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.int32 if a.dtype == np.int32 else torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _codes(case):
    return (PROFILE_REF if case["physics"] == "ref" else PROFILE_WCSPH,
            PREC_FP32_PAIR if case["precision"] == "fp32" else PREC_FP64)


def _cloud(case, seed):
    """Points of a square cloud, spacing 1, in an order that has nothing to do with place: (positions, fluid count,
    boundary index, radius^2).  The radius lies between two rings of the lattice and the points stay near their lattice
    places, so the number of pairs, and with it the outputs' shape, is the same for every seed."""
    rng = np.random.default_rng(seed)
    side = max(2, int(round(math.sqrt(case["n"]))))
    x, y = D.lattice(0.0, 0.0, side, side, 1.0)
    pos = np.stack([x, y], axis=1) + rng.uniform(-0.07, 0.07, (side * side, 2))
    pos = np.ascontiguousarray(pos[np.random.default_rng(case["n"]).permutation(side * side)])
    return pos, int(0.95 * side * side), side * side, case["radius"] ** 2


def _flume_frame(case, seed):
    """Training flumes (0.5 m deep, 4 m long, dx = 0.005; one shorter flume where the graph is small) in motion."""
    per = 4.0 * 0.5 / 0.005 ** 2
    count = max(1, int(round(case["n"] / per)))
    length = max(0.25, 4.0 * case["n"] / (per * count))
    rng = np.random.default_rng(seed)
    b = SG.flume_batch([(float(rng.uniform(0.02, 0.06)), float(rng.uniform(1.0, 1.6))) for _ in range(count)],
                       length=length)
    return b, _stir(b.deck, b.state, seed, 0.01)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        deck = _deck(case)
        st = _stir(deck, deck.initial_state(), seed, case["speed"])
        sim = Simulation(deck.uph_params(*_codes(case), knn_cap=case["cap"]))
        if deck.wall_table is not None:
            sim.set_wall_motion(*deck.wall_table)
        if case["graph"]:
            sim.set_graph(case["steps"])
        out = {k: _pinned(a) for k, a in empty_state(deck.n_fluid, deck.n_all).items() if k in STEP_OUTPUT_FIELDS}
        return {"case": case, "sim": sim, "in": {k: _pinned(st[k]) for k in STEP_INPUT_FIELDS}, "out": out}
    if kind == "rates":
        deck = _deck(case)
        st = _stir(deck, deck.initial_state(), seed, case["speed"])
        sim = Simulation(deck.uph_params(PROFILE_REF, PREC_FP64, knn_cap=case["cap"]))
        out = {k: _pinned(a) for k, a in empty_state(deck.n_fluid, deck.n_all).items() if k in RATE_OUTPUT_FIELDS}
        return {"case": case, "sim": sim, "in": {k: _pinned(st[k]) for k in RATE_INPUT_FIELDS}, "out": out}
    if kind == "search":
        return {"case": case, "cloud": _cloud(case, seed)}
    b, st = _flume_frame(case, seed)
    cfg, params = SG.Surrogate.load_file(WEIGHTS)
    nodes = SG.Nodes.from_state(st, b.deck.n_fluid, b.box)
    s = {"case": case, "net": SG.Surrogate(cfg, b.deck.n_all, params), "nodes": nodes}
    if kind == "train":
        s["target"] = _target(b.deck.n_fluid, seed)
    return s


def _target(nf, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((nf, SG.NOUT), generator=g, device="cuda", dtype=torch.float32)


# ---- one pass -------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        # a graph continues a run (it never holds a run's first step)
        s["sim"].upload(s["in"], 1 if case["graph"] else 0)
        s["sim"].step(case["steps"])
        return s["sim"].download(s["out"])
    if kind == "rates":
        s["sim"].upload(s["in"], 1)
        s["sim"].derivatives(0.0)
        return s["sim"].download(s["out"])
    if kind == "search":
        pos, nf, pb, dist = s["cloud"]
        i, j, r2 = search_neighbors(pos, nf, pb, dist, case["neighbors"])
        return {"i": i, "j": j, "r2": r2}
    if kind == "predict":
        return s["net"].forward(s["nodes"])
    loss, grad = s["net"].gradients(s["nodes"], s["target"])
    return {"loss": loss, "grad": grad}


# ---- the work a pass cannot do without --------------------------------------------
def work(case):
    """Bytes: the host arrays of the call each moved once, and per step the state a particle's step reads and writes
    (REF 23 FP64 values in and 20 out, WCSPH 8 and 8).  Operations: those of the pair terms (REF about 100 a pair side,
    WCSPH about 35) over the pairs of a full neighbourhood; for the network its multiply-adds, twice."""
    kind = case["kind"]
    if kind in ("step", "rates"):
        n = case["n"] or case["tanks"] * 11000
        h = math.sqrt(case["near"] / (4.0 * math.pi)) if case["near"] else 1.3
        sides = min(math.pi * (2.0 * h) ** 2 - 1.0, 2.0 * case["cap"] if case["cap"] else 1e9)
        if kind == "rates":
            return {"bytes": n * (13 * 8 + 4 + 12 * 8), "flops": n * sides * 100.0}
        ref = case["physics"] == "ref"
        per_step = 43 * 8 if ref else 16 * 8
        return {"bytes": n * (17 * 8 + 14 * 8 + case["steps"] * per_step),
                "flops": case["steps"] * n * sides * (100.0 if ref else 35.0)}
    if kind == "search":
        pairs = case["n"] * 0.475 * (math.pi * case["radius"] ** 2 - 1.0)
        return {"bytes": case["n"] * 16.0 + pairs * 16.0, "flops": pairs * 10.0}
    macs = 128 * 128 * 2 + 256 * 128 + 3 * (128 * 128 * 2 + 128 * 256 + 256 * 128)
    edges = case["n"] * 20.0
    flops = 2.0 * macs * case["n"] + 3 * edges * 128 * 7
    if kind == "predict":
        return {"bytes": case["n"] * (44 + 20), "flops": flops}
    return {"bytes": case["n"] * (44 + 20) + 4.0 * 3e5, "flops": 3.0 * flops}


# ---- the same in 64 bits, plain torch ----------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _neighbours(x, y, nq, r2cut):
    """Directed pairs (a, b) of points, a < nq, b != a, eps < r^2 < r2cut, by cells of one radius."""
    dev = x.device
    cell = math.sqrt(r2cut) * (1.0 + 1e-12)
    cx = torch.floor((x - x.min()) / cell).long() + 1
    cy = torch.floor((y - y.min()) / cell).long() + 1
    ncx = int(cx.max()) + 2
    key = cy * ncx + cx
    order = torch.argsort(key, stable=True)
    ncell = ncx * (int(cy.max()) + 2)
    start = torch.zeros(ncell + 2, dtype=torch.long, device=dev)
    start[1:ncell + 1] = torch.cumsum(torch.bincount(key, minlength=ncell), 0)
    start[ncell + 1] = start[ncell]
    got_a, got_b = [], []
    for oy in (-1, 0, 1):
        k = key[:nq] + oy * ncx
        lo, n = start[k - 1], start[k + 2] - start[k - 1]
        a = torch.repeat_interleave(torch.arange(nq, device=dev), n)
        at = torch.arange(a.numel(), device=dev) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
        b = order[lo[a] + at]
        dx, dy = x[a] - x[b], y[a] - y[b]
        r2 = dx * dx + dy * dy
        keep = (r2 < r2cut) & (r2 > np.finfo(np.float64).eps) & (a != b)
        got_a.append(a[keep])
        got_b.append(b[keep])
    return torch.cat(got_a), torch.cat(got_b)


def _cap(a, b, r2, nq, cap):
    """Of the directed pairs, those whose smaller index keeps the other among its `cap` nearest (r^2, index)."""
    o = torch.argsort(b, stable=True)
    o = o[torch.argsort(r2[o], stable=True)]
    o = o[torch.argsort(a[o], stable=True)]
    n = torch.bincount(a, minlength=nq)
    first = torch.cumsum(n, 0) - n
    rank = torch.empty_like(a)
    rank[o] = torch.arange(a.numel(), device=a.device) - first[a[o]]
    kept = rank < cap
    # the pair belongs to the query of its smaller index: look its entry up from the other side
    big = 1 << 32
    code = torch.sort(a[kept] * big + b[kept]).values
    want = torch.minimum(a, b) * big + torch.maximum(a, b)
    at = torch.searchsorted(code, want).clamp(max=max(0, code.numel() - 1))
    return code[at] == want


class _Exact:
    """The leapfrog of the two physics on plain FP64 tensors."""

    def __init__(self, deck, st, physics, cap):
        self.p = p = D.derive_params(deck.params, deck.eta_override)
        self.nf, self.n, self.ref, self.cap = deck.n_fluid, deck.n_all, physics == "ref", cap
        self.dev = _device()
        t = lambda k: torch.as_tensor(np.ascontiguousarray(st[k]), device=self.dev).clone()
        pos, vel, lv = t("Position"), t("Velocity"), t("localVelocity")
        self.x, self.y, self.u, self.v = pos[:, 0].clone(), pos[:, 1].clone(), vel[:, 0].clone(), vel[:, 1].clone()
        self.ut, self.vt = lv[:, 0].clone(), lv[:, 1].clone()
        self.rho, self.pr, self.m, self.itype = t("density"), t("DynamicPressure"), t("mass"), t("itype")
        self.rhot, self.pt = t("localDensity"), t("localPressure")
        self.rhot[self.nf:] = p["density0"]
        self.pt[self.nf:] = 0.0
        self.sponge = t("spongeFactor")
        self.rate = [torch.zeros(self.nf, dtype=torch.float64, device=self.dev) for _ in range(12)]
        self.table = deck.wall_table
        self.m0 = self.n - deck.moving.shape[0]
        if not self.ref:
            self.pr = self._tait(self.rho)

    def _tait(self, rho):
        return self.p["compression_factor"] * ((rho / self.p["density0"]) ** self.p["adiabatic_constant"] - 1.0)

    def _sum(self, a, v):
        return torch.zeros(self.nf, dtype=torch.float64, device=self.dev).index_add_(0, a, v)

    def _pairs(self):
        r2cut = self.p["h"] ** 2 * 4
        a, b = _neighbours(self.x, self.y, self.nf, r2cut)
        if self.cap:
            # the query of a pair is its smaller index, which is a fluid particle
            dx, dy = self.x[a] - self.x[b], self.y[a] - self.y[b]
            keep = _cap(a, b, dx * dx + dy * dy, self.nf, self.cap)
            a, b = a[keep], b[keep]
        keep = torch.maximum(a, b) < self.n - 1
        return a[keep], b[keep]

    def _spring(self, a, b, dx, dy, r, du, dv):
        """The spring and damper of fluid-wall pairs (selectBoundaryForce 3)."""
        p = self.p
        it = self.itype[b]
        w = (a < b) & ((it == 2) | (it == 3) | (it == 5)) & (r < 3.0 * p["dx"])
        a, dx, dy, r, du, dv = a[w], dx[w], dy[w], r[w], du[w], dv[w]
        ma = self.m[a]
        c = p["spring_constant0"] * (3.0 * p["dx"] - r) / (r * ma) + \
            p["damping_constant0"] * (dx * du + dy * dv) / (r * r * ma)
        return self._sum(a, -c * dx), self._sum(a, -c * dy)

    def rates(self):
        p, nf = self.p, self.nf
        h = p["h"]
        a, b = self._pairs()
        dx, dy = self.x[a] - self.x[b], self.y[a] - self.y[b]
        r2 = dx * dx + dy * dy
        r, q2 = torch.sqrt(r2), r2 / (h * h)
        du, dv = self.u[a] - self.u[b], self.v[a] - self.v[b]
        sx, sy = self._spring(a, b, dx, dy, r, du, dv)
        g = p["gravity"] if p["gravity_flag"] == 1 else 0.0
        damp = self.sponge * self.u[:nf] if p["moving_boundary"] == 1 else torch.zeros_like(sx)
        ma, mb = self.m[a], self.m[b]
        ra, rb, pa, pb = self.rho[a], self.rho[b], self.pr[a], self.pr[b]
        zero = torch.zeros_like(sx)
        if not self.ref:
            q = r / h
            sig = 10.0 / (7.0 * math.pi * h * h)
            F = torch.where(q < 1.0, sig * (-3.0 + 2.25 * q) / (h * h), -sig * 0.75 * (2.0 - q) ** 2 / (h * r))
            vr = du * dx + dv * dy
            pi = torch.where(vr < 0.0, -p["alpha"] * p["speed_of_sound"] * h * vr / (r2 + 0.01 * h * h) /
                             (0.5 * (ra + rb)), torch.zeros_like(vr))
            c = mb * (pa / ra ** 2 + pb / rb ** 2 + pi) * F
            drho = self._sum(a, mb * vr * F)
            ax = self._sum(a, -c * dx) + sx - damp
            ay = self._sum(a, -c * dy) + sy - g
            self.rate = [drho, zero, ax, ay, drho, zero, ax, ay, zero, zero, zero, zero]
            return
        t = 1.0 - 0.25 * q2
        W = 2145.0 / (1347584.0 * math.pi * h * h) * t ** 8 * _horner(
            q2, (305.0, -628.0, 1184.0, -1984.0, 2816.0, -3072.0, 2048.0))
        F = -2145.0 / (192512.0 * math.pi * h ** 4) * t ** 7 * _horner(
            q2, (305.0, -1106.0, 1912.0, -2912.0, 3712.0, -3584.0, 2048.0))
        is_i = a < b
        uta, vta, utb, vtb = self.ut[a], self.vt[a], self.ut[b], self.vt[b]
        rta, rtb, ptb = self.rhot[a], self.rhot[b], self.pt[b]
        gam, kap = p["adiabatic_constant"], p["thermal_diffusivity0"]
        Pa = p["density0"] * p["speed_of_sound"] ** 2 + gam * pa
        Pb = p["density0"] * p["speed_of_sound"] ** 2 + gam * pb
        ms = torch.where(is_i, mb, ma)
        Vb = mb / rb
        nu = F * r2 / (r2 + 0.01 * h * h)
        eu, ev = self.u[a] - utb, self.v[a] - vtb
        drho_a = ms * F * (torch.where(is_i, eu, uta - self.u[b]) * dx + torch.where(is_i, ev, vta - self.v[b]) * dy)
        mix = 4.0 * Pa / (Pa + Pb)
        inv = 1.0 / ra + 1.0 / rb
        dp_a = mb / ra * Pa * F * (du * dx + dv * dy) + gam * kap * ms / rb * (pa - pb) * nu * mix \
            - kap * Pa * ms / rb * (ra - rb) * inv * nu
        c1 = mb * (pa / ra ** 2 + pb / rb ** 2) * F
        drho = Vb * rtb * F * (eu * dx + ev * dy)
        dp = Vb * rtb / ra * Pa * F * (eu * dx + ev * dy) + gam * kap * Vb * (pa - ptb) * nu * mix \
            - kap * Pa * Vb * (ra - rtb) * inv * nu
        c2 = mb * (pa * rtb / (ra ** 2 * rb) + pb * rta / (rb ** 2 * ra)) * F
        mu = 2.0 * p["viscosity0"] * ra * rb / (ra + rb)
        vis = mb * mu / (r2 + 0.01 * h * h) * F * r2
        va = vis * (1.0 / ra ** 2 + 1.0 / rb ** 2)
        vc = torch.where(is_i, vis, -vis) * (rtb / (ra ** 2 * rb) - rta / (rb ** 2 * ra))
        cf = torch.where(is_i, (ma / rtb - mb / rta) * W, torch.zeros_like(W))
        self.rate = [self._sum(a, drho), self._sum(a, dp),
                     self._sum(a, -c2 * dx - vc * du) + sx - damp, self._sum(a, -c2 * dy - vc * dv) + sy - g,
                     self._sum(a, drho_a), self._sum(a, dp_a),
                     self._sum(a, -c1 * dx - va * du) + sx, self._sum(a, -c1 * dy - va * dv) + sy - g,
                     self._sum(a, -Vb * W * (ra - rb)), self._sum(a, -Vb * W * (pa - pb)),
                     self._sum(a, du * cf), self._sum(a, dv * cf)]

    def _walls(self, itime):
        if self.table is None:
            return
        x0, hs, om = (torch.as_tensor(np.ascontiguousarray(w), device=self.dev) for w in self.table)
        ph = om * (itime * self.p["time_step"])
        self.x[self.m0:] = x0 + hs * (1.0 - torch.cos(ph))
        self.u[self.m0:] = hs * om * torch.sin(ph)
        self.ut[self.m0:] = self.u[self.m0:]

    def step(self, steps, itime):
        nf, dt, eps = self.nf, self.p["time_step"], self.p["epsilon"]
        f = slice(0, nf)
        for _ in range(steps):
            itime += 1
            first = itime == 1
            base = [w[f].clone() for w in (self.rho, self.pr, self.u, self.v)]
            if not first:
                ra, pa, ua, va, fr, fp, fu, fv = self.rate[4:]
                k = 0.5 * dt
                self.rho[f] = base[0] + k * ra
                self.rhot[f] = self.rho[f] + fr
                p1 = base[1] + k * pa
                self.pt[f] = p1 + fp
                self.pr[f] = p1 if self.ref else self._tait(self.rho[f])
                self.u[f] = base[2] + k * ua
                self.v[f] = base[3] + k * va
                self.ut[f] = self.u[f] + k * ua + eps * fu
                self.vt[f] = self.v[f] + k * va + eps * fv
            self._walls(itime)
            self.rates()
            k = 0.5 * dt if first else dt
            r = self.rate
            self.rho[f] = base[0] + k * r[0]
            self.rhot[f] = self.rho[f] + r[8]
            p1 = base[1] + k * r[1]
            self.pr[f] = p1 if self.ref else self._tait(self.rho[f])
            self.pt[f] = p1 + r[9]
            self.u[f] = base[2] + k * r[2]
            self.v[f] = base[3] + k * r[3]
            self.ut[f] = self.u[f] + eps * r[10]
            self.vt[f] = self.v[f] + eps * r[11]
            self.x[f] += dt * self.u[f]
            self.y[f] += dt * self.v[f]

    def fields(self, names):
        two = lambda p, q: torch.stack([p, q], dim=1)
        r = self.rate
        all_ = {"Position": two(self.x, self.y), "Velocity": two(self.u, self.v), "density": self.rho,
                "DynamicPressure": self.pr, "ddensitydt": r[0], "dpdt": r[1], "dvdt": two(r[2], r[3]),
                "ddensitydt_approx": r[4], "dpdt_approx": r[5], "dvdt_approx": two(r[6], r[7]),
                "densityFluctuation": r[8], "pressureFluctuation": r[9], "velocityFluctuation": two(r[10], r[11])}
        return {k: all_[k] for k in names}


def _horner(q, c):
    v = torch.full_like(q, c[0])
    for k in c[1:]:
        v = v * q + k
    return v


def _exact_network(params, cfg, b, st):
    """The network on FP64 tensors; `params` one flat FP64 tensor (BF16-rounded matrices).  Returns the outputs."""
    dev = _device()
    W, at = {}, 0
    for name, shape in SG.param_layout(cfg.rounds):
        k = int(np.prod(shape))
        W[name] = params[at:at + k].view(shape)
        at += k
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev)
    x, y, rho, it = t(st["Position"][:, 0]), t(st["Position"][:, 1]), t(st["density"]), t(st["itype"])
    n = x.numel()
    F = torch.zeros((n, SG.FEAT), dtype=torch.float64, device=dev)
    F[:, 0], F[:, 1] = t(st["Velocity"][:, 0]) / cfg.vel_scale, t(st["Velocity"][:, 1]) / cfg.vel_scale
    F[:, 2] = (rho / cfg.rho0 - 1.0) / cfg.rho_scale
    F[:, 3], F[:, 4], F[:, 5] = it == 1, (it != 1) & (it != 3), it == 3
    i, j = _neighbours(x, y, n, cfg.radius ** 2)
    dx, dy = (x[j] - x[i]) / cfg.radius, (y[j] - y[i]) / cfg.radius
    e = torch.stack([dx, dy, torch.sqrt(dx * dx + dy * dy), (rho[j] - rho[i]) / (cfg.rho0 * cfg.edge_rho_scale)], 1)
    lin = lambda v, k: v @ W[k + ".w"].T + W[k + ".b"]
    h = lin(torch.relu(lin(F, "enc1")), "enc2")
    for r in range(cfg.rounds):
        pq = lin(h, f"r{r}.pq")
        parts = []
        for c in range(0, SG.LATENT, 32):  # the edge tensors in slices of the channels
            z = pq[:, c:c + 32][i] + pq[:, SG.LATENT + c:SG.LATENT + c + 32][j] + e @ W[f"r{r}.we"][c:c + 32].T
            parts.append(torch.zeros((n, 32), dtype=torch.float64, device=dev).index_add(0, i, torch.relu(z)))
        m = torch.cat(parts, 1) @ W[f"r{r}.w2"].T
        h = h + lin(torch.relu(lin(torch.cat([h, m], 1), f"r{r}.n1")), f"r{r}.n2")
    return lin(torch.relu(lin(h, "dec1")), "dec2")[:, :SG.NOUT]


def _bf16_matrices(flat, rounds):
    out, at = torch.as_tensor(flat, dtype=torch.float32).clone(), 0
    for name, shape in SG.param_layout(rounds):
        k = int(np.prod(shape))
        if len(shape) == 2 and not name.endswith(".we"):
            out[at:at + k] = out[at:at + k].bfloat16().float()
        at += k
    return out.double().to(_device())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "rates"):
        deck = _deck(case)
        st = _stir(deck, deck.initial_state(), seed, case["speed"])
        if kind == "step":
            # an upload without the local fields: the step derives them
            st["localVelocity"][:] = st["Velocity"]
            st["localDensity"][:deck.n_fluid] = st["density"][:deck.n_fluid]
            st["localPressure"][:] = 0.0
        e = _Exact(deck, st, case.get("physics", "ref"), case["cap"])
        if kind == "rates":
            e.rates()
            return e.fields(RATE_OUTPUT_FIELDS)
        e.step(case["steps"], 1 if case["graph"] else 0)
        return e.fields(STEP_OUTPUT_FIELDS)
    if kind == "search":
        pos, nf, pb, dist = _cloud(case, seed)
        t = torch.as_tensor(pos, device=_device())
        a, b = _neighbours(t[:, 0], t[:, 1], nf, dist)
        dx, dy = t[a, 0] - t[b, 0], t[a, 1] - t[b, 1]
        r2 = dx * dx + dy * dy
        keep = _cap(a, b, r2, nf, case["neighbors"]) & (a < b) & (b < pb)
        a, b, r2 = a[keep], b[keep], r2[keep]
        o = torch.argsort(a * (1 << 32) + b)
        return {"i": a[o].int(), "j": b[o].int(), "r2": r2[o]}
    b, st = _flume_frame(case, seed)
    cfg, flat = SG.Surrogate.load_file(WEIGHTS)
    params = _bf16_matrices(flat, cfg.rounds)
    if kind == "predict":
        with torch.no_grad():
            return _exact_network(params, cfg, b, st)
    params.requires_grad_(True)
    out = _exact_network(params, cfg, b, st)
    loss = (out[:b.deck.n_fluid] - _target(b.deck.n_fluid, seed).double()).square().mean()
    loss.backward()
    return {"loss": float(loss), "grad": params.grad}
