"""The framework's workloads as timed cases.

Each case is one pass of a program that uses the library: a state on the host
goes in, the model steps, and the fields (and, where such a program asks for
them, the integrals) come out.  Sizes are the icosahedral levels, time steps
and options of the configurations and experiments: icos level 3 (642 cells)
to level 9 (2,621,442 cells), dt = 110 s at level 8 scaled by the spacing.
``exact`` restates the same scheme in plain torch, in 64 bits, on the grid's
arrays.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from imodel_gb300 import learned, learned_weights
from imodel_gb300.mesh import ERAD, GRAV, OMEGA, meshbuild
from imodel_gb300.moist import FIELDS, Moist
from imodel_gb300.swm import SWM, Ensemble

DEV = "cuda:0"
INTEGRALS = ("mass", "penergy", "kenergy", "pot_enstrophy", "rms_div")


def listed():
    return [
        # one tendency of the smallest grid, from host arrays: the operator
        # tests and a host program that does its own time stepping
        {"name": "tendency_fp64_l3", "kind": "tendency", "level": 3, "precision": "fp64"},
        # short-range FP32 run of a coarse grid with diagnostics: launches
        # and their latency count
        {"name": "run_fp32_l5", "kind": "run", "level": 5, "precision": "fp32", "steps": 96,
         "diag": True},
        # the reference's own test run: case-2-like flow, level 5, FP64, a
        # tenth of the 960 steps of 5 days
        {"name": "run_fp64_l5", "kind": "run", "level": 5, "precision": "fp64", "steps": 96,
         "diag": True},
        # flow over mountains at the level of the Williamson cases
        {"name": "mountains_fp32_l7", "kind": "run", "level": 7, "precision": "fp32",
         "steps": 160, "mountains": True, "diag": True},
        # the headline configuration: level 9, FP32 with the learned TRSK
        # weights, page-locked host arrays
        {"name": "weights_fp32_l9", "kind": "run", "level": 9, "precision": "fp32", "steps": 32,
         "weights": True, "pinned": True},
        # the reference-order FP64 run of the balanced configuration's grid
        {"name": "run_fp64_l8", "kind": "run", "level": 8, "precision": "fp64", "steps": 16},
        # PV stabilisation and hyperdiffusion, as a production run sets them
        {"name": "apvm_k4_fp32_l8", "kind": "run", "level": 8, "precision": "fp32", "steps": 48,
         "apvm": 0.5, "k4": 1.0e12},
        # another method wrapper in the reference's order
        {"name": "pxt16_fp64_l6", "kind": "run", "level": 6, "precision": "fp64", "steps": 16,
         "scheme": "pxt16"},
        # the moist model, both precisions
        {"name": "moist_fp32_l8", "kind": "moist", "level": 8, "precision": "fp32", "steps": 48,
         "advection": "trsk"},
        {"name": "moist_fp64_l6", "kind": "moist", "level": 6, "precision": "fp64", "steps": 32,
         "advection": "trsk"},
        # many members on two grids in one launch
        {"name": "ensemble_l6_l7", "kind": "ensemble", "level": 6, "members": 32, "members2": 8,
         "steps": 32},
        # training of the correction network: Adam steps on one level-7
        # field set
        {"name": "train_network", "kind": "train", "rows": 983040, "steps": 100, "batch": 65536},
    ]


def draw(rng):
    """One more case of the same ranges: a kind, a level, options and a
    number of steps that keeps the pass below the largest listed one."""
    kind = rng.choice(["tendency", "run", "run", "run", "run", "moist", "moist", "ensemble",
                       "train"])
    prec = rng.choice(["fp32", "fp64"])

    def steps(level, most):
        cells = 10 * 4 ** level + 2
        hi = max(1, min(160, most // cells))
        return int(round(math.exp(rng.uniform(0.0, math.log(hi))))) if hi > 1 else 1

    if kind == "tendency":
        return {"kind": kind, "level": rng.randint(2, 7), "precision": prec}
    if kind == "run":
        level = rng.randint(3, 9 if prec == "fp32" else 8)
        c = {"kind": kind, "level": level, "precision": prec,
             "steps": steps(level, 40_000_000 if prec == "fp32" else 8_000_000)}
        extra = rng.choice(["plain", "plain", "mountains", "weights", "apvm", "k4", "pxt16"])
        if extra == "mountains":
            c["mountains"] = True
        elif extra == "weights" and prec == "fp32":
            c["weights"] = True
        elif extra == "apvm":
            c["apvm"] = round(rng.uniform(0.25, 1.0), 3)
        elif extra == "k4":
            c["k4"] = 1.0e12 * 8.0 ** (8 - level) if level >= 6 else 5.12e14
        elif extra == "pxt16":
            c["scheme"] = "pxt16"
            c["steps"] = max(1, c["steps"] // 4)
        c["diag"] = rng.random() < 0.5
        c["pinned"] = rng.random() < 0.3
        return c
    if kind == "moist":
        level = rng.randint(4, 8 if prec == "fp32" else 7)
        return {"kind": kind, "level": level, "precision": prec,
                "steps": steps(level, 16_000_000 if prec == "fp32" else 2_000_000),
                "advection": rng.choice(["trsk", "trsk", "upw1"])}
    if kind == "ensemble":
        level = rng.randint(4, 6)
        m = rng.randint(1, 48 if level < 6 else 32)
        return {"kind": kind, "level": level, "members": m, "members2": rng.randint(1, 8),
                "steps": rng.randint(4, 32)}
    return {"kind": "train", "rows": rng.randint(70_000, 983_040), "steps": rng.randint(10, 100),
            "batch": rng.choice([8192, 16384, 32768, 65536])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _grid(level):
    return meshbuild(level)


def _dt(level):
    # 110 s at level 8, halved per level; the coarsest grids stay below 900 s
    return min(900.0, 110.0 * 2.0 ** (8 - level))


def _waves(rng, n=10, kmax=12.0):
    k = rng.normal(size=(n, 3))
    k *= (rng.uniform(2.0, kmax, n) / np.linalg.norm(k, axis=1))[:, None]
    a = rng.normal(size=n) / np.sum(k * k, axis=1)
    return k, a, rng.uniform(0.0, 2.0 * math.pi, n)


def _flow(g, seed, umax=35.0):
    """A seeded smooth rotational flow near geostrophic balance: the
    streamfunction psi is a sum of plane waves in space, u = k x grad psi at
    the velocity points, g h = g h0 + f psi at the cells (f frozen locally)."""
    rng = np.random.default_rng(seed)
    k, a, ph = (torch.as_tensor(x, device=DEV) for x in _waves(rng))
    pe = torch.as_tensor(g.ed_c, device=DEV)
    pv = torch.as_tensor(g.v_p, device=DEV)
    grad = torch.zeros_like(pe)
    psi = torch.zeros(g.nv, dtype=torch.float64, device=DEV)
    for i in range(len(a)):
        grad += (a[i] * torch.cos(pe @ k[i] + ph[i]))[:, None] * k[i]
        psi += a[i] * torch.sin(pv @ k[i] + ph[i])
    v = torch.linalg.cross(pe, grad)
    # the level-independent scale: the sum of the waves' largest slopes
    scale = umax / float(torch.sqrt(torch.sum((a * torch.linalg.norm(k, dim=1)) ** 2)))
    u = (v * torch.as_tensor(g.ed_tg, device=DEV)).sum(1) * scale
    f = 2.0 * OMEGA * pv[:, 2]
    h = (2.94e4 + f * psi * (scale * ERAD) * 0.5) / GRAV
    return h.cpu().numpy(), u.cpu().numpy()


def _mountains(g, seed):
    rng = np.random.default_rng(seed + 77)
    b = np.zeros(g.nv)
    for _ in range(4):
        c = rng.normal(size=3)
        c /= np.linalg.norm(c)
        d2 = np.sum((g.v_p - c) ** 2, axis=1)
        b += rng.uniform(300.0, 900.0) * np.exp(-d2 / rng.uniform(0.02, 0.1))
    return b


def _moist_state(g, seed):
    """Moist flow: theta warm at the equator, vapour from 70 to 130 % of
    saturation (so that both condensation and evaporation act), some cloud
    and rain everywhere."""
    rng = np.random.default_rng(seed + 5)
    h, u = _flow(g, seed)
    k, a, ph = _waves(rng, 4, 6.0)
    s = sum(np.sin(g.v_p @ k[i] + ph[i]) for i in range(4)) / 4.0
    c2 = np.cos(g.v_lat) ** 2
    theta = 0.05 + 0.05 * c2
    q0 = 0.02
    qsat = q0 * np.exp(20.0 * theta) / (h * GRAV)
    qv = qsat * (1.0 + 0.3 * s)
    qc = 2e-4 * (1.0 + 0.5 * s * s)
    qr = 1e-4 * (1.0 + 0.2 * s)
    tr = np.exp(-5.0 * np.sum((g.v_p - [1.0, 0.0, 0.0]) ** 2, axis=1))
    return {"h": h, "u": u, "bt": np.zeros(g.nv), "theta": theta, "q0": q0, "qv": qv, "qc": qc,
            "qr": qr, "htheta": h * theta, "hqv": h * qv, "hqc": h * qc, "hqr": h * qr,
            "htracer": h * tr}


def _train_set(case, seed):
    """Inputs of unit scale (BF16 bits), targets from a fixed smooth function
    of them plus noise, positive weights of mean one."""
    r = torch.Generator(device=DEV).manual_seed(seed)
    n = case["rows"]
    x = torch.randn((n, learned.NFEAT), generator=r, device=DEV).to(torch.bfloat16)
    c = torch.linspace(-1.0, 1.0, learned.NFEAT, device=DEV)
    t = 0.2 * torch.tanh(x.float() @ c) + 0.05 * torch.randn(n, generator=r, device=DEV)
    w = torch.rand(n, generator=r, device=DEV) + 0.5
    return (x.view(torch.int16).cpu().numpy().view(np.uint16), t.cpu().numpy(), w.cpu().numpy())


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t, w = _train_set(case, seed)
        p0 = learned.init_params(seed)
        net = learned.Mlp(params=p0)
        net.load_dataset(x, t, w)
        return {"case": case, "net": net, "p0": p0, "seed": seed % 1000 + 1}
    level = case["level"]
    g = _grid(level)
    if kind == "ensemble":
        g2 = _grid(level + 1)
        ens = Ensemble([g, g2], [case["members"], case["members2"]])
        states = [[_flow(gr, 1000 * seed + 100 * k + j) for j in range(n)]
                  for k, (gr, n) in enumerate(((g, case["members"]), (g2, case["members2"])))]
        return {"case": case, "ens": ens, "states": states}
    if kind == "moist":
        st = _moist_state(g, seed)
        m = Moist(g, 3, st, advection=case["advection"], precision=case["precision"])
        return {"case": case, "m": m, "state": st}
    h, u = _flow(g, seed)
    kw = {}
    if case.get("mountains"):
        kw["bt"] = _mountains(g, seed)
        h = h - kw["bt"]
    if case.get("weights"):
        kw["learned_weights"] = learned_weights.trained_params()
    m = SWM(g, precision=case["precision"], scheme=case.get("scheme", "trsk10"), **kw)
    if case.get("apvm"):
        m.set_apvm(case["apvm"], _dt(level))
    if case.get("k4"):
        m.set_diffusion(0.0, case["k4"])
    if case.get("pinned"):
        h, u = _pin(h), _pin(u)
    s = {"case": case, "m": m, "h": h, "u": u}
    if case.get("pinned"):
        s["ho"], s["uo"] = _pin(np.zeros_like(h)), _pin(np.zeros_like(u))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _f64p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _fields(case, *arrays):
    """The fields as a program keeps them: FP32 fields of an FP32 run (the
    output files' type), FP64 of an FP64 run."""
    if case.get("precision", "fp32") == "fp64":
        return [torch.from_numpy(a) for a in arrays]
    return [torch.from_numpy(a).to(torch.float32) for a in arrays]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        net = state["net"]
        net.set_params(state["p0"])
        losses = net.train(case["steps"], batch=case["batch"], lr=1e-3, seed=state["seed"])
        return {"losses": losses, "params": net.get_params()}
    if kind == "ensemble":
        ens = state["ens"]
        for k, members in enumerate(state["states"]):
            for j, (h, u) in enumerate(members):
                ens.set_state(k, j, h, u)
        lv = case["level"]
        ens.advance([_dt(lv), _dt(lv + 1)], [case["steps"], 2 * case["steps"]])
        out = []
        for k, members in enumerate(state["states"]):
            got = [ens.get_state(k, j) for j in range(len(members))]
            out.append(torch.from_numpy(np.stack([h for h, _ in got])).to(torch.float32))
            out.append(torch.from_numpy(np.stack([u for _, u in got])).to(torch.float32))
        return out
    m = state["m"]
    if kind == "moist":
        m.set_state(state["state"])
        m.advance(_dt(case["level"]), case["steps"])
        r = m.get_state()
        return dict(zip(FIELDS, _fields(case, *[r[k] for k in FIELDS])))
    if kind == "tendency":
        return _fields(case, *m.tendency(state["h"], state["u"]))
    m.set_state(state["h"], state["u"])
    m.advance(_dt(case["level"]), case["steps"])
    out = []
    if case.get("diag"):
        d = m.diagnostics()
        out = _fields(case, *[np.array([d[k]]) for k in INTEGRALS])
    if case.get("pinned"):
        rc = m.lib.imodel_swm_get_state(m.handle, _f64p(state["ho"]), _f64p(state["uo"]))
        if rc:
            raise RuntimeError(f"imodel_swm_get_state: {rc}")
        return _fields(case, state["ho"], state["uo"]) + out
    return _fields(case, *m.get_state()) + out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """One RK4 step reads the geometry and the state once and writes the new
    state once: per cell 6 edges, 3 edge records (two cells, two triangles,
    two lengths), 2 triangle records (three edges, three kites, area,
    Coriolis parameter); members share their grid's geometry."""
    kind = case["kind"]
    if kind == "train":
        rows = case["steps"] * case["batch"]
        return {"bytes": rows * (2 * learned.NFEAT + 8),
                "flops": rows * 6.0 * (24 * 64 + 64 * 64 + 64)}
    w = 8 if case.get("precision", "fp32") == "fp64" else 4
    cells = 10 * 4 ** case["level"] + 2

    def per_step(nv, members, nfield):
        geo = nv * (24 + 8 * w + 3 * (16 + 2 * w) + 2 * (12 + 5 * w))
        return geo + members * nv * 2 * w * nfield

    flop = 4 * 420.0
    if kind == "tendency":
        return {"bytes": per_step(cells, 1, 4) + cells * 4 * 2 * 8, "flops": cells * 420.0}
    n = case["steps"]
    io = 8 * 2 * 4 * cells
    if kind == "ensemble":
        c2 = 4 * cells
        m1, m2 = case["members"], case["members2"]
        return {"bytes": n * per_step(cells, m1, 4) + 2 * n * per_step(c2, m2, 4) +
                (m1 + 4 * m2) * io,
                "flops": flop * n * cells * (m1 + 8 * m2)}
    if kind == "moist":
        return {"bytes": n * per_step(cells, 1, 12) + 8 * 18 * cells,
                "flops": (flop + 4 * 200.0) * n * cells}
    f = flop * (1.4 if case.get("apvm") else 1.0) * (1.4 if case.get("k4") else 1.0)
    return {"bytes": n * per_step(cells, 1, 4) + io, "flops": f * n * cells}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    """The TRSK shallow-water tendency on a grid's arrays; fields carry a
    trailing member axis."""

    def __init__(self, g, bt=None, scheme="trsk10", apvm=0.0, k4=0.0, trskw=None):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)  # noqa: E731
        idx = lambda a: t(a).long() - 1  # noqa: E731
        col = lambda a: t(a).double()[..., None]  # noqa: E731
        self.g, self.scheme, self.apvm, self.k4 = g, scheme, apvm, k4
        self.nnb = t(g.nnb).long()
        live = torch.arange(6, device=DEV)[None, :] < self.nnb[:, None]
        self.ved = torch.where(live, idx(g.v_ed), 0)
        self.edv, self.edt = idx(g.ed_v), idx(g.ed_sh)
        self.trv, self.tred = idx(g.tr_v), idx(g.tr_ed)
        self.out = torch.where(live, t(g.hx_ttgout).double(), 0.0)
        self.ccw = torch.where(live, t(g.hx_tnrccw).double(), 0.0)
        self.A, self.At = col(g.hx_areag), col(g.tr_areag)
        self.l, self.d = col(g.ed_leng), col(g.edhx_leng)
        self.tg = t(g.tr_tg).double()
        self.kite = t(g.tr_trhx_area).double()
        self.f = 2.0 * OMEGA * torch.sin(col(g.tr_c_lat))
        self.bt = col(bt) if bt is not None else 0.0
        # trskw(i, j) at [c, j, i]
        self.w = t(g.hx_trskw if trskw is None else trskw).double()
        pair = live[:, :, None] & live[:, None, :] & ~torch.eye(6, dtype=torch.bool, device=DEV)
        self.w = torch.where(pair, self.w, 0.0)
        e = torch.arange(g.ne, device=DEV)
        self.slot = [6 * self.edv[:, s] + torch.argmax(
            ((self.ved[self.edv[:, s]] == e[:, None]) & live[self.edv[:, s]]).int(), 1)
            for s in range(2)]
        if scheme == "pxt16" or apvm or k4:
            p = t(g.v_p).double()
            a, b, c = (p[self.trv[:, s]] for s in range(3))
            n = torch.linalg.cross(b - a, c - a)
            n = n / torch.linalg.norm(n, dim=1, keepdim=True)
            self.tc = n * torch.sign((n * a).sum(1, keepdim=True))
            self.p, self.ec, self.nr = p, t(g.ed_c).double(), t(g.ed_nr).double()
            dc = self.tc[self.edt[:, 1]] - self.tc[self.edt[:, 0]]
            self.sg = torch.sign((self.nr * dc).sum(1))[:, None]
            det = lambda x, y, z: (x * torch.linalg.cross(y, z)).sum(1).abs()  # noqa: E731
            bary = torch.stack([det(self.tc, b, c), det(self.tc, c, a), det(self.tc, a, b)], 1)
            self.bary = bary / bary.sum(1, keepdim=True)

            def arc(x, y):
                return 2.0 * torch.atan2(torch.linalg.norm(x - y, dim=1),
                                         torch.linalg.norm(x + y, dim=1))
            self.dist = [arc(self.ec, self.tc[self.edt[:, s]])[:, None] for s in range(2)]

    def perot_cell(self, x):
        """sum_j ttgout x_j (ed%c - v%p) d / A on the tangent plane, [nv, 3, M]"""
        v = 0.0
        for j in range(6):
            e = self.ved[:, j]
            r = (self.ec[e] - self.p)[:, :, None]
            v = v + (self.out[:, j, None] * x[e] * self.d[e])[:, None, :] * r
        v = v / self.A[:, None]
        return v - (v * self.p[:, :, None]).sum(1, keepdim=True) * self.p[:, :, None]

    def lap(self, u, kc):
        div = sum(self.out[:, j, None] * u[self.ved[:, j]] * self.d[self.ved[:, j]]
                  for j in range(6)) / self.A / ERAD
        z = sum(u[self.tred[:, s]] * self.l[self.tred[:, s]] * self.tg[:, s, None]
                for s in range(3)) / self.At / ERAD
        kt = math.sqrt(kc) * torch.sqrt(self.kite.sum(1, keepdim=True) / self.At)
        cd, cv = math.sqrt(kc) * div, kt * z
        return (cd[self.edv[:, 1]] - cd[self.edv[:, 0]]) / self.l / ERAD - \
            self.sg * (cv[self.edt[:, 1]] - cv[self.edt[:, 0]]) / (self.d * ERAD)

    def tendency(self, h, u, dt):
        pxt = self.scheme == "pxt16"
        he = 0.5 * (h[self.edv[:, 0]] + h[self.edv[:, 1]])
        F = u * he
        eta = sum(u[self.tred[:, s]] * self.l[self.tred[:, s]] * self.tg[:, s, None]
                  for s in range(3)) / self.At / ERAD + self.f
        if pxt:
            ht = sum(self.bary[:, s, None] * h[self.trv[:, s]] for s in range(3))
        else:
            ht = sum(self.kite[:, s, None] * h[self.trv[:, s]] for s in range(3)) / self.At
        q = eta / ht
        q1, q2 = q[self.edt[:, 0]], q[self.edt[:, 1]]
        if pxt:
            qe = (self.dist[1] * q1 + self.dist[0] * q2) / (self.dist[0] + self.dist[1])
        else:
            qe = 0.5 * (q1 + q2)
        if self.apvm:
            ge = self.sg * (q2 - q1) / self.d / ERAD
            v = 0.0
            for s in range(3):
                e = self.tred[:, s]
                r = (self.ec[e] - self.tc)[:, :, None]
                v = v - (self.tg[:, s, None] * ge[e] * self.l[e])[:, None, :] * r
            v = v / self.At[:, None]
            gt = v - (v * self.tc[:, :, None]).sum(1, keepdim=True) * self.tc[:, :, None]
            vc = self.perot_cell(u)
            qe = qe - self.apvm * dt * ((gt[self.edt[:, 0]] + gt[self.edt[:, 1]]) *
                                        (vc[self.edv[:, 0]] + vc[self.edv[:, 1]])).sum(1)
        G, Q, div, ke, area = [], [], 0.0, 0.0, 0.0
        for j in range(6):
            e = self.ved[:, j]
            G.append(F[e] * self.d[e] * self.out[:, j, None])
            Q.append(qe[e])
            div = div + G[j]
            a = 0.25 * self.l[e] * self.d[e] * self.out[:, j, None].abs()
            ke, area = ke + a * u[e] ** 2, area + a
        mass = -div / self.A / ERAD
        ke = (self.perot_cell(u) ** 2).sum(1) * 0.5 if pxt else ke / area
        B = GRAV * (h + self.bt) + ke
        Z = torch.empty((h.shape[0], 6, h.shape[1]), dtype=torch.float64, device=DEV)
        if pxt:
            # pered: half of the cell's Perot vector of F (q_e + q_k) / 2,
            # along ed%nr of each of its edges
            for i in range(6):
                v = 0.0
                for j in range(6):
                    r = (self.ec[self.ved[:, j]] - self.p)[:, :, None]
                    v = v + (G[j] * 0.5 * (Q[i] + Q[j]))[:, None, :] * r
                v = v / self.A[:, None]
                v = v - (v * self.p[:, :, None]).sum(1, keepdim=True) * self.p[:, :, None]
                e = self.ved[:, i]
                v = v - (v * self.ec[e][:, :, None]).sum(1, keepdim=True) * self.ec[e][:, :, None]
                Z[:, i] = -0.5 * (v * self.nr[e][:, :, None]).sum(1) * self.l[e]
        else:
            for i in range(6):
                z = 0.0
                for j in range(6):
                    z = z + self.w[:, j, i, None] * G[j] * (0.5 * (Q[i] + Q[j]))
                Z[:, i] = z * self.ccw[:, i, None]
        Z = Z.view(-1, h.shape[1])
        mom = -(B[self.edv[:, 1]] - B[self.edv[:, 0]]) / self.l / ERAD - \
            (Z[self.slot[0]] + Z[self.slot[1]]) / self.l
        if self.k4:
            mom = mom - self.lap(self.lap(u, self.k4), self.k4)
        return mass, mom, he

    def rk4(self, y, dt, rhs):
        k1 = rhs(y)
        k2 = rhs([a + 0.5 * dt * b for a, b in zip(y, k1)])
        k3 = rhs([a + 0.5 * dt * b for a, b in zip(y, k2)])
        y4 = [a + dt * b for a, b in zip(y, k3)]
        k4 = rhs(y4)
        self.last = (y4[0], y4[1])
        return [a + dt * (b + 2.0 * c + 2.0 * d + e) / 6.0
                for a, b, c, d, e in zip(y, k1, k2, k3, k4)]

    def steps(self, h, u, dt, n):
        y = [h, u]
        for _ in range(n):
            y = self.rk4(y, dt, lambda z: self.tendency(z[0], z[1], dt)[:2])
        return y

    def integrals(self, h, u):
        """mass, potential and kinetic energy, potential enstrophy and RMS
        divergence, with h_e, div u and q of the last stage input"""
        hs, us = self.last
        he = 0.5 * (hs[self.edv[:, 0]] + hs[self.edv[:, 1]])
        pe = (self.A * GRAV * h * (0.5 * h + self.bt)).sum()
        ke = (0.5 * self.l * self.d * he * u * u).sum()
        z = sum(us[self.tred[:, s]] * self.l[self.tred[:, s]] * self.tg[:, s, None]
                for s in range(3)) / self.At / ERAD + self.f
        ht = sum(self.kite[:, s, None] * hs[self.trv[:, s]] for s in range(3)) / self.At
        div = sum(self.out[:, j, None] * us[self.ved[:, j]] * self.d[self.ved[:, j]]
                  for j in range(6)) / self.A / ERAD
        both = [(self.A * h).sum() / self.A.sum(), pe, ke, (0.5 * self.At * z * z / ht).sum(),
                torch.sqrt((self.A * div * div).sum() / self.A.sum())]
        return [v.reshape(1).cpu() for v in both]


def _exact_moist(case, g, st):
    X = _Exact(g, st["bt"])
    t = lambda a: torch.as_tensor(a, device=DEV).double()[:, None]  # noqa: E731
    dt = _dt(case["level"])
    theta, ex = t(st["theta"]), torch.exp(20.0 * t(st["theta"]))
    y = [t(st[k]) for k in FIELDS]
    q = [t(st[k]) for k in ("qv", "qc", "qr")]
    upw = case["advection"] == "upw1"
    a, b = X.edv[:, 0], X.edv[:, 1]
    # the cell the flux u > 0 leaves: the one whose ttgout on the edge is +1
    o = X.out.reshape(-1)[X.slot[0]][:, None] > 0

    def rhs(z):
        h, u = z[0], z[1]
        mass, mom, he = X.tendency(h, u, dt)
        qv, qc, _ = q
        qs = st["q0"] * ex / ((h + X.bt) * GRAV)
        gam = 1.0 / (1.0 + 10.0 * (20.0 * qs))
        dqv = torch.clamp(gam * (qv - qs), min=0.0) / dt
        dqc = torch.minimum(qc, torch.clamp(-gam * (qv - qs), min=0.0)) / dt
        dqr = torch.clamp(0.001 * (qc - 0.0001), min=0.0) / dt
        src = [h * 10.0 * (dqv - dqc), h * (dqc - dqv), h * (dqv - dqc - dqr), h * dqr]
        gp = (h[b] * z[2][b] - h[a] * z[2][a]) / X.l / ERAD / he
        mom = mom + 0.5 * GRAV * gp
        bt = X.bt.expand_as(h) if torch.is_tensor(X.bt) else torch.zeros_like(h)
        mom = mom + GRAV * 0.5 * (theta[a] + theta[b]) * (bt[b] - bt[a]) / X.l / ERAD
        out = [mass, mom]
        for k in range(4):
            c = z[2 + k]
            ce = torch.where(o == (u > 0), c[a], c[b]) if upw else 0.5 * (c[a] + c[b])
            fl = u * ce
            div = sum(X.out[:, j, None] * fl[X.ved[:, j]] * X.d[X.ved[:, j]] for j in range(6))
            out.append(-div / X.A / ERAD + src[k])
        return out + [torch.zeros_like(h)]

    for _ in range(case["steps"]):
        y = X.rk4(y, dt, rhs)
        q = [y[3] / y[0], y[4] / y[0], y[5] / y[0]]
    return {k: v[:, 0].cpu() for k, v in zip(FIELDS, y)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # the batches come from the library's own random row draw
    g = _grid(case["level"])
    t = lambda a: torch.as_tensor(a, device=DEV).double()  # noqa: E731
    if kind == "ensemble":
        out = []
        for k, n in enumerate((case["members"], case["members2"])):
            gr = _grid(case["level"] + k)
            s = [_flow(gr, 1000 * seed + 100 * k + j) for j in range(n)]
            X = _Exact(gr)
            h, u = X.steps(t(np.stack([a for a, _ in s], 1)), t(np.stack([b for _, b in s], 1)),
                           _dt(case["level"] + k), case["steps"] * (k + 1))
            out += [h.T.cpu(), u.T.cpu()]
        return out
    if kind == "moist":
        return _exact_moist(case, g, _moist_state(g, seed))
    h, u = _flow(g, seed)
    kw = {}
    if case.get("mountains"):
        kw["bt"] = _mountains(g, seed)
        h = h - kw["bt"]
    if case.get("weights"):
        # the corrected weights are data of the scheme, like the grid's
        m = SWM(g, precision="fp64", learned_weights=learned_weights.trained_params())
        kw["trskw"] = m.learned_weights()[1]
        m.close()
    X = _Exact(g, scheme=case.get("scheme", "trsk10"), apvm=case.get("apvm", 0.0),
               k4=case.get("k4", 0.0), **kw)
    dt = _dt(case["level"])
    h, u = t(h)[:, None], t(u)[:, None]
    if kind == "tendency":
        a, b, _ = X.tendency(h, u, dt)
        return [a[:, 0].cpu(), b[:, 0].cpu()]
    h, u = X.steps(h, u, dt, case["steps"])
    out = X.integrals(h, u) if case.get("diag") else []
    return [h[:, 0].cpu(), u[:, 0].cpu()] + out
