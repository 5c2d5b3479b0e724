"""Performance cases of the grid thermal model, through its Python entry points.

A case is one call that a simulation makes again and again: a sampling
interval (``compute_temp``), a run of intervals (``compute_trace``), a steady
solve (``steady``) or a batch of chips (``Batch.trace``).  ``exact`` restates
the same physics in FP64 with torch: the RC network of the layer stack and its
package, the step-doubling RK4 of the transient and the linear system of the
steady state.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from hotspot_b200 import FORM_FAST, FORM_PARITY, STEADY_AUTO, STEADY_BICGSTAB
from hotspot_b200 import batch as hb
from hotspot_b200 import model as hm
from hotspot_b200 import workloads as W

FORMS = {"fast": FORM_FAST, "parity": FORM_PARITY}
ROWS = 4            # power rows (or sets of rows) a simulation cycles through


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def chip(**kw):
    """`layers` chip layers of alternating silicon and TIM (0: the default
    silicon + TIM pair without a layer file) over the spreader and the sink."""
    c = {"kind": "interval", "form": "fast", "rows": 64, "cols": 64, "layers": 0, "blocks": 15, "die_mm": 16.0,
         "dt": 3.333e-6, "intervals": 1, "chips": 1, "map": "center", "tol": 1e-8}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call of the library: one 3.3 us sampling interval of a
        # single 2-D chip, as a cycle-level simulator makes it after every
        # power sample; the fast form, and the form a caller gets by default
        chip(name="chip64_interval_fast"),
        chip(name="chip64_interval_default", form="parity"),
        # the 3-D stack of the headline benchmark, one 10 us interval at a time
        chip(name="stack256_interval_fast", rows=256, cols=256, layers=4, blocks=40, die_mm=20.0, dt=1e-5),
        chip(name="stack256_interval_default", form="parity", rows=256, cols=256, layers=4, blocks=40, die_mm=20.0,
             dt=1e-5),
        # a power trace replayed in runs of intervals on a deep stack
        chip(name="stack128x7_trace_fast", kind="trace", rows=128, cols=128, layers=7, blocks=37, intervals=24),
        # steady states: the 2-D chip in both forms (the default form's grid
        # is dumped, as with a grid steady file), the stack, the largest chip
        # of the serving mix; the fast form's tolerance is one at which the
        # differences between two floorplans can be taken
        chip(name="chip64_steady_fast", kind="steady"),
        chip(name="chip32_steady_default", kind="steady", form="parity", rows=32, cols=32),
        chip(name="stack256_steady_fast", kind="steady", rows=256, cols=256, layers=4, blocks=40, die_mm=20.0),
        chip(name="chip1024_steady_fast", kind="steady", rows=1024, cols=1024, layers=3, blocks=55),
        # liquid cooling: an interval with advection and per-cell coefficients
        # in the default form, and the non-symmetric steady system
        chip(name="uchan128_interval_default", kind="uchan_interval", form="parity", rows=128, cols=128, layers=2,
             blocks=1024, die_mm=2.56, map="avg"),
        chip(name="uchan512_steady", kind="uchan_steady", rows=512, cols=512, layers=2, blocks=4096, die_mm=10.24,
             map="avg"),
        # design-space exploration: many different chips advanced together
        chip(name="batch32_trace", kind="batch", rows=256, cols=256, layers=8, blocks=0, chips=32, intervals=24),
    ]


def draw(rng):
    kind = rng.choice(["interval", "interval", "interval", "trace", "steady", "steady", "steady", "uchan_interval",
                       "uchan_steady", "batch"])
    form = "fast"
    if kind == "interval":
        form = rng.choice(["fast", "parity"])
    elif kind == "uchan_interval":
        form = "parity"
    elif kind == "steady":
        form = rng.choice(["fast", "fast", "parity"])
    dt = math.exp(rng.uniform(math.log(2e-6), math.log(1.2e-5)))
    if kind.startswith("uchan"):
        side = rng.choice([128, 256]) if kind == "uchan_interval" else rng.choice([128, 256, 512])
        return chip(kind=kind, form=form, rows=side, cols=side, layers=2, blocks=(side // rng.choice([2, 4, 8])) ** 2,
                    die_mm=side * 0.02, dt=dt, map="avg", tol=rng.choice([1e-8, 1e-9]))
    if kind == "batch":
        side = rng.choice([64, 128, 256])
        return chip(kind=kind, rows=side, cols=side, layers=rng.randint(3, 8), blocks=0, chips=rng.randint(5, 32),
                    intervals=rng.randint(3, 24), dt=dt)
    if kind == "steady" and form == "parity":
        rows, cols = rng.choice([16, 32]), rng.choice([16, 32])
        layers = rng.randint(0, 2)
    elif kind == "steady":
        rows = rng.choice([64, 128, 256, 512])
        cols = rng.choice([rows, rows, rows // 2])
        layers = rng.randint(0, 8)
    else:
        rows = rng.choice([32, 64, 128, 256])
        cols = rng.choice([rows, rows, rows // 2, min(256, 2 * rows)])
        layers = rng.randint(0, 7)
    return chip(kind=kind, form=form, rows=rows, cols=cols, layers=layers, blocks=rng.randint(9, 60),
                die_mm=round(rng.uniform(10.0, 20.0), 2), dt=dt,
                intervals=rng.randint(5, 31) if kind == "trace" else 1, map=rng.choice(["center", "center", "avg"]),
                tol=rng.choice([1e-8, 1e-9]))


# ---------------------------------------------------------------------------
# inputs: the stack's floorplans and power rows, from the seed alone
# ---------------------------------------------------------------------------
def _stack(case, seed, which=0):
    """(layers, power rows) of one chip: a layer is (power, specific heat,
    resistivity, thickness, units)."""
    rng = np.random.default_rng([int(seed), which, 271])
    die = case["die_mm"] * 1e-3
    blocks, layers = case["blocks"], case["layers"]
    side = (case["rows"], case["cols"])
    if case["kind"] == "batch":                       # its own size for every chip, the case's own mix
        mix = np.random.default_rng([which, case["rows"], case["layers"], case["chips"]])
        s = int(2 ** mix.integers(5, int(math.log2(case["rows"])) + 1))
        side, layers, blocks = (s, s), int(mix.integers(1, case["layers"] + 1)), int(mix.integers(10, 101))
    stack, means = [], []
    for l in range(max(layers, 1)):
        if l % 2 == 0:
            units = W.guillotine_floorplan(rng, die, die, blocks, prefix=f"l{l}_")
            stack.append((True, 1.75e6, 0.01, 1.5e-4 if layers == 0 else 1e-4, units))
            # 0.1..2 W/mm^2 spread over the powered layers
            dens = rng.uniform(0.1, 2.0, len(units)) / ((max(layers, 1) + 1) // 2)
            means.append(dens * np.array([u.width * u.height * 1e6 for u in units]))
        else:
            stack.append((False, 4e6, 0.25, 2e-5, [W.Unit("tim", die, die, 0.0, 0.0)]))
    if layers == 0:                                   # the default pair: the TIM under the same floorplan
        stack.append((False, 4e6, 0.25, 2e-5, stack[0][4]))
    n = ROWS * case["intervals"]
    return side, stack, W.ar1_power(rng, np.concatenate(means), n)


def _scenario(case, seed, which, workdir):
    side, stack, rows = _stack(case, seed, which)
    cfg = {"model_type": "grid", "grid_rows": str(side[0]), "grid_cols": str(side[1]), "grid_map_mode": case["map"],
           "sampling_intvl": repr(case["dt"])}
    names = [[u.name for u in s[4]] if s[0] else [] for s in stack]
    flps = [W.write_flp(os.path.join(workdir, f"c{which}_{l}.flp"), s[4]) for l, s in enumerate(stack)]
    if case["layers"] == 0:
        return W.Scenario("chip", cfg, flp=flps[0], power_layers=names[:1], dt=case["dt"]), rows
    lcf = W.write_lcf(os.path.join(workdir, f"c{which}.lcf"),
                      [W.Layer(True, s[0], s[1], s[2], s[3], f) for s, f in zip(stack, flps)])
    cfg["grid_layer_file"] = lcf
    return W.Scenario("stack", cfg, lcf=lcf, power_layers=names, dt=case["dt"]), rows


def _uchan(case, seed, workdir):
    sc = W.scenario_microchannel(workdir, seed=int(seed), grid=case["rows"], die=case["die_mm"] * 1e-3,
                                 blocks=int(round(math.sqrt(case["blocks"]))))
    rng = np.random.default_rng([int(seed), 577])
    return sc, sc.block_power[0] * rng.uniform(0.7, 1.3, (ROWS, 1))


def prepare(case, seed):
    st = {"case": case, "k": 0}
    with tempfile.TemporaryDirectory() as d:
        if case["kind"] == "batch":
            models, rows = [], []
            for c in range(case["chips"]):
                sc, r = _scenario(case, seed, c, d)
                m = hm.from_scenario(sc)
                m.set_solver(FORM_FAST)
                m.set_grid("trans", np.full(m.n_cells + m.n_extra, m.config.init_temp))
                models.append(m)
                rows.append([m.power_vector(x) for x in r])
            n = case["intervals"]
            st["rows"] = [[[rows[c][q * n + k] for c in range(len(models))] for k in range(n)] for q in range(ROWS)]
            st["models"], st["batch"] = models, hb.Batch(models)
            return st
        sc, r = _uchan(case, seed, d) if case["kind"].startswith("uchan") else _scenario(case, seed, 0, d)
        m = hm.from_scenario(sc)
    m.set_solver(FORMS[case["form"]], STEADY_BICGSTAB if case["kind"] == "uchan_steady" else STEADY_AUTO,
                 steady_tol=case["tol"])
    rows = np.stack([m.power_vector(x) for x in r])
    if case["kind"] == "trace":
        rows = rows.reshape(ROWS, case["intervals"], -1)
    st.update(model=m, rows=rows, temp=m.vector(m.config.init_temp))
    return st


def run(st):
    case, k = st["case"], st["k"]
    st["k"] = k + 1
    row = st["rows"][k % ROWS]
    kind = case["kind"]
    if kind == "batch":
        st["batch"].trace(row, case["dt"])
        return [m.grid("trans") for m in st["models"]]
    m = st["model"]
    if kind in ("interval", "uchan_interval"):
        # the first interval starts from the block temperatures, the later
        # ones go on from the grid's own state
        m.compute_temp(row, st["temp"] if k == 0 else None, case["dt"])
        return st["temp"]
    if kind == "trace":
        return m.compute_trace(row, st["temp"] if k == 0 else None, case["dt"])[0]
    out = m.vector()
    m.steady(row, out)
    return {"block": out, "grid": m.grid("steady")} if case["form"] == "parity" else out


def _cells(case):
    """Grid cells of the case; a batch has chips of half the largest layer
    count and sides log-uniform from 32."""
    if case["kind"] == "batch":
        sides = [2 ** e for e in range(5, int(math.log2(case["rows"])) + 1)]
        return case["chips"] * (sum(s * s for s in sides) / len(sides)) * ((1 + case["layers"]) / 2 + 2)
    return case["rows"] * case["cols"] * ((case["layers"] or 2) + 2)


def work(case):
    """An interval reads the state and the power and writes the state (FP64);
    its four RK4 steps evaluate eleven seven-point slopes each.  A steady
    solve reads the power and writes the temperatures, and applies the operator some tens
    of times."""
    n = _cells(case)
    if "steady" in case["kind"]:
        return {"bytes": 16.0 * n, "flops": 14.0 * 30 * n}
    return {"bytes": 24.0 * n, "flops": 14.0 * 44 * n * case["intervals"]}


# ---------------------------------------------------------------------------
# the same results in FP64
# ---------------------------------------------------------------------------
def _near(x, y):
    return np.abs(x - y) < 1e-6


def _tol(x, up):
    near = np.floor(x + 0.5)
    return np.where(_near(x, near), near, np.ceil(x) if up else np.floor(x)).astype(int)


class _Grid:
    """The RC network: conductances gE, gS, gB between neighbouring cells,
    heat capacities, ambient and package couplings, advection."""

    def __init__(self, rows, cols, die, stack, dev, detailed=None):
        self.nr, self.nc = nr, nc = rows, cols
        self.dev = dev
        cw, ch = die / nc, die / nr
        self.cell_area = die * die / (nr * nc)
        self.die = die
        amb_r = 0.1 * 60e-3 ** 2 / (cw * ch)
        k = [1 / s[2] for s in stack] + [400.0, 400.0]
        t = [s[3] for s in stack] + [1e-3, 6.9e-3]
        sp = [s[1] for s in stack] + [3.55e6, 3.55e6]
        self.units = [s[4] for s in stack] + [stack[-1][4]] * 2
        self.nl = nl = len(k)
        rx = [cw / (k[n] * ch * t[n]) for n in range(nl)]
        ry = [ch / (k[n] * cw * t[n]) for n in range(nl)]
        rz = [t[n] / (k[n] * cw * ch) for n in range(nl)]
        cap = [0.333 * sp[n] * t[n] * cw * ch for n in range(nl)]
        rz[-1] += amb_r
        cap[-1] += 0.333 * 140.4 * (cw * ch) / 60e-3 ** 2
        full = lambda v, a, b: torch.full((a, b), v, dtype=torch.float64)  # noqa: E731
        self.adv = None
        if detailed is None:
            gE = [full(1 / ry[n], nr, nc - 1) for n in range(nl)]
            gS = [full(1 / rx[n], nr - 1, nc) for n in range(nl)]
            gB = [full(1 / rz[n], nr, nc) for n in range(nl - 1)]
            self.cap = torch.stack([full(c, nr, nc) for c in cap])
        else:
            # detailed 3-D: half resistances of the two cells (all of layer
            # 0's), and a heat transfer coefficient between fluid and solid
            fl = torch.zeros((nl, nr, nc), dtype=torch.bool)
            X, Y, Z = (torch.stack([full(v[n], nr, nc) for n in range(nl)]) for v in (rx, ry, rz))
            self.cap = torch.stack([full(c, nr, nc) for c in cap])
            u = detailed["layer"]
            fl[u][:, torch.from_numpy(detailed["fluid"])] = True
            res = torch.where(fl[u], torch.tensor(detailed["r_fluid"], dtype=torch.float64),
                              torch.tensor(detailed["r_wall"], dtype=torch.float64))
            X[u], Y[u], Z[u] = res * cw / (ch * t[u]), res * ch / (cw * t[u]), res * t[u] / (cw * ch)
            vol = torch.where(fl[u], torch.tensor(detailed["c_fluid"], dtype=torch.float64),
                              torch.tensor(detailed["c_wall"], dtype=torch.float64))
            self.cap[u] = 0.333 * vol * t[u] * cw * ch
            htc = detailed["htc"]

            def pair(ra, rb, fa, fb, rh):
                mixed = torch.where(fa, rb, ra) / 2 + rh
                return 1 / torch.where(fa != fb, mixed, ra / 2 + rb / 2)
            gE = [pair(Y[n][:, :-1], Y[n][:, 1:], fl[n][:, :-1], fl[n][:, 1:], 1 / (htc * ch * t[n])) for n in range(nl)]
            gS = [pair(X[n][:-1], X[n][1:], fl[n][:-1], fl[n][1:], 1 / (htc * cw * t[n])) for n in range(nl)]
            gB = []
            for n in range(nl - 1):
                g = pair(Z[n], Z[n + 1], fl[n], fl[n + 1], 1 / (htc * ch * cw))
                if n == 0:
                    g = 1 / torch.where(fl[0] != fl[1], Z[0] + 1 / (htc * ch * cw), Z[0] + Z[1] / 2)
                gB.append(g)
            # straight channels: the same flow F through every link of a lane
            F = torch.zeros((nl, nr, nc), dtype=torch.float64)
            F[fl] = detailed["heat_flow"]
            self.adv = F.to(dev)
            self.t_in = 300.0
        self.gE, self.gS, self.gB = (torch.stack(g).to(dev) for g in (gE, gS, gB))
        self.cap = self.cap.to(dev)
        self.g_amb = 1 / rz[-1]
        # package: 12 nodes W E N S of the spreader, the sink's inner and its
        # outer periphery (temperature.c's package R and C)
        w, ss, sp_, ts, tp, ks = die, 60e-3, 30e-3, 6.9e-3, 1e-3, 400.0
        per, out = (sp_ + w) * (sp_ - w) / 4, (ss ** 2 - sp_ ** 2) / 4
        side = (sp_ - w) / 4
        r_sp1 = side / (ks * (sp_ + 3 * w) / 4 * tp)
        r_hs1 = side / (ks * (sp_ + 3 * w) / 4 * ts)
        r_hs2 = side / (ks * (3 * sp_ + w) / 4 * ts) + (ss - sp_) / 4 / (ks * (ss + 3 * sp_) / 4 * ts)
        area = 0.1 * ss ** 2
        G = np.zeros((12, 12))
        amb = np.zeros(12)
        for q in range(4):
            for a, b, r in ((q, 4 + q, tp / (ks * per)), (4 + q, 8 + q, r_hs2)):
                G[a, b] += 1 / r
                G[b, a] += 1 / r
            amb[4 + q] = 1 / (ts / (ks * per) + area / per)
            amb[8 + q] = 1 / (ts / (ks * out) + area / out)
        conv = 0.333 * 140.4 / ss ** 2
        pcap = [0.333 * 3.55e6 * tp * per] * 4 + [0.333 * 3.55e6 * ts * per + conv * per] * 4 + \
               [0.333 * 3.55e6 * ts * out + conv * out] * 4
        d64 = lambda v: torch.tensor(np.asarray(v), dtype=torch.float64, device=dev)  # noqa: E731
        self.plink, self.pamb, self.pcap = d64(G), d64(amb), d64(pcap)
        self.edge = []                                   # (layer, first node, conductance N/S, E/W)
        for n, first, r in ((nl - 2, 0, r_sp1), (nl - 1, 4, r_hs1)):
            self.edge.append((n, first, 1 / (ry[n] / 2 + nc * r), 1 / (rx[n] / 2 + nr * r)))
        # block occupancy of the rows and columns, per layer
        self.maps = []
        for units in self.units:
            l, b = np.array([u.leftx for u in units]), np.array([u.bottomy for u in units])
            r, tp_ = l + np.array([u.width for u in units]), b + np.array([u.height for u in units])
            i, j = np.arange(nr), np.arange(nc)
            oh = np.minimum(tp_[:, None], die - i * ch) - np.maximum(b[:, None], die - (i + 1) * ch)
            ow = np.minimum(r[:, None], (j + 1) * cw) - np.maximum(l[:, None], j * cw)
            oh, ow = (np.where(_near(o, 0), 0, np.where(_near(o, 1), 1, np.clip(o, 0, 1))) for o in (oh / ch, ow / cw))
            box = (nr - _tol(tp_ / ch, True), nr - _tol(b / ch, False), _tol(l / cw, False), _tol(r / cw, True))
            self.maps.append((d64(oh), d64(ow), d64([u.width * u.height for u in units]), np.stack(box, 1)))

    def to_grid(self, values, power):
        """One value per unit, layer by layer, spread over the cells."""
        out = []
        for v, (oh, ow, area, _) in zip(values, self.maps):
            v = v / area * self.cell_area if power else v
            out.append((oh * v[:, None]).T @ ow)
        return torch.stack(out)

    def to_blocks(self, T, x, mode):
        out = []
        for n, (_, _, _, box) in enumerate(self.maps):
            g = T[n].cpu().numpy()
            for i1, i2, j1, j2 in box:
                if mode == "avg":
                    out.append(g[i1:i2, j1:j2].mean())
                    continue
                a, b = (i1 + i2) // 2, (j1 + j2) // 2
                c, d = a - (0 if (i2 - i1) % 2 else 1), b - (0 if (j2 - j1) % 2 else 1)
                out.append((g[a, b] + g[c, b] + g[a, d] + g[c, d]) / 4)
        return np.concatenate([np.array(out), x.cpu().numpy()])

    def flow(self, T, x, amb):
        """Net heat flow into every cell and package node (no power)."""
        q = torch.zeros_like(T)
        f = self.gE * (T[:, :, 1:] - T[:, :, :-1])
        q[:, :, :-1] += f
        q[:, :, 1:] -= f
        f = self.gS * (T[:, 1:] - T[:, :-1])
        q[:, :-1] += f
        q[:, 1:] -= f
        f = self.gB * (T[1:] - T[:-1])
        q[:-1] += f
        q[1:] -= f
        q[-1] += self.g_amb * (amb - T[-1])
        px = self.plink @ x - self.plink.sum(1) * x + self.pamb * (amb - x)
        for n, k, gn, ge in self.edge:
            for node, cells, g in ((k + 2, (n, 0), gn), (k + 3, (n, -1), gn), (k, (n, slice(None), 0), ge),
                                   (k + 1, (n, slice(None), -1), ge)):
                f = g * (x[node] - T[cells])
                q[cells] += f
                px[node] -= f.sum()
        if self.adv is not None:
            F = self.adv
            up = torch.cat([torch.full_like(T[:, :1], self.t_in if amb else 0.0), (T[:, :-1] + T[:, 1:]) / 2], 1)
            q += F * up
            q[:, :-1] -= F[:, :-1] * (T[:, :-1] + T[:, 1:]) / 2
            q[:, -1] -= F[:, -1] * T[:, -1]
        return q, px

    def interval(self, T, x, P, dt, amb):
        """The step-doubling RK4 over one interval, as the transient defines it."""
        shape, n = T.shape, T.numel()
        y = torch.cat([T.reshape(-1), x])
        icap = torch.cat([self.cap.reshape(-1), self.pcap])
        pw = torch.cat([P.reshape(-1), torch.zeros_like(x)])

        def f(y):
            q, px = self.flow(y[:n].reshape(shape), y[n:], amb)
            return (torch.cat([q.reshape(-1), px]) + pw) / icap

        def core(y, k1, h):
            k2 = f(y + h / 2 * k1)
            k3 = f(y + h / 2 * k2)
            return y + h * (k1 + 2 * k2 + 2 * k3 + f(y + h * k3)) / 6
        t, new_h = 0.0, 1e-7
        while t < dt and new_h >= 1e-13:
            k1 = f(y)
            while True:
                h = new_h
                one = core(y, k1, h)
                t1 = core(y, k1, h / 2)
                k1 = f(t1)
                err = float((one - core(t1, k1, h / 2)).abs().max())
                if err <= 0.01:
                    new_h = min(0.95 * h * abs(0.01 / err) ** 0.2, 5 * h)
                else:
                    new_h = max(0.95 * h * abs(0.01 / err) ** 0.25, h / 10)
                if new_h >= h:
                    break
            y = one
            new_h = min(new_h, dt - t - h)
            t += h
        return y[:n].reshape(shape), y[n:]

    # -- the steady system A theta = P, theta = T - ambient -----------------
    def _apply(self, v, shape):
        q, px = self.flow(v[:-12].reshape(shape), v[-12:], 0.0)
        return -torch.cat([q.reshape(-1), px])

    def steady(self, P, amb):
        """Conjugate gradients (Jacobi), restarted on the true residual."""
        shape = P.shape
        b = torch.cat([P.reshape(-1), torch.zeros(12, dtype=torch.float64, device=self.dev)])
        D = torch.zeros_like(P)
        for g, a, c in ((self.gE, (slice(None), slice(None), slice(0, -1)), (slice(None), slice(None), slice(1, None))),
                        (self.gS, (slice(None), slice(0, -1)), (slice(None), slice(1, None))),
                        (self.gB, (slice(0, -1),), (slice(1, None),))):
            D[a] += g
            D[c] += g
        D[-1] += self.g_amb
        pd = self.plink.sum(1) + self.pamb
        for n, k, gn, ge in self.edge:
            D[n, 0] += gn
            D[n, -1] += gn
            D[n, :, 0] += ge
            D[n, :, -1] += ge
            pd[k + 2:k + 4] += gn * self.nc
            pd[k:k + 2] += ge * self.nr
        M = 1 / torch.cat([D.reshape(-1), pd])
        v = torch.zeros_like(b)
        for _ in range(3):
            r = b - self._apply(v, shape)
            z = M * r
            p, rz = z.clone(), torch.dot(r, z)
            stop, e = float(rz) * 1e-24, torch.zeros_like(b)
            for it in range(40000):
                Ap = self._apply(p, shape)
                a = rz / torch.dot(p, Ap)
                e += a * p
                r -= a * Ap
                z = M * r
                new = torch.dot(r, z)
                if it % 50 == 49 and not float(new) > stop:
                    break
                p = z + (new / rz) * p
                rz = new
            v += e
        return v[:-12].reshape(shape) + amb, v[-12:] + amb

    def steady_rows(self, P, amb):
        """Block elimination over the rows of the grid (channels run along
        the rows, so the system is not symmetric), the package as a border."""
        nl, nr, nc = P.shape
        m = nl * nc
        zero = torch.zeros_like(P)
        x0 = torch.zeros(12, dtype=torch.float64, device=self.dev)
        b0, p0 = self.flow(torch.zeros_like(P), x0, amb)      # what ambient and the inlet bring in
        self_in = self.t_in
        # border columns: the effect of each package node
        cols, pcols = [], []
        for k in range(12):
            e = x0.clone()
            e[k] = 1.0
            self.t_in = 0.0
            q, px = self.flow(zero, e, 0.0)
            cols.append(q)
            pcols.append(px)
        self.t_in = self_in
        F = self.adv
        low = torch.zeros((nr, m), dtype=torch.float64, device=self.dev)
        upp = torch.zeros_like(low)
        gS, f = self.gS.transpose(0, 1).reshape(nr - 1, m), F.transpose(0, 1).reshape(nr, m)
        low[1:] = -gS - f[1:] / 2
        upp[:-1] = -gS + f[:-1] / 2
        D = torch.zeros((nl, nr, nc), dtype=torch.float64, device=self.dev)
        D[:, :, :-1] += self.gE
        D[:, :, 1:] += self.gE
        D[:, :-1] += self.gS + F[:, :-1] / 2
        D[:, 1:] += self.gS - F[:, 1:] / 2
        D[:, -1] += F[:, -1]
        D[:-1] += self.gB
        D[1:] += self.gB
        D[-1] += self.g_amb
        for n, k, gn, ge in self.edge:
            D[n, 0] += gn
            D[n, -1] += gn
            D[n, :, 0] += ge
            D[n, :, -1] += ge
        rhs = torch.stack([P + b0] + cols, -1).permute(1, 0, 2, 3).reshape(nr, m, 13)
        inv, y = [], []
        at = torch.arange(m, device=self.dev).reshape(nl, nc)
        for i in range(nr):
            A = torch.diag(D[:, i].reshape(-1))
            A[at[:, :-1], at[:, 1:]] = -self.gE[:, i]
            A[at[:, 1:], at[:, :-1]] = -self.gE[:, i]
            A[at[:-1], at[1:]] = -self.gB[:, i]
            A[at[1:], at[:-1]] = -self.gB[:, i]
            r = rhs[i]
            if i:
                A -= low[i][:, None] * inv[-1] * upp[i - 1][None, :]
                r = r - low[i][:, None] * y[-1]
            inv.append(torch.linalg.inv(A))
            y.append(inv[-1] @ r)
        for i in range(nr - 2, -1, -1):
            y[i] = y[i] - inv[i] @ (upp[i][:, None] * y[i + 1])
        S = torch.stack(y).reshape(nr, nl, nc, 13).permute(1, 0, 2, 3)
        # package rows: pcols x + (effect of the cells) + p0 = 0
        E = torch.zeros((12, 13), dtype=torch.float64, device=self.dev)
        for c in range(13):
            self.t_in = 0.0
            E[:, c] = self.flow(S[..., c].contiguous(), x0, 0.0)[1]
        self.t_in = self_in
        x = torch.linalg.solve(torch.stack(pcols, 1) + E[:, 1:], -(p0 + E[:, 0]))
        return S[..., 0] + S[..., 1:] @ x, x


def _grid_of(case, seed, which, dev):
    """(network, power rows as lists of one value per unit and layer)."""
    if case["kind"].startswith("uchan"):
        with tempfile.TemporaryDirectory() as d:
            sc, rows = _uchan(case, seed, d)
        side, die = case["rows"], case["die_mm"] * 1e-3
        cw, n = die / side, int(round(math.sqrt(case["blocks"])))
        fluid = np.fmod((np.arange(side) + 0.5) * cw, 200e-6) < 100e-6
        # W/m^3/K times the flow of one lane of cells, laminar in a 200 um tall duct
        hc = (1 - 0.63 * (cw / 200e-6)) * cw ** 3 * 200e-6 / (12 * 0.000889 * cw)
        flow = 4172638.0 * hc * float(sc.config["pumping_pressure"]) / (side - 1)
        # the channel layer's floorplan is one unit per cell, written with "%e"
        e7 = lambda v: float("%e" % v)  # noqa: E731
        cells = [W.Unit("", cw, cw, j * cw, die - (i + 1) * cw) for i in range(side) for j in range(side)]
        stack = [(True, 1.75e6, 0.01, 1e-4, W.uniform_tiling(die, die, n, n)),
                 (False, 1.75e6, 0.01, 200e-6, cells[:1])]
        net = _Grid(side, side, die, stack, dev,
                    {"layer": 1, "fluid": fluid, "r_fluid": e7(1 / 0.6069), "r_wall": e7(0.0076923077),
                     "c_fluid": e7(4172638.0), "c_wall": e7(1635660.0), "htc": 27132.0, "heat_flow": flow})
        net.per_cell = True
        return net, [[torch.tensor(r, device=dev)] for r in rows]
    side, stack, rows = _stack(case, seed, which)
    net = _Grid(side[0], side[1], case["die_mm"] * 1e-3, stack, dev)
    net.per_cell = False
    out = []
    for r in rows:
        v, k = [], 0
        for s in stack + [(False, 0, 0, 0, stack[-1][4])] * 2:
            n = len(s[4])
            v.append(torch.tensor(r[k:k + n] if s[0] else np.zeros(n), device=dev))
            k += n if s[0] else 0
        out.append(v)
    return net, out


def _power(net, row):
    if not net.per_cell:
        return net.to_grid(row, True)
    P = torch.zeros((net.nl, net.nr, net.nc), dtype=torch.float64, device=net.dev)
    oh, ow, area, _ = net.maps[0]
    P[0] = (oh * (row[0] / area * net.cell_area)[:, None]).T @ ow
    return P


def _blocks(net, T, x, mode):
    if not net.per_cell:
        return net.to_blocks(T, x, mode)
    keep, net.maps = net.maps, net.maps[:1]
    first = net.to_blocks(T, x, mode)[:-12]
    net.maps = keep
    return np.concatenate([first, T[1:].reshape(-1).cpu().numpy(), x.cpu().numpy()])


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    amb, init, kind = 318.15, 333.15, case["kind"]
    outs = []
    for c in range(case["chips"]):
        net, rows = _grid_of(case, seed, c, dev)
        if "steady" in kind:
            P = _power(net, rows[0])
            T, x = net.steady_rows(P, amb) if kind == "uchan_steady" else net.steady(P, amb)
            out = _blocks(net, T, x, case["map"])
            if case["form"] == "parity":
                return {"block": out, "grid": np.concatenate([T.reshape(-1).cpu().numpy(), x.cpu().numpy()])}
            return out
        if net.per_cell or kind == "batch":
            T = torch.full((net.nl, net.nr, net.nc), init, dtype=torch.float64, device=dev)
        else:
            T = net.to_grid([torch.full((len(u),), init, dtype=torch.float64, device=dev) for u in net.units], False)
        x = torch.full((12,), init, dtype=torch.float64, device=dev)
        for k in range(case["intervals"]):
            T, x = net.interval(T, x, _power(net, rows[k]), case["dt"], amb)
        if kind != "batch":
            return _blocks(net, T, x, case["map"])
        outs.append(np.concatenate([T.reshape(-1).cpu().numpy(), x.cpu().numpy()]))
    return outs
