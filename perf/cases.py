"""The work a user of this engine has it do, as measurable cases.

A case is a plain dict; `prepare` makes what a user's program holds before the
call (problem set up on the GPU, probes, network, traces), `run` is one pass
through the public entry points, `work` counts what a pass cannot do without
and `exact` restates the result in plain FP64 torch.

Kinds of case:

  solve      one whole `B200Backend.run(problem)` of the backend contract:
             set-up, every step, a snapshot every 50 steps, then the fields,
             ports and far field are read back.
  step       `Engine.run(steps)` on a problem already on the GPU, then the port
             traces and the far field are read, as a program does between
             checkpoints and at the end of a run.
  batch      `Batch.run(steps)` on a sweep of antennas, then every member's
             port traces and the far field of the first are read.
  pattern    `Engine.farfield_post`: power and directivity from the far-field sums.
  train      `EsNet.loss_grad`: loss and gradients of one minibatch.
  port       `postproc.port_s11`: S11 and Zin from one port's traces.

Each seed has its own material (and blocks, weights or traces); the grids and
counts are the case's, so every seed of a case costs the same.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """This repository's package (its folder's name is not an identifier)."""
    name = "special_topics_b200"
    if name not in sys.modules:
        d = os.path.join(os.getcwd(), "special-topics_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules[name] = m
        spec.loader.exec_module(m)
    return sys.modules[name]


def _mod(name):
    _package()
    return importlib.import_module("special_topics_b200." + name)


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed() -> list:
    return [
        # S11 and Zin of one port after a 7000-step run on the scenarios' 500-point frequency grid: the
        # smallest call, made once per antenna of a sweep
        {"name": "port-s11-7000x500", "kind": "port", "samples": 7000, "freqs": 500},
        # a small problem through the backend contract in FP64, host-built coefficient arrays: set-up,
        # launch latency and snapshots count as much as the kernels
        {"name": "solve-64-f64", "kind": "solve", "scene": "box", "nx": 64, "ny": 64, "nz": 64,
         "precision": "f64", "host": True, "steps": 300},
        # the reference's antenna on 0.5 mm cells in FP64, its drop-in precision, with uploaded arrays
        {"name": "ifa-0p5mm-f64", "kind": "step", "scene": "ifa-0.5mm", "precision": "f64", "host": True,
         "steps": 500, "warm": 200, "block": 0, "cuts": False},
        # the same antenna in FP32 with material tables: a design loop's everyday run
        {"name": "ifa-0p5mm-table", "kind": "step", "scene": "ifa-0.5mm", "precision": "f32-table", "host": False,
         "steps": 500, "warm": 200, "block": 0, "cuts": False},
        # 0.25 mm cells, 64 far-field frequencies, time-blocked surface sums, pattern cuts at the end
        {"name": "ifa-0p25mm-table-64f", "kind": "step", "scene": "ifa-0.25mm", "precision": "f32-table",
         "host": False, "steps": 320, "warm": 400, "block": 16, "cuts": True},
        # per-cell FP32 arrays (the reference's own GPU precision) on an odd-sized box
        {"name": "box-97x131x118-f32", "kind": "step", "scene": "box", "nx": 97, "ny": 131, "nz": 118,
         "precision": "f32", "host": True, "steps": 400, "warm": 200, "block": 0, "cuts": False},
        # FP64 larger than the caches, coefficients built on the device
        {"name": "box-256-f64", "kind": "step", "scene": "box", "nx": 256, "ny": 256, "nz": 256,
         "precision": "f64", "host": False, "steps": 160, "warm": 320, "block": 0, "cuts": False},
        # the largest: the benchmark's headline box
        {"name": "box-512x512x640-table", "kind": "step", "scene": "box", "nx": 512, "ny": 512, "nz": 640,
         "precision": "f32-table", "host": False, "steps": 128, "warm": 640, "block": 16, "cuts": False},
        # a sweep of antennas on uneven grids advanced together
        {"name": "batch-32-spread-table", "kind": "batch", "first": 40000, "members": 32, "spread": True,
         "precision": "f32-table", "steps": 160, "warm": 160, "block": 16},
        # the FP64 reference runs of a sweep
        {"name": "batch-6-f64", "kind": "batch", "first": 41000, "members": 6, "spread": False,
         "precision": "f64", "steps": 160, "warm": 160, "block": 0},
        # radiated power and directivity on a 2-degree grid from the far-field sums of a run
        {"name": "pattern-2deg-12f", "kind": "pattern", "freqs": 12, "degrees": 2.0, "warm": 600},
        # one minibatch of the early-stop network's training, forward and backward
        {"name": "train-256", "kind": "train", "batch": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("port", "solve", "antenna", "box", "box", "box", "batch", "batch", "pattern", "train"))
    if kind == "port":
        return {"kind": "port", "samples": _log(rng, 200, 20000), "freqs": _log(rng, 16, 2000)}
    if kind == "train":
        return {"kind": "train", "batch": _log(rng, 16, 512)}
    if kind == "pattern":
        return {"kind": "pattern", "freqs": rng.randint(1, 12), "degrees": rng.choice((2.0, 3.0, 5.0)),
                "warm": rng.randint(300, 700)}
    prec = rng.choice(("f64", "f32-table", "f32-table", "f32"))
    if kind == "antenna":
        return {"kind": "step", "scene": "variant", "first": rng.randint(0, 9999), "spread": rng.random() < 0.5,
                "precision": prec, "host": prec == "f32" or rng.random() < 0.3, "steps": rng.randint(100, 400),
                "warm": rng.randint(150, 300), "block": rng.choice((0, 16)) if prec != "f64" else 0, "cuts": False}
    if kind == "batch":
        prec = rng.choice(("f64", "f32-table", "f32-table"))
        return {"kind": "batch", "first": rng.randint(0, 9999), "members": _log(rng, 2, 6 if prec == "f64" else 32),
                "spread": rng.random() < 0.5, "precision": prec, "steps": rng.randint(60, 160), "warm": 160,
                "block": rng.choice((0, 16)) if prec != "f64" else 0}
    top = 96 if kind == "solve" else 180 if prec == "f32" else 280 if prec == "f64" else 400
    n = [_log(rng, 64, top) for _ in range(3)]
    case = {"kind": kind, "scene": "box", "nx": n[0], "ny": n[1], "nz": n[2], "precision": prec,
            "host": prec == "f32" or (kind == "solve" and prec == "f64")}
    if kind == "solve":
        return dict(case, steps=rng.randint(60, 300))
    return dict(case, kind="step", steps=max(40, min(400, 2_000_000_000 // (n[0] * n[1] * n[2]))), warm=80 + max(n),
                block=rng.choice((0, 16)) if prec != "f64" else 0, cuts=False)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _total_steps(case) -> int:
    """numberOfTimeSteps of a problem whose passes advance it: room for many of them."""
    if case["kind"] == "solve":
        return case["steps"]
    if case["kind"] == "pattern":
        return case["warm"]
    big = case["kind"] == "batch" or case["scene"] in ("box", "ifa-0.25mm")
    return case["warm"] + case["steps"] * (160 if big else 500)


def _scenario(case, seed, member=0) -> dict:
    W = _mod("workloads")
    rng = np.random.default_rng([seed, member, 77])
    scene = case.get("scene", "variant")
    steps = _total_steps(case)
    if case["kind"] == "pattern":
        scn = W.ifa_config0(steps)
        scn["farfield"]["frequencies"] = list(np.linspace(1e9, 4e9, case["freqs"]))
    elif scene == "box":
        return W.scaling_box((case["nx"], case["ny"], case["nz"]), seed=seed, steps=steps)
    elif scene == "ifa-0.5mm":
        scn = W.ifa_config0(steps)
    elif scene == "ifa-0.25mm":
        scn = W.ifa_config2(steps)
    else:
        scn = W.ifa_variant(case["first"] + member, steps=steps, spread=case["spread"])
    scn["materialTypes"][2]["eps_r"] = float(rng.uniform(2.2, 6.15))    # this seed's substrate
    return scn


def _problem(case, seed, member=0):
    return _package().build_problem_from_scenario(_scenario(case, seed, member), _total_steps(case),
                                                  per_cell=bool(case.get("host")))


def _engine(case, seed, member=0):
    return _mod("backend").Engine(_problem(case, seed, member), case.get("precision", "f64"),
                                  dft_block=case.get("block", 0))


def _ringing(rng, samples, dt):
    """A port transient: the pulse and two damped resonances."""
    t = np.arange(samples) * dt
    t0 = 0.08 * samples * dt
    x = np.exp(-((t - t0) / (0.25 * t0)) ** 2)
    for _ in range(2):
        f, a = rng.uniform(1.5e9, 3.5e9), rng.uniform(0.3e9, 1.5e9)
        on = t > t0
        x = x + rng.uniform(0.1, 0.5) * np.where(on, np.exp(-a * (t - t0)) * np.sin(2 * np.pi * f * (t - t0)), 0.0)
    return x


def _port_inputs(case, seed):
    rng = np.random.default_rng(seed)
    dt = 8.66e-13
    V, I = _ringing(rng, case["samples"], dt), 0.02 * _ringing(rng, case["samples"], dt)
    return V, I, dt, (1 + np.arange(case["freqs"])) * (10e9 / case["freqs"])


def _train_inputs(case, seed):
    """Inputs as earlystop makes them (each channel scaled to 1), standardised targets, weights."""
    ES = _mod("earlystop")
    rng = np.random.default_rng(seed)
    L, D, B = ES.ARCH["in_length"], 4, case["batch"]
    x = np.stack([np.stack([_ringing(rng, L, 3.46e-12) for _ in range(2)], axis=1) for _ in range(B)])
    x = (x / np.abs(x).max(axis=1, keepdims=True)).astype(np.float32)
    params = []
    cin = ES.ARCH["in_channels"]
    ch, k, n = ES.ARCH["channels"], ES.ARCH["kernel"], L
    for _ in range(ES.ARCH["conv_layers"]):
        params += [rng.uniform(-1, 1, ch * k * cin) / math.sqrt(k * cin), rng.uniform(-1, 1, ch) / math.sqrt(k * cin)]
        cin, n = ch, (n + 2 * (k // 2) - k) // ES.ARCH["stride"] + 1
    feat = n * ch
    for o in [ES.ARCH["mlp_width"]] * ES.ARCH["mlp_layers"] + [D]:
        params += [rng.uniform(-1, 1, o * feat) / math.sqrt(feat), rng.uniform(-1, 1, o) / math.sqrt(feat)]
        feat = o
    return x, rng.standard_normal((B, D)).astype(np.float32), np.concatenate(params).astype(np.float32), D


def _angles(degrees):
    th = np.radians(np.arange(0, 181, degrees))
    ph = np.radians(np.arange(0, 360, degrees))
    T, P = np.meshgrid(th, ph, indexing="ij")
    return T.ravel(), P.ravel()


def _cuts():
    angles, th_xy, th_xz, ph_xz = _mod("postproc").cut_angles()
    return np.concatenate([th_xy, th_xz]), np.concatenate([angles, ph_xz])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "port":
        return {"kind": kind, "in": _port_inputs(case, seed)}
    if kind == "train":
        x, t, params, D = _train_inputs(case, seed)
        net = _mod("earlystop").EsNet(out_dim=D, max_batch=512)
        net.params = params
        return {"kind": kind, "net": net, "x": x, "t": t}
    if kind == "solve":
        return {"kind": kind, "problem": _problem(case, seed), "precision": case["precision"]}
    if kind == "pattern":
        eng = _engine(case, seed)
        eng.run(case["warm"])
        return {"kind": kind, "engine": eng, "angles": _angles(case["degrees"])}
    if kind == "batch":
        engs = [_engine(case, seed, m) for m in range(case["members"])]
        b = _mod("backend").Batch(engs)
        b.run(case["warm"])
        return {"kind": kind, "batch": b, "engines": engs, "steps": case["steps"]}
    eng = _engine(case, seed)
    eng.run(case["warm"])                  # the pulse is in the box
    return {"kind": kind, "engine": eng, "steps": case["steps"], "angles": _cuts() if case["cuts"] else None}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
FIELDS = ("Hx", "Hy", "Hz", "Ex", "Ey", "Ez")


def run(state):
    kind = state["kind"]
    if kind == "port":
        return _mod("postproc").port_s11(*state["in"])
    if kind == "train":
        loss, grad = state["net"].loss_grad(state["x"], state["t"])
        return {"loss": loss, "grad": grad}
    if kind == "pattern":
        return list(state["engine"].farfield_post(*state["angles"]))
    if kind == "solve":
        be = _mod("backend").B200Backend(state["precision"])
        snapshots = [s["voltage"] for s in be.run(state["problem"])]
        eng = be.engine
        out = {"snapshots": np.array(snapshots), "V": eng.voltages()[0], "I": eng.currents()[0],
               "far": eng.farfield(), "fields": [eng.field(f) for f in FIELDS]}
        eng.close()
        return out
    if kind == "batch":
        state["batch"].run(state["steps"])
        engs = state["engines"]
        return {"V": [np.concatenate([e.voltages()[0] for e in engs])],
                "I": [np.concatenate([e.currents()[0] for e in engs])], "far": engs[0].farfield()}
    eng = state["engine"]
    eng.run(state["steps"])
    far = eng.farfield() if state["angles"] is None else list(eng.farfield_post(*state["angles"]))
    return {"V": eng.voltages()[0], "I": eng.currents()[0], "far": far}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
_EXTENT: dict = {}


def _extent(case, member=0):
    """(nx, ny, nz, CPML cells, far-field frequencies, Huygens box margin) of a problem."""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name")) + str(member)
    if key not in _EXTENT:
        S = _mod("scenario")
        scn = _scenario(case, 0, member)
        c = scn["cell"]
        g = S.build_grid(c["dx"], c["dy"], c["dz"], scn["boundary"], scn["bricks"], [], 0.9, 1)
        _EXTENT[key] = (g.nx, g.ny, g.nz, scn["boundary"]["cpml_cells_xn"], len(scn["farfield"]["frequencies"]),
                        scn["farfield"]["number_of_cells_from_outer_boundary"])
    return _EXTENT[key]


def _surface(nx, ny, nz, off):
    """Point pairs on the Huygens box."""
    a, b, c = nx - 2 * off, ny - 2 * off, nz - 2 * off
    return a * b + b * c + a * c


def _step_work(case, member=0):
    """Bytes and operations of one step: every field and Psi value read and written once, one byte that
    names each value's material, and the surface sums read and written once a step (once a block when
    they are time-blocked)."""
    nx, ny, nz, nc, nf, off = _extent(case, member)
    cells = nx * ny * nz
    size = 8 if case.get("precision", "f64") == "f64" else 4
    psi = 2 * 4 * nc * (nx * ny + ny * nz + nx * nz)
    pts = _surface(nx, ny, nz, off) * nf
    block = max(1, case.get("block", 0))
    return (cells * 6 * (2 * size + 1) + psi * 2 * size + pts * 8 * 16 * 2 / block,
            cells * 6 * 7 + psi * 5 + pts * 8 * 4)


def work(case) -> dict:
    kind = case["kind"]
    if kind == "port":
        n, m = case["samples"], case["freqs"]
        return {"bytes": 2 * 8 * n + 8 * m + 8 * 6 * m, "flops": 2 * n * m * 8}
    if kind == "train":
        ES = _mod("earlystop").ARCH
        n, cin, macs, params = ES["in_length"], ES["in_channels"], 0, 0
        for _ in range(ES["conv_layers"]):
            n = (n + 2 * (ES["kernel"] // 2) - ES["kernel"]) // ES["stride"] + 1
            macs += n * ES["channels"] * ES["kernel"] * cin
            params += ES["channels"] * (ES["kernel"] * cin + 1)
            cin = ES["channels"]
        feat = n * cin
        for o in [ES["mlp_width"]] * ES["mlp_layers"] + [4]:
            macs += feat * o
            params += o * (feat + 1)
            feat = o
        return {"bytes": params * 6 + case["batch"] * 4 * (ES["in_length"] * ES["in_channels"] + 4),
                "flops": 6 * macs * case["batch"]}
    if kind == "pattern":
        nx, ny, nz, _, nf, off = _extent(case)
        pts = 2 * _surface(nx, ny, nz, off)
        ang = _angles(case["degrees"])[0].size
        return {"bytes": nf * (pts * 4 * 16 + ang * 16) + 16 * ang, "flops": float(nf) * pts * ang * 38}
    if kind == "batch":
        per = [_step_work(case, m) for m in range(case["members"])]
        return {"bytes": case["steps"] * sum(p[0] for p in per), "flops": case["steps"] * sum(p[1] for p in per)}
    b, f = _step_work(case)
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


# ---------------------------------------------------------------------------
# The same results in plain FP64 torch
# ---------------------------------------------------------------------------
EPS0, MU0, C0, ETA0 = 8.854187817e-12, 4 * math.pi * 1e-7, 2.99792458e8, 376.73031346177066
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=_DEV).to(dtype)


class _Fdtd:
    """The Yee loop with CPML on a problem's material grid, profiles, source, probes and far-field box.
    Component order Hx Hy Hz Ex Ey Ez; component (h, a) has its curl over the axes b = a + 1, c = a + 2."""

    def __init__(self, p, wall):
        g = self.g = p.grid
        self.p, self.wall = p, wall
        self.n = n = (g.nx, g.ny, g.nz)
        self.d = d = (g.dx, g.dy, g.dz)
        mat = _t(p.meta["material_grid"], torch.int64)
        eps, mu, se, sm = (_t(p.meta["material_props"][:, c]) for c in range(4))
        self.H = [torch.zeros([n[q] + (q == a) for q in range(3)], dtype=torch.float64, device=_DEV) for a in range(3)]
        self.E = [torch.zeros([n[q] + (q != a) for q in range(3)], dtype=torch.float64, device=_DEV) for a in range(3)]
        self.cE, self.cH = [], []      # per axis: self, and the coefficient of the difference along b and along c
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3
            # E: mean of the four cells around an edge, away from the outer walls
            e, s = torch.ones_like(self.E[a]), torch.zeros_like(self.E[a])
            inner = tuple(slice(None) if q == a else slice(1, n[q]) for q in range(3))
            e[inner] = s[inner] = 0
            for sb in (0, 1):
                for sc in (0, 1):
                    sl = [slice(None)] * 3
                    sl[b], sl[c] = slice(sb, n[b] - 1 + sb), slice(sc, n[c] - 1 + sc)
                    m = mat[tuple(sl)]
                    e[inner] += 0.25 * eps[m]
                    s[inner] += 0.25 * se[m]
            for comp, i0, i1, j0, j1, k0, k1, sigma in p.meta["plates"]:
                if comp == a:
                    s[i0:i1 + 1, j0:j1 + 1, k0:k1 + 1] = sigma
            den = 2 * EPS0 * e + g.dt * s
            self.cE.append([(2 * EPS0 * e - g.dt * s) / den, 2 * g.dt / d[b] / den, -2 * g.dt / d[c] / den])
            # H: harmonic mean of the two cells beside a face
            m1, s1 = torch.ones_like(self.H[a]), torch.zeros_like(self.H[a])
            inner = tuple(slice(1, n[q]) if q == a else slice(None) for q in range(3))
            lo, hi = ([slice(None)] * 3 for _ in range(2))
            lo[a], hi[a] = slice(0, n[a] - 1), slice(1, n[a])
            u, v = mat[tuple(hi)], mat[tuple(lo)]
            m1[inner] = 2 * mu[u] * mu[v] / (mu[u] + mu[v])
            s1[inner] = 2 * sm[u] * sm[v] / (sm[u] + sm[v])
            den = 2 * MU0 * m1 + g.dt * s1
            self.cH.append([(2 * MU0 * m1 - g.dt * s1) / den, -2 * g.dt / d[b] / den, 2 * g.dt / d[c] / den])
        for v in p.voltage_sources:
            for w, col in ((0, 0), (1, 1), (2, 2)):
                self.cE[v.axis][w].view(-1)[_t(v.field_indices, torch.int64)] = _t(v.override[:, col])
        # CPML: (field, component, axis of the difference) -> band, profile, CPsi, Psi
        self.bands = {"E": [], "H": []}
        for fid, f in enumerate(p.cpml):
            if f is None or f.nc == 0:
                continue
            ax = fid // 2
            for kind, cs, start, pb, pa, kap in (("H", self.cH, f.m_start, f.b_m, f.a_m, f.kappa_m),
                                                 ("E", self.cE, f.e_start, f.b_e, f.a_e, f.kappa_e)):
                shape = [1, 1, 1]
                shape[ax] = f.nc
                pb, pa, kap = (_t(x).reshape(shape) for x in (pb, pa, kap))
                for a in range(3):
                    if a == ax:
                        continue
                    w = 1 if (a + 1) % 3 == ax else 2
                    sl = [slice(None)] * 3
                    sl[ax] = slice(start, start + f.nc)
                    sl = tuple(sl)
                    cp = cs[a][w][sl] * self.d[ax]
                    cs[a][w][sl] /= kap
                    self.bands[kind].append((a, w, sl, pb, pa, cp, torch.zeros_like(cp)))
        self.src = [(v.axis, _t(v.field_indices, torch.int64), _t(v.coef), v.voltage_per_e_field)
                    for v in p.voltage_sources]
        self.vp = [(q.axis, _t(q.field_indices, torch.int64), q.Csvf) for q in p.sampled_voltages]
        self.ip = [(_t(q.comp, torch.int64), _t(q.idx, torch.int64), _t(q.w)) for q in p.sampled_currents]
        self.ts, self.V, self.I = 0, [], []
        ff = self.ff = p.farfield
        self.lo, self.up = (ff.li - 1, ff.lj - 1, ff.lk - 1), (ff.ui - 1, ff.uj - 1, ff.uk - 1)
        self.acc, self.held = {}, []

    def step(self):
        H, E, n = self.H, self.E, self.n
        diffs = {}
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3
            diffs[a] = (None, torch.diff(E[c], dim=b), torch.diff(E[b], dim=c))
            H[a].mul_(self.cH[a][0]).addcmul_(self.cH[a][1], diffs[a][1]).addcmul_(self.cH[a][2], diffs[a][2])
        for a, w, sl, pb, pa, cp, psi in self.bands["H"]:
            psi.mul_(pb).addcmul_(pa, diffs[a][w][sl])
            H[a][sl].addcmul_(cp, psi)
        if self.ip:
            comp, idx, w = self.ip[0]
            flat = torch.stack([torch.take(H[q], idx.clamp(max=H[q].numel() - 1)) for q in range(3)])
            self.I.append((w * flat[comp, torch.arange(idx.numel(), device=_DEV)]).sum())
        # E: differences of H padded with zeros at the walls, where only the CPML reads them.  Without the
        # wall, Hz and Hy one plane past x = max are Ex(i=0) after its bulk update and the start of Hz.
        def pad_diff(x, ax):
            out = torch.zeros([s + (q == ax) for q, s in enumerate(x.shape)], dtype=x.dtype, device=_DEV)
            inner = [slice(None)] * 3
            inner[ax] = slice(1, x.shape[ax])
            out[tuple(inner)] = torch.diff(x, dim=ax)
            return out
        diffs = {a: (None, pad_diff(H[(a + 2) % 3], (a + 1) % 3), pad_diff(H[(a + 1) % 3], (a + 2) % 3))
                 for a in range(3)}
        old = [E[1][n[0]].clone(), E[2][n[0]].clone()]
        inner = (slice(None), slice(1, n[1]), slice(1, n[2]))
        E[0][inner] = (self.cE[0][0][inner] * E[0][inner] + self.cE[0][1][inner] * diffs[0][1][inner]
                       + self.cE[0][2][inner] * diffs[0][2][inner])
        top = n[0] if self.wall else n[0] + 1
        if not self.wall:
            diffs[1][2][n[0]] = E[0][0, :n[1]] - H[2][n[0] - 1]
            diffs[2][1][n[0]] = H[2].reshape(-1)[:(n[1] + 1) * n[2]].reshape(n[1] + 1, n[2]) - H[1][n[0] - 1]
        for a, sl in ((1, (slice(1, top), slice(None), slice(1, n[2]))), (2, (slice(1, top), slice(1, n[1]), slice(None)))):
            E[a][sl] = (self.cE[a][0][sl] * E[a][sl] + self.cE[a][1][sl] * diffs[a][1][sl]
                        + self.cE[a][2][sl] * diffs[a][2][sl])
        for a, w, sl, pb, pa, cp, psi in self.bands["E"]:
            psi.mul_(pb).addcmul_(pa, diffs[a][w][sl])
            E[a][sl].addcmul_(cp, psi)
        if self.wall:
            E[1][n[0]], E[2][n[0]] = old[0], old[1]
        for axis, idx, cs, wave in self.src:
            E[axis].view(-1)[idx] += cs * float(wave[self.ts])
        if self.vp:
            axis, idx, csvf = self.vp[0]
            self.V.append(csvf * torch.take(E[axis], idx).sum())
        self.surface()
        self.ts += 1

    def surface(self):
        """Tangential field averages on the six faces; every 64 steps they enter the running sums."""
        H, E, lo, up = self.H, self.E, self.lo, self.up
        out = {}
        for a, nm in enumerate("xyz"):
            b, c = sorted(q for q in range(3) if q != a)
            for side, at, sg in (("p", up[a], 1.0), ("n", lo[a], -1.0)):
                def e_avg(t, other):    # E along t, averaged over its two edges in the other tangential axis
                    sl = [slice(lo[q], up[q]) for q in range(3)]
                    sl[a] = at
                    s2 = list(sl)
                    s2[other] = slice(lo[other] + 1, up[other] + 1)
                    return 0.5 * (E[t][tuple(sl)] + E[t][tuple(s2)])

                def h_avg(t, other):    # H along t, averaged over both planes beside the face and along t
                    tot = 0
                    for pl in (at, at - 1):
                        for s in (0, 1):
                            sl = [slice(lo[q], up[q]) for q in range(3)]
                            sl[a], sl[t] = pl, slice(lo[t] + s, up[t] + s)
                            tot = tot + H[t][tuple(sl)]
                    return 0.25 * tot
                if a == 0:
                    v = {"cmy": sg * e_avg(2, 1), "cmz": -sg * e_avg(1, 2), "cjy": -sg * h_avg(2, 1), "cjz": sg * h_avg(1, 2)}
                elif a == 1:
                    v = {"cmx": -sg * e_avg(2, 0), "cmz": sg * e_avg(0, 2), "cjz": -sg * h_avg(0, 2), "cjx": sg * h_avg(2, 0)}
                else:
                    v = {"cmx": sg * e_avg(1, 0), "cmy": -sg * e_avg(0, 1), "cjx": -sg * h_avg(1, 0), "cjy": sg * h_avg(0, 1)}
                    if side == "p":
                        v["cjx"] = -h_avg(1, 0)
                        v["cjy"] = h_avg(0, 1)
                out.update({k + nm + side: x.reshape(-1) for k, x in v.items()})
        self.held.append(out)
        if len(self.held) == 64:
            self.flush()

    def flush(self):
        if not self.held:
            return
        t = np.arange(self.ts + 1 - len(self.held), self.ts + 1) if len(self.held) == 64 else \
            np.arange(self.ts - len(self.held), self.ts)
        w = 2 * math.pi * np.asarray(self.ff.frequencies)[:, None] * self.g.dt
        ph = {"cj": _t(w * (t + 0.5)), "cm": _t(w * (t + 1))}
        for k in self.held[0]:
            s = torch.stack([h[k] for h in self.held])
            re, im = torch.cos(ph[k[:2]]) @ s, -torch.sin(ph[k[:2]]) @ s
            if k in self.acc:
                self.acc[k][0].add_(re)
                self.acc[k][1].add_(im)
            else:
                self.acc[k] = [re, im]
        self.held = []

    def advance(self, steps):
        for _ in range(steps):
            self.step()
        self.flush()
        return self

    def ports(self):
        return torch.stack(self.V), torch.stack(self.I)

    def far(self):
        return {k: (v[0].reshape(-1), v[1].reshape(-1)) for k, v in self.acc.items()}

    def pattern(self, theta, phi):
        """Radiated power and directivity of every frequency."""
        lo, up, d = self.lo, self.up, self.d
        th, ph = _t(theta), _t(phi)
        st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
        u = (st * cp, st * sp, ct)
        th_hat, ph_hat = (ct * cp, ct * sp, -st), (-sp, cp, torch.zeros_like(st))
        A = {k: torch.complex(v[0], v[1]) for k, v in self.acc.items()}
        radp, dth, dph = [], [], []
        for f, freq in enumerate(self.ff.frequencies):
            k = 2 * math.pi * float(freq) / C0
            power = 0.0
            N = [torch.zeros(th.shape, dtype=torch.complex128, device=_DEV) for _ in range(4)]
            for a, nm in enumerate("xyz"):
                b, c = sorted(q for q in range(3) if q != a)
                area = d[b] * d[c]
                centre = [0.5 * (up[q] + lo[q]) for q in range(3)]
                # the reference counts the points from one cell below the faces' origin
                pos = [(torch.arange(lo[q], up[q], device=_DEV, dtype=torch.float64) - 0.5 - centre[q]) * d[q] for q in range(3)]
                for side, at, sg in (("p", up[a], 1), ("n", lo[a], -1)):
                    get = lambda s, q: A[s + "xyz"[q] + nm + side][f].reshape(up[b] - lo[b], up[c] - lo[c])  # noqa: E731
                    J, M = {q: get("cj", q) for q in (b, c)}, {q: get("cm", q) for q in (b, c)}
                    q1, q2 = {0: (2, 1), 1: (0, 2), 2: (1, 0)}[a]
                    power = power + sg * area * ((M[q1] * J[q2].conj()).real - (M[q2] * J[q1].conj()).real).sum()
                    e0 = torch.exp(1j * k * (at - centre[a]) * d[a] * u[a])
                    eb = torch.exp(1j * k * u[b][:, None] * pos[b][None, :])
                    ec = torch.exp(1j * k * u[c][:, None] * pos[c][None, :])
                    for q in (b, c):
                        for X, at_ in ((J, 0), (M, 2)):
                            s = area * e0 * ((eb @ X[q]) * ec).sum(1)
                            N[at_] = N[at_] + th_hat[q] * s
                            N[at_ + 1] = N[at_ + 1] + ph_hat[q] * s
            power = 0.5 * power
            scale = k * k / (8 * math.pi * ETA0 * power)
            radp.append(power)
            dth.append(scale * (N[3] + ETA0 * N[0]).abs() ** 2)
            dph.append(scale * (N[2] - ETA0 * N[1]).abs() ** 2)
        return [torch.stack(radp), torch.stack(dth), torch.stack(dph)]


def _exact_port(case, seed):
    V, I, dt, freqs = _port_inputs(case, seed)
    n = torch.arange(1, V.size + 1, dtype=torch.float64, device=_DEV)
    w = 2 * math.pi * _t(freqs)[:, None]

    def spectrum(x, shift):
        a = w * (n[None, :] * dt + shift)
        return dt * torch.complex(torch.cos(a) @ _t(x), -(torch.sin(a) @ _t(x)))
    v, i = spectrum(V, 0.0), spectrum(I, -dt / 2)
    a, b = 0.5 * (v + 50.0 * i), 0.5 * (v - 50.0 * i)
    s = b / a
    return {"re": s.real, "im": s.imag, "mag_dB": 20 * torch.log10(s.abs()), "phase_deg": torch.angle(s) * 180 / math.pi,
            "zin": v / i}


def _exact_train(case, seed):
    arch = _mod("earlystop").ARCH
    x, target, params, D = _train_inputs(case, seed)
    # the network computes with BF16 copies of its weights and FP32 biases
    parts, at = [], 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        v = torch.as_tensor(params[at:at + n].copy(), device=_DEV)
        at += n
        v = (v.to(torch.bfloat16) if len(shape) > 1 else v).double().reshape(shape).requires_grad_(True)
        parts.append(v)
        return v
    h, cin = _t(x).transpose(1, 2), arch["in_channels"]
    for _ in range(arch["conv_layers"]):
        w = take(arch["channels"], arch["kernel"], cin)
        h = torch.relu(torch.nn.functional.conv1d(h, w.transpose(1, 2), take(arch["channels"]), stride=arch["stride"],
                                                  padding=arch["kernel"] // 2))
        cin = arch["channels"]
    h = h.transpose(1, 2).reshape(x.shape[0], -1)
    for layer in range(arch["mlp_layers"] + 1):
        o = arch["mlp_width"] if layer < arch["mlp_layers"] else D
        w = take(o, h.shape[1])
        h = h @ w.T + take(o)
        if layer < arch["mlp_layers"]:
            h = torch.relu(h)
    loss = ((h - _t(target)) ** 2).sum(1).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": torch.cat([v.grad.reshape(-1) for v in parts])}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "port":
            return _exact_port(case, seed)
        if kind == "train":
            with torch.enable_grad():
                return _exact_train(case, seed)
        case = dict(case, host=False)
        wall = case.get("precision", "f64") != "f64"
        if kind == "pattern":
            return _Fdtd(_problem(case, seed), wall).advance(case["warm"]).pattern(*_angles(case["degrees"]))
        if kind == "batch":
            # the members one after another: the first two, the rest would take too long
            runs = [_Fdtd(_problem(case, seed, m), wall).advance(case["warm"] + case["steps"])
                    for m in range(min(2, case["members"]))]
            if case["members"] > 2:
                return {"V": [None], "I": [None], "far": runs[0].far()}
            return {"V": [torch.cat([r.ports()[0] for r in runs])], "I": [torch.cat([r.ports()[1] for r in runs])],
                    "far": runs[0].far()}
        nx, ny, nz = _extent(case)[:3]
        if nx * ny * nz * (case.get("warm", 0) + case["steps"]) > 1.2e10:
            return None                    # over about 20 seconds
        r = _Fdtd(_problem(case, seed), wall).advance(case.get("warm", 0) + case["steps"])
        V, I = r.ports()
        if kind == "solve":
            at = [min(q + 50, case["steps"]) - 1 for q in range(0, case["steps"], 50)]
            return {"snapshots": V[at], "V": V, "I": I, "far": r.far(),
                    "fields": [x.reshape(-1) for x in r.H + r.E]}
        far = r.pattern(*_cuts()) if case["cuts"] else r.far()
        return {"V": V, "I": I, "far": far}
