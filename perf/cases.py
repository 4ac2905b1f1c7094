"""Performance cases of rumdeed_gb300: the calls that its users make, at the sizes they make them.

A case is one of five kinds of call on an engine that the user keeps:

    accel   Calculate_Acceleration_Particles: the all-pair forces of one system
    field   Calc_Field_at_Batch: the field of one system at a list of points
    step    a few time steps of one diode, resumed from its checkpoint, and the particles read back
    idle    time steps of a diode that has no electron in flight
    serve   one iteration of the continuous-batching server over its resident diodes

`listed` holds the sizes of the repository's own configurations (the one-diode deck, the request
stream of the server, the force and field microbenchmark, hyperboloid tips); `draw` gives more of
the same ranges.  Results of the FP32-compensated engine carry single precision and are kept so,
except for the counters and particle states that a run goes on from.
"""
import math

import numpy as np
import torch

import rumdeed_gb300 as rg

NM = 1.0e-9
FP = {"fp32c": rg.PREC_FP32C, "fp64": rg.PREC_FP64}

# largest emitter of the request stream: 100 panels of 4 x 4 supply nodes per side
MAX_SUPPLY_POINTS = 400 * 400


def listed():
    return [
        # The reference's one-diode deck as specified (1 um gap, 2 kV, 4.7 eV): nothing is emitted and a
        # step is a chain of small launches.  The smallest call.
        {"name": "deck-empty", "kind": "idle", "prec": "fp32c", "V": 2.0e3, "gap": 1000.0, "side": 1000.0, "phi": 4.7,
         "jumps": 100, "steps": 20},
        # The populated deck (2.0 eV): thousands of electrons, most of them close to the cathode, and as many
        # Metropolis-Hastings chains.  The ordinary run of one diode.
        {"name": "deck-populated", "kind": "step", "geometry": "planar", "prec": "fp32c", "n": 4500, "V": 2.0e3,
         "gap": 1000.0, "side": 1000.0, "phi": 2.0, "jumps": 100, "steps": 4, "profile": "layer", "serial": False},
        # The same in FP64, for users who check against the reference.
        {"name": "deck-fp64", "kind": "step", "geometry": "planar", "prec": "fp64", "n": 1200, "V": 2.0e3,
         "gap": 1000.0, "side": 500.0, "phi": 2.0, "jumps": 100, "steps": 1, "profile": "layer", "serial": False},
        # The reference's default sampler (mh_batch = .false.), one chain after another, on a small emitter.
        {"name": "serial-small", "kind": "step", "geometry": "planar", "prec": "fp32c", "n": 400, "V": 2.0e3,
         "gap": 1000.0, "side": 100.0, "phi": 2.0, "jumps": 100, "steps": 1, "profile": "layer", "serial": True},
        # A hyperboloid tip that emits.
        {"name": "tip-step", "kind": "step", "geometry": "tip", "prec": "fp32c", "n": 10007, "V": 2.0e3, "gap": 1000.0,
         "apex": 30.0, "phi": 4.5, "jumps": 80, "steps": 1, "profile": "cloud", "serial": False},
        # The server's headline load: 128 resident requests of the stream, each filled to its peak count.
        {"name": "serve-128", "kind": "serve", "slots": 128, "cap_lo": 256, "cap_hi": 32768},
        # A small load with small diodes.
        {"name": "serve-24", "kind": "serve", "slots": 24, "cap_lo": 256, "cap_hi": 4096},
        # The force microbenchmark: one image partner, and the long series (29 partners).
        {"name": "accel-65536", "kind": "accel", "geometry": "planar", "prec": "fp32c", "n": 65536, "nic": 0,
         "V": 2.0e3, "gap": 1000.0, "side": 1000.0},
        {"name": "accel-series-8191", "kind": "accel", "geometry": "planar", "prec": "fp32c", "n": 8191, "nic": 7,
         "V": 2.0e3, "gap": 1000.0, "side": 1000.0},
        # Forces in the reference's precision.
        {"name": "accel-fp64-6000", "kind": "accel", "geometry": "planar", "prec": "fp64", "n": 6000, "nic": 0,
         "V": 2.0e3, "gap": 1000.0, "side": 1000.0},
        # Forces around a tip, sphere image included.
        {"name": "accel-tip-20001", "kind": "accel", "geometry": "tip", "prec": "fp32c", "n": 20001, "nic": 0,
         "V": 2.0e3, "gap": 1000.0, "apex": 30.0},
        # The field on a 64 x 64 cathode grid, the field microbenchmark's points.
        {"name": "field-grid", "kind": "field", "geometry": "planar", "prec": "fp32c", "n": 65536, "points": 4096,
         "nic": 0, "V": 2.0e3, "gap": 1000.0, "side": 1000.0, "at": "cathode"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["accel", "accel", "accel", "field", "field", "step", "step", "step", "idle", "serve"])
    c = {"kind": kind}
    if kind == "serve":
        c.update(slots=rng.randint(8, 64), cap_lo=256, cap_hi=int(_log(rng, 1024, 16384)))
        return c
    prec = "fp64" if rng.random() < 0.25 else "fp32c"
    V, gap, side = round(_log(rng, 500.0, 5000.0), 1), round(rng.uniform(200.0, 2000.0), 1), round(rng.uniform(100.0, 2000.0), 1)
    c.update(prec=prec, V=V, gap=gap)
    if kind == "idle":
        c.update(side=side, phi=round(rng.uniform(4.6, 5.5), 3), jumps=rng.choice([100, 200]), steps=rng.randint(5, 40))
        c.update(V=round(rng.uniform(1.0, 2.0) * gap, 1))   # fields at which such cathodes hardly emit
        return c
    tip = rng.random() < 0.25
    c.update(geometry="tip" if tip else "planar")
    if tip:
        c.update(apex=round(rng.uniform(10.0, 50.0), 1), gap=1000.0, V=round(rng.uniform(1000.0, 3000.0), 1))
    else:
        c.update(side=side)
    if kind == "step":
        serial = not tip and rng.random() < 0.2
        hi = 1000 if serial else 2000 if prec == "fp64" else 16000
        c.update(n=int(_log(rng, 200, hi)), phi=round(rng.uniform(2.0, 4.0), 3), jumps=rng.choice([80, 100, 200]),
                 steps=1 if serial or tip or prec == "fp64" else rng.randint(1, 4), serial=serial,
                 profile="cloud" if tip else rng.choice(["layer", "cloud"]))
        if serial:
            c.update(side=round(rng.uniform(60.0, 150.0), 1))
        return c
    nic = 0 if tip or rng.random() < 0.7 else rng.choice([1, 7, 8])
    hi = (6000 if prec == "fp64" else 65536) / math.sqrt(1 + nic)
    c.update(nic=nic, n=int(_log(rng, 100, hi)))
    if kind == "field":
        c.update(points=int(_log(rng, 1, 2000 if prec == "fp64" else 8192)), at="gap" if tip else rng.choice(["cathode", "gap"]))
    return c


# ---- inputs ----------------------------------------------------------------------------------
def _tip_dims(c):
    """(d_tip, R_base, h_tip) of a hyperboloid with the case's apex radius, 500 nm high."""
    h, d = 500.0 * NM, c["gap"] * NM
    return d, math.sqrt(c["apex"] * NM * ((h * h) / d + 2.0 * h)), h


def _tip_shape(c):
    d, R, h = _tip_dims(c)
    a = math.sqrt((d * d * R * R) / (h * h + 2.0 * d * h) + d * d)
    eta = -d / a
    theta = math.acos(d / a)
    return {"d": d, "h": h, "a": a, "eta": eta, "max_xi": h / d + 1.0, "r": a * math.sin(theta) * math.tan(theta),
            "shift": abs(a * eta * (h / d + 1.0))}


def _positions(c, rng):
    """Electrons in flight (m): a cloud that fills the gap, the layers of a space-charge limited
    current (density ~ z^(-2/3)), or the cloud in front of a tip."""
    n = c["n"]
    if c["geometry"] == "tip":
        t = _tip_shape(c)
        xi = 1.0 + 0.6 * (t["max_xi"] - 1.0) * rng.uniform(0.0, 1.0, n)
        eta = t["eta"] * rng.uniform(0.2, 0.995, n)
        phi = rng.uniform(0.0, 2.0 * np.pi, n)
        xy = t["a"] * np.sqrt((xi * xi - 1.0) * (1.0 - eta * eta))
        return np.column_stack([xy * np.cos(phi), xy * np.sin(phi), t["a"] * xi * eta + t["shift"]])
    s, d = c["side"], c["gap"]
    z = 1.0 + (d - 2.0) * rng.uniform(0.0, 1.0, n) ** (3 if c.get("profile") == "layer" else 1)
    return np.column_stack([rng.uniform(-s / 2, s / 2, n), rng.uniform(-s / 2, s / 2, n), z]) * NM


def _velocities(c, pos):
    """Speeds of electrons that fell freely from the cathode in the vacuum field."""
    v = np.zeros_like(pos)
    if c["geometry"] == "planar":
        v[:, 2] = np.sqrt(2.0 * rg.q_0 / rg.m_0 * c["V"] * pos[:, 2] / (c["gap"] * NM))
    return v


def _points(c, rng):
    m = c["points"]
    if c["geometry"] == "tip":
        return _positions(dict(c, n=m), rng)
    s = c["side"]
    k = int(math.isqrt(m))
    if c["at"] == "cathode" and k * k == m:
        g = ((np.arange(k) + 0.5) / k - 0.5) * s + rng.uniform(-0.2, 0.2) * s / k
        x, y = np.meshgrid(g, g, indexing="ij")
        x, y = x.ravel(), y.ravel()
    else:
        x, y = rng.uniform(-s / 2, s / 2, m), rng.uniform(-s / 2, s / 2, m)
    z = np.zeros(m) if c["at"] == "cathode" else rng.uniform(0.0, c["gap"], m)
    return np.column_stack([x, y, z]) * NM


def _diode(c, capacity, **more):
    if c.get("geometry", "planar") == "tip":
        return dict(geometry=rg.GEOM_TIP, V_s=c["V"], tip_dim=_tip_dims(c), tip_work_function=c.get("phi", 4.5),
                    image_charge=True, capacity=capacity, **more)
    s = c["side"] * NM
    return dict(V_s=c["V"], gap=c["gap"] * NM, time_step=0.25e-15, image_charge=True, N_ic_max=c.get("nic", 0),
                capacity=capacity, emitter_pos=(-s / 2, -s / 2), emitter_dim=(s, s), work=[[c.get("phi", 4.7)]], **more)


def _engine(c, kw, capacity):
    return rg.Engine(precision=FP[c["prec"]], max_diodes=1, particle_capacity=capacity + 64,
                     chain_capacity=capacity + 64, quad_capacity=rg.supply_points(**kw) + 64)


def _requests(c, rng):
    """Requests of the serving stream: peak electrons log-U, V U[0.5, 5] kV, gap U[200, 2000] nm, work
    function U[2.5, 5.5] eV, emitter side U[100, 2000] nm."""
    out = []
    for _ in range(c["slots"]):
        cap = int(round(math.exp(rng.uniform(math.log(c["cap_lo"]), math.log(c["cap_hi"])))))
        s, d = float(rng.uniform(100.0, 2000.0)), float(rng.uniform(200.0, 2000.0))
        kw = dict(V_s=float(rng.uniform(500.0, 5000.0)), gap=d * NM, time_step=0.25e-15, image_charge=True, N_ic_max=0,
                  capacity=cap, emitter_pos=(-s / 2 * NM, -s / 2 * NM), emitter_dim=(s * NM, s * NM),
                  work=[[float(rng.uniform(2.5, 5.5))]], emission=True, seed=int(rng.integers(1, 2 ** 62)))
        pos = np.column_stack([rng.uniform(-s / 2, s / 2, cap), rng.uniform(-s / 2, s / 2, cap),
                               rng.uniform(1.0, d - 1.0, cap)]) * NM
        out.append((kw, pos))
    return out


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    if c["kind"] == "serve":
        reqs = _requests(c, rng)
        S, cap = c["slots"], sum(-(-kw["capacity"] // 32) * 32 for kw, _ in reqs) + 64
        eng = rg.Engine(precision=rg.PREC_FP32C, max_diodes=S, particle_capacity=cap, chain_capacity=cap,
                        quad_capacity=S * MAX_SUPPLY_POINTS + 4096)
        ids = [eng.submit(20000, pos=pos, **kw) for kw, pos in reqs]
        eng.serve(1)   # admits them: the server is running
        return {"case": c, "engine": eng, "ids": ids}
    if c["kind"] == "idle":
        swept = dict(c, V=c["V"] * rng.uniform(0.98, 1.02))   # one voltage of a sweep around the deck's
        kw = _diode(swept, 20000, emission=True, seed=seed + 1, mh_jumps=c["jumps"])
        eng = _engine(c, kw, 20000)
        return {"case": c, "engine": eng, "diode": eng.add_diode(**kw), "next": 1}
    pos = _positions(c, rng)
    if c["kind"] == "step":
        cap = max(4096, 2 * c["n"])
        kw = _diode(c, cap, emission=True, seed=seed + 1, mh_jumps=c["jumps"], mh_serial=c["serial"])
        eng = _engine(c, kw, cap)
        d = eng.add_diode(**kw)
        d.add_particles(pos, _velocities(c, pos), step=0)
        return {"case": c, "engine": eng, "diode": d, "capacity": cap, "checkpoint": d.save_state()}
    kw = _diode(c, c["n"])
    eng = _engine(c, kw, c["n"])
    d = eng.add_diode(**kw)
    d.add_particles(pos)
    state = {"case": c, "engine": eng, "diode": d}
    if c["kind"] == "field":
        state["points"] = _points(c, rng)
    return state


# ---- the calls -------------------------------------------------------------------------------
REALS = ("N_sup", "MH_std", "a_rate", "residual", "df_avg", "ramo_current", "avg_mob")
VECTORS = ("F_avg", "avg_part_vel", "avg_elec_vel")
WHOLE = ("n", "emitted_step", "dropped_step", "absorbed_top_step", "absorbed_bot_step", "chains", "chains_failed",
         "chains_capped", "emitted_total", "electron_steps", "steps_done")


def _counters(rows):
    """The counters of one or more diodes, each kind as one array."""
    out = {k: np.array([r[k] for r in rows]) for k in REALS + VECTORS}
    out["whole"] = np.array([[r[k] for k in WHOLE] for r in rows], dtype=np.int64)
    return out


def _rows(state, a):
    """The particles of a diode in an array of its capacity."""
    out = np.zeros((state["capacity"],) + a.shape[1:], dtype=a.dtype)
    out[:len(a)] = a
    return out


def _kept(c, a):
    return a if c["prec"] == "fp64" else a.astype(np.float32)


def run(state):
    c, eng = state["case"], state["engine"]
    if c["kind"] == "accel":
        return {"acc": _kept(c, state["diode"].calculate_acceleration_particles())}
    if c["kind"] == "field":
        return {"field": _kept(c, state["diode"].calc_field_at_batch(state["points"]))}
    if c["kind"] == "serve":
        eng.serve(1)
        return _counters([eng.poll(i)["counters"] for i in state["ids"]])
    d = state["diode"]
    if c["kind"] == "idle":
        eng.run(state["next"], c["steps"])
        state["next"] += c["steps"]
        return _counters([d.counters()])
    d.load_state(state["checkpoint"])
    eng.run(1, c["steps"])
    return {"particles": {k: _rows(state, a) for k, a in d.particles().items()}, "counters": _counters([d.counters()])}


# ---- what a pass cannot do without -----------------------------------------------------------
def work(case):
    """Bytes: state in and results out.  Operations, 20 per Coulomb-like term: the forces, the supply
    integral's field at its points and one field value per chain (a serving request counts with the mean
    electron count and supply grid of its range); the emission of an idle diode, its random walk."""
    c = case
    if c["kind"] == "serve":
        lo, hi = math.log(c["cap_lo"]), math.log(c["cap_hi"])
        n = (c["cap_hi"] - c["cap_lo"]) / (hi - lo)
        n2 = (c["cap_hi"] ** 2 - c["cap_lo"] ** 2) / (2.0 * (hi - lo))
        return {"bytes": 400.0 * n * c["slots"], "flops": c["slots"] * (40.0 * n2 + 20.0 * n * 5.6e4)}
    pts = 0 if c["kind"] in ("accel", "field") else 10000 if c.get("geometry") == "tip" else \
        (4 * min(256, max(16, math.ceil(c["side"] / 20.0)))) ** 2
    if c["kind"] == "idle":
        return {"bytes": 24.0 * pts * c["steps"], "flops": c["steps"] * (20.0 * pts + 1000.0 * 60.0 * c["jumps"])}
    n, terms = c["n"], 2.0 + 4.0 * c.get("nic", 0)
    if c["kind"] == "accel":
        return {"bytes": 56.0 * n, "flops": 20.0 * terms * n * n}
    if c["kind"] == "field":
        return {"bytes": 32.0 * n + 48.0 * c["points"], "flops": 20.0 * terms * n * c["points"]}
    return {"bytes": 400.0 * n * c["steps"], "flops": c["steps"] * (20.0 * terms * n * n + 20.0 * n * (pts + 1000.0))}


# ---- the same in 64 bits ---------------------------------------------------------------------
_C2 = 299792458.0 ** 2
_EPS0 = 1.0 / (1.25663706212e-6 * _C2)
_KC = 1.0 / (4.0 * math.pi * _EPS0)
_L2 = NM * NM


def _cube(x2):
    r = torch.sqrt(x2) + _L2
    return 1.0 / (r * r * r)


def _tip_vacuum(c, p):
    t = _tip_shape(c)
    a, x, y, z = t["a"], p[:, 0], p[:, 1], p[:, 2]
    rp = torch.sqrt(x * x + y * y + (z + a - t["shift"]) ** 2)
    rm = torch.sqrt(x * x + y * y + (z - a - t["shift"]) ** 2)
    xi, eta = (rp + rm) / (2.0 * a), (rp - rm) / (2.0 * a)
    pre_E = 2.0 * c["V"] / (a * math.log((1.0 + t["eta"]) / (1.0 - t["eta"])))
    pre = pre_E / (xi * xi - eta * eta)
    fac = torch.where((xi - 1.0).abs() < 1.0e-6, torch.zeros_like(xi), eta * torch.sqrt((xi * xi - 1.0) / (1.0 - eta * eta)))
    rho = torch.sqrt(x * x + y * y).clamp_min(1.0e-30)
    return torch.stack([-pre * fac * x / rho, -pre * fac * y / rho, pre * xi], 1)


def _pair_sum(c, src, at, own):
    """Sum over the sources of the Coulomb and image terms at `at` (unit charges, without k).  own: the
    points are the sources themselves (no self term; the lower index in the image function's first
    role), else every point is in the first role."""
    out = torch.zeros_like(at)
    idx = torch.arange(len(src), device=src.device)
    block = max(1, (1 << 25) // len(src))
    for i0 in range(0, len(at), block):
        p = at[i0:i0 + block]
        i = idx[i0:i0 + len(p), None] if own else None
        upper = idx[None, :] > i if own else None
        live = (idx[None, :] != i).to(p.dtype) if own else 1.0
        dx, dy, dz = (p[:, k, None] - src[None, :, k] for k in range(3))
        d2 = dx * dx + dy * dy
        inv = _cube(d2 + dz * dz) * live
        inv = torch.nan_to_num(inv, posinf=0.0)
        sx, sy, sz = inv * dx, inv * dy, inv * dz
        if c["geometry"] == "planar":
            zs = p[:, 2, None] + src[None, :, 2]
            za = torch.where(upper, dz, -dz) if own else dz   # height of the first role above the second
            d = c["gap"] * NM
            terms = [(-1.0, zs)]
            for n in range(1, c.get("nic", 0) + 1):
                terms += [(-1.0, zs - 2.0 * n * d), (-1.0, zs + 2.0 * n * d), (1.0, za - 2.0 * n * d), (1.0, za + 2.0 * n * d)]
            for sign, h in terms:
                w = sign * _cube(d2 + h * h) * live
                sx += w * dx
                sy += w * dy
                sz += w * h
        else:
            t, K = _tip_shape(c), rg.q_0 * _KC
            z0, R = t["h"] - t["r"], t["r"]

            def image(q):
                h = q[:, 2] - z0
                dis = torch.sqrt(q[:, 0] ** 2 + q[:, 1] ** 2 + h * h)
                s = R * R / (dis * dis)   # along the ray from the sphere's centre
                return q[:, 0] * s * torch.sign(h), q[:, 1] * s * torch.sign(h), z0 + h.abs() * s, dis

            def term(xa, ya, za, m, xb, yb, zb):
                xm, ym, zm, dis = m
                a3 = ((xb - xa) ** 2 + (yb - ya) ** 2 + (zb - za) ** 2) ** -1.5
                b3 = R / dis * ((xb - xm) ** 2 + (yb - ym) ** 2 + (zb - zm) ** 2) ** -1.5
                return [torch.nan_to_num(K * ((u - v) * a3 - (w - v) * b3), posinf=0.0, neginf=0.0)
                        for u, v, w in ((xa, xb, xm), (ya, yb, ym), (za, zb, zm))]

            P = [p[:, k, None] for k in range(3)]
            Q = [src[None, :, k] for k in range(3)]
            up = term(*P, [m[:, None] for m in image(p)], *Q)
            if own:
                lo = term(*Q, [m[None, :] for m in image(src)], *P)
                up = [torch.where(upper, u, s * v) * live for u, v, s in zip(up, lo, (-1.0, -1.0, 1.0))]
            sx, sy, sz = sx + up[0], sy + up[1], sz + up[2]
        out[i0:i0 + len(p)] = torch.stack([sx.sum(1), sy.sum(1), sz.sum(1)], 1)
    return out


def exact(case, seed):
    c = case
    if c["kind"] not in ("accel", "field"):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    src = torch.from_numpy(_positions(c, rng)).to(dev)
    at = src if c["kind"] == "accel" else torch.from_numpy(_points(c, rng)).to(dev)
    E = -rg.q_0 * _KC * _pair_sum(c, src, at, c["kind"] == "accel")
    if c["geometry"] == "tip":
        E += _tip_vacuum(c, at)
    else:
        E[:, 2] -= c["V"] / (c["gap"] * NM)
    if c["kind"] == "field":
        return {"field": E.cpu().numpy()}
    return {"acc": (E * (-rg.q_0 / rg.m_0)).cpu().numpy()}
