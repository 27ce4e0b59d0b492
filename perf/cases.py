"""Performance cases: whole calls of the thin-film framework, as programs make them.

Every pass goes through the public Python API (drivers, ``time_loop``, ``Batch``,
``Server``): host films in, host results out, as a script does it.  Heights of
Float32 and Float16-storage states come back from the API widened to Float64;
the passes hand them on as the Float32 values they are.

Kinds of case and what they stand for:

  random    ``run_random``: a driver call that makes its own state (short runs, tests, sweeps)
  droplet   a relaxing droplet with the wetted-area record (``run_dropletrelax``'s loop)
  rt        a Rayleigh-Taylor film with the height-difference record (the headline run)
  film      a rough film levelling, no record but the mass (long production runs)
  pattern   a droplet on a chemically patterned substrate (contact-angle field)
  sliding   a droplet under a body force, heights and velocities read back
  callback  a Python callback between the forces and the collision (per-op path)
  ensemble  a batch of coalescing droplet pairs advanced together
  serve     a server with a burst of moving-wettability requests
  gamma1d   ``run_gamma``: 1D droplets on a surface-tension gradient
"""
import math
import os
import sys
import time

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "swalbe.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import swalbe_gb300 as sw  # noqa: E402

TYPES = {"f64": np.float64, "f32": np.float32, "f16": np.float16}
# lattices whose populations (two copies) fit in this stay on the chip between iterations
ON_CHIP = 129e6


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a driver call from a test or a parameter scan: state creation, launches and host work count
        {"name": "random_f64_56x40", "kind": "random", "T": "f64", "Lx": 56, "Ly": 40, "steps": 200, "tau": 1.0},
        # the reference's droplet relaxation (256², Float64 is the default element type)
        {"name": "droplet_f64_256", "kind": "droplet", "T": "f64", "Lx": 256, "Ly": 256, "steps": 600},
        # the headline film, 512² Float32, max(h) - min(h) every iteration
        {"name": "rt_f32_512", "kind": "rt", "T": "f32", "Lx": 512, "Ly": 512, "steps": 600},
        # the large rough film in Float32 and with FP16 storage
        {"name": "film_f32_2048", "kind": "film", "T": "f32", "Lx": 2048, "Ly": 2048, "steps": 300},
        {"name": "film_f16_2048", "kind": "film", "T": "f16", "Lx": 2048, "Ly": 2048, "steps": 300},
        # a large film in the default Float64, sides that are no power of two
        {"name": "film_f64_1000x1030", "kind": "film", "T": "f64", "Lx": 1000, "Ly": 1030, "steps": 60},
        # a patterned substrate, odd sides, Float64
        {"name": "pattern_f64_301x257", "kind": "pattern", "T": "f64", "Lx": 301, "Ly": 257, "steps": 400},
        # a sliding droplet in Float32
        {"name": "sliding_f32_384x250", "kind": "sliding", "T": "f32", "Lx": 384, "Ly": 250, "steps": 700},
        # a script with its own force between the reference's ops
        {"name": "callback_f64_128x96", "kind": "callback", "T": "f64", "Lx": 128, "Ly": 96, "steps": 50},
        # coalescence ensemble (128² .. 1024 x 256), Float32
        {"name": "ensemble_f32_24", "kind": "ensemble", "T": "f32", "count": 24, "steps": 150},
        # a burst of requests to the server
        {"name": "serve_f32_8", "kind": "serve", "T": "f32", "count": 8, "side": 512, "steps": 500},
        # 1D coalescence on a surface-tension gradient, Float64
        {"name": "gamma1d_f64_1024", "kind": "gamma1d", "T": "f64", "Lx": 1024, "steps": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["random", "droplet", "rt", "film", "film", "pattern", "sliding", "callback", "ensemble",
                       "serve", "gamma1d"])
    if kind == "random":
        return {"kind": kind, "T": rng.choice(["f64", "f64", "f32"]), "Lx": _log(rng, 16, 160), "Ly": _log(rng, 16, 160),
                "steps": rng.randint(50, 400), "tau": rng.choice([1.0, 1.0, 0.8])}
    if kind in ("droplet", "pattern", "sliding"):
        return {"kind": kind, "T": rng.choice(["f64", "f32"]), "Lx": _log(rng, 96, 420), "Ly": _log(rng, 96, 420),
                "steps": rng.randint(200, 700)}
    if kind == "rt":
        return {"kind": kind, "T": rng.choice(["f64", "f32", "f16"]), "Lx": _log(rng, 100, 620), "Ly": _log(rng, 100, 620),
                "steps": rng.randint(200, 600)}
    if kind == "film":
        t = rng.choice(["f64", "f32", "f16"])
        if t == "f64":
            return {"kind": kind, "T": t, "Lx": _log(rng, 200, 1100), "Ly": _log(rng, 200, 1100), "steps": rng.randint(30, 70)}
        return {"kind": kind, "T": t, "Lx": _log(rng, 300, 2048), "Ly": _log(rng, 300, 2048), "steps": rng.randint(60, 300)}
    if kind == "callback":
        return {"kind": kind, "T": rng.choice(["f64", "f32"]), "Lx": _log(rng, 32, 200), "Ly": _log(rng, 32, 200),
                "steps": rng.randint(20, 60)}
    if kind == "ensemble":
        return {"kind": kind, "T": "f32", "count": rng.randint(4, 24), "steps": rng.randint(60, 150)}
    if kind == "serve":
        return {"kind": kind, "T": "f32", "count": rng.randint(2, 10), "side": 64 * rng.randint(2, 8), "steps": rng.randint(100, 500)}
    return {"kind": kind, "T": rng.choice(["f64", "f64", "f32"]), "Lx": _log(rng, 256, 2400), "steps": rng.randint(200, 800)}


# ---------------------------------------------------------------- inputs
def _cap(Lx, Ly, radius, theta, cx, cy, floor=0.05):
    """A spherical cap of sphere radius `radius` and contact angle `theta` (units of pi) on a precursor film."""
    x = np.arange(1, Lx + 1)[:, None] - cx
    y = np.arange(1, Ly + 1)[None, :] - cy
    r2 = np.minimum(x * x + y * y, radius * radius)
    return np.asfortranarray(np.maximum(np.sqrt(radius * radius - r2) - radius * math.cos(math.pi * theta), floor))


def _rand_film(Lx, Ly, amp, rng):
    return np.asfortranarray(1.0 + rng.uniform(-amp, amp, (Lx, Ly)))


def _inputs(case, seed):
    """Films and parameters of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    k = case["kind"]
    if k == "random":
        return {"eps": 0.01, "seed": int(rng.integers(1 << 30)), "par": {"tau": case["tau"], "Tmax": case["steps"]}}
    if k in ("droplet", "pattern", "sliding", "callback"):
        Lx, Ly = case["Lx"], case["Ly"]
        # apex height at most 20, contact radius about a quarter of the shorter side
        side = min(Lx, Ly)
        th0 = 1 / 6
        radius = min(side * rng.uniform(0.45, 0.5), 20 / (1 - math.cos(math.pi * th0)))
        h = _cap(Lx, Ly, radius, th0, Lx / 2 + rng.uniform(-2, 2), Ly / 2 + rng.uniform(-2, 2))
        d = {"h": h, "par": {"Tmax": case["steps"]}}
        if k == "pattern":
            # boxes of lower wettability, as the pattern generators paint them
            th = np.full((Lx, Ly), 1 / 9)
            for _ in range(4):
                cx, cy, w = rng.integers(0, Lx), rng.integers(0, Ly), int(rng.integers(10, 40))
                th[max(cx - w, 0):cx + w, max(cy - w, 0):cy + w] += 1 / 36
            d["theta"] = np.asfortranarray(np.minimum(th, 1 / 4))
        if k in ("sliding", "callback"):
            d["alpha"] = [float(rng.uniform(1e-4, 2e-4)), float(rng.uniform(-1e-4, 1e-4))]
            d["par"]["delta"] = 2.0
        return d
    if k == "rt":
        return {"h": _rand_film(case["Lx"], case["Ly"], 0.01, rng),
                "par": {"Tmax": case["steps"], "g": -0.001, "gamma": 0.0005}}
    if k == "film":
        return {"h": _rand_film(case["Lx"], case["Ly"], 0.1, rng), "par": {"Tmax": case["steps"]}}
    if k == "ensemble":
        sizes = [(128, 128), (256, 256), (512, 512), (1024, 256)]
        out = []
        for i in range(case["count"]):
            Lx, Ly = sizes[i % 4]
            th = float(rng.uniform(1 / 18, 1 / 4))
            sn, cs = math.sin(math.pi * th), math.cos(math.pi * th)
            r1, r2 = rng.uniform(0.15, 0.40, 2) * Ly
            gap = int(rng.integers(2, 11))
            f = min(1.0, (Lx - gap - 8) / (2 * (r1 + r2) * sn), 20 / (max(r1, r2) * (1 - cs)))
            r1, r2 = r1 * f, r2 * f
            left = (Lx - 2 * (r1 + r2) * sn - gap) / 2
            h = np.maximum(_cap(Lx, Ly, r1, th, left + r1 * sn, Ly / 2),
                           _cap(Lx, Ly, r2, th, left + 2 * r1 * sn + gap + r2 * sn, Ly / 2))
            out.append({"h": np.asfortranarray(h), "Lx": Lx, "Ly": Ly, "par": {"Tmax": case["steps"], "theta": th}})
        return {"members": out}
    if k == "serve":
        out = []
        for i in range(case["count"]):
            # sides and lengths of the burst spread over their range, the same for every seed
            Lx = max(64, (case["side"] * (i % 4 + 1) // 4) // 64 * 64)
            Ly = max(64, (case["side"] * ((3 * i) % 4 + 1) // 4) // 64 * 64)
            par = {"Tmax": case["steps"] * (i % 3 + 2) // 4, "theta": float(rng.uniform(1 / 18, 1 / 4)),
                   "g": float(rng.uniform(-1e-3, 0.0))}
            out.append({"h": _rand_film(Lx, Ly, 0.05, rng), "Lx": Lx, "Ly": Ly, "par": par})
        return {"members": out}
    L = case["Lx"]
    x = 2 * math.pi * (np.arange(L) / L + rng.uniform())
    return {"gamma": 0.01 * (1 + rng.uniform(0.05, 0.15) * np.sin(x)), "r": 0.11 * L, "dump": max(1, case["steps"] // 4),
            "par": {"Tmax": case["steps"]}}


# ---------------------------------------------------------------- passes
def prepare(case, seed):
    d = _inputs(case, seed)
    k, T = case["kind"], TYPES[case["T"]]
    s = {"case": case, "in": d, "T": T}
    if k == "ensemble":
        s["batch"] = sw.Batch([sw.SysConst(m["Lx"], m["Ly"], sw.Taumucs(**m["par"])) for m in d["members"]], T=T)
    elif k == "serve":
        s["server"] = sw.Server(2 << 30, T=T, steps_per_tick=100)
        s["sys"] = [sw.SysConst(m["Lx"], m["Ly"], sw.Taumucs(**m["par"])) for m in d["members"]]
    elif k == "gamma1d":
        s["sys"] = sw.SysConst_1D(case["Lx"], sw.Taumucs(**d["par"]))
    else:
        s["sys"] = sw.SysConst(case["Lx"], case["Ly"], sw.Taumucs(**d["par"]))
        if k != "random":
            s["state"] = sw.Sys(s["sys"], "GB300", T=T)
            s["rest"] = np.zeros((case["Lx"], case["Ly"]), order="F")
    return s


def _out(s, a):
    return a if s["T"] is np.float64 else a.astype(np.float32)


def _push(measure, state):
    """A script's own force: a constant body force added by the reference's op."""
    sw.inclination_(measure, state)


def run(s):
    k, d = s["case"]["kind"], s["in"]
    if k == "random":
        h = sw.run_random(s["sys"], "GB300", ϵ=d["eps"], verbos=False, T=s["T"], rng=np.random.default_rng(d["seed"]))
        return {"h": _out(s, h)}
    if k == "gamma1d":
        r = d["r"]
        return {"h": _out(s, sw.run_gamma(s["sys"], d["gamma"], r1=r, r2=r, verbos=False, dump=d["dump"], T=s["T"]))}
    if k == "ensemble":
        b = s["batch"]
        for i, m in enumerate(d["members"]):
            b.set_height(i, m["h"])
        b.step(s["case"]["steps"])
        b.sync()
        return {"h": [_out(s, b.get_height(i)) for i in range(len(d["members"]))]}
    if k == "serve":
        sv, got = s["server"], {}
        ids = [sv.submit(c, m["h"], m["par"]["Tmax"], dtheta=1 / 36, v=1 / 98) for c, m in zip(s["sys"], d["members"])]
        while len(got) < len(ids):
            for i, rid in enumerate(ids):
                if i not in got:
                    done, h, info = sv.poll(rid, (d["members"][i]["Lx"], d["members"][i]["Ly"]))
                    if done:
                        got[i] = _out(s, h)
                    elif info.status < 0:
                        raise RuntimeError(f"request {rid} failed: {info.status}")
                    else:
                        time.sleep(1e-4)
                        break
        return {"h": [got[i] for i in range(len(ids))]}
    # a film uploaded to the program's state, the time loop, the results read back
    st, c = s["state"], s["sys"]
    st.height = d["h"]
    st.velx = s["rest"]
    st.vely = s["rest"]
    if k == "droplet":
        area = []
        sw.time_loop(c, st, sw.wetted_, area)
        # a Float32 height beside the threshold may fall on either side of it by its last bit
        return {"h": _out(s, st.height), "area": np.array(area, dtype=np.int64 if s["T"] is np.float64 else np.float32)}
    if k == "rt":
        dh = []
        sw.time_loop(c, st, dh)
        return {"h": _out(s, st.height), "dh": _out(s, np.array(dh))}
    if k == "film":
        sw.time_loop(c, st)
        return {"h": _out(s, st.height)}
    if k == "pattern":
        sw.time_loop(c, st, d["theta"])
        return {"h": _out(s, st.height)}
    if k == "sliding":
        sw.time_loop(c, st, sw.inclination_, d["alpha"])
    else:
        sw.time_loop(c, st, _push, d["alpha"])
    return {"h": _out(s, st.height), "ux": _out(s, st.velx), "uy": _out(s, st.vely)}


# ---------------------------------------------------------------- work
def work(case):
    k = case["kind"]
    # operations of one cell and iteration (D2Q9 / D1Q3), and a population set in bytes
    ops = 60 if k == "gamma1d" else 165
    pop = (3 if k == "gamma1d" else 9) * 8
    if case["T"] == "f32":
        pop //= 2
    elif case["T"] == "f16":
        pop = 20
    if k in ("ensemble", "serve"):
        cells = [(m["Lx"] * m["Ly"], m["par"]["Tmax"]) for m in _sizes(case)]
    else:
        cells = [(case["Lx"] * case.get("Ly", 1), case["steps"])]
    resident = 2 * pop * sum(n for n, _ in cells) <= ON_CHIP
    # films in and results out once; the populations through memory every iteration where they do not stay on the chip
    fields = {"sliding": 6, "callback": 6, "gamma1d": 6}.get(k, 4)
    b = sum(n * (8 * fields + (0 if resident else 2 * pop * t)) for n, t in cells)
    return {"bytes": b, "flops": sum(n * t * ops for n, t in cells)}


def _sizes(case):
    if case["kind"] == "ensemble":
        sizes = [(128, 128), (256, 256), (512, 512), (1024, 256)]
        return [{"Lx": sizes[i % 4][0], "Ly": sizes[i % 4][1], "par": {"Tmax": case["steps"]}} for i in range(case["count"])]
    return [{"Lx": max(64, (case["side"] * (i % 4 + 1) // 4) // 64 * 64),
             "Ly": max(64, (case["side"] * ((3 * i) % 4 + 1) // 4) // 64 * 64),
             "par": {"Tmax": case["steps"] * (i % 3 + 2) // 4}} for i in range(case["count"])]


# ---------------------------------------------------------------- the same in 64 bits
_C = [(0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1)]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _nb(a):
    """Neighbours of every cell: a[i+dx, j+dy] by (dx, dy)."""
    return {c: torch.roll(a, (-c[0], -c[1]), (0, 1)) for c in _C}


def _kappa(theta, P):
    c = torch.cos(math.pi * theta) if torch.is_tensor(theta) else math.cos(math.pi * theta)
    return (1 - c) * (P["n"] - 1) * (P["m"] - 1) / ((P["n"] - P["m"]) * P["hmin"])


def _params(par):
    P = {"tau": 1.0, "delta": 1.0, "gamma": 0.01, "n": 9, "m": 3, "hmin": 0.1, "hcrit": 0.05, "theta": 1 / 9, "g": 0.0}
    P.update(par)
    P["mu"] = (P["tau"] - 0.5) / 3
    return P


def _loop2d(h0, par, theta=None, alpha=None, wave=None, record=None):
    """The thin-film lattice Boltzmann loop in Float64; `record(h)` sees every iteration's height at its start."""
    P = _params(par)
    h = torch.as_tensor(np.ascontiguousarray(h0), dtype=torch.float64, device=_dev())
    ux, uy = torch.zeros_like(h), torch.zeros_like(h)
    f = [torch.zeros_like(h) for _ in range(9)]
    th = P["theta"] if theta is None else torch.as_tensor(np.ascontiguousarray(theta), device=h.device)
    kap = _kappa(th, P)
    x = torch.arange(h.shape[0], dtype=torch.float64, device=h.device)[:, None]
    om, g, mu6, d = 1 - 1 / P["tau"], P["g"], 6 * P["mu"], P["delta"]
    for t in range(1, P["Tmax"] + 1):
        if record is not None:
            record(h)
        if wave is not None:
            kap = _kappa(th + wave[0] * torch.sin(2 * math.pi * (x - wave[1] * t) / h.shape[0]), P)
        n = _nb(h)
        lap = 2 / 3 * (n[1, 0] + n[-1, 0] + n[0, 1] + n[0, -1]) + \
            1 / 6 * (n[1, 1] + n[-1, 1] + n[1, -1] + n[-1, -1]) - 10 / 3 * h
        q = P["hmin"] / (h + P["hcrit"])
        p = -P["gamma"] * (kap * (q ** P["n"] - q ** P["m"]) + lap)
        n = _nb(p)
        gx = (n[1, 0] - n[-1, 0]) / 3 + (n[1, 1] - n[-1, 1] + n[1, -1] - n[-1, -1]) / 12
        gy = (n[0, 1] - n[0, -1]) / 3 + (n[1, 1] + n[-1, 1] - n[1, -1] - n[-1, -1]) / 12
        slip = mu6 * h / (2 * h * h + 6 * d * h + 3 * d * d)
        Fx, Fy = -h * gx - slip * ux, -h * gy - slip * uy
        if alpha is not None:
            Fx, Fy = Fx + h * alpha[0], Fy + h * alpha[1]
        v2 = ux * ux + uy * uy
        out = []
        for c, (cx, cy) in enumerate(_C):
            if c == 0:
                e = h * (1 - 5 / 6 * g * h - 2 / 3 * v2)
                out.append(om * f[0] + e / P["tau"])
                continue
            w, ws = (1 / 9, 1 / 3) if c < 5 else (1 / 36, 1 / 24)
            cu = cx * ux + cy * uy
            e = w * h * (1.5 * g * h + 3 * cu + 4.5 * cu * cu - 1.5 * v2)
            v = om * f[c] + e / P["tau"] + ws * (cx * Fx + cy * Fy)
            out.append(torch.roll(v, (cx, cy), (0, 1)))
        f = out
        h = sum(f[1:], f[0])
        ux = (f[1] - f[3] + f[5] - f[6] - f[7] + f[8]) / h
        uy = (f[2] - f[4] + f[5] + f[6] - f[7] - f[8]) / h
    return h.cpu().numpy(), ux.cpu().numpy(), uy.cpu().numpy()


def _loop1d(h0, gamma, par, dump):
    P = _params(par)
    h, u = h0.copy(), np.zeros_like(h0)
    f = [np.zeros_like(h0) for _ in range(3)]
    kap, om, it, d = _kappa(P["theta"], P), 1 - 1 / P["tau"], 1 / P["tau"], P["delta"]
    dg = -0.75 * (np.roll(gamma, 1) - np.roll(gamma, -1))
    rows = []
    for t in range(1, P["Tmax"] + 1):
        q = P["hmin"] / (h + P["hcrit"])
        p = -gamma * (kap * (q ** P["n"] - q ** P["m"]) + np.roll(h, 1) - 2 * h + np.roll(h, -1))
        F = 0.5 * h * (np.roll(p, 1) - np.roll(p, -1)) - \
            6 * P["mu"] * h * u / (2 * h * h + 6 * d * h + 3 * d * d) - dg
        e0 = h * (1 - 0.5 * P["g"] * h - u * u)
        e1 = h * (0.25 * P["g"] * h + 0.5 * u + 0.5 * u * u)
        e2 = h * (0.25 * P["g"] * h - 0.5 * u + 0.5 * u * u)
        f = [om * f[0] + it * e0, np.roll(om * f[1] + it * e1 + 0.5 * F, 1), np.roll(om * f[2] + it * e2 - 0.5 * F, -1)]
        h = f[0] + f[1] + f[2]
        u = (f[1] - f[2]) / h
        if t % dump == 0:
            rows.append(h)
    return np.stack(rows)


def _caps1d(L, r, theta):
    i = np.arange(1, L + 1)

    def cap(c):
        a = np.abs(i - c)
        v = np.where(a <= r, (np.sqrt(1 - np.minimum(a / r, 1.0) ** 2) - math.cos(math.pi * theta)) * r, 0.05)
        return np.where(v < 0, 0.05, v)

    h = cap(L / 3) + cap(2 * L / 3) - 0.05
    return np.where(h < 0, 0.05, h)


def exact(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    if k == "random":
        h0 = 1.0 + d["eps"] * np.random.default_rng(d["seed"]).standard_normal((case["Lx"], case["Ly"]))
        return {"h": _loop2d(h0, d["par"])[0]}
    if k == "gamma1d":
        return {"h": _loop1d(_caps1d(case["Lx"], d["r"], 1 / 9), d["gamma"], d["par"], d["dump"])}
    if k == "ensemble":
        return {"h": [_loop2d(m["h"], m["par"])[0] for m in d["members"]]}
    if k == "serve":
        return {"h": [_loop2d(m["h"], m["par"], wave=(1 / 36, 1 / 98))[0] for m in d["members"]]}
    if k == "droplet":
        area = []
        h = _loop2d(d["h"], d["par"], record=lambda v: area.append((v > 0.055).sum()))[0]
        return {"h": h, "area": None if case["T"] == "f64" else np.array([float(a) for a in area])}
    if k == "rt":
        dh = []
        h = _loop2d(d["h"], d["par"], record=lambda v: dh.append(v.max() - v.min()))[0]
        return {"h": h, "dh": np.array([float(a) for a in dh])}
    if k == "pattern":
        return {"h": _loop2d(d["h"], d["par"], theta=d["theta"])[0]}
    if k in ("sliding", "callback"):
        h, ux, uy = _loop2d(d["h"], d["par"], alpha=d["alpha"])
        return {"h": h, "ux": ux, "uy": uy}
    return {"h": _loop2d(d["h"], d["par"])[0]}
