"""Workloads of the engine as its users run it, for timing and comparison.

Each case goes through the public Python entry points (`Engine`, the seeded
population generator, the host breakup model) over the ranges the engine is
used in:

  screen     one-shot screening of given start / end states: the call behind
             the reference's Screener::screen, once per step of its own loop,
             on host arrays
  propagate  one-shot propagation of host arrays, no screening (the CLI
             without --screen)
  run        a chunk of a long run with the population resident on the
             device: steps, the records and counters they gave, the states
  trial      one Monte Carlo trial: population uploaded, a forced impact
             fragmented, the steps after it, everything read back
  ensemble   realisations of a breakup study stepped as one batch
  cascade    realisations of a dense population with fragmentation on the
             device inside every step

A case is a dict of plain values. `prepare` makes what a program holds before
the call (inputs from the seed alone), `run` makes one pass, `work` states the
bytes and operations a pass cannot do without, `exact` gives the same values
from plain 64-bit torch where such values exist.
"""
import importlib
import math

import numpy as np
import torch

ks = importlib.import_module("kessler-syndrom-simulation_b200")

EPOCH_JD = 2461253.916666667
CATALOGUE = 28340      # objects of the reference's shipped catalogue
CLOUDS = 200           # parents of the fragment clouds of larger populations
CLOUD_AGE_S = 86400.0  # the clouds were released within the last day
MOST_FRAGMENTS = 12000  # of one collision of bodies up to 4 t, down to 5 cm


def listed():
    return [
        # A constellation against its neighbourhood, screened on request: latency.
        {"name": "screen_2k", "kind": "screen", "n": 2111, "dt": 10.0, "km": 5.0, "precision": "fp64"},
        # One step of the reference's own loop behind its Screener::screen.
        {"name": "screen_catalogue", "kind": "screen", "n": CATALOGUE, "dt": 10.0, "km": 5.0, "precision": "fp64"},
        # The same call late in a cascade (the reference's 28 h cascade passes 250 000 objects).
        {"name": "screen_250k", "kind": "screen", "n": 250007, "dt": 10.0, "km": 5.0, "precision": "fp64"},
        # Ephemeris service: the catalogue carried six hours ahead, no screening.
        {"name": "propagate_6h", "kind": "propagate", "n": CATALOGUE, "dt": 10.0, "steps": 2160, "precision": "fp64"},
        # The reference's headline run, an hour of it: catalogue, dt 10 s, 5 km.
        {"name": "hour_fp64", "kind": "run", "n": CATALOGUE, "dt": 10.0, "km": 5.0, "steps": 360, "precision": "fp64"},
        # The same hour in split precision at the reference's coarse step (60 times the candidate pairs).
        {"name": "hour_dt60_split", "kind": "run", "n": CATALOGUE, "dt": 60.0, "km": 5.0, "steps": 60,
         "precision": "split"},
        # A mid-size debris population at the step the reference's cascades use.
        {"name": "250k_dt30_fp64", "kind": "run", "n": 250007, "dt": 30.0, "km": 5.0, "steps": 30, "precision": "fp64"},
        # The million-object workload, both precisions.
        {"name": "1m_fp64", "kind": "run", "n": 1000000, "dt": 10.0, "km": 5.0, "steps": 32, "precision": "fp64"},
        {"name": "1m_split", "kind": "run", "n": 1000000, "dt": 10.0, "km": 5.0, "steps": 64, "precision": "split"},
        # One trial of a breakup study: a satellite struck, the six minutes after it.
        {"name": "trial_fp64", "kind": "trial", "n": CATALOGUE, "dt": 10.0, "km": 5.0, "steps": 36, "precision": "fp64",
         "lc": 0.05},
        # The 64-realisation breakup study as one batch.
        {"name": "ensemble_64", "kind": "ensemble", "n": CATALOGUE, "realisations": 64, "dt": 10.0, "km": 5.0,
         "steps": 16, "precision": "split", "lc": 0.05},
        # A cascade study with fragmentation in the loop on the device.
        {"name": "cascade_4x1m", "kind": "cascade", "n": 1000000, "realisations": 4, "dt": 10.0, "km": 5.0,
         "steps": 16, "precision": "split", "lc": 0.1, "radius_scale": 5.0},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges; candidate pairs per step grow with n^2 and about dt^2.3."""
    kind = rng.choice(["screen", "screen", "propagate", "run", "run", "run", "trial", "ensemble", "cascade"])
    prec = rng.choice(["fp64", "split"])
    km = round(rng.uniform(1.0, 10.0), 2)
    if kind == "propagate":
        n = int(_log_uniform(rng, 700, 900000))
        most = min(2160, int(5e7 / n))
        return {"kind": kind, "n": n, "dt": rng.choice([5.0, 10.0, 30.0, 60.0]),
                "steps": int(_log_uniform(rng, 2, max(3, most))), "precision": prec}
    if kind in ("screen", "run"):
        n = int(_log_uniform(rng, 1200, 300000 if kind == "screen" else 950000))
        widest = 10.0 * (1e6 / n) ** 0.87  # as many candidate pairs as the million-object step
        dt = rng.choice([d for d in (5.0, 10.0, 20.0, 30.0, 60.0) if d <= max(10.0, widest)])
        if kind == "screen":
            return {"kind": kind, "n": n, "dt": dt, "km": km, "precision": prec}
        most = min(360, int(4e7 / (n + 100000)))
        return {"kind": kind, "n": n, "dt": dt, "km": km, "steps": int(_log_uniform(rng, 4, most)), "precision": prec}
    if kind == "trial":
        return {"kind": kind, "n": int(_log_uniform(rng, 3000, 100000)), "dt": rng.choice([5.0, 10.0]), "km": km,
                "steps": rng.randrange(6, 40), "precision": prec, "lc": rng.choice([0.05, 0.1])}
    if kind == "ensemble":
        n = int(_log_uniform(rng, 2000, CATALOGUE))
        return {"kind": kind, "n": n, "realisations": rng.randrange(3, 49), "dt": 10.0, "km": km,
                "steps": rng.randrange(4, 17), "precision": prec, "lc": rng.choice([0.05, 0.1])}
    n = int(_log_uniform(rng, 50000, 800000))
    return {"kind": kind, "n": n, "realisations": rng.randrange(1, 5), "dt": 10.0, "km": km,
            "steps": rng.randrange(4, 17), "precision": prec, "lc": 0.1, "radius_scale": rng.choice([1.0, 3.0, 5.0])}


def _population(case, seed):
    """The mixed catalogue, with clouds of fragments above its size."""
    n = case["n"]
    return ks.generate_population(seed & 0x7FFFFFFF, min(n, CATALOGUE), n, CLOUDS, CLOUD_AGE_S)


def _leo(states):
    return np.flatnonzero(np.linalg.norm(states[:, :3], axis=1) < 6378.137 + 2000.0)


def _engine(case):
    eng = ks.Engine(0)
    eng.set_precision(ks.PRECISION_SPLIT if case["precision"] == "split" else ks.PRECISION_FP64)
    eng.set_clock(EPOCH_JD, 0.0, case["dt"])
    if "km" in case:
        eng.set_screening(True, case["km"], case.get("radius_scale", 1.0), 0.01)
    return eng


def _pinned(n):
    """Result buffers of a program that reads the population back often; rows past its size stay zero."""
    return torch.zeros((n, 6), dtype=torch.float64).pin_memory().numpy(), np.zeros(n, dtype=np.uint8)


def _ensemble_population(case, seed):
    """Realisations of one catalogue, each with one collision of its own fragmented by the host model."""
    st, sz, al = _population(case, seed)
    rng = np.random.default_rng(seed)
    leo = _leo(st)
    states, sizes, alive, offsets = [], [], [], [0]
    for r in range(case["realisations"]):
        target = int(rng.choice(leo))
        _, fs, fz, _, _, after = ks.sbm_impact(st[target], float(rng.uniform(100.0, 2000.0)), float(sz[target]),
                                               float(rng.uniform(100.0, 2000.0)), 10.0, 0.0, int(rng.integers(1 << 30)),
                                               case["lc"])
        a = al.copy()
        a[target] = int(after[0])
        states += [st, fs]
        sizes += [sz, fz]
        alive += [a, np.ones(len(fz), np.uint8)]
        offsets.append(offsets[-1] + len(sz) + len(fz))
    return np.array(offsets), np.concatenate(states), np.concatenate(sizes), np.concatenate(alive)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "eng": _engine(case)}
    eng = s["eng"]
    if kind == "screen":
        st, sz, al = _population(case, seed)
        after, alive_after = eng.propagate(st, al, EPOCH_JD, 0.0, case["dt"], 1)
        s.update(before=st, after=after, alive=alive_after, size=sz)
    elif kind == "propagate":
        s["states"], _, s["alive"] = _population(case, seed)
    elif kind == "run":
        st, sz, al = _population(case, seed)
        eng.set_population(st, sz, al)
        s["out"] = _pinned(len(sz))
    elif kind == "trial":
        st, sz, al = _population(case, seed)
        rng = np.random.default_rng(seed)
        target = int(rng.choice(_leo(st)))
        mass = np.zeros(len(sz))
        mass[target] = rng.uniform(500.0, 2000.0)
        s.update(states=st, size=sz, alive=al, mass=mass, target=target, projectile=float(rng.uniform(50.0, 500.0)))
        eng.set_breakup(True, case["lc"], 40.0, 1 + (seed & 0xFFFF))
        s["out"] = _pinned(len(sz) + MOST_FRAGMENTS)
        s["objects"] = {f: np.zeros(len(sz) + MOST_FRAGMENTS) for f in ("size_m", "mass_kg", "area_to_mass")}
    elif kind == "ensemble":
        offsets, st, sz, al = _ensemble_population(case, seed)
        eng.set_population_batch(offsets, st, sz, al)
        s["out"] = _pinned(case["realisations"] * (case["n"] + MOST_FRAGMENTS))
    elif kind == "cascade":
        r, n = case["realisations"], case["n"]
        st, sz, al = _population(case, seed)
        budget = r * n * 5 // 4
        eng.set_breakup_mode(ks.BREAKUP_DEVICE, budget)
        eng.set_breakup(True, case["lc"], 40.0, 1 + (seed & 0xFFFF))
        eng.set_population_batch(np.arange(r + 1) * n, np.tile(st, (r, 1)), np.tile(sz, r), np.tile(al, r))
        s["out"] = _pinned(budget)
    if "km" in case:
        s["room"] = _record_room(case)
    if "lc" in case:
        s["events"] = np.zeros(1024, ks.BREAKUP_DTYPE)
    return s


def _record_room(case):
    """The program's buffer of records, reused from pass to pass: several times what a pass gives."""
    n = case["n"] * case.get("realisations", 1)
    room = int(5e-4 * case["km"] ** 2 * n * case.get("steps", 1)) + 4096
    if case["kind"] in ("trial", "ensemble"):  # fresh clouds: many approaches among a collision's fragments
        room += 3 * MOST_FRAGMENTS * case.get("realisations", 1)
    return np.zeros(room, ks.CONJ_DTYPE)


def _records(s):
    """Every record found, moved into the program's own buffer; field by field, with their number."""
    rec = s["eng"].take_conjunctions(s["room"])
    if len(rec) == len(s["room"]):
        raise RuntimeError("record buffer too small")
    return {"count": len(rec), **{f: s["room"][f] for f in ks.CONJ_DTYPE.names}}


def _events(s):
    """The breakup events of a pass, in the program's buffer."""
    ev = s["eng"].take_breakups()
    s["events"][: len(ev)] = ev
    return {"count": len(ev), **{f: s["events"][f] for f in ("step", "t", "realisation", "target", "projectile",
                                                            "fragments", "fragments_mass_kg")}}


def _counters(st):
    return {f: st[f] for f in ks.STATS_DTYPE.names}


def _read_back(s):
    n = s["eng"].population_size()
    states, alive = s["out"]
    s["eng"].get_population(states[:n], alive[:n])
    return {"states": states, "alive": alive}


def run(s):
    case, eng = s["case"], s["eng"]
    kind = case["kind"]
    if kind == "screen":
        conj, st = eng.screen(s["before"], s["after"], s["alive"], s["size"], 0.0, case["dt"])
        s["room"][: len(conj)] = conj
        return {"records": {"count": len(conj), **{f: s["room"][f] for f in ks.CONJ_DTYPE.names}},
                "counters": _counters(st)}
    if kind == "propagate":
        states, alive = eng.propagate(s["states"], s["alive"], EPOCH_JD, 0.0, case["dt"], case["steps"])
        return {"states": states, "alive": alive}
    if kind == "trial":
        eng.set_clock(EPOCH_JD, 0.0, case["dt"])
        eng.set_population(s["states"], s["size"], s["alive"])
        eng.set_masses(s["mass"])
        eng.impact(s["target"], s["projectile"], 10.0)
    eng.run(case["steps"])
    out = {"records": _records(s), "counters": _counters(eng.take_step_stats()), **_read_back(s)}
    if kind in ("trial", "cascade"):
        out["events"] = _events(s)
    if kind == "trial":
        found = eng.objects()
        for f, room in s["objects"].items():
            room[: len(found[f])] = found[f]
        out["objects"] = s["objects"]
    return out


# Floating-point operations of one object-step (four evaluations of the point-mass, J2 and lunar
# accelerations and the Runge-Kutta sums, divisions and roots counted once).
STEP_FLOPS = 326
# Cell key and the tests of an object against what shares its neighbourhood, at the least.
SCREEN_FLOPS = 100


def work(case):
    """States in and out once, sizes and alive flags in, one set of operations per object and step."""
    n = case["n"] * case.get("realisations", 1)
    steps = case.get("steps", 1)
    if case["kind"] == "screen":
        return {"bytes": n * (2 * 48 + 9), "flops": n * SCREEN_FLOPS}
    per_step = STEP_FLOPS + (SCREEN_FLOPS if "km" in case else 0)
    return {"bytes": n * (2 * 48 + 10), "flops": n * steps * per_step}


# --- the same values in plain 64-bit arithmetic ---

MU, RE, J2, MU_MOON = 398600.4418, 6378.137, 1.08262668e-3, 4902.800066


def _moon(jd):
    """Lunar position, km: Meeus, Astronomical Algorithms, ch. 47, principal terms."""
    T = (jd - 2451545.0) / 36525.0
    rad = math.pi / 180.0
    Lp = math.fmod(math.fmod(218.3164477 + 481267.88123421 * T, 360.0) + 360.0, 360.0)
    D, M, Mp, F = (math.fmod(c0 + c1 * T, 360.0) * rad for c0, c1 in
                   ((297.8501921, 445267.1114034), (357.5291092, 35999.0502909), (134.9633964, 477198.8675055),
                    (93.2720950, 483202.0175233)))
    s, c = math.sin, math.cos
    lon = (Lp + 6.288774 * s(Mp) + 1.274027 * s(2 * D - Mp) + 0.658314 * s(2 * D) + 0.213618 * s(2 * Mp)
           - 0.185116 * s(M) - 0.114332 * s(2 * F) + 0.058793 * s(2 * D - 2 * Mp) + 0.057066 * s(2 * D - M - Mp)
           + 0.053322 * s(2 * D + Mp) + 0.045758 * s(2 * D - M)) * rad
    lat = (5.128122 * s(F) + 0.280602 * s(Mp + F) + 0.277693 * s(Mp - F) + 0.173237 * s(2 * D - F)
           + 0.055413 * s(2 * D - Mp + F) + 0.046271 * s(2 * D - Mp - F)) * rad
    dist = (385000.56 - 20905.355 * c(Mp) - 3699.111 * c(2 * D - Mp) - 2955.968 * c(2 * D) - 569.925 * c(2 * Mp)
            + 48.888 * c(M) - 3.149 * c(2 * F) + 246.158 * c(2 * D - 2 * Mp) - 152.138 * c(2 * D - M - Mp)
            - 170.733 * c(2 * D + Mp) - 204.586 * c(2 * D - M))
    eps = (23.439291 - 0.0130042 * T) * rad
    xe, ye, ze = dist * c(lat) * c(lon), dist * c(lat) * s(lon), dist * s(lat)
    return xe, ye * c(eps) - ze * s(eps), ye * s(eps) + ze * c(eps)


def _acceleration(r, jd):
    x, y, z = r
    r2 = x * x + y * y + z * z
    rn = r2.sqrt()
    central = -MU / (r2 * rn)
    j = 1.5 * J2 * MU * RE * RE / (r2 * r2 * rn)
    z2 = 5.0 * z * z / r2
    m = _moon(jd)
    mn = math.sqrt(m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
    d = [m[q] - r[q] for q in range(3)]
    dn = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
    sd = MU_MOON / (dn * dn * dn)
    si = MU_MOON / mn ** 3
    return [r[q] * central + j * r[q] * (z2 - (3.0 if q == 2 else 1.0)) + d[q] * sd - m[q] * si for q in range(3)]


def _truth_states(st, al, dt, steps):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = [c.clone() for c in torch.from_numpy(st).to(dev).t()]
    live = torch.from_numpy(al).to(dev).bool()
    t = 0.0
    for _ in range(steps):
        jd = [EPOCH_JD + (t + f * dt) / 86400.0 for f in (0.0, 0.5, 1.0)]
        k, total = None, [0.0] * 6
        for f, w, e in ((0.0, 1.0, 0), (0.5, 2.0, 1), (0.5, 2.0, 1), (1.0, 1.0, 2)):
            y = s if k is None else [s[q] + k[q] * (f * dt) for q in range(6)]
            k = y[3:] + _acceleration(y[:3], jd[e])
            total = [total[q] + w * k[q] for q in range(6)]
        s = [torch.where(live, s[q] + total[q] * (dt / 6.0), s[q]) for q in range(6)]
        live = live & ~((s[0] * s[0] + s[1] * s[1] + s[2] * s[2]).sqrt() < RE)
        t += dt
    return torch.stack(s, 1)


def _truth_screen(case, st, al):
    """Closest approaches inside the step below the threshold, from the cubic through both ends' states."""
    dt, km = case["dt"], case["km"]
    after = _truth_states(st, al, dt, 1)
    dev = after.device
    b = torch.from_numpy(st).to(dev)
    live = torch.from_numpy(al).to(dev).bool() & ((after[:, :3] ** 2).sum(1).sqrt() >= RE)
    index = torch.nonzero(live).flatten()
    index = index[torch.argsort(b[index, 0])]
    p, v = b[index, :3], b[index, 3:]
    speed = v.norm(dim=1).max().item()
    reach = 2.0 * speed * dt * (1.0 + 2e-6 * dt * dt) + km + 1.0
    left = torch.searchsorted(p[:, 0].contiguous(), p[:, 0].contiguous() + reach).cpu().tolist()
    pairs = []
    rows = 512
    for r0 in range(0, len(index), rows):
        r1 = min(len(index), r0 + rows)
        end = left[r1 - 1]
        dr = p[None, r0:end] - p[r0:r1, None]
        near = (dr[..., 0].abs() < reach) & (dr[..., 1].abs() < reach) & (dr[..., 2].abs() < reach)
        near &= torch.arange(r0, end, device=dev)[None] > torch.arange(r0, r1, device=dev)[:, None]
        a, c = torch.nonzero(near, as_tuple=True)
        d = dr[a, c]
        w = v[r0 + c] - v[r0 + a]
        w2 = (w * w).sum(1)
        ts = torch.clamp(-(d * w).sum(1) / w2.clamp(min=1e-300), 0.0, dt)
        gap = (d + w * ts[:, None]).norm(dim=1)
        keep = (gap <= km + 2e-6 * w2.sqrt() * dt ** 3 + 1e-3) & (w2 >= 1e-4)
        keep &= ~(((d * w).sum(1) >= 0) & (w2 > 2e-6 * (d * d).sum(1)))
        pairs.append(torch.stack([index[r0 + a[keep]], index[r0 + c[keep]]], 1))
    pairs = torch.cat(pairs)
    i, j = pairs.min(1).values, pairs.max(1).values
    p0, m0 = b[j, :3] - b[i, :3], (b[j, 3:] - b[i, 3:]) * dt
    p1, m1 = after[j, :3] - after[i, :3], (after[j, 3:] - after[i, 3:]) * dt

    def at(u):
        u = u[:, None]
        return (p0 * (2 * u ** 3 - 3 * u ** 2 + 1) + m0 * (u ** 3 - 2 * u ** 2 + u) + p1 * (-2 * u ** 3 + 3 * u ** 2)
                + m1 * (u ** 3 - u ** 2))

    lo, hi = torch.zeros(len(i), dtype=torch.float64, device=dev), torch.ones(len(i), dtype=torch.float64, device=dev)
    g = (math.sqrt(5.0) - 1.0) / 2.0
    for _ in range(60):
        c, d = hi - g * (hi - lo), lo + g * (hi - lo)
        smaller = (at(c) ** 2).sum(1) < (at(d) ** 2).sum(1)
        lo, hi = torch.where(smaller, lo, c), torch.where(smaller, d, hi)
    u = 0.5 * (lo + hi)
    miss = at(u).norm(dim=1)
    keep = (u > 1e-9) & (u < 1.0 - 1e-9) & (miss <= km)
    i, j, u, miss = i[keep], j[keep], u[keep], miss[keep]
    p0, m0, p1, m1 = p0[keep], m0[keep], p1[keep], m1[keep]
    w = u[:, None]
    rate = (p0 * (6 * w ** 2 - 6 * w) + m0 * (3 * w ** 2 - 4 * w + 1) + p1 * (-6 * w ** 2 + 6 * w)
            + m1 * (3 * w ** 2 - 2 * w))
    t, vrel = u * dt, rate.norm(dim=1) / dt
    order = np.lexsort((j.cpu().numpy(), i.cpu().numpy(), t.cpu().numpy()))
    out = {}
    for f, x in (("t", t), ("miss_km", miss), ("v_rel_km_s", vrel)):
        out[f] = np.zeros(len(_record_room(case)))
        out[f][: len(order)] = x.cpu().numpy()[order]
    return out


def exact(case, seed):
    """64-bit values of what `run` computes: states of runs without fragmentation, records of one-shot screening."""
    kind = case["kind"]
    if kind in ("trial", "cascade"):
        return None  # random fragments: no value but the engine's own draws
    if kind == "ensemble":
        _, st, _, al = _ensemble_population(case, seed)
        states = _truth_states(st, al, case["dt"], case["steps"]).cpu().numpy()
        out = np.zeros((case["realisations"] * (case["n"] + MOST_FRAGMENTS), 6))
        out[: len(states)] = states
        return {"states": out}
    st, _, al = _population(case, seed)
    if kind == "screen":
        return {"records": _truth_screen(case, st, al)}
    return {"states": _truth_states(st, al, case["dt"], case["steps"])}
