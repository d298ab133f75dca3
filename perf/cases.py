"""Performance cases of the Hermite force path, through the Python entry points.

Four kinds of call make up what a program does with this library:

* "step"       one block step of a host-driven integrator: the corrected
               particles go in (set_jp_records on the first nact slots), every
               particle is predicted, the force on the first nact slots comes
               back.  nact = n is the start-up pass over all particles.
* "potential"  the potential of every particle (each energy diagnostic).
* "integrate"  a whole run on the device: start-up, block steps to t, the
               records back.
* "ensemble"   the same for many independent clusters together.

A case holds the kind, the scheme's order, the sizes, the precision ("fp64",
"mixed", or "dd": 8th order with double-double positions) and, for runs, the
end time 1 / tinv.  Runs are 4th order: there a record holds what the force
gives.  At 6th and 8th order it also holds derivatives that the corrector forms
from differences of forces over powers of the step, so the last bits of a sum's
order show in them; the steps above cover those orders' arithmetic.
"""
import math

import numpy as np
import torch

from hermite_b200 import Ensemble, Gravity
from hermite_b200.ic import plummer, power_law_masses, records

# Floating-point operations per interaction as the Hermite literature counts
# them, by order.
FLOPS = {4: 60, 6: 97, 8: 144}
POT_FLOPS = 14
# Sizes of random derivatives acc, jrk, snp, crk, d4a, d5a in N-body units.
DERIV_SCALES = (1.0, 3.0, 10.0, 30.0, 100.0, 300.0)
TNOW = 1.0 / 256


def _step(name, order, n, nact, prec="fp64"):
    return {"name": name, "kind": "step", "order": order, "n": n, "nact": nact, "prec": prec}


def listed():
    return [
        # the bulk of a 1k star cluster's block steps: a few tens of particles
        _step("step o4 n1024 a19", 4, 1024, 19),
        # the innermost block steps of a quarter-million-body run: one particle
        _step("step o6 n262144 a1", 6, 262144, 1),
        # and the next levels up, some tens of particles
        _step("step o6 n262144 a45", 6, 262144, 45),
        # the mean block step of a 64k-body 4th-order run
        _step("step o4 n65536 a1044", 4, 65536, 1044),
        # an upper level of a 6th-order run, not a multiple of any tile
        _step("step o6 n262144 a3001", 6, 262144, 3001),
        # a middle level of the largest 8th-order configuration
        _step("step o8 n1048576 a2100", 8, 1 << 20, 2100),
        # the start-up pass of a 6th-order run: every particle active
        _step("step o6 n131072 all", 6, 131072, 131072),
        # the same in mixed precision, an odd size
        _step("step o4 n65537 all mixed", 4, 65537, 65537, "mixed"),
        # the energy diagnostic of a 100k-body run
        {"name": "potential o6 n100003", "kind": "potential", "order": 6, "n": 100003, "prec": "fp64"},
        # a small cluster to its first synchronised time
        {"name": "integrate o4 n1024", "kind": "integrate", "order": 4, "n": 1024, "prec": "fp64",
         "tinv": 8},
        # a window of a medium run
        {"name": "integrate o4 n16384", "kind": "integrate", "order": 4, "n": 16384, "prec": "fp64",
         "tinv": 128},
        # an ensemble of small clusters with a mass spectrum
        {"name": "ensemble o4 32x256-4096", "kind": "ensemble", "order": 4, "clusters": 32,
         "nmin": 256, "nmax": 4096, "prec": "fp64", "tinv": 128},
    ]


def _log_int(rng, lo, hi):
    """An integer, uniform in its logarithm over [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    u = rng.random()
    order = rng.choice([4, 6, 6, 8])
    if u < 0.62:
        v = rng.random()
        prec = "fp64" if v < 0.72 else "mixed"
        if order == 8 and v > 0.93:
            prec = "dd"
        n = _log_int(rng, 512, {4: 1 << 18, 6: 1 << 19, 8: 1 << 20}[order])
        # as many active particles as cost no more than the largest listed case
        cap = max(1, min(n, int(131072 * 131072 * FLOPS[6] * 0.8 / FLOPS[order] / n)))
        nact = cap if rng.random() < 0.15 else _log_int(rng, 1, cap)
        return {"kind": "step", "order": order, "n": n, "nact": nact, "prec": prec}
    if u < 0.77:
        return {"kind": "potential", "order": order, "n": _log_int(rng, 512, 160000), "prec": "fp64"}
    if u < 0.90:
        n = _log_int(rng, 256, 12000)
        return {"kind": "integrate", "order": 4, "n": n, "prec": "fp64",
                "tinv": 16 if n < 3000 else 128}
    lo = _log_int(rng, 128, 1024)
    return {"kind": "ensemble", "order": 4, "clusters": rng.randint(5, 32), "nmin": lo,
            "nmax": _log_int(rng, lo + 1, 4096), "prec": "fp64", "tinv": 128}


def _eps2(n):
    return (4.0 / n) ** 2


def _records(case, seed):
    """Particles of a Plummer sphere between their own times and now: every
    derivative non-zero, block-step spread of tlast."""
    order, n = case["order"], case["n"]
    rng = np.random.default_rng([seed, 1])
    rec = records(plummer(n, seed), order)
    for k in range(order - 2):
        rec[:, 8 + 3 * k:11 + 3 * k] = rng.standard_normal((n, 3)) * DERIV_SCALES[k]
    rec[:, 7] = rng.choice([0.0, 1 / 512, 3 / 1024, TNOW], size=n)
    if case["prec"] == "dd":
        low = rec[:, 0:3] * rng.uniform(-2.0 ** -53, 2.0 ** -53, (n, 3))
        rec = np.ascontiguousarray(np.concatenate([rec, low], axis=1))
    return rec


def _sizes(case):
    """Cluster sizes, uniform in their logarithm (the same for every seed)."""
    rng = np.random.default_rng([case["nmin"], case["nmax"], case["clusters"]])
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return [int(round(math.exp(x))) for x in rng.uniform(lo, hi, case["clusters"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "potential"):
        rec = _records(case, seed)
        g = Gravity(case["order"], case["n"], case["prec"])
        g.set_jp_records(rec)
        g.predict_all(TNOW)
        g.synchronize()
        if kind == "potential":
            return {"case": case, "g": g, "out": np.empty(case["n"])}
        nact = case["nact"]
        return {"case": case, "g": g, "new": np.ascontiguousarray(rec[:nact]),
                "out": np.empty((nact, g.F))}
    if kind == "integrate":
        rec = records(plummer(case["n"], seed), case["order"])
        return {"case": case, "g": Gravity(case["order"], case["n"], case["prec"]), "rec": rec}
    sizes = _sizes(case)
    recs = []
    for c, n in enumerate(sizes):
        m = power_law_masses(n, np.random.default_rng([seed, 3, c]))
        recs.append(records(plummer(n, seed * 1000 + c, masses=m), case["order"]))
    return {"case": case, "e": Ensemble(case["order"], sizes, case["prec"]), "recs": recs}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        g = state["g"]
        g.set_jp_records(state["new"])
        g.predict_all(TNOW)
        return g.calc_force_on_first_nact(case["nact"], _eps2(case["n"]), out=state["out"])
    if kind == "potential":
        return state["g"].calc_potential(_eps2(case["n"]), out=state["out"])
    eta = 0.01
    t = 1.0 / case["tinv"]
    if kind == "integrate":
        g = state["g"]
        g.set_jp_records(state["rec"])
        g.integrator_init(0.0, _eps2(case["n"]), eta, eta / 4, t)
        g.integrator_run(t)
        return g.get_records()
    e = state["e"]
    for c, rec in enumerate(state["recs"]):
        e.set_cluster(c, rec, _eps2(e.sizes[c]))
    e.init(0.0, eta, eta / 4, t)
    e.run(t)
    return np.concatenate([e.get_cluster(c) for c in range(len(e.sizes))])


def _words(case):
    """Doubles of a particle's record and of its force record."""
    order = case["order"]
    return 8 + 3 * (order - 2) + (3 if case["prec"] == "dd" else 0), 3 * (order // 2)


def work(case):
    """Interactions at the counts above; bytes: what comes from the caller and
    goes back, and one read of the particles where they stay on the device.
    Runs: the mean particle takes about 6000 steps per time unit."""
    R, F = _words(case)
    kind, order = case["kind"], case["order"]
    if kind == "step":
        n, nact = case["n"], case["nact"]
        return {"bytes": 8.0 * (n * R + nact * R + nact * F), "flops": float(FLOPS[order]) * n * nact}
    if kind == "potential":
        n = case["n"]
        return {"bytes": 8.0 * n * 5, "flops": float(POT_FLOPS) * n * n}
    rate = 6000.0
    if kind == "integrate":
        n = float(case["n"])
        nn = n * n
    else:
        a, b, k = case["nmin"], case["nmax"], case["clusters"]
        ln = math.log(b / a)
        n = k * (b - a) / ln
        nn = k * (b * b - a * a) / (2.0 * ln)
    return {"bytes": 8.0 * 2 * n * R, "flops": FLOPS[order] * (1.0 + rate / case["tinv"]) * nn}


def _predict(rec, order, dd, t):
    """Positions, velocities, ... at time t, and low parts of the positions."""
    dt = (t - rec[:, 7])[:, None]
    der = [rec[:, 0:3], rec[:, 4:7]] + [rec[:, 8 + 3 * k:11 + 3 * k] for k in range(order - 2)]
    out = []
    for q in range(order // 2):
        low = torch.zeros_like(dt)
        for k in range(len(der) - 1, q, -1):
            low = (der[k] + low) * dt / (k - q)
        out.append((der[q] + low) if q or not dd else der[0])
        if q == 0:
            taylor = low
    xl = rec[:, 26:29] + taylor if dd else None
    return out, xl


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("step", "potential"):
        return None          # a whole run: thousands of dependent steps
    n = case["n"]
    rows = case["nact"] if kind == "step" else n
    order, dd = case["order"], case["prec"] == "dd"
    if rows * n * (FLOPS[order] if kind == "step" else POT_FLOPS) > 1.8e12:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rec = torch.from_numpy(_records(case, seed)).to(dev)
    eps2 = _eps2(n)
    m = rec[:, 3]
    if kind == "step":
        q, xl = _predict(rec, order, dd, TNOW)
    else:
        q, xl = [rec[:, 0:3]], None
    q = [v.T.contiguous() for v in q]                 # 3 x n each
    xl = xl.T.contiguous() if xl is not None else None
    out = torch.empty((rows, 3 * (order // 2)) if kind == "step" else (rows,), dtype=torch.float64,
                      device=dev)
    block = max(1, (1 << 21) // n)
    for i0 in range(0, rows, block):
        i1 = min(rows, i0 + block)
        d = [[v[k][None, :] - v[k][i0:i1, None] for k in range(3)] for v in q]
        if xl is not None:
            d[0] = [d[0][k] + (xl[k][None, :] - xl[k][i0:i1, None]) for k in range(3)]

        def dot(a, b):
            return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

        r2 = dot(d[0], d[0])
        ri2 = 1.0 / (r2 + eps2)
        if kind == "potential":
            w = m * ri2.sqrt()
            w[torch.arange(i1 - i0, device=dev), torch.arange(i0, i1, device=dev)] = 0.0
            out[i0:i1] = -w.sum(1)
            continue
        mr3 = m * ri2 * ri2.sqrt()
        if dd:
            mr3 = torch.where(r2 == 0.0, torch.zeros_like(mr3), mr3)
        dr, dv = d[0], d[1]
        al = dot(dr, dv) * ri2
        t = [dv[k] - 3.0 * al * dr[k] for k in range(3)]
        terms = [dr, t]
        if order >= 6:
            da = d[2]
            be = (dot(dv, dv) + dot(dr, da)) * ri2 + al * al
            u = [da[k] - 6.0 * al * t[k] - 3.0 * be * dr[k] for k in range(3)]
            terms.append(u)
        if order >= 8:
            dj = d[3]
            ga = (3.0 * dot(dv, da) + dot(dr, dj)) * ri2 + al * (3.0 * be - 4.0 * al * al)
            terms.append([dj[k] - 9.0 * al * u[k] - 9.0 * be * t[k] - 3.0 * ga * dr[k]
                          for k in range(3)])
        for c, w in enumerate(terms):
            for k in range(3):
                out[i0:i1, 3 * c + k] = (mr3 * w[k]).sum(1)
    return out.cpu().numpy()
