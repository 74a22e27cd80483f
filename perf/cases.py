"""The work that is timed: force evaluations, time steps, ensembles, planetary
systems, recorded runs and adjoints, each through the calls a user's program
makes (aster_b200.api), on the seeded distributions of aster_b200.gen.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program has in hand before the call, run() is one pass, work()
what the pass cannot do without, exact() the same outputs in 64 bits by plain
torch and numpy. The states of the stepping cases move on from pass to pass,
as a running simulation's do.
"""
import math

import numpy as np
import torch

from aster_b200 import gen
from aster_b200.api import (COLLECT_CENTER, COLLECT_ENERGY, COLLECT_ENERGY_ERROR, COLLECT_MOMENTUM, EIH, FP64,
                            LEAPFROG, MIXED, NEWTON, PN1, PN2, PN25, SOLVER_ALLPAIRS, SOLVER_LBVH, UPDATER_KDK,
                            UPDATER_SABA, YOSHIDA4, Context, CudaLBVH, Params, Simulation)

PREC = {"fp64": FP64, "mixed": MIXED}
LAW = {"newton": NEWTON, "pn1": NEWTON | PN1, "pn": NEWTON | PN1 | PN2 | PN25, "eih": NEWTON | PN1 | EIH}
COLLECT = COLLECT_ENERGY | COLLECT_ENERGY_ERROR | COLLECT_MOMENTUM | COLLECT_CENTER


def listed():
    return [
        # one force evaluation of a small cluster: the call a host program makes every step (latency)
        dict(name="forces_small", kind="forces", dist="plummer", n=1000, precision="fp64", law="newton", eps=0.01),
        # the cold disk with a central mass, plain FP64: the largest direct sum
        dict(name="forces_disk", kind="forces", dist="disk", n=262144, precision="fp64", law="newton", eps=0.002),
        # a relativistic cluster, unsoftened, odd size
        dict(name="forces_pn1", kind="forces", dist="plummer", n=30011, precision="fp64", law="pn1", eps=0.0),
        # the mixed-precision direct sum at an odd middle size
        dict(name="forces_mixed", kind="forces", dist="disk", n=100003, precision="mixed", law="newton", eps=0.002),
        # the 4096-body Plummer sphere, 100 KDK steps with the energy before and after
        dict(name="integrate_plummer", kind="integrate", n=4096, precision="fp64", steps=100, eps=0.01, dt=1e-3),
        # a recorded run: SABA4 with energy, momentum and centre of mass after every second step
        dict(name="record_saba4", kind="record", n=12001, precision="fp64", order=4, steps=6, rate=2, eps=0.01,
             dt=1e-3),
        # Barnes-Hut at 2^20 bodies, lognormal masses, ten steps on host-resident (pinned) state
        dict(name="tree_steps_1m", kind="tree", n=1048576, precision="mixed", steps=10, host=True, law="newton",
             eps=0.005, dt=5e-4, theta=0.5),
        # Barnes-Hut at an interactive size: fifty device-resident steps, then a snapshot
        dict(name="tree_steps_20k", kind="tree", n=20011, precision="mixed", steps=50, host=False, law="newton",
             eps=0.005, dt=5e-4, theta=0.5),
        # one FP64 tree step per call, the state kept by a host program
        dict(name="tree_host_fp64", kind="tree", n=131073, precision="fp64", steps=1, host=True, law="newton",
             eps=0.005, dt=5e-4, theta=0.5),
        # the batched few-body ensemble with 1PN terms
        dict(name="ensemble_pn1", kind="ensemble", systems=16384, precision="mixed", law="pn1", steps=100,
             integrator="yoshida4", dt=1e-4),
        # a star, eight planets and a belt of test particles
        dict(name="planets_belt", kind="planets", planets=8, particles=262144, precision="fp64", steps=20, dt=0.02),
        # gradients of a trajectory loss, forward and reverse
        dict(name="adjoint_plummer", kind="adjoint", n=16384, precision="mixed", steps=32, every=16, eps=0.01,
             dt=1e-3),
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    kind = rng.choice(["forces", "forces", "integrate", "record", "tree", "tree", "ensemble", "planets", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "forces":
        law = rng.choice(["newton", "newton", "pn1", "pn"])
        n = _size(rng, 300, {"newton": 250000, "pn1": 60000, "pn": 30000}[law])
        return dict(kind=kind, dist=rng.choice(["plummer", "disk"]), n=n, precision=precision, law=law,
                    eps=rng.choice([0.0, 0.002, 0.01]))
    if kind == "integrate":
        n = _size(rng, 500, 16000)
        return dict(kind=kind, n=n, precision=precision, steps=rng.randint(10, 100), eps=0.01, dt=1e-3)
    if kind == "record":
        n = _size(rng, 500, 16000)
        return dict(kind=kind, n=n, precision=precision, order=rng.choice([0, 2, 4, 6]), steps=rng.randint(4, 16),
                    rate=rng.randint(1, 4), eps=0.01, dt=1e-3)
    if kind == "tree":
        law = rng.choice(["newton", "newton", "newton", "pn1"])
        n = _size(rng, 2000, 1000000)
        steps = rng.randint(1, 50) if n < 50000 else rng.randint(1, 8)
        return dict(kind=kind, n=n, precision=precision, steps=steps, host=rng.random() < 0.5, law=law, eps=0.005,
                    dt=5e-4, theta=rng.choice([0.4, 0.5, 0.7]))
    if kind == "ensemble":
        s = _size(rng, 64, 16000)
        return dict(kind=kind, systems=s, precision=precision, law=rng.choice(["newton", "pn1", "pn", "eih"]),
                    steps=rng.randint(10, 60), integrator=rng.choice(["yoshida4", "leapfrog"]), dt=1e-4)
    if kind == "planets":
        return dict(kind=kind, planets=rng.randint(2, 12), particles=_size(rng, 100, 250000), precision="fp64",
                    steps=rng.randint(2, 40), dt=rng.choice([0.01, 0.02, 0.05]))
    n = _size(rng, 300, 16000)
    return dict(kind="adjoint", n=n, precision=precision, steps=rng.randint(8, 24), every=rng.choice([4, 8, 16]),
                eps=0.01, dt=1e-3)


def _bodies(case, seed):
    """Initial conditions of a case: positions, velocities, masses."""
    if case["kind"] == "forces" and case["dist"] == "disk":
        return gen.exponential_disk(case["n"], seed)
    return gen.plummer(case["n"], seed, masses="lognormal" if case["kind"] == "tree" else "equal")


def _params(case):
    return Params(G=1.0, c=100.0, eps2=case.get("eps", 0.0) ** 2, theta=case.get("theta", 0.5),
                  dt=case.get("dt", 1e-3), force_law=LAW[case.get("law", "newton")])


def _ensemble(case, seed):
    """Systems of 3 to 64 bodies, every size as often, in a mixed order that the seed does not change."""
    sizes = np.random.default_rng(0).permutation(3 + np.arange(case["systems"]) % 62)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    pos, vel, m = np.empty((off[-1], 3)), np.empty((off[-1], 3)), np.empty(off[-1])
    for k in range(3, 65):
        which = np.nonzero(sizes == k)[0]
        if len(which):
            at = (off[which][:, None] + np.arange(k)).ravel()
            pos[at], vel[at], m[at], _ = gen.hierarchical_ensemble(len(which), seed * 64 + k, k, k)
    return pos, vel, m, off


def _target(case, pos, seed):
    return pos + np.random.default_rng(seed + 1).normal(0.0, 1e-2, pos.shape)


def _pinned(a):
    """A copy of `a` in page-locked host memory, as a numpy array."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "ensemble":
        pos, vel, m, off = _ensemble(case, seed)
        s["ctx"] = Context(0).ensemble_upload(off, pos, vel, m)
        s["p"] = _params(case)
        return s
    if kind == "planets":
        pos, vel, m = gen.planetary_system(case["planets"], case["particles"], seed)
        s["ctx"] = Context(0).upload(pos, vel, m)
        s["p"] = _params(case)
        return s
    pos, vel, m = _bodies(case, seed)
    if kind == "integrate":
        sim = Simulation(pos, vel, m, dt=case["dt"], softening=case["eps"] ** 2)
        sim.solver.precision = PREC[case["precision"]]
        s["sim"] = sim.load()
        return s
    s["p"] = _params(case)
    s["ctx"] = Context(0).upload(pos, vel, m)
    if kind == "tree" and case["host"]:
        acc = s["ctx"].lbvh_forces(s["p"], PREC[case["precision"]])
        s["host"] = [_pinned(a) for a in (pos, vel, acc, m)]
    if kind == "adjoint":
        s["target"] = _target(case, pos, seed)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "integrate":
        sim = state["sim"]
        r = sim.integrate(case["steps"], precision_test=True)
        b = sim.bodies
        # (the report's relative energy change follows from the two energies)
        return dict(pos=b.positions, vel=b.velocities, acc=b.accs, e0=r["initial_energy"], e1=r["final_energy"])
    ctx, p, prec = state["ctx"], state["p"], PREC[case["precision"]]
    if kind == "forces":
        return ctx.allpairs(p, prec)
    if kind == "record":
        rows, _ = ctx.record(p, case["steps"], updater=UPDATER_SABA if case["order"] else UPDATER_KDK,
                             order=case["order"] or 2, solver=SOLVER_ALLPAIRS, precision=prec, rate=case["rate"],
                             collect=COLLECT)
        pos, vel, _ = ctx.download()
        return dict(rows=rows, pos=pos, vel=vel)
    if kind == "tree":
        if case["host"]:
            pos, vel, acc, m = state["host"]
            ctx.kdk_steps_host(p, case["steps"], pos, vel, acc, m, CudaLBVH.kind, prec)
        else:
            ctx.kdk_steps(p, case["steps"], SOLVER_LBVH, prec)
            pos, vel, acc = ctx.download()
        return dict(pos=pos, vel=vel, acc=acc)
    if kind == "ensemble":
        ctx.ensemble_run(p, case["steps"], YOSHIDA4 if case["integrator"] == "yoshida4" else LEAPFROG, prec)
        pos, vel = ctx.ensemble_download()
        return dict(pos=pos, vel=vel)
    if kind == "planets":
        ctx.wh_steps(p, case["steps"], prec)
        pos, vel, _ = ctx.download()
        return dict(pos=pos, vel=vel)
    loss, gx, gv, gm = ctx.adjoint(p, case["steps"], state["target"], prec, case["every"])
    return dict(loss=loss, gx=gx, gv=gv, gm=gm)


#: operations of one unordered pair whose force is formed once and applied to both bodies: separation 3, squared
#: distance 6, inverse cube 4, and per body a product and a three-component update (7)
PAIR = {"newton": 27.0, "pn1": 100.0, "pn": 300.0, "eih": 140.0}


def work(case):
    kind = case["kind"]
    law = PAIR[case.get("law", "newton")]
    if kind == "ensemble":
        mean = 0.5 * (3 + 64)
        pairs = case["systems"] * sum(k * (k - 1) / 2 for k in range(3, 65)) / 62
        stages = 3 if case["integrator"] == "yoshida4" else 1
        return dict(bytes=case["systems"] * mean * (56 + 48), flops=pairs * law * stages * case["steps"])
    if kind == "planets":
        n = 1 + case["planets"] + case["particles"]
        # per body and step: a Kepler drift of about 250 operations and the planets' pull
        return dict(bytes=n * (56.0 + 48.0), flops=case["steps"] * n * (250.0 + 20.0 * case["planets"]))
    n = float(case["n"])
    pair = n * (n - 1) / 2
    if kind == "forces":
        vel = 24 if case["law"] != "newton" else 0
        return dict(bytes=n * (32 + vel + 24), flops=pair * law)
    if kind == "integrate":  # one evaluation a step and the two energies
        return dict(bytes=n * (56 + 72), flops=pair * (law * case["steps"] + 2 * 14.0))
    if kind == "record":
        rows = case["steps"] // case["rate"] + 1
        return dict(bytes=n * (56 + 48), flops=pair * (law * max(1, case["order"]) * case["steps"] + rows * 14.0))
    if kind == "tree":
        # interactions per body: about 160 log2(n) at theta 0.5, falling as theta^-2
        inter = n * min(n, 160.0 * math.log2(n) * (0.5 / case["theta"]) ** 2 - 700.0)
        return dict(bytes=case["steps"] * n * 240.0, flops=case["steps"] * inter * 20.0 * law / 27.0)
    # adjoint: a forward and a recomputed force evaluation and one tidal sweep (about 60 a pair) a step
    return dict(bytes=n * (56 + 24 + 56), flops=pair * case["steps"] * (2 * law + 60.0))


# ---- the same outputs in 64 bits ------------------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


def _chunks(rows, cols):
    step = max(1, int(3.2e7) // max(1, cols))
    return [(a, min(rows, a + step)) for a in range(0, rows, step)]


def _pn_terms(n, dv, inv, mi, mj, vi, vj, c, law):
    """Post-Newtonian accelerations (G = 1) of pairs: n the unit vectors from j to i, dv = v_i - v_j, inv = 1/r."""
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    v1, v2, v12, a1, a2 = dot(vi, vi), dot(vj, vj), dot(vi, vj), dot(n, vi), dot(n, vj)
    q = mj * inv * inv
    A = -v1 - 2 * v2 + 4 * v12 + 1.5 * a2 * a2 + (5 * mi + 4 * mj) * inv
    B = 4 * a1 - 3 * a2
    out = [q / c ** 2 * (n[k] * A + dv[k] * B) for k in range(3)]
    if law != "pn":
        return out
    p1, p2 = mi * inv, mj * inv
    S = (-2 * v2 ** 2 + 4 * v2 * v12 - 2 * v12 ** 2 + 1.5 * v1 * a2 ** 2 + 4.5 * v2 * a2 ** 2 - 6 * v12 * a2 ** 2
         - 1.875 * a2 ** 4 + p1 * (-3.75 * v1 + 1.25 * v2 - 2.5 * v12 + 19.5 * a1 ** 2 - 39 * a1 * a2 + 8.5 * a2 ** 2)
         + p2 * (4 * v2 - 8 * v12 + 2 * a1 ** 2 - 4 * a1 * a2 - 6 * a2 ** 2)
         - 14.25 * p1 ** 2 - 9 * p2 ** 2 - 34.5 * p1 * p2)
    W = (v1 * a2 + 4 * v2 * a1 - 5 * v2 * a2 - 4 * v12 * a1 + 4 * v12 * a2 - 6 * a1 * a2 ** 2 + 4.5 * a2 ** 3
         + p1 * (-15.75 * a1 + 13.75 * a2) + p2 * (-2 * a1 - 2 * a2))
    d2 = dot(dv, dv)
    I1 = -d2 + 2 * p1 - 8 * p2
    I2 = (a1 - a2) * (3 * d2 - 6 * p1 + 52.0 / 3.0 * p2)
    for k in range(3):
        out[k] = out[k] + q / c ** 4 * (n[k] * S + dv[k] * W) + 0.8 * p1 * q / c ** 5 * (dv[k] * I1 + n[k] * I2)
    return out


def _forces(x, v, m, eps2, law="newton", c=100.0):
    """Accelerations of all bodies by the direct sum."""
    out = torch.empty_like(x)
    for a, b in _chunks(len(x), len(x)):
        d = [x[None, :, k] - x[a:b, None, k] for k in range(3)]
        r2 = d[0] * d[0]
        r2 += d[1] * d[1]
        r2 += d[2] * d[2]
        r2 += eps2
        if eps2 == 0.0:
            r2[r2 == 0.0] = math.inf
        inv = r2.rsqrt_()
        s = inv * inv
        s *= inv
        s *= m[None, :]
        for k in range(3):
            out[a:b, k] = (s * d[k]).sum(1)
        if law != "newton":
            n = [-dk * inv for dk in d]
            vi, vj = [v[a:b, None, k] for k in range(3)], [v[None, :, k] for k in range(3)]
            pn = _pn_terms(n, [vi[k] - vj[k] for k in range(3)], inv, m[a:b, None], m[None, :], vi, vj, c, law)
            for k in range(3):
                out[a:b, k] += pn[k].sum(1)
    return out


def _energy(x, v, m, eps2, ref_form):
    pot = torch.zeros((), dtype=torch.float64, device=x.device)
    for a, b in _chunks(len(x), len(x)):
        r2 = sum((x[None, :, k] - x[a:b, None, k]) ** 2 for k in range(3))
        r = r2.sqrt() + eps2 if ref_form else (r2 + eps2).sqrt()
        w = m[a:b, None] * m[None, :] / r
        i = torch.arange(a, b, device=x.device)
        w[i - a, i] = 0.0
        pot += w.sum()
    return float(0.5 * (m * (v * v).sum(1)).sum() - 0.5 * pot)


def _kdk(x, v, m, steps, dt, force):
    a = force(x, v)
    for _ in range(steps):
        v = v + a * (0.5 * dt)
        x = x + v * dt
        a = force(x, v)
        v = v + a * (0.5 * dt)
    return x, v, a


def _saba(x, v, order, steps, dt, force):
    z, w = np.polynomial.legendre.leggauss(order)
    t = 0.5 * (1.0 + z)
    c = np.diff(np.concatenate([[0.0], t, [1.0]]))
    for _ in range(steps):
        x = x + v * (c[0] * dt)
        for k in range(order):
            v = v + force(x, v) * (0.5 * w[k] * dt)
            x = x + v * (c[k + 1] * dt)
    return x, v


def _exact_record(case, x, v, m):
    eps2, dt = case["eps"] ** 2, case["dt"]
    force = lambda y, u: _forces(y, u, m, eps2)  # noqa: E731
    rows, e0, done = [], None, 0

    def sample():
        nonlocal e0
        e = _energy(x, v, m, eps2, True)
        e0 = e if e0 is None else e0
        mom, cen = (m[:, None] * v).sum(0), (m[:, None] * x).sum(0) / m.sum()
        rows.append([float(done), e, abs(e - e0) / abs(e0)] + mom.tolist() + cen.tolist())

    sample()
    while done < case["steps"]:
        k = min(case["rate"], case["steps"] - done)
        if case["order"]:
            x, v = _saba(x, v, case["order"], k, dt, force)
        else:
            x, v, _ = _kdk(x, v, m, k, dt, force)
        done += k
        if k == case["rate"]:
            sample()
    return dict(rows=np.array(rows), pos=x, vel=v)


def _ens_acc(x, v, m, law, c=100.0):
    """Accelerations of systems padded to one size: x (systems, size, 3); padding has no mass."""
    d = [x[:, None, :, k] - x[:, :, None, k] for k in range(3)]
    r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
    r2[r2 == 0.0] = math.inf
    inv = r2.rsqrt()
    mi, mj = m[:, :, None].expand_as(inv), m[:, None, :].expand_as(inv)
    s = mj * inv ** 3
    acc = torch.stack([(s * d[k]).sum(2) for k in range(3)], 2)
    if law == "newton":
        return acc
    vi = [v[:, :, None, k].expand_as(inv) for k in range(3)]
    vj = [v[:, None, :, k].expand_as(inv) for k in range(3)]
    dv = [vi[k] - vj[k] for k in range(3)]
    n = [-d[k] * inv for k in range(3)]
    if law != "eih":
        pn = _pn_terms(n, dv, inv, mi, mj, vi, vj, c, law)
        return acc + torch.stack([p.sum(2) for p in pn], 2)
    dot = lambda a, b: a[0] * b[0] + a[1] * b[1] + a[2] * b[2]  # noqa: E731
    phi = (mj * inv).sum(2)
    aj = [acc[:, None, :, k].expand_as(inv) for k in range(3)]
    B = (-4 * phi[:, :, None] - phi[:, None, :] + dot(vi, vi) + 2 * dot(vj, vj) - 4 * dot(vi, vj)
         - 1.5 * dot(n, vj) ** 2 + 0.5 * dot(d, aj))
    W = 4 * dot(n, vi) - 3 * dot(n, vj)
    q = mj * inv * inv
    return acc + torch.stack([(q * (d[k] * inv * B + W * dv[k]) + 3.5 * mj * aj[k] * inv).sum(2)
                              for k in range(3)], 2) / c ** 2


def _exact_ensemble(case, pos, vel, m, off):
    sizes = np.diff(off)
    if case["integrator"] == "yoshida4":
        cb = 2.0 ** (1.0 / 3.0)
        w1, w0 = 1.0 / (2.0 - cb), -cb / (2.0 - cb)
        cs, ds = [w1 / 2, (w0 + w1) / 2, (w0 + w1) / 2, w1 / 2], [w1, w0, w1]
    else:
        cs, ds = [0.5, 0.5], [1.0]
    out_x, out_v = np.empty_like(pos), np.empty_like(vel)
    for lo, hi in ((1, 16), (17, 28), (29, 40), (41, 52), (53, 64)):
        which = np.nonzero((sizes >= lo) & (sizes <= hi))[0]
        for part in np.array_split(which, max(1, len(which) * hi * hi // 2000000 + 1)):
            if not len(part):
                continue
            idx = off[part][:, None] + np.arange(hi)[None]
            ok = np.arange(hi)[None] < sizes[part][:, None]
            idx = np.where(ok, idx, 0)
            x, v = _t(pos[idx]), _t(vel[idx])
            mm = _t(np.where(ok, m[idx], 0.0))
            # padding sits apart from every body and from one another, at rest
            far = _t(np.where(ok, 0.0, 1e6 + np.arange(hi)[None]))[:, :, None].expand(-1, -1, 3)
            keep = _t(ok.astype(float))[:, :, None]
            x, v = x * keep + far, v * keep
            for _ in range(case["steps"]):
                for k, dk in enumerate(ds):
                    x = x + v * (cs[k] * case["dt"])
                    v = v + _ens_acc(x, v, mm, case["law"]) * (dk * case["dt"])
                x = x + v * (cs[-1] * case["dt"])
            out_x[idx[ok]], out_v[idx[ok]] = x.cpu().numpy()[ok], v.cpu().numpy()[ok]
    return dict(pos=out_x, vel=out_v)


def _kepler(r, v, mu, dt):
    """(r, v) after dt on its conic about mu: Newton's method on the universal Kepler equation. Steps here are short
    against the orbits, so the Stumpff functions are their series (argument below 1 in size)."""
    r0, s0 = r.norm(dim=1), (r * v).sum(1) / math.sqrt(mu)
    alpha = 2.0 / r0 - (v * v).sum(1) / mu
    x = math.sqrt(mu) * dt / r0
    for it in range(13):
        z = alpha * x * x
        c2 = sum((-z) ** k * (1.0 / math.factorial(2 * k + 2)) for k in range(11))
        c3 = sum((-z) ** k * (1.0 / math.factorial(2 * k + 3)) for k in range(11))
        rx = x * x * c2 + s0 * x * (1.0 - z * c3) + r0 * (1.0 - z * c2)
        if it == 12:
            break
        x = x - (x ** 3 * c3 + s0 * x * x * c2 + r0 * x * (1.0 - z * c3) - math.sqrt(mu) * dt) / rx
    f, g = 1.0 - x * x * c2 / r0, dt - x ** 3 * c3 / math.sqrt(mu)
    rn = f[:, None] * r + g[:, None] * v
    r1 = rn.norm(dim=1)
    fd, gd = math.sqrt(mu) / (r1 * r0) * x * (z * c3 - 1.0), 1.0 - x * x * c2 / r1
    return rn, fd[:, None] * r + gd[:, None] * v


def _exact_planets(case, x, v, m):
    """Wisdom-Holman in democratic heliocentric coordinates, kick and linear drift of half a step at either end."""
    dt, massive = case["dt"], int((m > 0).sum())
    M = m.sum()
    xc, vc = (m[:, None] * x).sum(0) / M, (m[:, None] * v).sum(0) / M
    q, u, mp = x[1:] - x[0], v[1:] - vc, m[1:]

    def pull(q):
        a = torch.zeros_like(q)
        for j in range(massive - 1):
            d = q[j] - q
            r2 = (d * d).sum(1)
            r2[j] = math.inf
            a += (mp[j] / (r2 * r2.sqrt()))[:, None] * d
        return a

    for _ in range(case["steps"]):
        q = q + (mp[:, None] * u).sum(0) / m[0] * (0.5 * dt)
        u = u + pull(q) * (0.5 * dt)
        q, u = _kepler(q, u, float(m[0]), dt)
        q = q + (mp[:, None] * u).sum(0) / m[0] * (0.5 * dt)
        u = u + pull(q) * (0.5 * dt)
    x0 = xc + vc * (dt * case["steps"]) - (mp[:, None] * q).sum(0) / M
    v0 = vc - (mp[:, None] * u).sum(0) / m[0]
    return dict(pos=torch.cat([x0[None], q + x0]), vel=torch.cat([v0[None], u + vc]))


def _tidal(x, m, w, eps2):
    """J(x)^T w and (dA/dm)^T w of the softened accelerations."""
    gx, gm = torch.empty_like(x), torch.empty_like(m)
    for a, b in _chunks(len(x), len(x)):
        d = [x[None, :, k] - x[a:b, None, k] for k in range(3)]
        s2 = 1.0 / (d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + eps2)
        s3 = s2 * s2.sqrt()
        u = [m[a:b, None] * w[None, :, k] - m[None, :] * w[a:b, None, k] for k in range(3)]
        t = 3 * s3 * s2 * (d[0] * u[0] + d[1] * u[1] + d[2] * u[2])
        for k in range(3):
            gx[a:b, k] = (s3 * u[k] - t * d[k]).sum(1)
        gm[a:b] = -(s3 * (d[0] * w[None, :, 0] + d[1] * w[None, :, 1] + d[2] * w[None, :, 2])).sum(1)
    return gx, gm


def _exact_adjoint(case, x, v, m, target):
    eps2, dt, h = case["eps"] ** 2, case["dt"], 0.5 * case["dt"]
    path, a = [], _forces(x, v, m, eps2)
    for _ in range(case["steps"]):
        path.append(x)
        v = v + a * h
        x = x + v * dt
        a = _forces(x, v, m, eps2)
        v = v + a * h
    r = x - target
    lx, lv, lm = 2.0 / len(x) * r, torch.zeros_like(x), torch.zeros_like(m)
    for t in range(case["steps"] - 1, -1, -1):
        lv = lv + dt * lx
        gx, gm = _tidal(path[t], m, (2.0 if t else 1.0) * h * lv, eps2)
        lx, lm = lx + gx, lm + gm
    return dict(loss=float((r * r).sum() / len(x)), gx=lx, gv=lv, gm=lm)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return _exact_ensemble(case, *_ensemble(case, seed))
    if kind == "planets":
        x, v, m = (_t(a) for a in gen.planetary_system(case["planets"], case["particles"], seed))
        return _exact_planets(case, x, v, m)
    # the value that a tree walk approximates is the direct sum: too long for large trees
    if kind == "tree" and float(case["n"]) ** 2 * (case["steps"] + 1) * (8 if case["law"] != "newton" else 1) > 6e10:
        return None
    pos, vel, m = _bodies(case, seed)
    x, v, m = _t(pos), _t(vel), _t(m)
    eps2, dt = case["eps"] ** 2, case.get("dt", 0.0)
    if kind == "forces":
        return _forces(x, v, m, eps2, case["law"])
    if kind == "integrate":
        y, u, a = _kdk(x, v, m, case["steps"], dt, lambda y, u: _forces(y, u, m, eps2))
        return dict(pos=y, vel=u, acc=a, e0=_energy(x, v, m, eps2, False), e1=_energy(y, u, m, eps2, False))
    if kind == "record":
        return _exact_record(case, x, v, m)
    if kind == "adjoint":
        return _exact_adjoint(case, x, v, m, _t(_target(case, pos, seed)))
    law = case["law"]
    y, u, a = _kdk(x, v, m, case["steps"], dt, lambda y, u: _forces(y, u, m, eps2, law))
    return dict(pos=y, vel=u, acc=a)
