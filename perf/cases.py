"""The force evaluations and integration steps that this engine is measured on.

Every case goes through the public entry points of `fmms_b200` as a program
that uses the engine calls them: `refresh` / `run` on host arrays (the
reference solver's interface), `build_device` + `evaluate_device` on resident
bodies (an external integrator), `build_ensemble_device` (many systems in one
forest), `kdk_step_device` (a serving tick), `leapfrog_device` (a resident
simulation) and `direct_targets` (the accuracy check). The bodies come from
the seeded generators of the package; sizes, orders and opening criteria are
those of the benchmark configurations, the tests and the serving loop.

Keys of a case:
  call       which entry points a pass goes through (see `run`)
  gen        body distribution: plummer, hernquist, uniform, clusters
  n          bodies (all systems together)
  systems    independent systems in one forest (1: a single tree)
  precision  plain (FP64) or mixed
  mac        theta (opening angle `theta`) or dehnen (accuracy `eps`)
  p, n_leaf, softening, soft_gap   expansion order, leaf capacity, ...
  dt, steps, refresh               time step (short, so that thousands of passes leave the distribution as it is),
                                   steps a pass, tree rebuild interval
  targets                          targets of the direct sum
"""

import math

import numpy as np
import torch

import fmms_b200 as fx

DEFAULTS = dict(systems=1, mac="theta", theta=0.5, eps=1e-5, softening=1e-3, soft_gap=0.0, dt=1e-6, steps=1,
                refresh=1, targets=0)

# the largest system whose exact forces (an O(n^2) sum in FP64) are computed
EXACT_MAX = 140_000


def listed():
    return [
        # a serving tick of the smallest session: launches and read-backs
        dict(name="tick_1k", call="tick", gen="plummer", n=1000, precision="mixed", p=8, n_leaf=64),
        # a serving tick of an ordinary session, an odd number of bodies
        dict(name="tick_30k", call="tick", gen="uniform", n=30_011, precision="mixed", p=8, n_leaf=64),
        # a resident simulation that rebuilds its tree every 8th step
        dict(name="reuse_64k", call="leapfrog", gen="plummer", n=65_536, precision="mixed", p=8, n_leaf=64, steps=8,
             refresh=8),
        # the reference's own call with its defaults: host arrays, error-controlled MAC, FP64
        dict(name="host_16k", call="host", gen="plummer", n=16_384, precision="plain", mac="dehnen", eps=1e-5, p=8,
             n_leaf=16, softening=0.0),
        # an FP64 evaluation under the error-controlled MAC at low order, cuspy profile, ragged size
        dict(name="hernquist_100k", call="eval", gen="hernquist", n=100_003, precision="plain", mac="dehnen", eps=1e-4,
             p=6, n_leaf=16, softening=0.0),
        # an FP64 evaluation of a large uniform system
        dict(name="uniform_fp64_256k", call="eval", gen="uniform", n=1 << 18, precision="plain", p=10, n_leaf=64,
             softening=1e-4),
        # the force evaluation of the million-body benchmark, mixed precision
        dict(name="uniform_1m", call="eval", gen="uniform", n=1 << 20, precision="mixed", p=10, n_leaf=64,
             softening=1e-4),
        # strongly clustered bodies at high order, ragged size
        dict(name="clusters_p12_300k", call="eval", gen="clusters", n=300_007, precision="mixed", theta=0.4, p=12,
             n_leaf=32, softening=1e-5),
        # the headline: one rebuilt kick-drift-kick step of four million clustered bodies
        dict(name="clusters_4m", call="leapfrog", gen="clusters", n=1 << 22, precision="mixed", p=10, n_leaf=32,
             softening=1e-5, soft_gap=200.0),
        # fast low-accuracy forces (previews, collisionless runs)
        dict(name="low_order_200k", call="eval", gen="plummer", n=200_003, precision="mixed", theta=0.7, p=4,
             n_leaf=64, softening=1e-2),
        # a batch of independent systems in one forest, at the autotuner's pick for them
        dict(name="forest_1m", call="forest", gen="plummer", n=1_000_003, systems=48, precision="mixed", theta=0.4,
             p=12, n_leaf=128, soft_gap=400.0),
        # the accuracy check: FP64 direct sum at sampled targets
        dict(name="direct_256k", call="direct", gen="uniform", n=1 << 18, precision="plain", p=1, n_leaf=64,
             softening=1e-4, targets=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["tick", "leapfrog", "host", "eval", "eval", "eval", "forest", "direct"])
    mixed = call in ("tick", "leapfrog", "forest") or (call == "eval" and rng.random() < 0.6)
    c = dict(call=call, precision="mixed" if mixed else "plain")
    c["gen"] = rng.choice(["plummer", "uniform", "clusters"] + ([] if mixed else ["hernquist"]))
    c["p"] = rng.choice([4, 6, 8, 8, 9, 10, 10, 11, 12, 14])
    c["n_leaf"] = rng.choice([16, 32, 48, 64, 64, 96, 128])
    # well below the distances at which the (unsoftened) far field takes over
    c["softening"] = rng.choice({"plummer": [1e-2, 1e-3, 1e-3, 1e-4], "hernquist": [1e-3, 1e-4],
                                 "uniform": [1e-3, 1e-4, 1e-4], "clusters": [1e-4, 1e-5]}[c["gen"]])
    if not mixed and call in ("host", "eval") and rng.random() < 0.6:
        c.update(mac="dehnen", eps=rng.choice([1e-4, 1e-5, 1e-6]), softening=0.0, n_leaf=rng.choice([16, 32, 48]))
        c["n"] = _log_int(rng, 1_000, 150_000)
    else:
        c["theta"] = rng.choice([0.4, 0.5, 0.5, 0.6, 0.7])
        c["n"] = _log_int(rng, 1_000, 1_100_000 if mixed else 270_000)
        if c["softening"] <= 1e-4 and c["n"] > 50_000:
            c["soft_gap"] = rng.choice([0.0, 100.0, 200.0])
    if call == "leapfrog":
        c.update(rng.choice([dict(steps=1), dict(steps=4, refresh=4), dict(steps=8, refresh=8), dict(steps=6, refresh=3)]))
        c["n"] = max(1_000, c["n"] // c["steps"])
        if c["steps"] > 1 and c["gen"] == "clusters":
            c["gen"] = "plummer"  # a reused tree does not suit cores that turn over within a few steps
    elif call == "forest":
        c["systems"] = rng.randint(2, max(2, min(200, c["n"] // 500)))
    elif call == "direct":
        c["targets"] = _log_int(rng, 100, 5_000)
    return c


def _full(case):
    return {**DEFAULTS, **case}


def _bodies(c, seed):
    """(mass, pos, vel, offsets) as host arrays; vel is zero where the generator has none."""
    if c["systems"] > 1:
        g = np.random.default_rng(seed)
        cut = np.exp(g.uniform(np.log(1e3), np.log(1e5), c["systems"]))  # sizes log-uniform over two decades
        sizes = np.maximum(1, np.floor(cut / cut.sum() * c["n"])).astype(np.int64)
        sizes[int(np.argmax(sizes))] += c["n"] - int(sizes.sum())
        parts = [_bodies({**c, "systems": 1, "n": int(k)}, seed * 1009 + i) for i, k in enumerate(sizes)]
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        return tuple(np.concatenate([q[j] for q in parts]) for j in range(3)) + (off,)
    n, seed = c["n"], int(seed) + 1
    vel = None
    if c["gen"] == "plummer":
        mass, pos, vel = fx.gen_plummer_ic(n, 1.0, 1.0, 20.0, seed)
    elif c["gen"] == "clusters":
        mass, pos, vel = fx.gen_clusters(n, 64 if n >= 64_000 else 8, seed=seed)
    elif c["gen"] == "hernquist":
        # truncated at 50 scale radii (4 % of the bodies lie beyond): the profile has no edge of its own
        mass, pos = fx.gen_hernquist(n + n // 16 + 100, seed=seed)
        keep = np.flatnonzero((pos * pos).sum(1) < 2500.0)[:n]
        mass, pos = mass[keep], pos[keep]
        assert len(mass) == n
    else:
        mass, pos = fx.gen_uniform_lognormal(n, seed=seed)
    return mass, pos, np.zeros_like(pos) if vel is None else vel, np.array([0, n], dtype=np.uint64)


def _targets(c, seed):
    return np.sort(np.random.default_rng(seed).choice(c["n"], size=min(c["targets"], c["n"]), replace=False)).astype(np.uint32)


def prepare(case, seed):
    c = _full(case)
    mass, pos, vel, off = _bodies(c, seed)
    s = dict(c=c, mass=mass, pos=pos, off=off)
    if c["call"] == "direct":
        s["targets"] = _targets(c, seed)
        return s
    # the engine context, kept by the program for all its evaluations
    s["g"] = g = fx.Fmm(None, None, c["p"], c["eps"], c["n_leaf"], mac=c["mac"], theta=c["theta"],
                        softening=c["softening"], precision=c["precision"], soft_gap=c["soft_gap"])
    if c["call"] == "host":
        return s
    for k, v in (("d_mass", mass), ("d_pos", pos), ("d_vel", vel)):
        s[k] = torch.from_numpy(v).cuda()
    s["d_acc"] = torch.empty((c["n"], 3), dtype=torch.float64, device="cuda")
    s["d_pot"] = torch.empty(c["n"], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    if c["call"] in ("tick", "leapfrog"):  # a running simulation: forces at the present positions
        s["d_dt"] = torch.full((c["n"],), c["dt"], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        g.build_device(s["d_pos"].data_ptr(), s["d_mass"].data_ptr(), c["n"])
        g.evaluate_device(s["d_pos"].data_ptr(), s["d_mass"].data_ptr(), s["d_acc"].data_ptr(), s["d_pot"].data_ptr())
        g.synchronize()
    return s


def run(s):
    c, call = s["c"], s["c"]["call"]
    if call == "direct":
        acc, pot, f = fx.direct_targets(s["mass"], s["pos"], s["targets"], softening=c["softening"])
        return dict(acc=acc, pot=pot, f=f)
    g = s["g"]
    if call == "host":
        g.refresh(s["mass"], s["pos"])
        r = g.run()
        return dict(acc=r.accel, pot=r.pot)
    pos, vel, mass, acc, pot = (s[k].data_ptr() for k in ("d_pos", "d_vel", "d_mass", "d_acc", "d_pot"))
    if call == "tick":
        g.kdk_step_device(pos, vel, mass, acc, pot, s["d_dt"].data_ptr(), offsets=s["off"])
    elif call == "leapfrog":
        g.leapfrog_device(pos, vel, mass, acc, pot, c["dt"], c["steps"], "kdk", c["refresh"])
    else:
        if call == "forest":
            g.build_ensemble_device(s["off"], pos, mass)
        else:
            g.build_device(pos, mass, c["n"])
        g.evaluate_device(pos, mass, acc, pot)
        return dict(acc=s["d_acc"], pot=s["d_pot"])
    return dict(pos=s["d_pos"], vel=s["d_vel"], acc=s["d_acc"], pot=s["d_pot"])


def work(case):
    """Bytes: bodies in and results out, once per evaluation. Flops: an estimate of the method's arithmetic from the
    opening angle alone, for a uniform system with half-full leaves -- a leaf's near field holds the leaves within
    2 rho / theta of it (16 flops a body pair) and a cell translates the multipoles of about four times as many cells
    (of the order of 6 (p + 1)^3 flops each, rotation-accelerated)."""
    c = _full(case)
    n, state = c["n"], 8
    if c["call"] in ("tick", "leapfrog"):
        state = 17  # positions, velocities and forces in and out, masses in
    evals = c["steps"]
    if c["call"] == "direct":
        t = min(c["targets"], n)
        return dict(bytes=32 * n + 44 * t, flops=18 * n * t)
    # half-full leaves, and never more of them than bodies
    leaves = max(c["systems"], 2 * n / c["n_leaf"])
    theta = c["theta"] if c["mac"] == "theta" else 0.6
    near = min(leaves / c["systems"], 4.19 * (1.43 / theta) ** 3)
    far = min(leaves / c["systems"], 4 * near)
    flops = 16 * n * near * (n / leaves) + 1.15 * leaves * far * 6 * (c["p"] + 1) ** 3
    return dict(bytes=8 * n * state * evals, flops=flops * evals)


def tolerance(case):
    """Plain: FP64 sums in another order. Measured with the O(p^4) M2L against the rotation M2L: rel up to 8e-16, max
    up to 4e-15 at 1e3 to 3e5 bodies; near-field sums of 1e5 terms in another order move more than that.
    Mixed: FP32 expansions and FP32 partial sums. Measured against the plain form with the same lists: rel up to 1.6e-6,
    max up to 2.1e-4 (a body where large forces cancel)."""
    c = _full(case)
    if c["precision"] == "plain":
        return {"rel": 1e-13, "max": 1e-11}
    return {"rel": 6e-6, "max": 8e-4}


def _exact_forces(c, mass, pos, off, targets=None):
    """(acc, pot, sum m / r^2) by direct summation in FP64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    acc, pot, fsc = [], [], []
    for s in range(len(off) - 1):
        a, b = int(off[s]), int(off[s + 1])
        x, m = torch.as_tensor(pos[a:b]).to(dev), torch.as_tensor(mass[a:b]).to(dev)
        ids = torch.arange(b - a, device=dev) if targets is None else torch.as_tensor(targets.astype(np.int64)).to(dev)
        rows = max(1, 60_000_000 // (b - a))
        for r0 in range(0, len(ids), rows):
            t = ids[r0:r0 + rows]
            d = [x[None, :, k] - x[t, k][:, None] for k in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + c["softening"] ** 2
            inv = 1.0 / torch.sqrt(r2)
            inv[torch.arange(len(t), device=dev), t] = 0.0  # not the body itself
            mi = m[None, :] * inv
            pot.append(mi.sum(1))
            mi *= inv
            fsc.append(mi.sum(1))
            mi *= inv
            acc.append(torch.stack([(mi * q).sum(1) for q in d], 1))
    return torch.cat(acc), torch.cat(pot), torch.cat(fsc)


def exact(case, seed):
    c = _full(case)
    mass, pos, vel, off = _bodies(c, seed)
    if c["call"] == "direct":
        acc, pot, f = _exact_forces(c, mass, pos, off, _targets(c, seed))
        return dict(acc=acc.cpu().numpy(), pot=pot.cpu().numpy(), f=f.cpu().numpy())
    if int((np.diff(off.astype(np.int64)).astype(np.float64) ** 2).sum() * (1 + c["steps"])) > 2 * EXACT_MAX ** 2:
        return None
    if c["call"] not in ("tick", "leapfrog"):
        acc, pot, _ = _exact_forces(c, mass, pos, off)
        if c["call"] == "host":
            return dict(acc=acc.cpu().numpy(), pot=pot.cpu().numpy())
        return dict(acc=acc, pot=pot)
    acc, pot, _ = _exact_forces(c, mass, pos, off)
    x, v, dt = torch.as_tensor(pos).to(acc.device), torch.as_tensor(vel).to(acc.device), c["dt"]
    for _ in range(c["steps"]):
        v = v + 0.5 * dt * acc
        x = x + dt * v
        acc, pot, _ = _exact_forces(c, mass, x, off)
        v = v + 0.5 * dt * acc
    return dict(pos=x, vel=v, acc=acc, pot=pot)
