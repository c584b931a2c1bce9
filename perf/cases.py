"""Workloads of the retaining-wall framework, for timing one build against another.

Each case is what a user's program has the framework do through its public entry points:
steps of a single case (a column collapse or a retaining wall, FP32, FP64 or the precision
form), a host program that calls the stage methods itself, a batched sweep, steps with the
learned closure, the closure network's training and gradient, and the cell-key sort.  Sizes
run from the smallest test cases to the 1.92M-particle retaining wall.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from retainwall_code_b200 import LoquatSph, _abi, cases
from retainwall_code_b200._lib import check, lib
from retainwall_code_b200.closure import IN, NPARAM, OUT, TRAIN_RANGES, Mlp
from retainwall_code_b200.sph import Batch

# What a program reads back after a run of steps: in-cell positions and pressure, velocities
# and densities, stresses (all particles, boundary rows included).
STATE = ("pospres", "velrhop", "str")


def _column(name, nx, ny, nz, precision, steps, lead=0, dx=0.005, model="hypo_cs"):
    return dict(name=name, kind="column", nx=nx, ny=ny, nz=nz, precision=precision, steps=steps, lead=lead, dx=dx,
                model=model)


def _wall(name, nx, ny, nz, steps, mode="active", drift=0.0, form="plain", dx=0.0025):
    return dict(name=name, kind="wall", nx=nx, ny=ny, nz=nz, steps=steps, mode=mode, drift=drift, form=form, dx=dx)


def listed():
    return [
        # a small collapse, as the tests and a first try of a case file run it: launches count
        _column("column_small", 9, 7, 11, 4, 20),
        # the 27,648-particle column collapse in FP64, as its reference build runs it
        _column("column_f64", 24, 24, 48, 8, 100),
        # the same column once it flows: particles change cell, lists are updated, keys sorted
        _column("column_f64_flow", 24, 24, 48, 8, 60, lead=600),
        # a host program that calls the stage methods, stress filter every fifth step, a
        # rotating wall (a case of the size of the batched sweep's smaller ones)
        _wall("wall_stages", 61, 25, 37, 15, mode="rotation", form="stages", dx=0.004),
        # precision form, wall pushed into the soil, wall force read after every step
        _wall("wall_mixed", 111, 45, 67, 40, mode="passive", form="mixed", dx=0.003),
        # steps with the trained closure in place of the hypoplastic rate
        _wall("wall_closure", 97, 39, 59, 40, form="closure", dx=0.003),
        # a wall whose soil moves through the cells, as late in a long run: sorted sections
        _wall("wall_drift", 133, 53, 79, 40, drift=0.05),
        # the 1.92M-particle retaining wall, steps between two reads of the state
        _wall("wall_full", 200, 80, 120, 100),
        # a sweep of uneven walls in one graph per step
        dict(name="sweep", kind="batch", n_cases=12, spec=5, n_lo=50_000, n_hi=130_000, steps=50),
        # one epoch of training the closure network on solver samples
        dict(name="train", kind="train", samples=400_000, batch=8192, epochs=1),
        # loss gradient of the network over a set of samples
        dict(name="gradient", kind="grad", samples=50_001),
        # stable sort of cell keys with its permutation, caller's device arrays
        dict(name="cell_sort", kind="sort", n=1_000_003, max_key=2_000_000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["column", "column", "wall", "wall", "wall", "batch", "train", "grad", "sort"])
    if kind == "column":
        s = _log(rng, 700, 60_000) ** (1.0 / 3.0)  # nx : ny : nz about 1 : 1 : 2
        nx, ny, nz = (max(4, int(round(s * k * rng.uniform(0.9, 1.1)))) for k in (0.79, 0.79, 1.59))
        precision, flow = rng.choice([4, 8]), rng.random() < 0.3
        c = _column("", nx, ny, nz, precision, rng.randint(20, 100), rng.randint(300, 600) if flow else 0,
                    model=rng.choice(["hypo_cs", "hypo_cs", "hypo_basic", "dp", "mui_dp"]))
    elif kind == "wall":
        s = (_log(rng, 20_000, 1_500_000) / 30.0) ** (1.0 / 3.0)  # nx : ny : nz = 5 : 2 : 3
        nx, ny, nz = (max(6, int(round(s * k * rng.uniform(0.93, 1.07)))) for k in (5, 2, 3))
        c = _wall("", nx, ny, nz, rng.randint(15, 50), mode=rng.choice(["active", "passive", "rotation"]),
                  drift=0.05 if rng.random() < 0.25 else 0.0,
                  form=rng.choice(["plain", "plain", "mixed", "stages", "closure"]), dx=rng.uniform(0.0025, 0.005))
    elif kind == "batch":
        lo = rng.randint(20_000, 80_000)
        c = dict(kind=kind, n_cases=rng.randint(2, 14), spec=rng.randint(1, 10_000), n_lo=lo,
                 n_hi=lo + rng.randint(10_000, 60_000), steps=rng.randint(8, 25))
    elif kind == "train":
        c = dict(kind=kind, samples=rng.randint(50_000, 500_000), batch=rng.choice([2048, 8192, 19456, 20000]),
                 epochs=rng.randint(1, 2))
    elif kind == "grad":
        c = dict(kind=kind, samples=int(_log(rng, 100, 200_000)))
    else:
        c = dict(kind=kind, n=int(_log(rng, 1000, 1 << 20)), max_key=int(_log(rng, 200, (1 << 24) - 1)))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------
def _case(case, seed):
    """The particle case of a column or wall workload."""
    if case["kind"] == "column":
        return cases.column_collapse(case["nx"], case["ny"], case["nz"], dx=case["dx"], seed=seed,
                                     model=case["model"])
    c = cases.retaining_wall(case["nx"], case["ny"], case["nz"], dx=case["dx"], seed=seed, mode=case["mode"])
    if case["drift"]:  # soil moving along +x, a band of particles close to the cells' x faces
        c.pospres[c.npb:, 0] += 0.1 * c.params["dr"]
        c.velrhop[c.npb:, 0] = case["drift"]
    return c


def _specs(case):
    return cases.batch_sweep(case["n_cases"], case["spec"], case["n_lo"], case["n_hi"])


def _samples(n, seed):
    """n training samples of the solver's own states, the same ones in the same order from
    run to run (the device appends them in any order)."""
    c = cases.column_collapse(20, 20, 40, seed=seed)
    net = Mlp(seed=seed, sample_capacity=n + c.npm)
    sim = LoquatSph(case=c)
    k = 0
    while net.sample_count() < n:
        sim.step(25)
        net.collect(sim, 1, TRAIN_RANGES, seed * 1000003 + k)
        k += 1
    sim.close()
    x, t = net.samples()
    net.close()
    order = np.lexsort((x[:, 12], x[:, 0], x[:, 6]))
    order = order[np.random.default_rng(seed).permutation(len(order))[:n]]
    return x[order], t[order]


def _trained(n, epochs, seed):
    x, t = _samples(n, seed)
    net = Mlp(seed=seed, sample_capacity=n)
    net.add_samples(x, t)
    net.train(epochs, 8192, 2e-3, seed)
    return net


def _weights(seed):
    """Network parameters drawn as rw_mlp_create draws them, with small biases."""
    rng = np.random.default_rng(seed)
    p = []
    for i, o in ((IN, 64), (64, 64), (64, 64), (64, 64), (64, OUT)):
        p += [rng.uniform(-1, 1, i * o) * math.sqrt(6.0 / (i + o)), rng.uniform(-0.1, 0.1, o)]
    return np.concatenate(p).astype(np.float32)


def _grad_data(case, seed):
    """Features within the ranges of the closure's and targets of their size."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (case["samples"], IN)).astype(np.float32)
    x[:, 0:3] -= 1.0  # normal stresses over p: compressive
    x[:, 15] = 0.0
    return x, rng.normal(0.0, 0.5, (case["samples"], OUT)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("column", "wall"):
        c = _case(case, seed)
        form = case.get("form", "plain")
        if form == "stages":
            c.params["stress_shepard_filter"] = 5
        sim = LoquatSph(case=c, precision=case.get("precision", 4))
        state = dict(case=case, sim=sim)
        if form == "mixed":
            sim.set_option(_abi.OPT_MIXED_PRECISION, 1)
        if form == "closure":
            state["net"] = _trained(400_000, 150, 7)
            sim.set_closure(state["net"], 0.05)
        sim.step(1 + case.get("lead", 0))  # the program has begun its run: the step graph is captured
        sim.synchronize()
        return state
    if kind == "batch":
        sims = [LoquatSph(case=cases.retaining_wall(**dict(s, seed=seed + k))) for k, s in enumerate(_specs(case))]
        batch = Batch(sims)
        batch.step(1)
        batch.synchronize()
        return dict(case=case, sims=sims, batch=batch)
    if kind == "train":
        x, t = _samples(case["samples"], seed)
        net = Mlp(seed=seed, sample_capacity=case["samples"])
        net.add_samples(x, t)
        return dict(case=case, net=net, seed=seed)
    if kind == "grad":
        net = Mlp(seed=seed)
        net.set_params(_weights(seed))
        x, t = _grad_data(case, seed)
        return dict(case=case, net=net, x=x, t=t)
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.randint(0, case["max_key"] + 1, (case["n"],), device="cuda", dtype=torch.int32, generator=g)
    return dict(case=case, keys=keys, sorted=torch.empty_like(keys), perm=torch.empty_like(keys))


# ------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("column", "wall"):
        sim, out = state["sim"], {}
        form = case.get("form", "plain")
        if form == "stages":
            for k in range(case["steps"]):
                sim.step_calculation()
                sim.predictor_section(shepard=k % 5 == 4)
                sim.corrector_section()
                sim.end_step()
        elif form == "mixed":
            force = []
            for _ in range(case["steps"]):
                sim.step(1)
                force.append(sim.wall_force(0))
            out["force"] = np.stack(force)
        else:
            sim.step(case["steps"])
        for name in STATE:
            out[name] = sim.get(name)
        return out
    if kind == "batch":
        state["batch"].step(case["steps"])
        state["batch"].synchronize()
        out = {"force": state["batch"].wall_force(0)}
        for k, sim in enumerate(state["sims"]):
            out["str%d" % k] = sim.get("str")
        return out
    if kind == "train":
        loss = state["net"].train(case["epochs"], case["batch"], 5e-4, state["seed"])
        return {"loss": loss, "params": state["net"].params()}
    if kind == "grad":
        loss, grad = state["net"].grad(state["x"], state["t"])
        return {"loss": loss, "grad": grad}
    stream = torch.cuda.current_stream().cuda_stream
    check(lib().rw_cell_sort_noalloc(state["keys"].data_ptr(), case["n"], case["max_key"],
                                     state["sorted"].data_ptr(), state["perm"].data_ptr(), stream),
          "rw_cell_sort_noalloc")
    return {"keys": state["sorted"], "perm": state["perm"]}


# ------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------
_LAYERS = 3  # wall and floor layers of the generator at h = 1.2 dx


def _counts(nx, ny, nz, kind="wall"):
    """(soil, boundary) particles of a generated case."""
    top = nz + 2
    if kind == "column":
        floor = (5 * nx + _LAYERS) * (3 * ny + 2 * _LAYERS) * _LAYERS
        walls = _LAYERS * (ny + 2 * _LAYERS) * top + 2 * nx * _LAYERS * top
    else:
        floor = (nx + 2 * _LAYERS) * (ny + 2 * _LAYERS) * _LAYERS
        walls = 2 * nx * _LAYERS * top + 2 * _LAYERS * (ny + 2 * _LAYERS) * top
    return nx * ny * nz, floor + walls


def _steps_work(npm, npb, steps, scalar):
    """Two sections' own state in and out, every neighbour record once (1276 bytes per soil
    and 644 per boundary particle in FP32), about 27 kFLOP of pair terms and material law."""
    return steps * (1276.0 * npm + 644.0 * npb) * scalar / 4.0, steps * 27.0e3 * npm


def work(case):
    kind = case["kind"]
    if kind in ("column", "wall"):
        npm, npb = _counts(case["nx"], case["ny"], case["nz"], kind)
        b, f = _steps_work(npm, npb, case["steps"], case.get("precision", 4))
        if case.get("form") == "closure":
            f += case["steps"] * 2 * npm * 2.0 * NPARAM
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for s in _specs(case):
            npm, npb = _counts(s["nx"], s["ny"], s["nz"])
            x, y = _steps_work(npm, npb, case["steps"], 4)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind == "train":
        n = case["epochs"] * (case["samples"] // case["batch"]) * case["batch"]
        return {"bytes": 4.0 * (IN + OUT) * n, "flops": 6.0 * NPARAM * n}
    if kind == "grad":
        return {"bytes": 4.0 * (IN + OUT) * case["samples"], "flops": 6.0 * NPARAM * case["samples"]}
    return {"bytes": 12.0 * case["n"], "flops": 0.0}


# ------------------------------------------------------------------------------------
# The same outputs in 64 bits
# ------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        keys = prepare(case, seed)["keys"].long()
        s, perm = torch.sort(keys, stable=True)
        return {"keys": s.int(), "perm": perm.int()}
    if kind == "grad":
        return _exact_grad(case, seed)
    # A column's steps from the start.  Beside a contact wall a decision (which wall particle
    # is nearest, is a particle in contact) turns on one rounding, and a trained network or a
    # long run carries such differences on: those have no 64-bit value to be held to.
    if kind == "column" and not case["lead"] and case["model"] == "hypo_cs" and _counts(
            case["nx"], case["ny"], case["nz"], "column")[0] <= 70_000:
        return _exact_column(_case(case, seed), 1 + case["steps"])
    return None


def _exact_grad(case, seed):
    x, t = (torch.from_numpy(a).double() for a in _grad_data(case, seed))
    p = torch.from_numpy(_weights(seed)).double().requires_grad_()
    h, at = x, 0
    dims = ((IN, 64), (64, 64), (64, 64), (64, 64), (64, OUT))
    for k, (i, o) in enumerate(dims):
        h = h @ p[at:at + i * o].reshape(i, o) + p[at + i * o:at + i * o + o]
        at += i * o + o
        if k < 4:
            h = h * torch.sigmoid(h)
    loss = ((h - t) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grad": p.grad.numpy()}


class _Pairs:
    """Pairs (i, j) within 2h for targets i among the sources j, from a cell list."""

    def __init__(self, cell, pos, n_cell, h, src_lo, src_hi):
        self.cell, self.pos, self.nc, self.h = cell, pos, n_cell, h
        key = (cell[src_lo:src_hi, 0] * n_cell[1] + cell[src_lo:src_hi, 1]) * n_cell[2] + cell[src_lo:src_hi, 2]
        self.key, self.order = torch.sort(key, stable=True)
        self.order = self.order + src_lo
        cells = torch.arange(n_cell[0] * n_cell[1] * n_cell[2], device=key.device)
        self.beg = torch.searchsorted(self.key, cells)
        self.end = torch.searchsorted(self.key, cells, right=True)

    def of(self, lo, hi):
        ii, jj, dd = [], [], []
        c = self.cell[lo:hi]
        for off in range(27):
            o = torch.tensor([off % 3 - 1, off // 3 % 3 - 1, off // 9 - 1], device=c.device)
            cj = c + o
            inside = ((cj >= 0) & (cj < self.nc)).all(1)
            k = ((cj[:, 0] * self.nc[1] + cj[:, 1]) * self.nc[2] + cj[:, 2]).clamp(0, len(self.beg) - 1)
            n = torch.where(inside, self.end[k] - self.beg[k], torch.zeros_like(k))
            i = torch.repeat_interleave(torch.arange(len(c), device=c.device), n)
            first = torch.cumsum(n, 0) - n
            j = self.order[self.beg[k][i] + torch.arange(len(i), device=c.device) - first[i]]
            d = self.pos[lo + i] - self.pos[j] - o.double() * (2.0 * self.h)
            near = (d * d).sum(1) < 4.0 * self.h * self.h
            ii.append(i[near]), jj.append(j[near]), dd.append(d[near])
        return torch.cat(ii), torch.cat(jj), torch.cat(dd)


def _full(s):
    xx, yy, zz, xy, xz, yz = s.unbind(-1)
    return torch.stack([xx, xy, xz, xy, yy, yz, xz, yz, zz], -1).reshape(-1, 3, 3)


def _sym(f):
    f = 0.5 * (f + f.transpose(1, 2))
    return torch.stack([f[:, 0, 0], f[:, 1, 1], f[:, 2, 2], f[:, 0, 1], f[:, 0, 2], f[:, 1, 2]], -1)


def _tr(a):
    return a[:, :3].sum(1)


def _tr2(a, b):
    return (a[:, :3] * b[:, :3]).sum(1) + 2.0 * (a[:, 3:] * b[:, 3:]).sum(1)


def _hypo_cs(dt, rho, om, D, sig, mp):
    """HypoCS stress update (constitutive_model.h:209-299), no cohesion."""
    Ei, Vi, phi, _, p_ref, e_co, lam, xi, alpha, e_min, e_max, e_0, rho_0 = mp[:13]
    C1 = -Ei / (3.0 * p_ref * (1.0 + Vi))
    a = 3.0 / (math.sqrt(2.0) * math.sin(phi))
    C2 = C1 * ((3.0 * Vi + a * math.sqrt(1.0 + Vi * Vi)) / (1.0 - Vi) - a * a / 3.0)
    C3, C4 = a * a * C1, a * C1
    one = torch.tensor([1.0, 1.0, 1.0, 0.0, 0.0, 0.0], device=sig.device, dtype=sig.dtype)
    z = torch.zeros_like(om[:, 0])
    W = torch.stack([z, -om[:, 2], om[:, 1], om[:, 2], z, -om[:, 0], -om[:, 1], om[:, 0], z], -1).reshape(-1, 3, 3)
    F = _full(sig)
    I1 = _tr(sig)
    reset = I1 > -4.0
    I1 = torch.where(reset, torch.full_like(I1, -4.0), I1)
    dev = sig - one * (I1 / 3.0)[:, None]
    nD = _tr2(D, D).sqrt()
    p = -I1 / 3.0
    e = ((1.0 + e_0) * rho_0 / rho - 1.0).clamp(e_min, e_max)
    e_c = e_co * torch.exp(-lam * (p / p_ref) ** xi)
    fd = ((e - e_min) / (e_c - e_min)) ** alpha
    rate = _sym(W @ F - F @ W) + D * (C1 * I1)[:, None] + sig * (C2 * _tr(D))[:, None] + sig * (
        C3 * _tr2(sig, D) / I1)[:, None] + (sig + dev) * (fd * C4 * nD)[:, None]
    s = sig + rate * dt
    sph = _tr(s) / 3.0
    dev = s - one * sph[:, None]
    fa, fb, fc = C2 / C1, C3 / C1, C4 / C1
    t1 = 1.0 + fa + fb / 3.0
    g = (fd * fc) ** 2
    A = g / 3.0 - t1 * t1
    B = 2.0 * g * (t1 * t1 + 2.0 * fa + 3.0) - 4.0 * fb * (1.0 + fa + fb / 3.0)
    C = 4.0 / 3.0 * g * fb * fb - 4.0 * fb * fb
    k_phi = 3.0 / ((-B - (B * B - 4.0 * A * C).sqrt()) / (2.0 * A)).sqrt()
    tau = (0.5 * _tr2(dev, dev)).sqrt()
    ratio = torch.where(tau + sph * k_phi > 0.0, -k_phi * sph / tau.clamp_min(1e-300), torch.ones_like(tau))
    out = dev * ratio[:, None] + one * sph[:, None]
    low = torch.tensor([-1.0, -1.0, -2.0, 0.0, 0.0, 0.0], device=sig.device, dtype=sig.dtype)
    return torch.where((reset | (sph > 0.0))[:, None], low, out)


def _exact_column(c, steps):
    """Steps of a column collapse (fixed walls, no contact walls) in FP64: the reference's
    cell sort, Adami boundary, particle interaction, predictor and corrector."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).double().to(dev)  # noqa: E731
    q = c.params
    npb, dr = c.npb, q["dr"]
    h = dr * q["hdr"]
    dt = q["cfl"] * h / q["cs_m"]
    mp = [q["model-0-par-%d" % k] for k in range(15)]
    nc = torch.tensor([int(0.5 / h * q["domain_size_%s" % a]) + 1 for a in "xyz"], device=dev)
    grav = torch.tensor([q["gravity_%s" % a] for a in "xyz"], device=dev, dtype=torch.float64)
    knorm, kgrad = 42.0 / (256.0 * math.pi * h ** 3), -5.0 * 42.0 / (256.0 * math.pi * h ** 5)
    k_0, k_dr = knorm * 8.0, knorm * (2.0 - dr / h) ** 4 * (dr / h + 0.5)
    pabs = f(c.pospres[:, :3])
    cell = (pabs * (0.5 / h)).long()
    S = dict(cell=cell, pos=pabs - cell.double() * (2.0 * h), pres=f(c.pospres[:, 3]), vr=f(c.velrhop), mass=f(c.idmassidx[:, 1]),
             sig=f(c.stress), normal=torch.cat([f(c.normal), torch.zeros(c.npm, 4, device=dev, dtype=torch.float64)]))

    def search():
        key = (S["cell"][:, 0] * nc[1] + S["cell"][:, 1]) * nc[2] + S["cell"][:, 2]
        key[npb:] += nc.prod()
        order = torch.sort(key, stable=True)[1]
        for k in S:
            S[k] = S[k][order]

    def adami():
        soil = _Pairs(S["cell"], S["pos"], nc, h, npb, len(S["pos"]))
        i, j, d = soil.of(0, npb)
        qq = d.norm(dim=1) / h
        ker = knorm * (2.0 - qq) ** 4 * (qq + 0.5)
        kv = ker * S["mass"][j] / S["vr"][j, 3]
        z = lambda n: torch.zeros(npb, n, device=dev, dtype=torch.float64)  # noqa: E731
        rs = z(6).index_add_(0, i, S["sig"][j] * kv[:, None])
        rd = z(3).index_add_(0, i, d * (ker * S["mass"][j])[:, None])
        rv = z(4).index_add_(0, i, S["vr"][j] * kv[:, None])
        w = z(1).index_add_(0, i, kv[:, None])
        on = w > 0.0
        w = torch.where(on, w, torch.ones_like(w))
        n, slip = S["normal"][:npb, :3], S["normal"][:npb, 3:]
        v = rv[:, :3] / w
        vn = n * (n * v).sum(1, keepdim=True)
        vt = v - vn
        ext = torch.cat([-vn + torch.where(slip == -1.0, -vt, vt), rv[:, 3:] / w], 1)
        S["vr"][:npb] = torch.where(on, ext, S["vr"][:npb])
        sig = rs / w
        sig[:, :3] -= grav * rd / w
        S["sig"][:npb] = torch.where(on, sig, torch.zeros_like(sig))

    def interaction():
        every = _Pairs(S["cell"], S["pos"], nc, h, 0, len(S["pos"]))
        i, j, d = every.of(npb, len(S["pos"]))
        I = i + npb
        r2 = (d * d).sum(1)
        qq = r2.sqrt() / h
        gk = d * (kgrad * (2.0 - qq) ** 3)[:, None]
        rho = S["vr"][:, 3]
        mass = torch.cat([dr ** 3 * rho[:npb], S["mass"][npb:]])
        vol, mj = (mass / rho)[j], mass[j][:, None]
        sor = S["sig"] / (rho * rho)[:, None]
        dv = S["vr"][I, :3] - S["vr"][j, :3]
        n = len(S["pos"]) - npb
        z = lambda *k: torch.zeros(n, *k, device=dev, dtype=torch.float64)  # noqa: E731
        gv = z(9).index_add_(0, i, -(dv[:, :, None] * (gk * vol[:, None])[:, None, :]).reshape(-1, 9)).reshape(-1, 3, 3)
        den = z().index_add_(0, i, rho[I] * (dv * gk).sum(1) * vol)
        t = ((_full(sor[I] + sor[j]) @ gk[:, :, None])[:, :, 0]) * mj
        x = (dv * d).sum(1).clamp_max(0.0)
        t += gk * mj * (q["artificial_viscosity_alpha_m"] * q["cs_m"] * h * x / (r2 + 0.01 * h * h) / (
            0.5 * (rho[I] + rho[j])))[:, None]
        R = _tr(sor).clamp_min(0.0) * q["artificial_pressure_coefficient_material"]
        ker = knorm * (2.0 - qq) ** 4 * (qq + 0.5)
        t -= gk * mj * ((R[I] + R[j]) * (ker / k_dr) ** (k_0 / k_dr))[:, None]
        acc = z(3).index_add_(0, i, t) - q["damping"] * S["vr"][npb:, :3] + grav
        om = 0.5 * torch.stack([gv[:, 1, 0] - gv[:, 0, 1], gv[:, 2, 0] - gv[:, 0, 2], gv[:, 2, 1] - gv[:, 1, 2]], -1)
        return torch.cat([acc, den[:, None]], 1), _sym(gv), om

    for _ in range(steps):
        search()
        adami()
        acc, D, om = interaction()
        pos0, vr0, sig0 = S["pos"][npb:].clone(), S["vr"][npb:].clone(), S["sig"][npb:].clone()
        vr = vr0 + acc * (0.5 * dt)
        S["pos"][npb:] = pos0 + vr[:, :3] * (0.5 * dt)
        vr[:, 3].clamp_(mp[13], mp[14])
        S["vr"][npb:], S["sig"][npb:] = vr, _hypo_cs(0.5 * dt, vr[:, 3], om, D, sig0, mp)
        adami()
        acc, D, om = interaction()
        vr = vr0 + acc * dt
        pos = pos0 + (vr[:, :3] + vr0[:, :3]) * (0.5 * dt)
        vr[:, 3].clamp_(mp[13], mp[14])
        move = (pos >= 2.0 * h).long() - (pos < 0.0).long()
        S["cell"][npb:] += move
        S["pos"][npb:] = pos - move.double() * (2.0 * h)
        S["vr"][npb:], S["sig"][npb:] = vr, _hypo_cs(dt, vr[:, 3], om, D, sig0, mp)
    return {"pospres": torch.cat([S["pos"], S["pres"][:, None]], 1), "velrhop": S["vr"], "str": S["sig"]}
