"""Workloads of the self-gravity engine as a user's program runs them, with
what each needs, and their results in 64-bit arithmetic.

listed() names the fixed workloads, draw(rng) makes another one of the same
ranges.  prepare(case, seed) makes the inputs on the GPU together with the
engine, solver or handle that a program keeps; run(state) is one pass
through the public entry points; work(case) is the memory traffic and the
arithmetic that a pass cannot do without; exact(case, seed) is what the
first run returns, computed in plain torch in float64.
"""
import importlib
import math
import random

import torch

PKG = "real-astronomy-simulation_gb300"
GALACTIC_G = 43009.1725  # kpc, km/s, 1e10 Msun
# A Miyamoto-Nagai disk in a Plummer halo (the analytic fixtures' first potential).
GAS_POTENTIAL = dict(M_d=5.0, a=3.0, b=0.3, M_h=12.0, a_h=8.0)


def _mod(name):
    return importlib.import_module(PKG + "." + name)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # An interactive or test-sized direct-sum run: one step per frame,
        # where the step's latency is all that counts.
        dict(name="direct_1k", kind="direct", ic="plummer", n=1000, steps=1, energies=False),
        # The plain direct-sum Plummer run, printing its energies every ten
        # steps.
        dict(name="direct_20k", kind="direct", ic="plummer", n=20000, steps=10, energies=True),
        # A merger of two Plummer spheres, 2 x 131,072 particles.
        dict(name="direct_merger_262k", kind="direct", ic="merger", n=262144, steps=1, energies=False),
        # A small tree run with the Engine's defaults (theta 0.6, 63-bit keys).
        dict(name="bh_10k", kind="bh", n=10000, theta=0.6, bits=21, shape=-1, steps=1, energies=False),
        # A middling tree run that prints its energies; an odd size.
        dict(name="bh_print_100k", kind="bh", n=100003, theta=0.5, bits=21, shape=-1, steps=5, energies=True),
        # The large stellar disk: theta 0.5, 30-bit keys.
        dict(name="bh_1m", kind="bh", n=1000000, theta=0.5, bits=10, shape=-1, steps=1, energies=False),
        # The same method with the opt-in group walk.
        dict(name="bh_group_300k", kind="bh", n=300000, theta=0.5, bits=10, shape=3, steps=1, energies=False),
        # The gravity call of a gas-disk engine: self-gravity of gas and
        # stars and the analytic galaxy added onto the hydro forces.
        dict(name="tree_ext_200k", kind="ext", n=200001, theta=0.6, bits=21),
        # Many small systems of uneven size in one launch per step.
        dict(name="batch_512", kind="batch", systems=512, n_lo=256, n_hi=16384, steps=4),
        # A training step through the integrator: forward, loss, gradients.
        dict(name="train_4k", kind="train", n=4096, steps=20, every=10, symmetric=True),
        # The same on a large disk, with the solver's default force pass.
        dict(name="train_65k", kind="train", n=65536, steps=5, every=5, symmetric=False),
        # The neighbour grid of a gas run's particles, rebuilt at each step.
        dict(name="grid_1m", kind="grid", n=1000000, stars=0.3),
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["direct", "direct", "bh", "bh", "bh", "ext", "batch", "train", "grid"])
    if kind == "direct":
        n = _log_int(rng, 300, 200000)
        few = n > 30000
        return dict(kind="direct", ic=rng.choice(["plummer", "merger"]), n=n, steps=1 if few else rng.choice([1, 4, 10]),
                    energies=(not few) and rng.random() < 0.4)
    if kind == "bh":
        return dict(kind="bh", n=_log_int(rng, 1000, 1000000), theta=rng.choice([0.5, 0.6, 0.7, 0.8]),
                    bits=rng.choice([10, 21]), shape=rng.choice([-1, -1, 3]), steps=rng.choice([1, 2]),
                    energies=rng.random() < 0.3)
    if kind == "ext":
        return dict(kind="ext", n=_log_int(rng, 2000, 500000), theta=rng.choice([0.5, 0.6, 0.8]), bits=rng.choice([10, 21]))
    if kind == "batch":
        return dict(kind="batch", systems=rng.randint(3, 300), n_lo=rng.choice([64, 100, 256]), n_hi=rng.choice([1000, 4096, 12000]),
                    steps=rng.choice([1, 4]))
    if kind == "train":
        return dict(kind="train", n=_log_int(rng, 200, 30000), steps=rng.randint(3, 12), every=rng.choice([3, 5, 20]),
                    symmetric=rng.random() < 0.5)
    return dict(kind="grid", n=_log_int(rng, 1000, 1000000), stars=rng.choice([0.0, 0.3, 0.6]))


# ----------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _directions(g, n):
    mu = 2.0 * _rand(g, n) - 1.0
    s = torch.sqrt(1.0 - mu * mu)
    phi = 2.0 * math.pi * _rand(g, n)
    return torch.stack((s * torch.cos(phi), s * torch.sin(phi), mu), 1)


def _plummer(g, n):
    """A unit Plummer sphere (M = a = G = 1), isotropic velocities with the
    local dispersion sigma^2 = 1 / (6 sqrt(1 + r^2))."""
    x = _rand(g, n).clamp(1e-9, 0.999)
    r = 1.0 / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)
    pos = _directions(g, n) * r[:, None]
    sigma = torch.sqrt(1.0 / (6.0 * torch.sqrt(1.0 + r * r)))
    return pos, _randn(g, n, 3) * sigma[:, None], torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")


def _merger(g, n):
    """Two Plummer spheres 10 apart, approaching on a parabolic orbit."""
    parts = [_plummer(g, n // 2), _plummer(g, n - n // 2)]
    v = math.sqrt(2.0 * 2.0 / 10.0)
    vel = torch.tensor([math.sqrt(0.96) * v, 0.2 * v, 0.0], dtype=torch.float64, device="cuda")
    off = torch.tensor([5.0, 0.0, 0.0], dtype=torch.float64, device="cuda")
    return (torch.cat((parts[0][0] - off, parts[1][0] + off)), torch.cat((parts[0][1] + 0.5 * vel, parts[1][1] - 0.5 * vel)),
            torch.cat((parts[0][2], parts[1][2])))


def _disk(g, n):
    """An exponential stellar disk (M = 5, Rd = 3, sech^2 height 0.3) with
    circular velocities from the enclosed mass and a 10% dispersion."""
    x = torch.linspace(0.0, 20.0, 20001, dtype=torch.float64, device="cuda")
    cdf = 1.0 - (1.0 + x) * torch.exp(-x)
    u = _rand(g, n)
    k = torch.searchsorted(cdf, u).clamp(1, 20000)
    f = (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp_min(1e-300)
    R = 3.0 * (x[k - 1] + f.clamp(0.0, 1.0) * (x[k] - x[k - 1]))
    phi = 2.0 * math.pi * _rand(g, n)
    z = 0.3 * torch.atanh((2.0 * _rand(g, n) - 1.0).clamp(-1 + 1e-12, 1 - 1e-12))
    pos = torch.stack((R * torch.cos(phi), R * torch.sin(phi), z), 1)
    mass = torch.full((n,), 5.0 / n, dtype=torch.float64, device="cuda")
    r = pos.norm(dim=1)
    order = torch.argsort(r)
    enc = torch.empty_like(r)
    enc[order] = torch.arange(1, n + 1, dtype=torch.float64, device="cuda") * (5.0 / n)
    vc = torch.sqrt(GALACTIC_G * enc / torch.sqrt(r * r + 0.0225))
    Rc = pos[:, :2].norm(dim=1) + 1e-6
    sig = 0.1 * vc[:, None] * _randn(g, n, 3)
    c, s = pos[:, 0] / Rc, pos[:, 1] / Rc
    vphi = vc + 0.5 * sig[:, 1]
    vel = torch.stack((c * sig[:, 0] - s * vphi, s * sig[:, 0] + c * vphi, 0.35 * sig[:, 2]), 1)
    return pos, vel, mass


def _f32(*arrays):
    return [a.float() for a in arrays]


def _sizes(case):
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [int(round(math.exp(random.Random(s).uniform(lo, hi)))) for s in range(case["systems"])]


def _inputs(case, seed):
    """The case's particles: float32 device tensors."""
    g, kind = _gen(seed), case["kind"]
    if kind == "direct":
        return _f32(*(_merger if case["ic"] == "merger" else _plummer)(g, case["n"]))
    if kind == "bh":
        return _f32(*_disk(g, case["n"]))
    if kind == "ext":
        pos, vel, mass = _disk(g, case["n"])
        hydro = 200.0 * _randn(g, case["n"], 3)  # pressure accelerations, (km/s)^2 / kpc
        return _f32(pos, mass, hydro)
    if kind == "batch":
        sizes = _sizes(case)
        pos, vel, _ = _plummer(g, sum(sizes))
        mass = torch.cat([torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda") for n in sizes])
        return _f32(pos, vel, mass)
    if kind == "train":
        pos, vel, mass = _disk(g, case["n"])
        mass = torch.full_like(mass, 5.0 / 65536)  # the large disk's particle mass at any n
        target = pos + 0.05 * _randn(g, case["n"], 3)  # an observed snapshot
        return _f32(pos, vel, mass, target)
    pos, _, mass = _disk(g, case["n"])
    h = 0.05 * (1.0 + 3.0 * _rand(g, case["n"]))
    star = (_rand(g, case["n"]) < case["stars"]).int()
    return _f32(pos, mass, h) + [star]


def _records(v, w=None):
    out = torch.zeros((v.shape[0], 4), dtype=torch.float32, device=v.device)
    out[:, :3] = v
    if w is not None:
        out[:, 3] = w
    return out


DIRECT = dict(G=1.0, softening=0.01)
BH_SOFT, BH_DT, DIRECT_DT, BATCH_DT, TRAIN_DT = 0.05, 1e-4, 5e-4, 1e-3, 1e-3


def prepare(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    if kind in ("direct", "bh"):
        Engine = importlib.import_module(PKG).Engine
        if kind == "direct":
            eng = Engine(gravity_mode="direct", **DIRECT)
        else:
            eng = Engine(softening=BH_SOFT, gravity_mode="bh", theta=case["theta"], key_bits=case["bits"],
                         bh_traversal=case["shape"])
        eng.load_device_state(*data)
        return dict(case=case, eng=eng)
    if kind == "ext":
        pos, mass, hydro = data
        bh = _mod("solvers.barnes_hut").BarnesHut(case["n"], theta=case["theta"], softening=BH_SOFT, key_bits=case["bits"])
        hydro = _records(hydro)
        pot = _mod("solvers.external").Potential.from_dict(GAS_POTENTIAL)
        return dict(case=case, bh=bh, xm=_records(pos, mass), hydro=hydro, acc=torch.empty_like(hydro), pot=pot)
    if kind == "batch":
        pos, vel, mass = (a.cpu().numpy() for a in data)
        systems, at = [], 0
        for n in _sizes(case):
            systems.append((pos[at:at + n], vel[at:at + n], mass[at:at + n]))
            at += n
        return dict(case=case, batch=_mod("batch").DirectBatch(systems, G=1.0, softening=0.02, variant=1))
    if kind == "train":
        pos, vel, mass, target = data
        solver = _mod("solvers.gravity").DirectGravity(case["n"])
        if case["symmetric"]:
            solver.set_variant(2)
        leaves = [t.requires_grad_(True) for t in (pos, vel, mass)]
        return dict(case=case, leaves=leaves, target=target, solver=solver)
    pos, mass, h, star = data
    grid = _mod("solvers.neighbor_grid").NeighborGrid(case["n"])
    return dict(case=case, grid=grid, xm=_records(pos, mass), h=h, star=star)


# -------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("direct", "bh"):
        eng = state["eng"]
        dt = DIRECT_DT if kind == "direct" else BH_DT
        if case["steps"] == 1:
            eng.step(dt)
        else:
            eng.run(dt, case["steps"])
        d = eng.to_device_state()
        out = dict(pos=d["pos"], vel=d["vel"], acc=d["acc"])
        if case["energies"]:
            out["kinetic"], out["potential"], _ = eng.energies()
        return out
    if kind == "ext":
        state["acc"].copy_(state["hydro"])
        _mod("solvers.external").tree_forces_ext(state["bh"], state["xm"], state["acc"], state["pot"], accumulate=True)
        return dict(acc=state["acc"])
    if kind == "batch":
        b = state["batch"]
        b.run(BATCH_DT, case["steps"])
        return dict(xm=b.xm, vel=b.v4, acc=b.a4)
    if kind == "train":
        x, v, m = state["leaves"]
        xt, vt = _mod("adjoint").simulate(x, v, m, G=GALACTIC_G, softening=0.05, dt=TRAIN_DT, nsteps=case["steps"],
                                          checkpoint_every=case["every"], solver=state["solver"])
        loss = ((xt - state["target"]) ** 2).mean()
        gx, gv, gm = torch.autograd.grad(loss, (x, v, m))
        return dict(pos=xt.detach(), vel=vt.detach(), gx=gx, gv=gv, gm=gm)
    g = state["grid"]
    ngas = g.rebuild(state["xm"], state["h"], state["star"])
    return dict(gsort=g.gsort, cell_start=g.cell_start, ngas=ngas)


# ------------------------------------------------------------------- work
# A pair's force on both its particles: 3 differences, the squared distance
# (6), the reciprocal square root and its cube (3), two weights (2) and six
# multiply-adds (12).  Its reverse pass takes about 60.
PAIR, PAIR_VJP = 26.0, 60.0


def _tree_terms(n, theta):
    """Accepted nodes per particle on the disk."""
    return 44.0 * math.log2(max(n, 2)) * (0.5 / theta) ** 2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case)
        pairs = sum(0.5 * n * n for n in sizes)
        return dict(bytes=96.0 * sum(sizes), flops=PAIR * pairs * case["steps"])
    n = case["n"]
    if kind == "direct":
        return dict(bytes=96.0 * n, flops=PAIR * 0.5 * n * n * case["steps"])
    if kind == "bh":
        return dict(bytes=96.0 * n, flops=20.0 * n * _tree_terms(n, case["theta"]) * case["steps"])
    if kind == "ext":
        return dict(bytes=48.0 * n, flops=20.0 * n * _tree_terms(n, case["theta"]))
    if kind == "train":
        return dict(bytes=(28.0 + 12.0 + 24.0 + 28.0) * n, flops=(PAIR + PAIR_VJP) * 0.5 * n * n * (case["steps"] + 1))
    return dict(bytes=44.0 * n, flops=30.0 * n)


# ------------------------------------------------------- 64-bit arithmetic
_CHUNK = 1 << 24


def _direct_acc(x, m, eps2, G):
    n = x.shape[0]
    acc = torch.empty_like(x)
    rows = max(1, _CHUNK // n)
    for i in range(0, n, rows):
        d = [x[None, :, k] - x[i:i + rows, None, k] for k in range(3)]
        w = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2).rsqrt_()
        w = w * w * w * m
        for k in range(3):
            acc[i:i + rows, k] = G * (w * d[k]).sum(1)
    return acc


def _direct_potential(x, m, eps2, G):
    n, total = x.shape[0], 0.0
    rows = max(1, _CHUNK // n)
    for i in range(0, n, rows):
        r2 = sum((x[None, :, k] - x[i:i + rows, None, k]) ** 2 for k in range(3)) + eps2
        w = r2.rsqrt_()
        part = (w * m).sum(1) - m[i:i + rows] / math.sqrt(eps2)
        total += float((m[i:i + rows] * part).sum())
    return -0.5 * G * total


def _force_vjp(x, m, w, eps2, G):
    """Gradients of sum(acc * w) by positions and masses."""
    n = x.shape[0]
    gx, gm = torch.zeros_like(x), torch.zeros_like(m)
    rows = max(1, (_CHUNK // 2) // n)
    for i in range(0, n, rows):
        X, M = x.detach().requires_grad_(True), m.detach().requires_grad_(True)
        with torch.enable_grad():
            d = [X[None, :, k] - X[i:i + rows, None, k] for k in range(3)]
            r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps2).rsqrt()
            t = sum(d[k] * w[i:i + rows, None, k] for k in range(3))
            s = G * (r * r * r * t * M).sum()
        a, b = torch.autograd.grad(s, (X, M))
        gx += a
        gm += b
    return gx, gm


def _spread(x, bits):
    r = torch.zeros_like(x)
    for b in range(bits):
        r |= ((x >> b) & 1) << (3 * b)
    return r


def _msb(x):
    """Position of the highest set bit of positive int64 values."""
    r = torch.zeros_like(x)
    for s in (32, 16, 8, 4, 2, 1):
        up = x >= (1 << s)
        r += torch.where(up, s, 0)
        x = torch.where(up, x >> s, x)
    return r


class _Tree:
    """The radix tree over stably sorted Morton keys: every node is a range
    of sorted leaves, split where the highest bit in which its keys (or, for
    equal keys, its indices) differ flips."""

    def __init__(self, x, m, bits):
        n = x.shape[0]
        lo = x.min(0).values
        span = float((x.max(0).values - lo).max())
        scale = ((1 << bits) - 1) / ((span if span > 0 else 1.0) * 1.0000001)
        q = ((x - lo) * scale).clamp(0, (1 << bits) - 1).long()
        key = _spread(q[:, 0], bits) | (_spread(q[:, 1], bits) << 1) | (_spread(q[:, 2], bits) << 2)
        self.key, self.order = torch.sort(key, stable=True)
        self.x, self.m = x[self.order], m[self.order]
        first = torch.zeros(1, dtype=torch.long, device=x.device)
        last = torch.full_like(first, n - 1)
        F, L, left, levels = [first], [last], [], []
        at, base = 1, 0
        while first.numel():
            kids = last > first  # nodes to split
            f, l = first[kids], last[kids]
            diff = self.key[f] ^ self.key[l]
            bit = _msb(torch.where(diff > 0, diff, 1))
            by_key = torch.searchsorted(self.key, ((self.key[f] >> bit) | 1) << bit)
            b2 = _msb(torch.where(f != l, f ^ l, 1))
            cut = torch.where(diff > 0, by_key, (l >> b2) << b2)  # first leaf of the right child
            ch = torch.full_like(first, -1)
            ch[kids] = at + 2 * torch.arange(f.numel(), device=x.device)
            left.append(ch)
            levels.append((base, base + first.numel()))
            base += first.numel()
            at += 2 * f.numel()
            first = torch.stack((f, cut), 1).reshape(-1)
            last = torch.stack((cut - 1, l), 1).reshape(-1)
            F.append(first)
            L.append(last)
        self.first, self.last, self.left = torch.cat(F), torch.cat(L), torch.cat(left)  # right child: left + 1
        z = torch.zeros(1, dtype=torch.float64, device=x.device)
        cm = torch.cat((z, self.m.cumsum(0)))
        cx = torch.cat((z[None].expand(1, 3), (self.m[:, None] * self.x).cumsum(0)))
        self.mass = cm[self.last + 1] - cm[self.first]
        self.com = (cx[self.last + 1] - cx[self.first]) / self.mass[:, None]
        leaf = self.left < 0
        self.com[leaf], self.mass[leaf] = self.x[self.first[leaf]], self.m[self.first[leaf]]
        self.mn = self.x[self.first].clone()
        self.mx = self.mn.clone()
        for a, b in reversed(levels):
            k = torch.nonzero(self.left[a:b] >= 0)[:, 0] + a
            c = self.left[k]
            self.mn[k] = torch.minimum(self.mn[c], self.mn[c + 1])
            self.mx[k] = torch.maximum(self.mx[c], self.mx[c + 1])
        self.size2 = (self.mx - self.mn).max(1).values ** 2

    def walk(self, theta, eps2, grouped):
        """Accelerations and potentials (no G) per particle.  A walker is one
        particle, or (grouped) a maximal subtree of at most 32 leaves, which
        tests nodes against its bounding box."""
        n = self.x.shape[0]
        if grouped:
            cnt = self.last - self.first + 1
            small = cnt <= 32
            top = small.clone()
            inner = torch.nonzero((self.left >= 0) & small)[:, 0]
            top[self.left[inner]] = False
            top[self.left[inner] + 1] = False
            w = torch.nonzero(top)[:, 0]
            w0, wc, wlo, whi = self.first[w], cnt[w], self.mn[w], self.mx[w]
        else:
            w0 = torch.arange(n, device=self.x.device)
            wc, wlo, whi = torch.ones_like(w0), self.x, self.x
        acc = torch.zeros_like(self.x)
        phi = torch.zeros_like(self.m)
        step = 8192 if grouped else 65536
        for s in range(0, w0.numel(), step):
            who = torch.arange(s, min(s + step, w0.numel()), device=self.x.device)
            node = torch.zeros_like(who)
            while who.numel():
                c = self.com[node]
                d = torch.maximum(torch.maximum(wlo[who] - c, c - whi[who]), torch.zeros_like(c))
                r2 = (d * d).sum(1) + eps2
                take = (self.left[node] < 0) | (self.size2[node] < theta * theta * r2)
                aw, an = who[take], node[take]
                reps = wc[aw]
                i = torch.repeat_interleave(w0[aw], reps)
                if grouped:
                    begin = torch.repeat_interleave(reps.cumsum(0) - reps, reps)
                    i = i + torch.arange(i.numel(), device=i.device) - begin
                    an = torch.repeat_interleave(an, reps)
                d = self.com[an] - self.x[i]
                inv = ((d * d).sum(1) + eps2).rsqrt()
                mw = self.mass[an]
                acc.index_add_(0, i, (mw * inv ** 3)[:, None] * d)
                own = (self.left[an] < 0) & (self.first[an] == i)
                phi.index_add_(0, i, torch.where(own, 0.0, mw * inv))
                kids = self.left[node[~take]]
                who = torch.repeat_interleave(who[~take], 2)
                node = torch.stack((kids, kids + 1), 1).reshape(-1)
        out, pot = torch.empty_like(acc), torch.empty_like(phi)
        out[self.order], pot[self.order] = acc, phi
        return out, pot


def _galaxy(x, G):
    p = GAS_POTENTIAL
    R2 = x[:, 0] ** 2 + x[:, 1] ** 2
    S = torch.sqrt(x[:, 2] ** 2 + p["b"] ** 2)
    aS = p["a"] + S
    cd = -G * p["M_d"] / (R2 + aS * aS) ** 1.5
    ch = -G * p["M_h"] / (R2 + x[:, 2] ** 2 + p["a_h"] ** 2) ** 1.5  # Plummer halo
    return torch.stack(((cd + ch) * x[:, 0], (cd + ch) * x[:, 1], (cd * aS / S + ch) * x[:, 2]), 1)


def _kdk(x, v, force, dt, steps):
    """KDK steps from freshly evaluated accelerations; positions are stored
    in float32 between steps, as the engine's records are."""
    a = force(x)
    for _ in range(steps):
        v = v + 0.5 * dt * a
        x = (x + dt * v).float().double()
        a = force(x)
        v = v + 0.5 * dt * a
    return x, v, a


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return None  # whole numbers
    with torch.no_grad():
        data = [t.double() for t in _inputs(case, seed)]
        if kind == "direct":
            x, v, m = data
            eps2 = DIRECT["softening"] ** 2
            x, v, a = _kdk(x, v, lambda p: _direct_acc(p, m, eps2, 1.0), DIRECT_DT, case["steps"])
            out = dict(pos=x, vel=v, acc=a)
            if case["energies"]:
                out["kinetic"] = 0.5 * float((m * (v * v).sum(1)).sum())
                out["potential"] = _direct_potential(x, m, eps2, 1.0)
            return out
        if kind == "bh":
            x, v, m = data
            last = {}

            def force(p):
                acc, last["phi"] = _Tree(p, m, case["bits"]).walk(case["theta"], BH_SOFT ** 2, case["shape"] == 3)
                return GALACTIC_G * acc

            x, v, a = _kdk(x, v, force, BH_DT, case["steps"])
            out = dict(pos=x, vel=v, acc=a)
            if case["energies"]:
                out["kinetic"] = 0.5 * float((m * (v * v).sum(1)).sum())
                out["potential"] = -0.5 * GALACTIC_G * float((m * last["phi"]).sum())
            return out
        if kind == "ext":
            x, m, hydro = data
            acc, _ = _Tree(x, m, case["bits"]).walk(case["theta"], BH_SOFT ** 2, False)
            acc = GALACTIC_G * acc + _galaxy(x, GALACTIC_G) + hydro
            return dict(acc=torch.cat((acc, torch.zeros_like(acc[:, :1])), 1))
        if kind == "batch":
            parts, at = [], 0
            for n in _sizes(case):
                x, v, m = (t[at:at + n] for t in data)
                at += n
                x, v, a = _kdk(x, v, lambda p: _direct_acc(p, m, 0.02 ** 2, 1.0), BATCH_DT, case["steps"])
                zero = torch.zeros_like(m)[:, None]
                parts.append((torch.cat((x, m[:, None]), 1), torch.cat((v, zero), 1), torch.cat((a, zero), 1)))
            return dict(zip(("xm", "vel", "acc"), (torch.cat(p) for p in zip(*parts))))
        x, v, m, target = data
        eps2, dt = 0.05 ** 2, TRAIN_DT
        h, path = 0.5 * dt, [x]
        a = _direct_acc(x, m, eps2, GALACTIC_G)
        for _ in range(case["steps"]):
            v = v + h * a
            x = x + dt * v
            a = _direct_acc(x, m, eps2, GALACTIC_G)
            v = v + h * a
            path.append(x)
        lx = 2.0 * (x - target) / x.numel()
        lv, la, lm = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(m)
        for p in reversed(path[1:]):
            gx, gm = _force_vjp(p, m, la + h * lv, eps2, GALACTIC_G)
            lx, lm = lx + gx, lm + gm
            lv = lv + dt * lx
            la = h * lv
        gx, gm = _force_vjp(path[0], m, la, eps2, GALACTIC_G)
        return dict(pos=x, vel=v, gx=lx + gx, gv=lv, gm=lm + gm)
