"""The work that a user of this library has it do, as measurable cases.

A case is a dict of plain values; ``op`` names the call that is made:

* ``step``   one force evaluation over device-resident lists
             (gravity.DeviceSystem.step; order 4 lists go through the
             hexadecapole build's entry);
* ``graph``  many independent systems as one replayed graph
             (gravity.GravityGraph);
* ``tree``   positions to forces on the GPU: tree build, walk, forces
             (gputree.DeviceTree, walk.gpu_walk, gravity.DeviceSystem);
* ``vjp``    one forward evaluation and its vector-Jacobian product
             (adjoint.TreeStep.accel and .vjp);
* ``host``   one evaluation from pinned host arrays, the particle lists as
             runs (gravity.gravity_step_host);
* ``dropin`` one evaluation through the HostCUDA.h / EwaldCUDA.h boundary,
             FP32 structs in pinned host memory (gravity.dropin_step).

``model`` is the particle distribution: an isolated Plummer sphere, or a
periodic unit box with the Ewald term holding NFW halos and a uniform
background, or a lattice hardly perturbed.  The lattice is evaluated in FP64
only: its net forces and potentials are the small rest of terms of order one,
of which FP32 leaves three or four digits.  The FP32-mixed form computes in FP32 and
returns FP64 arrays; its results are handed on here in FP32, the precision in
which ChaNGa's VariablePartData keeps them.  The FP64 form's stay FP64.

``exact`` evaluates the same interactions in FP64 with torch alone: its own
tree, walk, moments, spline and Ewald sums, written from the rules that the
package's host tree states.
"""
import itertools
import math

import numpy as np
import torch

DEV = "cuda"
BUCKETS = (8, 12, 16, 24, 32, 64)  # ChaNGa's default is 12; the workloads use 16 and 32
EW_CUT, EWH_CUT = 2.6, 2.8


def listed():
    return [
        # one small isolated system: a few dozen buckets, the latency of a call
        dict(name="plummer1k", op="step", model="plummer", n=1024, n_bucket=16, theta=0.6,
             form="mixed", order=2),
        # an isolated galaxy or cluster model
        dict(name="plummer32k", op="step", model="plummer", n=32768, n_bucket=16, theta=0.7,
             form="mixed", order=2),
        # a cosmological box at a late time, particles in halos
        dict(name="nfw1m", op="step", model="nfw", n=2 ** 20, n_bucket=32, theta=0.7,
             form="mixed", order=2),
        # the benchmark's box, the largest
        dict(name="nfw8m", op="step", model="nfw", n=2 ** 23, n_bucket=32, theta=0.7,
             form="mixed", order=2),
        # the plain FP64 form, used where forces are checked; a ragged count
        dict(name="nfw120k_fp64", op="step", model="nfw", n=120011, n_bucket=32, theta=0.7,
             form="fp64", order=2),
        # hexadecapole cells, ChaNGa's default build, ChaNGa's default bucket
        dict(name="plummer200k_hex", op="step", model="plummer", n=200003, n_bucket=12, theta=0.7,
             form="mixed", order=4),
        # many independent clusters in one launch
        dict(name="clusters40_graph", op="graph", model="plummer", n=40, n_bucket=16, theta=0.6,
             form="mixed", order=2, n_max=65536),
        # one time step of an isolated model: the tree is new each time
        dict(name="plummer64k_tree", op="tree", model="plummer", n=65536, n_bucket=16, theta=0.7,
             form="mixed", order=2),
        # one time step of a cosmological box, a ragged count
        dict(name="nfw1m_tree", op="tree", model="nfw", n=1000003, n_bucket=16, theta=0.7,
             form="mixed", order=2),
        # forward and backward of a differentiated step
        dict(name="plummer64k_vjp", op="vjp", model="plummer", n=65536, n_bucket=16, theta=0.7,
             form="mixed", order=2),
        # lists built on the host, forces wanted there
        dict(name="nfw1m_host", op="host", model="nfw", n=2 ** 20, n_bucket=32, theta=0.7,
             form="mixed", order=2),
        # ChaNGa's own boundary, a ragged count
        dict(name="nfw500k_dropin", op="dropin", model="nfw", n=500009, n_bucket=32, theta=0.7,
             form="fp32", order=2),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(("step", "step", "step", "step", "fp64", "hex", "graph", "tree", "tree", "vjp",
                       "host", "dropin"))
    c = dict(op=kind, model=rng.choice(("plummer", "nfw")), n=0,
             n_bucket=rng.choice(BUCKETS), theta=round(rng.uniform(0.55, 0.8), 3), form="mixed",
             order=2)
    if kind == "step":
        c["n"] = size(1024, 2 ** 21)
    elif kind == "fp64":
        c.update(op="step", model=rng.choice(("plummer", "nfw", "lattice")), form="fp64",
                 n=size(1024, 100000))
    elif kind == "hex":
        c.update(op="step", model="plummer", order=4, n=size(1024, 2 ** 18))
    elif kind == "graph":
        c.update(model="plummer", n=rng.randint(3, 40), n_max=rng.choice((4096, 16384, 32768)))
    elif kind == "tree":
        c["n"] = size(1024, 2 ** 20)
    elif kind == "vjp":
        c.update(model="plummer", n=size(1024, 2 ** 17))
    elif kind == "host":
        c["n"] = size(2048, 2 ** 20)
    else:
        c.update(n=size(2048, 2 ** 19), form="fp32")
    if c["model"] == "lattice":
        c["n"] = round(c["n"] ** (1 / 3)) ** 3
    return c


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _directions(g, n):
    u = 2 * _rand(g, n) - 1
    phi = 2 * math.pi * _rand(g, n)
    s = torch.sqrt(1 - u * u)
    return torch.stack((s * torch.cos(phi), s * torch.sin(phi), u), 1)


def _plummer(g, n, a=1.0):
    x = _rand(g, n).clamp_min(1e-12) * (1 + 1 / 400.0) ** -1.5  # truncated at 20 scale radii
    r = a / torch.sqrt(x ** (-2.0 / 3.0) - 1)
    return r[:, None] * _directions(g, n)


def _nfw(g, n, seed, n_halos=64, conc=10.0):
    rs = np.random.RandomState(seed % 2 ** 32)
    mh = np.exp(rs.normal(math.log(0.01), 1.0, n_halos))
    rvir = 0.02 * (mh / np.median(mh)) ** (1 / 3)
    n_in = round(0.8 * n)
    cum = torch.from_numpy(np.cumsum(mh / mh.sum())).to(DEV)
    halo = torch.searchsorted(cum, _rand(g, n_in).sort().values).clamp_max(n_halos - 1)
    target = _rand(g, n_in) * (math.log1p(conc) - conc / (1 + conc))
    lo, hi = torch.zeros_like(target), torch.full_like(target, conc)
    for _ in range(50):
        mid = 0.5 * (lo + hi)
        below = torch.log1p(mid) - mid / (1 + mid) < target
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    r = lo / conc * torch.from_numpy(rvir).to(DEV)[halo]
    centres = torch.from_numpy(rs.uniform(0, 1, (n_halos, 3))).to(DEV)
    inside = centres[halo] + r[:, None] * _directions(g, n_in)
    return torch.remainder(torch.cat((inside, _rand(g, n - n_in, 3))), 1.0)


def _lattice(g, n, rms):
    """A cubic lattice displaced by a Gaussian field, P(k) ~ k^-2."""
    ng = round(n ** (1 / 3))
    k = torch.fft.fftfreq(ng, device=DEV, dtype=torch.float64) * ng
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    amp = torch.where(k2 > 0, 1 / torch.sqrt(k2.clamp_min(1)), torch.zeros_like(k2))
    disp = torch.stack([torch.fft.ifftn(torch.fft.fftn(
        torch.randn(ng, ng, ng, generator=g, device=DEV, dtype=torch.float64)) * amp).real
        for _ in range(3)], -1)
    disp *= rms / torch.sqrt((disp ** 2).sum(-1).mean())
    x = (torch.arange(ng, device=DEV, dtype=torch.float64) + 0.5) / ng
    grid = torch.stack(torch.meshgrid(x, x, x, indexing="ij"), -1)
    return torch.remainder((grid + disp).reshape(-1, 3), 1.0)


def _particles(case, seed):
    """Positions, masses and softenings (FP64, on the GPU)."""
    n, model, g = case["n"], case["model"], _gen(seed)
    if model == "plummer":
        pos, soft = _plummer(g, n), 0.01
    elif model == "nfw":
        pos, soft = _nfw(g, n, seed), 2e-4
    else:
        ng = round(n ** (1 / 3))
        pos = _lattice(g, n, 0.2 / ng)
        soft = 1 / (50.0 * ng)
    if case["op"] == "dropin":
        pos = pos.float().double()  # snapshot files and this boundary hold FP32 coordinates
    full = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    return pos, full, torch.full_like(full, soft)


def _clusters(case, seed):
    """Independent Plummer spheres, sizes log-uniform in [1024, n_max] (the
    same for every seed, so that results have one shape)."""
    g, rs, out = _gen(seed), np.random.RandomState(case["n"]), []
    for _ in range(case["n"]):
        n = int(math.exp(rs.uniform(math.log(1024), math.log(case["n_max"]))))
        a = rs.uniform(0.5, 2.0)
        m = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
        out.append((_plummer(g, n, a), m, torch.full_like(m, 0.01 * a)))
    return out


def _period(case):
    return 0.0 if case["model"] == "plummer" else 1.0


def _ewald(case):
    from changa_gb300.gravity import EwaldConfig
    return EwaldConfig(_period(case), 1, EW_CUT, EWH_CUT) if _period(case) else None


class _Host:
    """A program's pinned host arrays, released with the state."""

    def __init__(self):
        self.held = []

    def pin(self, a):
        from changa_gb300.gravity import PinnedArray
        self.held.append(PinnedArray(a))
        return self.held[-1].array

    def __del__(self):
        for h in self.held:
            h.free()


class _Kept:
    """An array view that keeps the owner of its memory alive."""

    def __init__(self, a, owner):
        self.owner, self.__array_interface__ = owner, a.__array_interface__


def prepare(case, seed):
    from changa_gb300 import gravity, tree
    from changa_gb300.adjoint import TreeStep
    from changa_gb300.gputree import DeviceTree
    from changa_gb300.walk import gpu_walk
    op, nb, theta, per = case["op"], case["n_bucket"], case["theta"], _period(case)
    if op == "graph":
        systems = [tree.build_lists(*(a.cpu().numpy() for a in p), n_bucket=nb, theta=theta)
                   for p in _clusters(case, seed)]
        ds = gravity.DeviceSystem(tree.concat_systems(systems))
        return dict(case=case, ds=ds, graph=gravity.GravityGraph(ds, case["form"]))
    p = _particles(case, seed)
    if op == "tree":
        return dict(case=case, particles=p)
    if op == "vjp":
        lam = torch.randn(case["n"], 3, generator=_gen(seed + 1), device=DEV, dtype=torch.float64)
        return dict(case=case, lam=lam,
                    ts=TreeStep(*p, theta=theta, n_bucket=nb, builder="device"))
    if op == "step" and case["order"] == 2:
        t = DeviceTree(*p, n_bucket=nb, theta=theta, period=per)
        cells, plist, _ = gpu_walk(t)
        return dict(case=case, ds=gravity.DeviceSystem(t, ewald=_ewald(case),
                                                       device_reqs=[cells, plist]))
    lists = tree.build_lists(*(a.cpu().numpy() for a in p), n_bucket=nb, theta=theta, period=per,
                             order=case["order"])
    if op == "step":
        return dict(case=case, ds=gravity.DeviceSystem(lists))
    host = _Host()
    if op == "dropin":
        host.held.append(gravity.DropInInputs(lists, _ewald(case)))
        return dict(case=case, host=host, inputs=host.held[0])
    runs = tree.part_runs(lists.plist)
    for o, names in ((lists, ("moments", "parts")),
                     (lists.cells, ("list", "markers", "starts", "sizes")),
                     (runs, ("runs", "run_markers", "markers", "starts", "sizes"))):
        for name in names:
            setattr(o, name, host.pin(getattr(o, name)))
    return dict(case=case, host=host, lists=lists, runs=runs, ewald=_ewald(case),
                out=host.pin(np.zeros((lists.n, 5))))


# ---------------------------------------------------------------- the calls

def _columns(v):
    return {"acc": v[:, :3], "pot": v[:, 3], "dt": v[:, 4]}


def run(state):
    from changa_gb300 import gravity
    from changa_gb300.gputree import DeviceTree
    from changa_gb300.walk import gpu_walk
    case = state["case"]
    op = case["op"]
    if op == "step":
        v = state["ds"].step(case["form"])
        return _columns(v if case["form"] == "fp64" else v.float())
    if op == "graph":
        return _columns(state["graph"].launch().float())
    if op == "tree":
        t = DeviceTree(*state["particles"], n_bucket=case["n_bucket"], theta=case["theta"],
                       period=_period(case))
        cells, plist, _ = gpu_walk(t)
        ds = gravity.DeviceSystem(t, ewald=_ewald(case), device_reqs=[cells, plist])
        return dict(_columns(ds.step(case["form"]).float()), perm=t.perm)
    if op == "vjp":
        a = state["ts"].accel(case["form"])
        gx, gm = state["ts"].vjp(state["lam"])
        return {"acc": a.float(), "gx": gx.float(), "gm": gm.float()}
    if op == "host":
        v = gravity.gravity_step_host(state["lists"], case["form"], state["ewald"],
                                      vars=state["out"], overwrite=True, runs=state["runs"])
        return _columns(torch.from_numpy(v).float())
    v = gravity.dropin_step(state["inputs"])
    return _columns(np.asarray(_Kept(v, state["host"])))


# ---------------------------------------------------------------- FP64 with torch alone

class _Tree:
    """Tree, moments and interaction lists of one system in FP64: a binary
    Morton tree in a cubical box, buckets of at most n_bucket particles, and
    the dual walk's opening rules (gravity.h:652-723)."""

    def __init__(self, pos, mass, soft, n_bucket, theta, period, order=2):
        self.period, self.theta, self.order = period, theta, order
        f = pos.float()
        lo, hi = f.amin(0).cpu().numpy(), f.amax(0).cpu().numpy()
        half = np.float32(float(np.float32(1) + np.float32(1.91e-6)) * 0.5 * float((hi - lo).max()))
        mid = np.float32(0.5) * (lo + hi)
        b0, b1 = (torch.from_numpy(x.astype(np.float64)).to(DEV) for x in (mid - half, mid + half))
        q = (((pos - b0) / (b1 - b0)).clamp_min(0) * 2097152.0).clamp_max(2097151).long()
        key = torch.zeros_like(q[:, 0])
        for b in range(21):
            for k in range(3):
                key |= ((q[:, k] >> b) & 1) << (3 * b + 2 - k)
        key, self.perm = torch.sort(key, stable=True)
        self.pos, self.mass, self.soft = pos[self.perm], mass[self.perm], soft[self.perm]
        n = pos.shape[0]
        # nodes level by level
        first = torch.zeros(1, dtype=torch.long, device=DEV)
        count = torch.full_like(first, n)
        parent = torch.full_like(first, -1)
        levels, total, level = [], 0, 0
        while first.numel():
            ids = torch.arange(total, total + first.numel(), device=DEV)
            levels.append((first, count, parent, ids))
            total += first.numel()
            o = (count > n_bucket) & (level < 60)
            f0, c0, sh = first[o], count[o], 62 - level
            thr = (((key[f0] >> (sh + 1)) << 1) | 1) << sh
            at = torch.minimum(torch.maximum(torch.searchsorted(key, thr), f0), f0 + c0)
            first = torch.stack((f0, at), 1).reshape(-1)
            count = torch.stack((at - f0, f0 + c0 - at), 1).reshape(-1)
            parent = ids[o].repeat_interleave(2)
            keep = count > 0
            first, count, parent, level = first[keep], count[keep], parent[keep], level + 1
        self.first, self.count, self.parent = (torch.cat([x[j] for x in levels]) for j in range(3))
        self.levels = [x[3] for x in levels]
        self.child = torch.full((total, 2), -1, dtype=torch.long, device=DEV)
        kids = torch.arange(1, total, device=DEV)
        slot = (self.first[1:] != self.first[self.parent[1:]]).long()
        alone = torch.bincount(self.parent[1:], minlength=total)[self.parent[1:]] == 1
        self.child[self.parent[1:], torch.where(alone, torch.zeros_like(slot), slot)] = kids
        self.leaf = self.child[:, 0] < 0
        self.buckets = torch.nonzero(self.leaf)[:, 0]
        self.buckets = self.buckets[torch.argsort(self.first[self.buckets])]
        self.bstart, self.bsize = self.first[self.buckets], self.count[self.buckets]
        # buckets below a node: a contiguous range in key order
        self.b_lo = torch.searchsorted(self.bstart, self.first)
        self.b_hi = torch.searchsorted(self.bstart, self.first + self.count)
        self.of = torch.repeat_interleave(self.buckets, self.bsize)  # each particle's bucket
        inf = torch.full((total, 3), math.inf, dtype=torch.float64, device=DEV)
        at = self.of[:, None].expand(-1, 3)
        self.lo = inf.scatter_reduce(0, at, self.pos, "amin")
        self.hi = (-inf).scatter_reduce(0, at, self.pos, "amax")
        for ids in reversed(self.levels[1:]):
            p = self.parent[ids][:, None].expand(-1, 3)
            self.lo = self.lo.scatter_reduce(0, p, self.lo[ids], "amin")
            self.hi = self.hi.scatter_reduce(0, p, self.hi[ids], "amax")
        self.M, self.cm, self.Q = self.moments(self.pos, self.mass)
        ms = torch.zeros_like(self.M).index_add(0, self.of, self.mass * self.soft)
        for ids in reversed(self.levels[1:]):
            ms = ms.index_add(0, self.parent[ids], ms[ids])
        self.s = ms / self.M
        far = torch.maximum(self.cm - self.lo, self.hi - self.cm).square().sum(1)
        d2 = (self.pos - self.cm[self.of]).square().sum(1)
        r2 = torch.where(self.leaf, torch.zeros_like(far).scatter_reduce(0, self.of, d2, "amax"), far)
        self.radius = torch.sqrt(r2)
        self.walk()

    def moments(self, pos, mass):
        """Mass, centre of mass and second moments (xx xy xz yy yz zz) of
        every node, differentiable in pos and mass."""
        total = self.first.numel()

        def up(x):
            for ids in reversed(self.levels[1:]):
                x = x.index_add(0, self.parent[ids], x[ids])
            return x

        def zero(*k):
            return torch.zeros((total, *k), dtype=torch.float64, device=DEV)

        M = up(zero().index_add(0, self.of, mass))
        cm = up(zero(3).index_add(0, self.of, mass[:, None] * pos)) / M[:, None]

        def outer(d):
            return torch.stack([d[:, i] * d[:, j] for i in range(3) for j in range(i, 3)], 1)

        Q = zero(6).index_add(0, self.of, mass[:, None] * outer(pos - cm[self.of]))
        for ids in reversed(self.levels[1:]):
            p = self.parent[ids]
            Q = Q.index_add(0, p, Q[ids] + M[ids][:, None] * outer(cm[ids] - cm[p]))
        return M, cm, Q

    def offsets(self):
        r = range(-1, 2) if self.period else (0,)
        return self.period * torch.tensor(list(itertools.product(r, r, r)), dtype=torch.float64,
                                          device=DEV)

    def walk(self):
        """The accepted cells and opened source buckets as (local node,
        source node, replica), then per target bucket."""
        off = self.offsets()
        g = torch.zeros(off.shape[0], dtype=torch.long, device=DEV)
        loc, rep = torch.zeros_like(g), torch.arange(off.shape[0], device=DEV)
        geo = 2.0 / math.sqrt(3.0)
        big = torch.maximum(geo * self.radius / self.theta, self.radius)
        mono = geo * self.radius / self.theta ** 4
        cells, parts = [], []
        while g.numel():
            c = self.cm[g] + off[rep]
            lo, hi = self.lo[loc], self.hi[loc]
            near = torch.maximum((lo - c).clamp_min(0), (c - hi).clamp_min(0)).square().sum(1)
            far = torch.maximum((c - lo).abs(), (hi - c).abs()).square().sum(1)
            r2 = big[g] ** 2
            few = self.count[g] <= 6
            inter = near <= r2
            opened = few | (inter & (self.leaf[loc] | (far <= r2)))
            accept = ~few & ~inter
            if self.order == 4:
                again = accept & self.softened(g, loc, off[rep]) & (near <= mono[g] ** 2)
                opened, accept = opened | again, accept & ~again
            cells.append((loc[accept], g[accept], rep[accept]))
            part = ~accept & self.leaf[g]
            parts.append((loc[part], g[part], rep[part]))
            down = ~accept & ~self.leaf[g]
            o, u = down & opened, down & ~opened
            kid = self.child[g[o]].reshape(-1)
            lkid = self.child[loc[u]].reshape(-1)
            k0, k1 = kid >= 0, lkid >= 0
            rep = torch.cat((rep[o].repeat_interleave(2)[k0], rep[u].repeat_interleave(2)[k1]))
            loc = torch.cat((loc[o].repeat_interleave(2)[k0], lkid[k1]))
            g = torch.cat((kid[k0], g[u].repeat_interleave(2)[k1]))
        self.cells, self.parts = self.per_bucket(cells), self.per_bucket(parts)

    def softened(self, g, loc, off):
        """The cell's softening sphere meets the node's (gravity.h:252-260)."""
        c = self.cm[g] + off
        r = 2 * self.s[g]
        d2 = (c - self.cm[loc]).square().sum(1)
        near = torch.maximum((self.lo[loc] - c).clamp_min(0),
                             (c - self.hi[loc]).clamp_min(0)).square().sum(1)
        return (d2 <= (r + 2 * self.s[loc]) ** 2) | (near <= r * r)

    def per_bucket(self, found):
        loc, src, rep = (torch.cat(x) for x in zip(*found))
        nb = self.b_hi[loc] - self.b_lo[loc]
        e = torch.repeat_interleave(torch.arange(loc.numel(), device=DEV), nb)
        b = self.b_lo[loc][e] + torch.arange(e.numel(), device=DEV) - (torch.cumsum(nb, 0) - nb)[e]
        b, o = torch.sort(b, stable=True)
        return b, src[e][o], rep[e][o]

    def blocks(self, which, most=1 << 22):
        """The pairs of one kind, some buckets at a time: (buckets, list
        lengths, targets with -1 where a bucket has fewer, sources as node or
        particle indices, replica offsets)."""
        b, src, rep = self.cells if which == "cells" else self.parts
        off, width = self.offsets(), int(self.bsize.max())
        nb = self.buckets.numel()
        size = torch.ones_like(src) if which == "cells" else self.count[src]
        per = torch.zeros(nb, dtype=torch.long, device=DEV).index_add(0, b, size)
        part = torch.div(torch.cumsum(per, 0) * width, most, rounding_mode="floor")
        edges = [0] + (torch.nonzero(part[1:] != part[:-1])[:, 0] + 1).tolist() + [nb]
        ent = torch.searchsorted(b, torch.tensor(edges, device=DEV)).tolist()
        lane = torch.arange(width, device=DEV)
        for (b0, b1), (e0, e1) in zip(zip(edges, edges[1:]), zip(ent, ent[1:])):
            if e0 == e1:
                continue
            s, r, bb = src[e0:e1], rep[e0:e1], b[e0:e1]
            if which == "parts":
                k = size[e0:e1]
                e = torch.repeat_interleave(torch.arange(e1 - e0, device=DEV), k)
                s = self.first[s][e] + torch.arange(e.numel(), device=DEV) - (torch.cumsum(k, 0) - k)[e]
                r, bb = r[e], bb[e]
            tgt = self.bstart[bb][:, None] + lane
            tgt = torch.where(lane < self.bsize[bb][:, None], tgt, -1)
            yield (b0, b1), per[b0:b1], tgt, s, off[r]


def _spline(r2, twoh):
    """SPLINEQ's a, b, c, d (gravity.h:22-66)."""
    ir = 1 / torch.sqrt(r2)
    a, b = ir, ir ** 3
    c, d = 3 * ir ** 5, 15 * ir ** 7
    near = r2 < twoh * twoh
    if not bool(near.any()):
        return a, b, c, d
    h = torch.where(near, 2 / twoh, torch.ones_like(r2))
    u = torch.where(near, h * r2 * ir, torch.ones_like(r2))
    inner = (h * (7 / 5 - 2 / 3 * u ** 2 + 3 / 10 * u ** 4 - 1 / 10 * u ** 5),
             h ** 3 * (4 / 3 - 6 / 5 * u ** 2 + 0.5 * u ** 3), h ** 5 * (12 / 5 - 1.5 * u),
             1.5 * h ** 6 * ir)
    outer = (-ir / 15 + h * (8 / 5 - 4 / 3 * u ** 2 + u ** 3 - 3 / 10 * u ** 4 + u ** 5 / 30),
             -ir ** 3 / 15 + h ** 3 * (8 / 3 - 3 * u + 6 / 5 * u ** 2 - u ** 3 / 6),
             -ir ** 5 / 5 + 3 * h ** 4 * ir + h ** 5 * (-12 / 5 + 0.5 * u),
             -ir ** 7 + 3 * h ** 4 * ir ** 3 - 0.5 * h ** 6 * ir)
    return tuple(torch.where(near, torch.where(u < 1, i, o), f)
                 for i, o, f in zip(inner, outer, (a, b, c, d)))


def _point(r, r2, hit, m, twoh):
    """Softened point masses m at r = source - target: acceleration,
    potential and b."""
    a, b, _, _ = _spline(torch.where(hit, r2, torch.ones_like(r2)), twoh)
    a, b = a * hit, b * hit
    return [m * b * x for x in r], -m * a, b


def _quad(r, r2, hit, M, Q, twoh):
    """Quadrupole cells at r = target - cell (gravity.h:436-472)."""
    a, b, c, d = (x * hit for x in _spline(torch.where(hit, r2, torch.ones_like(r2)), twoh))
    xx, xy, xz, yy, yz, zz = Q
    q = (xx * r[0] + xy * r[1] + xz * r[2], xy * r[0] + yy * r[1] + yz * r[2],
         xz * r[0] + yz * r[1] + zz * r[2])
    qir = 0.5 * (q[0] * r[0] + q[1] * r[1] + q[2] * r[2])
    tr = 0.5 * (xx + yy + zz)
    g = b * M + d * qir - c * tr
    return [c * q[k] - g * r[k] for k in range(3)], -(M * a + c * qir - b * tr), b


_MONO = {k: list(itertools.combinations_with_replacement(range(3), k)) for k in (2, 3, 4)}


def _hex_moments(t):
    """Sums over each node's particles of m times the monomials of order 2 to
    4 about the centre of mass, and their traces."""
    total = t.first.numel()
    out = {k: torch.zeros((total, len(v)), dtype=torch.float64, device=DEV) for k, v in _MONO.items()}
    node = t.of.clone()
    while bool((node >= 0).any()):
        live = torch.nonzero(node >= 0)[:, 0]
        d = t.pos[live] - t.cm[node[live]]
        for k, v in _MONO.items():
            mono = torch.stack([d[:, list(ix)].prod(1) for ix in v], 1) * t.mass[live][:, None]
            out[k].index_add_(0, node[live], mono)
        node[live] = t.parent[node[live]]
    at = {k: {ix: i for i, ix in enumerate(v)} for k, v in _MONO.items()}

    def tr(k, ix):
        return sum(out[k][:, at[k][tuple(sorted(ix + (j, j)))]] for j in range(3))

    t3 = [tr(3, (i,)) for i in range(3)]
    t4 = {ix: tr(4, ix) for ix in _MONO[2]}
    return out, tr(2, ()), t3, t4, t4[(0, 0)] + t4[(1, 1)] + t4[(2, 2)]


def _hex(r, r2, hit, M, mo, src):
    """Cells expanded to the hexadecapole at r = target - cell: the Legendre
    sums to fourth order, the acceleration by differentiating them."""
    out, t2, t3, t4, u4 = mo
    r = [x.detach().requires_grad_(True) for x in r]
    with torch.enable_grad():
        ir = 1 / torch.sqrt(torch.where(hit, r[0] ** 2 + r[1] ** 2 + r[2] ** 2, 1.0))
        x = [c * ir for c in r]

        def full(k, tab):
            s = 0
            for i, ix in enumerate(_MONO[k]):
                w = math.factorial(k)
                for j in range(3):
                    w //= math.factorial(ix.count(j))
                term = w * (tab[ix][src] if isinstance(tab, dict) else tab[src, i])[:, None]
                for j in ix:
                    term = term * x[j]
                s = s + term
            return s

        n3 = sum(t3[j][src][:, None] * x[j] for j in range(3))
        pot = -(M * ir + (3 * full(2, out[2]) - t2[src][:, None]) * ir ** 3 / 2 +
                (5 * full(3, out[3]) - 3 * n3) * ir ** 4 / 2 +
                (35 * full(4, out[4]) - 30 * full(2, t4) + 3 * u4[src][:, None]) * ir ** 5 / 8)
        pot = pot * hit
        acc = torch.autograd.grad(-pot.sum(), r)
    return list(acc), pot.detach(), (ir ** 3 * hit).detach()


def _forces(t):
    """Accelerations, potentials and dtGrav of every particle (tree order)."""
    v = torch.zeros(t.pos.shape[0], 5, dtype=torch.float64, device=DEV)
    hexa = _hex_moments(t) if t.order == 4 else None

    def add(bk, per, tgt, acc, pot, idt):
        rows = torch.stack([*acc, pot], -1)
        s = torch.segment_reduce(rows.contiguous(), "sum", lengths=per, axis=0, unsafe=True)
        m = torch.segment_reduce(idt.contiguous(), "max", lengths=per, axis=0, unsafe=True, initial=0)
        lane = torch.arange(tgt.shape[1], device=DEV)
        at = t.bstart[bk[0]:bk[1]][:, None] + lane
        ok = lane < t.bsize[bk[0]:bk[1]][:, None]
        v[at[ok], :4] += s[ok]
        v[at[ok], 4] = torch.maximum(v[at[ok], 4], m[ok])

    for which in ("cells", "parts"):
        for bk, per, tgt, src, off in t.blocks(which, 1 << (20 if hexa and which == "cells" else 22)):
            live, k = tgt >= 0, tgt.clamp_min(0)
            if which == "cells":
                r = [t.pos[k, j] - (t.cm[src, j] + off[:, j])[:, None] for j in range(3)]
                M, twoh = t.M[src][:, None], t.s[src][:, None] + t.soft[k]
            else:
                r = [(t.pos[src, j] + off[:, j])[:, None] - t.pos[k, j] for j in range(3)]
                M, twoh = t.mass[src][:, None], t.soft[src][:, None] + t.soft[k]
            r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
            hit = (r2 != 0) & live
            if which == "parts":
                acc, pot, b = _point(r, r2, hit, M, twoh)
            elif hexa is None:
                acc, pot, b = _quad(r, r2, hit, M, [t.Q[src, i][:, None] for i in range(6)], twoh)
            else:
                bb = t.of[k[:, 0]]
                soft = t.softened(src, bb, off)[:, None]
                acc, pot, b = _hex(r, r2, hit & ~soft, M, hexa, src)
                a2, p2, b2 = _point([-x for x in r], r2, hit & soft, M, twoh)
                acc, pot, b = [x + y for x, y in zip(acc, a2)], pot + p2, b + b2
            add(bk, per, tgt, acc, pot, (M + t.mass[k]) * b)
    return v


def _add_ewald(v, t, form):
    """The Ewald correction about the root (Ewald.cpp:72-281, 285-383), L = 1:
    the FP64 form and the FP32 boundary keep the reference's two-term series
    near the root, each within its own radius."""
    M, cm = t.M[0], t.cm[0]
    xx, xy, xz, yy, yz, zz = t.Q[0]
    d = t.pos - cm
    alpha, ka = 2.0, 4.0 / math.sqrt(math.pi)
    a2 = alpha * alpha
    inner = {"fp64": 1.2e-3, "fp32": 1.1e-2}.get(form, 0.0)
    v[:, 3] += M * math.pi / a2
    n_e = math.ceil(EW_CUT)
    for i in itertools.product(range(-n_e, n_e + 1), repeat=3):
        hole = max(map(abs, i)) <= 1
        x, y, z = (d[:, k] + i[k] for k in range(3))
        r2 = x * x + y * y + z * z
        s = a2 * r2
        ir2 = 1 / r2.clamp_min(1e-30)
        e = ka * torch.exp(-s) * ir2
        g = [(torch.erfc(torch.sqrt(s)) - (1.0 if hole else 0.0)) * torch.sqrt(ir2)]
        for k in range(3):
            g.append((2 * k + 1 if k else 1) * g[k] * ir2 + (2 * a2) ** k * e)
        if hole:
            for k in range(4):
                terms = [(-1) ** j / (math.factorial(j) * (2 * j + 2 * k + 1)) for j in range(24)]
                ser = torch.zeros_like(s)
                for c in reversed(terms):
                    ser = ser * s + c
                two = terms[0] + terms[1] * s
                ser = torch.where(r2 < inner, two, ser)
                g[k] = torch.where((s < 1.0) if not inner else (s < 0.05) | (r2 < inner),
                                   -ka * (2 * a2) ** k * ser, g[k])
        else:
            g = [torch.where(r2 <= EW_CUT ** 2, x_, torch.zeros_like(x_)) for x_ in g]
        q = (xx * x + xy * y + xz * z, xy * x + yy * y + yz * z, xz * x + yz * y + zz * z)
        qir, tr = 0.5 * (q[0] * x + q[1] * y + q[2] * z), 0.5 * (xx + yy + zz)
        w = g[1] * M - g[2] * tr + g[3] * qir
        v[:, 3] -= g[0] * M - g[1] * tr + g[2] * qir
        for k, c in enumerate((x, y, z)):
            v[:, k] += g[2] * q[k] - c * w
    n_h = math.ceil(EWH_CUT)
    for h in itertools.product(range(-n_h, n_h + 1), repeat=3):
        h2 = sum(c * c for c in h)
        if not 0 < h2 <= EWH_CUT ** 2:
            continue
        g0 = math.exp(-math.pi ** 2 * h2 / a2) / (math.pi * h2)
        qh = 0.5 * (xx * h[0] ** 2 + yy * h[1] ** 2 + zz * h[2] ** 2) + xy * h[0] * h[1] + \
            xz * h[0] * h[2] + yz * h[1] * h[2]
        coef = 4 * math.pi ** 2 * g0 * qh - g0 * M
        ph = 2 * math.pi * (h[0] * d[:, 0] + h[1] * d[:, 1] + h[2] * d[:, 2])
        v[:, 3] += coef * torch.cos(ph)
        s = 2 * math.pi * coef * torch.sin(ph)
        for k in range(3):
            v[:, k] += h[k] * s


def _gradient(t, lam):
    """d(sum lam . a)/dx and d/dm through pairs and moments, lists and
    softenings fixed (tree order)."""
    pos, mass = t.pos.clone().requires_grad_(True), t.mass.clone().requires_grad_(True)
    with torch.enable_grad():
        mo = t.moments(pos, mass)
        M, cm, Q = (x.detach().requires_grad_(True) for x in mo)
        for which in ("cells", "parts"):
            for _, _, tgt, src, off in t.blocks(which, 1 << 21):
                live, k = tgt >= 0, tgt.clamp_min(0)
                if which == "cells":
                    r = [pos[k, j] - (cm[src, j] + off[:, j])[:, None] for j in range(3)]
                else:
                    r = [(pos[src, j] + off[:, j])[:, None] - pos[k, j] for j in range(3)]
                hit = (r[0].detach() ** 2 + r[1].detach() ** 2 + r[2].detach() ** 2 != 0) & live
                r2 = torch.where(hit, r[0] ** 2 + r[1] ** 2 + r[2] ** 2, 1.0)
                if which == "cells":
                    acc = _quad(r, r2, hit, M[src][:, None], [Q[src, i][:, None] for i in range(6)],
                                t.s[src][:, None] + t.soft[k])[0]
                else:
                    acc = _point(r, r2, hit, mass[src][:, None], t.soft[src][:, None] + t.soft[k])[0]
                sum((lam[k, j] * acc[j]).sum() for j in range(3)).backward()
        torch.autograd.backward(mo, (M.grad, cm.grad, Q.grad))
    return pos.grad, mass.grad


def exact(case, seed):
    if case["op"] == "graph":
        systems = _clusters(case, seed)
    elif case["n"] > 2 ** 20:
        return None  # the pairs of more particles take longer than a check should
    else:
        systems = [_particles(case, seed)]
    with torch.no_grad():
        rows, trees = [], []
        for p in systems:
            t = _Tree(*p, case["n_bucket"], case["theta"], _period(case), case["order"])
            v = _forces(t)
            if _period(case):
                _add_ewald(v, t, case["form"])
            rows.append(v)
            trees.append(t)
        v = torch.cat(rows)
        if case["op"] != "vjp":
            return _columns(v)
        t, lam = trees[0], torch.randn(case["n"], 3, generator=_gen(seed + 1), device=DEV,
                                       dtype=torch.float64)
        gx, gm = _gradient(t, lam[t.perm])
        back = torch.empty_like(t.perm)
        back[t.perm] = torch.arange(t.perm.numel(), device=DEV)
        return {"acc": v[back, :3], "gx": gx[back], "gm": gm[back]}


# ---------------------------------------------------------------- the work of one pass

def _interactions(n, n_bucket, theta, per):
    """Cell and particle list entries per particle: the counts that the walk
    gives on these models (n 1e5 to 8e6, buckets 8 to 64), as powers of the
    bucket size and the opening angle."""
    few = min(1.0, math.log2(n) / 20.0) if not per else 1.0
    cells = 640.0 * (0.7 / theta) ** 2.2 * (n_bucket / 32.0) ** -0.1 * few
    parts = 1180.0 * (0.7 / theta) ** 2.0 * (n_bucket / 32.0) ** 0.9 * few
    return min(cells, 2.0 * n), min(parts, 1.0 * n)


def work(case):
    n, per, op = case["n"], _period(case), case["op"]
    if op == "graph":  # the mean of the log-uniform sizes
        n = int(n * (case["n_max"] - 1024) / math.log(case["n_max"] / 1024))
    cells, parts = _interactions(n, case["n_bucket"], case["theta"], per)
    flops = n * (cells * (196 if case["order"] == 4 else 67) + parts * 23)
    if per:  # about 74 replica terms and 40 pairs of h-vectors per particle
        flops += n * (74 * 60 + 40 * 12)
    if op == "vjp":
        flops *= 3
    held = 20 if op == "dropin" else 40
    buckets = n / (0.7 * case["n_bucket"])
    nodes = 2 * buckets * (27 if case["order"] == 4 else 12) * held / 5
    lists = buckets * 8 * (cells + (parts / 14 if op == "host" else parts))
    if op == "tree":
        nodes = lists = 0  # made and used inside the pass
    moved = n * held * 2 + nodes + lists + (n * 7 * 8 if op == "vjp" else 0)
    return {"bytes": float(moved), "flops": float(flops)}
