"""What the framework is asked to do, at the sizes it is asked to do it.

A case is one call (or the few calls that belong together) of a user's
program through the public Python entry points: a start is uploaded, strained
affinely, relaxed, and the positions and the report come back.  Relaxations
carry a cap on the FIRE steps, so that a pass is a fixed amount of the work
that a full relaxation repeats 1e4 to 1e6 times; none of them converges
within its cap.  Networks are the diluted triangular lattices, Mikado
networks and gel composites of the benchmark and the tests.

Kinds of case:
  eval      forces, energies and stress of one network at given positions
  relax     Network: set_positions, affine_displace, relax, positions
  sweep     the compression-then-shear protocol as one CUDA graph
  batch     Batch: many uneven networks relaxed in one call
  gel       a network in a gel (network_mesh_relax.cu's program)
  response  the linear-response program (sparse_relax.cpp's): both unit
            loads solved, then three points of the protocol
"""
import math
import random

import numpy as np
import torch

import network_relaxation_gb300 as nr

GEL = (0.3, 1.0, 0.02)  # shear modulus, bulk modulus, dilation
TOL = 1e-12             # linear response: relative residual of the unit loads


def listed():
    return [
        # an optimiser of the user's own, or a check of a state: the smallest
        # call there is, one force / energy / stress evaluation of a 32 x 32
        # lattice (latency, launches, copies)
        dict(name="eval_32", kind="eval", nx=32, ny=32, p=0.65, jitter=0.0, line=False, kb=1e-3),
        # the reference's own use: a small network strained in ten steps,
        # FP64, here as one CUDA graph
        dict(name="sweep_fp64_32", kind="sweep", nx=32, ny=32, p=0.65, jitter=0.0, line=False, kb=1e-3,
             precision="fp64", strain_steps=10, steps=300),
        # the default precision on a network of ten thousand nodes, with
        # sizes that divide by nothing
        dict(name="relax_fp64_97x103", kind="relax", net="lattice", nx=97, ny=103, p=0.62, jitter=0.0, line=False,
             kb=1e-3, precision="fp64", criterion="rms", shear=0.02, compr=0.0, steps=400),
        # the default precision on a large jittered network with rest angles
        dict(name="relax_fp64_256", kind="relax", net="lattice", nx=256, ny=256, p=0.65, jitter=0.05, line=True,
             kb=1e-4, precision="fp64", criterion="max", shear=0.01, compr=0.0, steps=200),
        # mixed precision on one small network (an odd size)
        dict(name="relax_mixed_47x53", kind="relax", net="lattice", nx=47, ny=53, p=0.65, jitter=0.0, line=False,
             kb=1e-3, precision="mixed", criterion="max", shear=0.03, compr=0.0, steps=1000),
        # mixed precision on one network of 65 536 nodes
        dict(name="relax_mixed_256", kind="relax", net="lattice", nx=256, ny=256, p=0.65, jitter=0.05, line=True,
             kb=1e-4, precision="mixed", criterion="max", shear=0.01, compr=0.0, steps=1000),
        # a fibre network of 2e5 crossings under compression: per-bond and
        # per-triple stiffness, uneven node density.  In FP64: segments of
        # 1e-6 carry forces of 1e5, so that two FP32 trajectories part within
        # a few steps and cannot be compared
        dict(name="relax_fp64_mikado", kind="relax", net="mikado", fibres=15850, length=0.05, kb=1.0,
             precision="fp64", criterion="max", shear=0.0, compr=0.01, steps=100),
        # the largest single network: 1 048 576 nodes
        dict(name="relax_mixed_1024", kind="relax", net="lattice", nx=1024, ny=1024, p=0.65, jitter=0.05, line=True,
             kb=1e-4, precision="mixed", criterion="max", shear=0.0025, compr=0.0, steps=500),
        # throughput: an ensemble of uneven lattices, each with its own
        # dilution, stiffness and shear
        dict(name="batch_mixed_192", kind="batch", count=192, lmin=16, lmax=96, precision="mixed", steps=1000),
        # the same ensemble in the reference's precision
        dict(name="batch_fp64_64", kind="batch", count=64, lmin=16, lmax=96, precision="fp64", steps=100),
        # a network in a gel, FP64 (the only precision with a gel)
        dict(name="gel_192x144", kind="gel", nx=192, ny=144, p=0.65, kb=1e-4, shear=0.0025, steps=200),
        # linear response of a 160 x 160 lattice
        dict(name="response_160", kind="response", nx=160, ny=160, p=0.8, kb=1e-2, mu=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["eval", "sweep", "relax", "relax", "relax", "relax", "batch", "batch", "gel", "response"])
    lattice = dict(p=round(rng.uniform(0.55, 0.8), 3), jitter=rng.choice([0.0, 0.05]), kb=rng.choice([1e-4, 1e-3, 1e-2]))
    lattice["line"] = lattice["jitter"] > 0
    if kind == "eval":
        nx = _log(rng, 8, 500)
        return dict(kind=kind, nx=nx, ny=max(4, int(nx * rng.uniform(0.7, 1.4))), **lattice)
    if kind == "sweep":
        nx = _log(rng, 12, 60)
        return dict(kind=kind, nx=nx, ny=max(6, int(nx * rng.uniform(0.7, 1.4))), precision="fp64",
                    strain_steps=rng.randint(2, 10), steps=rng.randint(50, 300), **lattice)
    if kind == "relax":
        precision = rng.choice(["fp64", "mixed"])
        load = rng.choice([dict(shear=0.02, compr=0.0), dict(shear=0.005, compr=0.0), dict(shear=0.0, compr=0.01)])
        more = dict(precision=precision, criterion=rng.choice(["max", "rms"]), **load)
        if rng.random() < 0.2:
            more["precision"] = "fp64"
            return dict(kind=kind, net="mikado", fibres=_log(rng, 400, 15000), length=0.05, kb=1.0,
                        steps=rng.randint(30, 100), **more)
        nx = _log(rng, 16, 320 if precision == "fp64" else 800)
        return dict(kind=kind, net="lattice", nx=nx, ny=max(8, int(nx * rng.uniform(0.7, 1.25))),
                    steps=rng.randint(100, 400), **lattice, **more)
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed"])
        lmin = rng.randint(8, 40)
        return dict(kind=kind, count=_log(rng, 3, 100), lmin=lmin, lmax=rng.randint(lmin + 1, 96),
                    precision=precision, steps=rng.randint(50, 100 if precision == "fp64" else 500))
    if kind == "gel":
        nx = _log(rng, 16, 300)
        return dict(kind=kind, nx=nx, ny=max(8, int(nx * rng.uniform(0.6, 1.2))), p=lattice["p"], kb=lattice["kb"],
                    shear=rng.choice([0.0025, 0.02]), steps=rng.randint(50, 200))
    nx = _log(rng, 16, 200)
    return dict(kind=kind, nx=nx, ny=max(8, int(nx * rng.uniform(0.7, 1.4))), p=round(rng.uniform(0.75, 0.95), 3),
                kb=rng.choice([1e-3, 1e-2]), mu=rng.choice([0.02, 0.1]))


# ---------------------------------------------------------------- inputs

def _host(case, seed):
    """The network on the host, as a user's program reads or generates it."""
    if case["kind"] == "gel":
        return nr.HostNetwork.lattice_mesh(case["nx"], case["ny"], case["p"], 0.0, seed).get_triples()
    if case.get("net") == "mikado":
        # one realisation (its size depends on it); the start differs by seed
        return nr.HostNetwork.mikado(case["fibres"], case["length"], 1.0, 1e-5, 3)
    line = bool(case.get("line", False))
    h = nr.HostNetwork.lattice(case["nx"], case["ny"], case["p"], case.get("jitter", 0.0), seed, line_triples=line)
    return h if line else h.get_triples()


def _dt_max(case, h):
    """FIRE's largest step: 0.1 for unit springs; k = 1 / l0 makes the
    shortest Mikado segments stiff."""
    if case.get("net") == "mikado":
        return 0.05 * float(np.sqrt(h.arrays()["edge_l0"].min()))
    return 0.1


def _members(case, seed):
    """The networks of a batch: side (of the case), dilution, bending
    stiffness and shear (of the seed)."""
    r, sides = random.Random(seed), random.Random(case["count"])
    return [dict(L=sides.randint(case["lmin"], case["lmax"]), p=r.uniform(0.55, 0.75),
                 kb=math.exp(r.uniform(math.log(1e-5), math.log(1e-2))), gamma=r.uniform(0.0, 0.1),
                 seed=r.randint(1, 1 << 30)) for _ in range(case["count"])]


def _batch_hosts(case, seed):
    ms = _members(case, seed)
    return ms, [nr.HostNetwork.lattice(m["L"], m["L"], m["p"], 0.0, m["seed"]).get_triples() for m in ms]


def _params(case, dt_max=0.1):
    return nr.fire_params(alpha0=0.1, falpha=0.99, dt_max=dt_max, finc=1.1, fdec=0.5, nmin=5, mass=1.0, fcut=1e-12,
                          max_steps=case["steps"], criterion=case.get("criterion", "max"),
                          precision=case.get("precision", "fp64"))


def _start(case, points, seed):
    """Positions a user starts from: the network's own, thermally shaken a
    little in x (rows kept level for the clamps); a Mikado network, whose
    segments go down to 1e-6, is pre-strained a little instead."""
    g = np.random.default_rng(seed)
    x = points.copy()
    if case.get("net") == "mikado":
        x[:, 1] = x[:, 1].min() + (x[:, 1] - x[:, 1].min()) * (1 - 1e-3 * g.uniform(0.5, 1.0))
    else:
        x[:, 0] += g.normal(scale=1e-4, size=len(x)) * (points[:, 0].max() - points[:, 0].min()) / math.sqrt(len(x))
    return x


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "batch":
        ms, hosts = _batch_hosts(case, seed)
        b = nr.Batch(hosts, 1.0, np.array([m["kb"] for m in ms]))
        s.update(batch=b, x0=b.positions(), gamma=np.array([m["gamma"] for m in ms]) * (b.maxy - b.miny),
                 prm=_params(case))
        return s
    h = _host(case, seed)
    a = h.arrays()
    if kind == "response":
        s["spr"] = nr.Spr(h, ks=1.0, kb=case["kb"], mu=case["mu"])
        s["height"] = float(a["points"][:, 1].max() - a["points"][:, 1].min())
        return s
    net = nr.Network(h, ks=1.0, kb=case["kb"])
    s.update(net=net, H=net.maxy - net.miny, x0=_start(case, a["points"], seed))
    if kind == "eval":
        s["x0"] = a["points"] + np.random.default_rng(seed).normal(scale=0.03, size=a["points"].shape)
        return s
    if kind == "gel":
        net.set_gel(*GEL)
    s["prm"] = _params(case, _dt_max(case, h))
    return s


# ------------------------------------------------------------------ a pass

def _report(r):
    return {"e": np.array([r.e_stretch, r.e_bend, r.e_gel]), "f": np.array([r.rms_force, r.max_force]),
            "stress": np.array([r.stress_xx, r.stress_yy, r.stress_xy]), "n": np.array([r.steps, r.status])}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "batch":
        b = state["batch"]
        b.set_positions(state["x0"])
        b.affine_displace(state["gamma"], 0.0)
        reps = b.relax(state["prm"])
        return {"x": b.positions(), "e": np.array([[r.e_stretch, r.e_bend] for r in reps]),
                "f": np.array([[r.rms_force, r.max_force] for r in reps]),
                "stress": np.array([[r.stress_xx, r.stress_yy, r.stress_xy] for r in reps]),
                "n": np.array([[r.steps, r.status] for r in reps])}
    if kind == "response":
        spr, height = state["spr"], state["height"]
        spr.solve(affine=True, tol=TOL)
        out = []
        for c, g in ((0.01, 0.0), (0.0, 0.01), (0.01, 0.02)):
            rec, u = spr.point(c * height, g * height)
            out.append({"u": u, "e": np.array([rec.e_total, rec.e_ss, rec.e_bend])})
        return out
    net, H = state["net"], state["H"]
    net.set_positions(state["x0"])
    if kind == "eval":
        f = net.forces()
        es, eb = net.energies()
        stress, _ = net.stress()
        return {"f": f, "e": np.array([es, eb]), "stress": stress}
    if kind == "sweep":
        n = case["strain_steps"]
        recs, pos = net.sweep((0.0, 0.0, 0.0), (0.01, 0.01 * n, 0.01), state["prm"], keep_positions=True, graph=True)
        return {"x": pos, "e": np.array([[r.e_stretch, r.e_bend] for r in recs]),
                "f": np.array([[r.rms_force, r.max_force] for r in recs]),
                "stress": np.array([[r.stress_xx, r.stress_yy, r.stress_xy] for r in recs]),
                "n": np.array([[r.steps, r.status] for r in recs])}
    net.affine_displace(net.miny, H, case["shear"] * H, -case.get("compr", 0.0) * H)
    rep = net.relax(state["prm"])
    return {"x": net.positions(), **_report(rep)}


# -------------------------------------------------------------------- work

def _counts(case):
    """Expected nodes, bonds, triples, gel triangles of a case (one network,
    or the whole batch)."""
    if case["kind"] == "batch":
        n = case["count"] * (case["lmin"] ** 2 + case["lmin"] * case["lmax"] + case["lmax"] ** 2) / 3.0
        return n, 3 * 0.65 * n, 3 * 0.65 ** 2 * n, 0.0
    if case.get("net") == "mikado":
        n = 197246 * (case["fibres"] / 15850) ** 2
        return n, 1.92 * n, 1.84 * n, 0.0
    n, p = float(case["nx"] * case["ny"]), case["p"]
    return n, 3 * p * n, 3 * p * p * n, 2.0 * n if case["kind"] == "gel" else 0.0


def work(case):
    """Topology (17 B a bond, 14 B a triple, 20 B a gel triangle with its 48 B
    inverse and area), positions in and out; per FIRE step 36 operations a
    node, 40 a bond, 90 a triple, 120 a gel triangle."""
    n, e, t, g = _counts(case)
    data = 17.0 * e + 14.0 * t + 68.0 * g
    step = 36.0 * n + 40.0 * e + 90.0 * t + 120.0 * g
    if case["kind"] == "eval":
        return {"bytes": data + 32 * n, "flops": step}
    if case["kind"] == "response":
        # 2 x 2 blocks of a node, its neighbours and its second neighbours
        # along lines; two right-hand sides; about 12 iterations a side
        nnz, its = 4.0 * (n + 2 * e + 2 * t), 12.0 * max(case["nx"], case["ny"])
        return {"bytes": data + 12 * nnz + 64 * n, "flops": its * (4 * nnz + 64 * n)}
    if case["kind"] == "sweep":
        k = case["strain_steps"]
        return {"bytes": data + 16 * n * (1 + k), "flops": k * case["steps"] * step}
    return {"bytes": data + 32 * n, "flops": case["steps"] * step}


# ------------------------------------------------------------------- exact

def _seg(v, lens):
    """Sums of the consecutive groups of `lens` entries."""
    return v.sum().reshape(1) if len(lens) == 1 else torch.segment_reduce(v, "sum", lengths=lens)


def _segmax(v, lens):
    return v.max().reshape(1) if len(lens) == 1 else torch.segment_reduce(v, "max", lengths=lens)


class _Model:
    """Energies, forces and FIRE of several networks at once, in 64 bits:
    ks/2 (|r| - l0)^2 a bond, kb/2 (theta - theta0)^2 a triple, and a gel's
    smod A (|F|^2 / det F - 2) / 2 + bmod A (det F - 1 - d)^2 / 2 a triangle."""

    def __init__(self, arrays, kbs, gel=None):
        dev = torch.device("cuda")
        f64 = lambda v: torch.as_tensor(np.ascontiguousarray(v, np.float64), device=dev)  # noqa: E731
        i64 = lambda v: torch.as_tensor(np.ascontiguousarray(v, np.int64), device=dev)    # noqa: E731
        off = np.concatenate([[0], np.cumsum([len(a["points"]) for a in arrays])])
        cat = lambda f: np.concatenate([f(k, a) for k, a in enumerate(arrays)])           # noqa: E731
        self.m, self.n = len(arrays), int(off[-1])
        self.lens, self.elens, self.tlens = (i64([len(a[k]) for a in arrays]) for k in ("points", "edge_l0", "tri_hjk"))
        self.net = i64(cat(lambda k, a: np.full(len(a["points"]), k)))
        self.ij = i64(cat(lambda k, a: a["edge_ij"] + off[k]))
        self.hjk = i64(cat(lambda k, a: a["tri_hjk"].astype(np.int64) + off[k]))
        self.bw = f64(cat(lambda k, a: a["edge_wrap"] * a["offset"]))
        self.tw = f64(cat(lambda k, a: a["tri_wrap"] * a["offset"]))
        self.l0 = f64(cat(lambda k, a: a["edge_l0"]))
        self.k = f64(cat(lambda k, a: np.ones(len(a["edge_l0"])) if a["bond_k"] is None else a["bond_k"]))
        self.kb = f64(cat(lambda k, a: np.full(len(a["tri_hjk"]), kbs[k]) if a["tri_kb"] is None else a["tri_kb"]))
        self.phi0 = f64(cat(lambda k, a: np.zeros(len(a["tri_hjk"])) if a["tri_phi0"] is None else a["tri_phi0"]))
        self.free = f64(cat(lambda k, a: ((a["points"][:, 1] >= a["miny"] + 1e-10) &
                                          (a["points"][:, 1] <= a["maxy"] - 1e-10)).astype(float)))[:, None]
        self.area = f64([a["offset"] * (a["maxy"] - a["miny"]) for a in arrays])
        self.miny, self.H = f64([a["miny"] for a in arrays]), f64([a["maxy"] - a["miny"] for a in arrays])
        self.gel = None
        if gel is not None:
            a = arrays[0]
            v = f64(a["points"])[i64(a["facets"])]  # F, 3, 2
            (x1, y1), (x2, y2), (x3, y3) = ((v[:, r, 0], v[:, r, 1]) for r in range(3))
            det = x1 * (y2 - y3) + x2 * (y3 - y1) + x3 * (y1 - y2)
            inv = torch.stack([y2 - y3, x3 - x2, y3 - y1, x1 - x3, y1 - y2, x2 - x1], 1).reshape(-1, 3, 2) / det[:, None, None]
            self.gel = gel + (i64(a["facets"]), inv, f64(a["areas"]), i64(a["mpairs"]))

    def _bonds(self, x):
        r = x[self.ij[:, 1]] - x[self.ij[:, 0]]
        r[:, 0] += self.bw
        return r, r.square().sum(1).sqrt()

    def _triples(self, x):
        h = x[self.hjk[:, 0]]
        a, b = x[self.hjk[:, 1]] - h, x[self.hjk[:, 2]] - h
        a[:, 0] += self.tw[:, 0]
        b[:, 0] += self.tw[:, 1]
        th = torch.atan2(-(a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]), -(a * b).sum(1)) - self.phi0
        return a, b, th

    def _gel(self, x):
        smod, bmod, dil, el, inv, area, pairs = self.gel
        F = torch.einsum("fvi,fvj->fij", x[el], inv)
        det = F[:, 0, 0] * F[:, 1, 1] - F[:, 0, 1] * F[:, 1, 0]
        sq = F.square().sum((1, 2))
        return F, det, sq

    def forces(self, x, virial=False):
        r, l = self._bonds(x)
        fb = (self.k * (1 - self.l0 / l))[:, None] * r
        a, b, th = self._triples(x)
        g = self.kb * th
        fj = torch.stack([-a[:, 1], a[:, 0]], 1) * (g / a.square().sum(1))[:, None]
        fk = torch.stack([b[:, 1], -b[:, 0]], 1) * (g / b.square().sum(1))[:, None]
        if virial:
            w = torch.stack([_seg((r[:, p] * fb[:, q]).contiguous(), self.elens) -
                             _seg((a[:, p] * fj[:, q] + b[:, p] * fk[:, q]).contiguous(), self.tlens)
                             for p, q in ((0, 0), (1, 1), (1, 0))], 1)
            return w / self.area[:, None]
        f = torch.zeros_like(x)
        f.index_add_(0, self.ij[:, 0], fb)
        f.index_add_(0, self.ij[:, 1], -fb)
        f.index_add_(0, self.hjk[:, 1], fj)
        f.index_add_(0, self.hjk[:, 2], fk)
        f.index_add_(0, self.hjk[:, 0], -(fj + fk))
        if self.gel:
            smod, bmod, dil, el, inv, area, pairs = self.gel
            F, det, sq = self._gel(x)
            c1 = -smod * area / det
            c2 = area * (bmod * (dil + 1 - det) + smod * sq / (2 * det * det))
            cof = torch.stack([torch.stack([F[:, 1, 1], -F[:, 1, 0]], 1), torch.stack([-F[:, 0, 1], F[:, 0, 0]], 1)], 1)
            du = F * c1[:, None, None] + cof * c2[:, None, None]
            f.index_add_(0, el.reshape(-1), torch.einsum("fij,fvj->fvi", du, inv).reshape(-1, 2))
        f = f * self.free
        if self.gel and len(pairs):
            s = f[pairs[:, 0]] + f[pairs[:, 1]]
            f[pairs[:, 0]] = s
            f[pairs[:, 1]] = s
        return f

    def energies(self, x):
        _, l = self._bonds(x)
        _, _, th = self._triples(x)
        es = _seg(0.5 * self.k * (l - self.l0).square(), self.elens)
        eb = _seg(0.5 * self.kb * th.square(), self.tlens)
        eg = torch.zeros_like(es)
        if self.gel:
            smod, bmod, dil, _, _, area, _ = self.gel
            _, det, sq = self._gel(x)
            eg = (smod * area * (sq / det - 2) / 2 + bmod * area * (det - 1 - dil).square() / 2).abs().sum().reshape(1)
        return es, eb, eg

    def affine(self, x, dx, dy):
        """x += dx (y - miny) / H, y += dy (y - miny) / H, one pair a network."""
        s = ((x[:, 1] - self.miny[self.net]) / self.H[self.net])
        return torch.stack([x[:, 0] + dx[self.net] * s, x[:, 1] + dy[self.net] * s], 1)

    def fire(self, x, steps, dt_max):
        """`steps` iterations from v = 0 (Bitzek et al. 2006, velocity Verlet);
        returns positions and the last |F|^2 and max |F|^2."""
        z = lambda v: torch.full((self.m,), v, dtype=torch.float64, device=x.device)  # noqa: E731
        dt, al, since = z(dt_max), z(0.1), z(0.0)
        na, ca, keep = z(0.0), z(0.0), z(1.0)
        v, f = torch.zeros_like(x), self.forces(x)
        at = lambda s: s[self.net][:, None] if self.m > 1 else s  # noqa: E731
        for _ in range(steps):
            v = (v + at(na) * v + at(ca) * f) * at(keep)
            x = x + at(dt) * v + at(0.5 * dt * dt) * f
            v = v + at(0.5 * dt) * f
            f = self.forces(x)
            v = v + at(0.5 * dt) * f
            P, V2, F2 = _seg((v * f).sum(1), self.lens), _seg(v.square().sum(1), self.lens), _seg(f.square().sum(1), self.lens)
            ca, na, up = al * V2.sqrt() / F2.sqrt(), -al, P > 0
            since = torch.where(up, since + 1, 0.0)
            grow = up & (since > 5)
            dt = torch.where(up, torch.where(grow, torch.clamp(dt * 1.1, max=dt_max), dt), dt * 0.5)
            al = torch.where(up, torch.where(grow, al * 0.99, al), 0.1)
            keep = up.double()
        return x, F2, _segmax(f.square().sum(1), self.lens)


def _relaxed(m, x, steps, dt_max):
    x, F2, M2 = m.fire(x, steps, dt_max)
    rms = F2.sqrt() / (2 * m.lens.double()).sqrt()
    return x, m.energies(x), torch.stack([rms, M2.sqrt()], 1), m.forces(x, virial=True)


def _response(case, a):
    """K u = -K bc on the free nodes by conjugate gradients to the last bits."""
    dev, n = torch.device("cuda"), len(a["points"])
    x, l0 = a["points"], a["edge_l0"]
    i, j = a["edge_ij"].astype(np.int64).T
    d = x[j] - x[i]
    d[:, 0] += a["edge_wrap"] * a["offset"]
    l = np.sqrt((d ** 2).sum(1))
    h, tj, tk = a["tri_hjk"].astype(np.int64).T
    e = x[tj] - x[h]
    e[:, 0] += a["tri_wrap"][:, 0] * a["offset"]
    ln = np.sqrt((e ** 2).sum(1))
    zero = np.zeros(len(l))
    # every term is w w^T / its scale: stretch along the bond, shear per
    # component, bending across the line
    s1 = np.sqrt(1.0 / l) / l
    m1, m2 = (np.sqrt(case["mu"] * (1 - (d[:, c] / l0) ** 2)) for c in (0, 1))
    sb = np.sqrt(case["kb"]) / ln
    node = np.concatenate([np.stack([i, j], 1)] * 3)
    coef = np.concatenate([np.stack([s1 * d[:, 0], s1 * d[:, 1]], 1), np.stack([m1, zero], 1), np.stack([zero, m2], 1)])
    rows = np.concatenate([np.repeat(np.arange(len(node)), 4), np.repeat(len(node) + np.arange(len(h)), 6)])
    cols = np.concatenate([np.stack([2 * node[:, 0], 2 * node[:, 0] + 1, 2 * node[:, 1], 2 * node[:, 1] + 1], 1).reshape(-1),
                           np.stack([2 * h, 2 * h + 1, 2 * tj, 2 * tj + 1, 2 * tk, 2 * tk + 1], 1).reshape(-1)])
    b = sb[:, None] * np.stack([e[:, 1], -e[:, 0]], 1)
    vals = np.concatenate([np.concatenate([-coef, coef], 1).reshape(-1), np.concatenate([-2 * b, b, b], 1).reshape(-1)])
    t = lambda v: torch.as_tensor(v, device=dev)  # noqa: E731
    B = torch.sparse_coo_tensor(torch.stack([t(rows), t(cols)]), t(vals), (len(node) + len(h), 2 * n)).coalesce()
    Bt = B.t().coalesce().to_sparse_csr()
    B = B.to_sparse_csr()
    y = t(x[:, 1])
    lo, hi = y.min(), y.max()
    H = hi - lo
    free = ((y >= lo + 1e-10) & (y <= hi - 1e-10)).double().repeat_interleave(2)[:, None]
    K = lambda u: Bt @ (B @ u)  # noqa: E731
    diag = torch.zeros(2 * n, dtype=torch.float64, device=dev).index_add_(0, t(cols), t(vals) ** 2)[:, None]
    M = torch.where((diag > 0) & (free > 0), 1 / diag.clamp(min=1e-300), 0.0)
    bc = torch.zeros(2 * n, 2, dtype=torch.float64, device=dev)  # unit compression, unit shear
    bc[1::2, 0] = (lo - y) / H
    bc[0::2, 1] = (y - lo) / H
    r = -K(bc) * free
    u, z = torch.zeros_like(r), M * r
    p, rz, b2 = z.clone(), (r * z).sum(0), r.square().sum(0)
    for it in range(20000):
        q = K(p) * free
        al = rz / (p * q).sum(0).clamp(min=1e-300)
        u, r = u + al * p, r - al * q
        if it % 50 == 49 and bool((r.square().sum(0) <= 1e-29 * b2).all()):
            break
        z = M * r
        new = (r * z).sum(0)
        p, rz = z + (new / rz.clamp(min=1e-300)) * p, new
    out, height = [], float(H)
    for c, g in ((0.01, 0.0), (0.0, 0.01), (0.01, 0.02)):
        w = torch.tensor([c * height, g * height], dtype=torch.float64, device=dev)
        U = ((bc + u) @ w).reshape(n, 2)
        du = U[t(j)] - U[t(i)]
        de = (du * t(d)).sum(1) / t(l0)
        ess = (0.5 * de ** 2 + 0.5 * case["mu"] * (du.square().sum(1) - de ** 2)).sum()
        db = U[t(tj)] + U[t(tk)] - 2 * U[t(h)]
        cr = db[:, 0] * t(e[:, 1]) - db[:, 1] * t(e[:, 0])
        ebn = (0.5 * case["kb"] * cr ** 2 / t(ln ** 2)).sum()
        out.append({"u": U.cpu().numpy(), "e": torch.stack([ess + ebn, ess, ebn]).cpu().numpy()})
    return out


def exact(case, seed):
    """run()'s outputs from the definitions, in 64 bits, with torch."""
    kind = case["kind"]
    host = lambda v: v.cpu().numpy()  # noqa: E731
    if kind == "batch":
        ms, hosts = _batch_hosts(case, seed)
        arrays = [h.arrays() for h in hosts]
        m = _Model(arrays, [q["kb"] for q in ms])
        x = torch.as_tensor(np.concatenate([a["points"] for a in arrays]), device="cuda")
        gam = torch.as_tensor(np.array([q["gamma"] for q in ms]), device="cuda") * m.H
        x, e, f, s = _relaxed(m, m.affine(x, gam, torch.zeros_like(gam)), case["steps"], 0.1)
        return {"x": host(x), "e": host(torch.stack(e[:2], 1)), "f": host(f), "stress": host(s), "n": None}
    h = _host(case, seed)
    a = h.arrays()
    if kind == "response":
        return _response(case, a)
    m = _Model([a], [case["kb"]], GEL if kind == "gel" else None)
    if kind == "eval":
        x = torch.as_tensor(a["points"] + np.random.default_rng(seed).normal(scale=0.03, size=a["points"].shape), device="cuda")
        es, eb, _ = m.energies(x)
        return {"f": host(m.forces(x)), "e": host(torch.cat([es, eb])), "stress": host(m.forces(x, virial=True)[0])}
    x, dt = torch.as_tensor(_start(case, a["points"], seed), device="cuda"), _dt_max(case, h)
    if kind == "sweep":
        out = {"x": [], "e": [], "f": [], "stress": []}
        for _ in range(case["strain_steps"]):
            x, e, f, s = _relaxed(m, m.affine(x, 0.01 * m.H, 0 * m.H), case["steps"], dt)
            for key, v in (("x", x), ("e", torch.cat(e[:2])), ("f", f[0]), ("stress", s[0])):
                out[key].append(host(v))
        return {**{key: np.stack(v) for key, v in out.items()}, "n": None}
    x = m.affine(x, case["shear"] * m.H, -case.get("compr", 0.0) * m.H)
    x, e, f, s = _relaxed(m, x, case["steps"], dt)
    return {"x": host(x), "e": host(torch.cat(e)), "f": host(f[0]), "stress": host(s[0]), "n": None}
