"""What is measured: the calls that a BROMOC program makes on this framework.

Each case is one pass of such a program through the public entry points, over
the kinds of system that the repository's own workloads have: single ENERGY
evaluations, Brownian-dynamics (BD) runs, GCMC/BD cycles, Metropolis moves,
the ssDNA system, the MMIJ reaction field, replica batches and the adjoint of
a BD segment.  `kind` says which; the other keys are its sizes and options.

An engine made with FP32 precision computes forces, energies and moves in 32
bits and hands them over in the ABI's 64-bit arrays; a pass returns them as
the 32-bit numbers that they are (the width of the .btr frames that programs
save).  FP64 engines' results are returned as they come.

`exact` restates the physics in 64 bits with plain torch and numpy.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from bromoc_gb300 import _lib, abi, synth
from bromoc_gb300.adjoint import Adjoint, RdfLoss, knot_gradient, knot_jacobians
from bromoc_gb300.batch import Batch
from bromoc_gb300.deck import CELEC

SMALL = dict(nclx=28, ncly=28, nclz=40, radius=6.0, slab=10.0)
FULL = dict(nclx=120, ncly=120, nclz=180, radius=10.0, slab=30.0)


def listed():
    return [
        # one ENERGY of a handful of ions around a small pore with a membrane:
        # the smallest call (a test particle system, a check of a deck)
        dict(name="energy-80-fp64", kind="energy", n=80, fp32=False, maps="small",
             spline=False, membrane=True),
        # ENERGY and forces of a whole nanopore in the exact mode, with the
        # B-spline form of the repulsion map: re-scoring saved frames
        dict(name="energy-2000-fp64", kind="energy", n=2000, fp32=False, maps="full",
             spline=True, membrane=False),
        # the same of the largest pore that the pair tiles take, in FP32
        dict(name="energy-8000-fp32", kind="energy", n=8000, fp32=True, maps="full",
             spline=False, membrane=False),
        # bulk 1 M KCl in a 60 A cube, hard walls, FP64: a run of BD steps
        dict(name="bulk-260-fp64", kind="bulk", n=260, fp32=False, rcut=0.0, steps=50),
        # a large bulk system, periodic with a 20 A cutoff (the cell list)
        dict(name="periodic-20000-fp32", kind="bulk", n=20000, fp32=True, rcut=20.0, steps=5),
        # the nanopore's production loop: GRAND(4) + 10 BD steps + COUNT
        dict(name="cycle-2000-fp32", kind="cycle", n=2000, fp32=True, attempts=4, nbd=10,
             cycles=4, mmij=False),
        # GCMC/BD with the MMIJ reaction field (RECTBOX) in the exact mode
        dict(name="mmij-500-fp64", kind="cycle", n=500, fp32=False, attempts=4, nbd=5,
             cycles=1, mmij=True),
        # Metropolis moves of the nanopore's ions
        dict(name="metropolis-2000", kind="metropolis", n=2000, fp32=True, moves=20),
        # ssDNA, 40 nt x 3 free sites with bonded terms, in ~5000 ions
        dict(name="ssdna-5000-fp32", kind="ssdna", n=5000, fp32=True, nnuc=40, steps=10),
        # 256 uneven replicas of bulk KCl sharing the pore's maps
        dict(name="batch-256", kind="batch", nrep=256, nmin=200, nmax=8000, steps=4,
             attempts=0),
        # many small replicas with GCMC: GRAND + BD + COUNT on every replica
        dict(name="batch-gcmc-48", kind="batch", nrep=48, nmin=40, nmax=130, steps=10,
             attempts=4),
        # a fitting step's gradient: BD segment and its adjoint, 4096 ions
        dict(name="adjoint-4096-fp32", kind="adjoint", n=4096, fp32=True, steps=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["energy", "bulk", "cycle", "metropolis", "ssdna", "batch", "gcmc",
                       "adjoint"])
    if kind == "energy":
        fp32 = rng.random() < 0.5
        n = _log(rng, 60, 8000 if fp32 else 2500)
        return dict(kind=kind, n=n, fp32=fp32, maps="small" if n < 120 else "full",
                    spline=rng.random() < 0.5, membrane=rng.random() < 0.3)
    if kind == "bulk":
        fp32 = rng.random() < 0.5
        n = _log(rng, 300, 20000) if fp32 else _log(rng, 100, 1000)
        return dict(kind=kind, n=n, fp32=fp32, rcut=20.0 if rng.random() < 0.6 else 0.0,
                    steps=rng.randint(3, 8) if fp32 else rng.randint(10, 50))
    if kind == "cycle":
        mmij = rng.random() < 0.25
        fp32 = rng.random() < 0.75 and not mmij
        return dict(kind=kind, n=_log(rng, 300, 8000) if fp32 else _log(rng, 200, 1000),
                    fp32=fp32, attempts=rng.randint(1, 12), nbd=rng.randint(3, 10),
                    cycles=rng.randint(1, 4) if fp32 else 1, mmij=mmij)
    if kind == "metropolis":
        return dict(kind=kind, n=_log(rng, 150, 6000), fp32=rng.random() < 0.5,
                    moves=_log(rng, 4, 60))
    if kind == "ssdna":
        return dict(kind=kind, n=_log(rng, 500, 5000), fp32=True, nnuc=rng.randint(5, 40),
                    steps=rng.randint(3, 10))
    if kind == "batch":
        nmax = _log(rng, 400, 8000)
        return dict(kind="batch", nrep=_log(rng, 8, 200), nmin=max(60, nmax // 20), nmax=nmax,
                    steps=rng.randint(2, 4), attempts=0)
    if kind == "gcmc":
        return dict(kind="batch", nrep=_log(rng, 4, 96), nmin=40, nmax=rng.randint(60, 130),
                    steps=rng.randint(3, 10), attempts=rng.randint(1, 8))
    fp32 = rng.random() < 0.7
    return dict(kind=kind, n=_log(rng, 200, 4096) if fp32 else _log(rng, 100, 700),
                fp32=fp32, steps=rng.randint(10, 50))


# ---- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _maps(size):
    """The pore's maps: a file that a program reads once, the same for all."""
    g = SMALL if size == "small" else FULL
    return synth.pore_maps(seed=11, **g)


def _scatter(rng, n, half, ok=None, dmin=3.0):
    """n positions in the box of half lengths `half`, at least dmin apart: sites
    of a lattice in random order, each moved within its cell."""
    size = 2.0 * np.asarray(half, float)
    a = (np.prod(size) / n) ** (1.0 / 3.0)
    while True:
        m = np.maximum(1, np.floor(size / a).astype(int))
        cell = size / m
        site = rng.permutation(int(np.prod(m)))
        p = np.stack(np.unravel_index(site, m), 1) + 0.5
        p = p * cell - 0.5 * size + (cell - dmin) * (rng.random((len(site), 3)) - 0.5)
        if ok is not None:
            p = p[ok(p)]
        if len(p) >= n:
            return p[:n]
        a *= 0.97
        if a < dmin:
            raise ValueError("too many ions for the box")


def _place(spec, p, types):
    spec.x, spec.y, spec.z = (p[:, k].copy() for k in range(3))
    spec.typei = np.asarray(types, np.int32)


def _half(n):
    """K+ and Cl- by turns, as many of each as n allows."""
    return 1 + np.arange(n) % 2


def _precision(case):
    return abi.FP32 if case["fp32"] else abi.FP64


def _pore(case, seed, size, spline=False, membrane=False, rfpar=True):
    """n K+/Cl- around the pore of the given maps."""
    g = SMALL if size == "small" else FULL
    s = synth.pore(seed=1, nions=2, maps=_maps(size), radius=g["radius"], slab=g["slab"],
                   precision=_precision(case), buffers=False, membrane=membrane,
                   trilinear=not spline, rfpar=rfpar)

    def free(p):
        return ~((np.abs(p[:, 2]) <= 0.5 * g["slab"] + 1.0)
                 & (np.hypot(p[:, 0], p[:, 1]) >= g["radius"] - 1.0))

    half = [0.5 * s.lx - 0.5, 0.5 * s.ly - 0.5, 0.5 * s.lz - 0.5]
    _place(s, _scatter(np.random.default_rng(seed), case["n"], half, free), _half(case["n"]))
    return s


def _buffers(s, depth):
    """GCMC buffers of both ions at both ends, near the number that they hold."""
    zb = 0.5 * s.lz
    for name in ("K", "Cl"):
        for lo, hi in ((-zb, -zb + depth), (zb - depth, zb)):
            s.buffers.append(dict(ion=name, conc=1.0, lzmin=lo, lzmax=hi, mu=-0.5))
    s.count()
    for b in s.buffers:
        b["aver"] = max(1.0, float(b["nat"]))


def _bulk(case, seed, srpmf=True):
    n = case["n"]
    L = (n / (2 * 6.02214e-4)) ** (1.0 / 3.0)
    rcut = case.get("rcut", 0.0) or None
    if rcut is not None:
        L = max(L, 2.05 * rcut)
    s = synth.bulk_kcl(seed=1, n_per=1, L=L, srpmf=srpmf, precision=_precision(case),
                       periodic_rcut=rcut)
    h = 0.5 * L - (1.5 if rcut else 0.5)
    _place(s, _scatter(np.random.default_rng(seed), n, [h] * 3), _half(n))
    return s


def _spec(case, seed):
    """The deck of a case, and for a batch its replicas' decks."""
    kind = case["kind"]
    if kind == "energy":
        return _pore(case, seed, case["maps"], case["spline"], case["membrane"])
    if kind == "bulk":
        return _bulk(case, seed)
    if kind == "cycle":
        s = _pore(case, seed, "full", rfpar=not case["mmij"])
        if case["mmij"]:
            s.mmij = synth.mmij_rect(seed=12, half=(40.0, 40.0, 70.0))
        _buffers(s, 20.0)
        return s
    if kind == "metropolis":
        return _pore(case, seed, "full")
    if kind == "ssdna":
        s = synth.ssdna(seed=seed % 9973, nions=2, nnuc=case["nnuc"], maps=_maps("full"),
                        precision=_precision(case), bonded=True, free=True)
        ns = s.nsites
        sites = np.stack([s.x, s.y, s.z], 1)[:ns]
        # off the native structure, so that every bonded term carries force
        rng = np.random.default_rng(seed)
        sites = sites + rng.normal(0.0, 0.15, sites.shape)
        ions = _pore(dict(case, n=case["n"] + 2 * ns), seed, "full")
        p = np.stack([ions.x, ions.y, ions.z], 1)
        p = p[((p[:, None, :] - sites[None]) ** 2).sum(-1).min(1) > 9.0][:case["n"]]
        _place(s, np.concatenate([sites, p]),
               np.concatenate([np.zeros(ns), _half(len(p)) + s.ndna]))
        return s
    if kind == "adjoint":
        s = _bulk(case, seed, srpmf=False)
        rng = np.random.default_rng(7)
        s.efpot_res = 0.05
        for key, (sg, ep) in ((("K", "K"), (3.1, 0.09)), (("K", "Cl"), (3.6, 0.11)),
                              (("Cl", "Cl"), (4.0, 0.15))):
            s.efpot_knots[key] = synth.efpot_knots(rng, sg, ep, r0=1.05, r1=16.0, res=0.05)
        return s
    raise ValueError(kind)


def _replicas(case, seed):
    """The prototype's deck and one deck a replica."""
    rng = np.random.default_rng(seed)
    # the same sizes for every seed: the seed gives the coordinates
    counts = np.random.default_rng(4).integers(case["nmin"], case["nmax"] + 1, case["nrep"])
    one = dict(n=2, fp32=True)
    if case["attempts"]:
        out = []
        for r, n in enumerate(counts):
            s = _pore(dict(one, n=int(n)), seed + 7919 * (r + 1), "small")
            _buffers(s, 10.0)
            out.append(s)
        return out[0], out
    proto = _pore(one, seed, "full")
    out = []
    for n in counts:
        L = (n / (2 * 6.02214e-4)) ** (1.0 / 3.0)
        s = synth.bulk_kcl(seed=1, n_per=1, L=L, srpmf=True, precision=abi.FP32)
        s.phix, s.phiv, s.rfpar = proto.phix, proto.phiv, proto.rfpar
        _place(s, _scatter(rng, int(n), [0.5 * L - 0.5] * 3, synth.outside_pore_slab),
               _half(int(n)))
        out.append(s)
    return proto, out


ADJ_BINS, ADJ_R0, ADJ_DR, ADJ_SIGMA = 150, 0.05, 0.1, 0.1


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, seed=int(seed), done=0)
    if kind == "batch":
        proto, reps = _replicas(case, seed)
        eng = _lib.create(max(400, 2 * len(proto.x)), abi.FP32)
        proto.push(eng)
        caps = [len(s.x) + (64 + len(s.x) if case["attempts"] else 0) for s in reps]
        b = Batch(eng, caps)
        b.set_systems([s.system_struct() for s in reps])
        for r, s in enumerate(reps):
            b.set_particles(r, s.x, s.y, s.z, s.typei)
            if case["attempts"]:
                b.set_buffers(r, s.buffer_params(), s.ibuffer)
        st.update(eng=eng, batch=b, caps=caps,
                  seeds=np.arange(len(reps), dtype=np.uint64) + np.uint64(seed % 100003))
        return st
    s = _spec(case, seed)
    n = len(s.x)
    # room for the ions that GCMC may add
    eng = _lib.create(2 * n + 64 if kind == "cycle" else n + 16, _precision(case))
    s.push(eng)
    st.update(eng=eng)
    if kind == "energy":
        st.update(xyz=(s.x, s.y, s.z), typei=s.typei)
    if kind == "adjoint":
        adj = Adjoint(eng, n, _precision(case))
        adj.set_particles(s.x, s.y, s.z, s.typei)
        rb = ADJ_R0 + ADJ_DR * np.arange(ADJ_BINS)
        st.update(adj=adj, loss=RdfLoss(2, [(n + 1) // 2, n // 2], s.lx ** 3, case["steps"], rb,
                                        np.ones((3, ADJ_BINS))),
                  tables=s.pair_tables(), jac=knot_jacobians(s, eng.efpot_from_knots))
    return st


# ---- a pass -----------------------------------------------------------------

def _kept(case, a):
    """Results of an FP32 engine as 32-bit numbers."""
    return np.asarray(a, np.float32) if case.get("fp32", True) else np.asarray(a)


def _whole(arrays, cap):
    """Arrays over the live particles in arrays of the program's capacity."""
    out = [np.zeros(cap, a.dtype) for a in arrays]
    for o, a in zip(out, arrays):
        o[:len(a)] = a
    return out


def run(st):
    case, eng, seed, k = st["case"], st["eng"], st["seed"], st["done"]
    kind = case["kind"]
    st["done"] += 1
    if kind == "energy":
        # another frame's coordinates, then its energies and forces
        eng.set_particles(*st["xyz"], st["typei"])
        e, f, warn = eng.energy()
        return _kept(case, list(e.values())), _kept(case, f), warn
    if kind in ("bulk", "ssdna"):
        eng.bd_steps(case["steps"], seed, k * case["steps"], energies=False)
        return _kept(case, eng.get_particles()[:3])
    if kind == "cycle":
        dener = []
        for c in range(k * case["cycles"], (k + 1) * case["cycles"]):
            d = eng.grand(case["attempts"], seed, c + 1, dener=c + 1 == (k + 1) * case["cycles"])
            eng.bd_steps(case["nbd"], seed, c * case["nbd"], energies=False)
            eng.count()
        dener.append(d)
        x, y, z, t, ib = _whole(eng.get_particles(), eng.capacity)
        nat, nin, nrm, _ = eng.get_buffers()
        return _kept(case, dener), _kept(case, [x, y, z]), t, ib, nat, nin, nrm
    if kind == "metropolis":
        na, d = eng.metropolis(case["moves"], 1.0, seed, k + 1)
        return na, _kept(case, [d]), _kept(case, eng.get_particles()[:3])
    if kind == "batch":
        b, steps, seeds = st["batch"], case["steps"], st["seeds"]
        whole = []
        if case["attempts"]:
            whole.append(_kept(case, b.grand(case["attempts"], seeds, k + 1)))
        b.bd_steps(steps, seeds, k * steps)
        if case["attempts"]:
            b.count()
        frames = [b.get_particles(r, n) for r, n in enumerate(st["caps"])]
        if case["attempts"]:
            frames = [_whole(f, n) for f, n in zip(frames, st["caps"])]
        whole.append(np.concatenate([_kept(case, f) for f in frames], 1))
        if case["attempts"]:
            got = [b.get_buffers(r, 4, n) for r, n in enumerate(st["caps"])]
            got = [g[:3] + tuple(_whole(g[3:], n)) for g, n in zip(got, st["caps"])]
            whole += [np.concatenate([g[m] for g in got]) for m in range(5)]
        return whole
    adj, pt = st["adj"], st["tables"]
    hist = adj.forward(case["steps"], 25, seed, k * case["steps"], ADJ_BINS, ADJ_R0, ADJ_DR,
                       ADJ_SIGMA, 3)
    _, dl = st["loss"].loss_grad(hist)
    g_ep, g_sc = adj.backward(dl, int(pt["cnt"]), int(pt["ntc"]))
    grads = knot_gradient(st["jac"], g_ep, g_sc)
    return _kept(case, hist), _kept(case, list(grads.values())), _kept(case, adj.get_particles())


def work(case):
    """Bytes: coordinates in and out, forces, and the map nodes gathered.
    Operations: 38 a pair for the pair law, 32 for the reaction-field term, 33
    and a table entry for a tabulated law, ~150 an ion for maps and move."""
    kind = case["kind"]

    def pass_of(n, rf, law=38, rcut=0.0):
        pairs = 0.5 * n * (n - 1)
        if rcut:
            pairs = min(pairs, 0.5 * n * 4.19 * rcut ** 3 * 2 * 6.02214e-4)
        return dict(bytes=n * (72.0 + 104.0 * rf), flops=pairs * (law + 32 * rf) + 150.0 * n)

    def times(w, k):
        return dict(bytes=w["bytes"] * k, flops=w["flops"] * k)

    if kind == "energy":
        return pass_of(case["n"], 1)
    if kind == "bulk":
        return times(pass_of(case["n"], 0, rcut=case["rcut"]), case["steps"])
    if kind == "cycle":
        w = times(pass_of(case["n"], 0 if case["mmij"] else 1), case["nbd"] * case["cycles"])
        w["flops"] += 70.0 * case["n"] * case["attempts"] * case["cycles"]
        return w
    if kind == "metropolis":
        return dict(bytes=72.0 * case["n"], flops=140.0 * case["n"] * case["moves"])
    if kind == "ssdna":
        w = times(pass_of(case["n"], 1), case["steps"])
        w["flops"] += 33.0 * case["n"] * 3 * case["nnuc"] * case["steps"]
        return w
    if kind == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n, n2 = 0.5 * (lo + hi), (hi ** 2 + hi * lo + lo ** 2) / 3.0
        w = pass_of(math.sqrt(n2), 1)
        return dict(bytes=case["nrep"] * n * 176.0 * case["steps"],
                    flops=case["nrep"] * w["flops"] * case["steps"])
    return times(pass_of(case["n"], 0, law=33 * 4), case["steps"])


# ---- the same in 64 bits ----------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=_device())


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 on arrays of counters: four arrays of 32-bit words."""
    c = [np.asarray(v, np.uint64) + np.zeros(np.shape(c0), np.uint64) for v in (c0, c1, c2, c3)]
    k0, k1 = np.uint64(seed & 0xffffffff), np.uint64(seed >> 32)
    low = np.uint64(0xffffffff)
    for _ in range(10):
        a = np.uint64(0xD2511F53) * c[0]
        b = np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & low, (a >> np.uint64(32)) ^ c[3] ^ k1, a & low]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & low, (k1 + np.uint64(0xBB67AE85)) & low
    return [v.astype(np.float64) * 2.0 ** -32 for v in c]


def _normals(seed, step, n):
    """The noise of a BD step: [n, 3] normal deviates by slot."""
    slot = np.arange(n)
    out = np.zeros((n, 3))
    for block in (0, 1):
        u = _philox(slot, block, step & 0xffffffff, (step >> 32 & 0xffffff) | 1 << 24, seed)
        for m in range(2):
            if 2 * block + m < 3:
                out[:, 2 * block + m] = (np.cos(2 * math.pi * u[2 * m])
                                         * np.sqrt(-2 * np.log(1 - u[2 * m + 1])))
    return out


def _uniforms(seed, cycle, attempt, tag):
    """The uniform draws of a GCMC attempt (tag 2) or a Metropolis move (3)."""
    k = 0
    while True:
        yield from (float(u) for u in _philox(attempt, k, cycle & 0xffffffff,
                                              (cycle >> 32 & 0xffffff) | tag << 24, seed))
        k += 1


def _table(r, u, fct):
    """An effective-potential table's pieces [n, 3] and core and tail constants
    from its knots: averaged parabolas through three knots, their slopes joined
    linearly and integrated, then the end value put right over the pieces."""
    n, k = len(r), fct
    sc = np.zeros(3)
    sc[2] = (r[-1] * u[-1] - k) * r[-1] ** 5
    d2 = -k / r[-1] ** 2 - 6.0 * sc[2] / r[-1] ** 7
    dd2 = 2.0 * k / r[-1] ** 3 + 42.0 * sc[2] / r[-1] ** 8
    a, b = r[0] ** 12, r[1] ** 12
    sc[0] = (u[1] - u[0]) * b * a / (a - b)
    sc[1] = (u[0] * a - u[1] * b) / (a - b)
    d1 = -12.0 * sc[0] / r[0] ** 13
    slope = np.diff(u) / np.diff(r)
    p3, p2 = np.zeros(n), np.zeros(n)
    p3[0] = (slope[0] - d1) / (r[1] - r[0])
    p2[0] = d1 - 2.0 * p3[0] * r[0]
    p3[1:-1] = np.diff(slope) / (r[2:] - r[:-2])
    p2[1:-1] = slope[1:] - p3[1:-1] * (r[2:] + r[1:-1])
    p3[-1] = (d2 - slope[-1]) / (r[-1] - r[-2])
    p2[-1] = d2 - 2.0 * p3[-1] * r[-1]
    # a piece is the mean of its two ends' parabolas, but the first
    for p in (p2, p3):
        p[1:-1] = 0.5 * (p[1:-1] + p[2:])
    # slopes at the knots
    s = np.empty(n)
    s[0] = p2[0] + 2 * p3[0] * r[0]
    s[1:-1] = 0.5 * (p2[1:-1] + 2 * p3[1:-1] * r[1:-1] + p2[:-2] + 2 * p3[:-2] * r[1:-1])
    s[-1] = p2[-1] + 2 * p3[-1] * r[-1]
    # linear slopes between the knots, integrated from the first value
    g1 = np.empty(n)
    g1[:-1] = np.diff(s) / np.diff(r)
    g1[-1] = dd2
    g0 = s - g1 * r
    p3, p2, p1 = 0.5 * g1, g0.copy(), np.empty(n)
    p1[0] = u[0] - r[0] * (p2[0] + p3[0] * r[0])
    p1[1:] = p1[0] + np.cumsum(r[1:] * (p2[:-1] - p2[1:] + r[1:] * (p3[:-1] - p3[1:])))
    # the end value, spread with the table's nominal spacing
    end = p1[-1] + r[-1] * (p2[-1] + r[-1] * p3[-1])
    b = 2.0 * (u[-1] - end) / (r[-1] - r[0])
    h = (r[1] - r[0]) / (n - 1)
    p1 += -0.5 * b * r[0]
    p2 += b
    at = r + h * np.arange(n)
    at[-1] = r[-1]
    p3 += -0.5 * b / at
    return np.stack([p1, p2, p3], 1), sc


class _Map:
    """Gathers from one grid map, differentiable in the positions."""

    def __init__(self, grid, data):
        self.n = torch.tensor([grid["nclx"], grid["ncly"], grid["nclz"]], device=_device())
        self.d = grid["dcel"]
        self.half = 0.5 * (self.n - 1).double() * self.d
        self.c = _t([grid["xbcen"], grid["ybcen"], grid["zbcen"]])
        self.data = _t(np.asarray(data, np.float64))

    def inside(self, p, margin=0.0):
        return ((p - self.c).abs() <= self.half - margin).all(1)

    def _nodes(self, base, width):
        o = torch.arange(width, device=base.device)
        i, j, k = (base[:, a, None] + o for a in range(3))
        at = ((i[:, :, None, None] * self.n[1] + j[:, None, :, None]) * self.n[2]
              + k[:, None, None, :])
        return self.data[at]

    @staticmethod
    def _sum(w, v):
        return torch.einsum("ni,nj,nk,nijk->n", w[:, 0], w[:, 1], w[:, 2], v)

    def linear(self, p):
        """Value and sum of the eight nodes."""
        u = (p - self.c + self.half) / self.d
        base = torch.minimum(u.detach().long(), self.n - 2)
        f = u - base
        # the model takes no slope along an axis within 1e-3 of a node
        f = torch.where((f > 1e-3) & (f < 1 - 1e-3), f, f.detach())
        v = self._nodes(base, 2)
        return self._sum(torch.stack([1 - f, f], 2), v), v.sum((1, 2, 3))

    def spline(self, p):
        """The quadratic B-spline value over 27 nodes and the nodes' sum."""
        u = (p - self.c + self.half) / self.d
        base = (u.detach() + 0.5).floor().long()
        base = torch.minimum(base.clamp_min(1), self.n - 2) - 1
        x = 1.5 - (u[:, :, None] - (base[:, :, None] + torch.arange(3, device=u.device)))

        def hat(y):
            return (1 - (y - 1).abs()).clamp_min(0)

        w = torch.where((x >= 0) & (x <= 3), 0.5 * x * hat(x) + 0.5 * (3 - x) * hat(x - 1), 0 * x)
        v = self._nodes(base, 3)
        used = (w != 0).double()
        return self._sum(w, v), self._sum(used, v)


class _System:
    """A deck in 64 bits: ENERGY, INTERACT and the moves."""

    def __init__(self, s):
        self.s = s
        self.ns = s.nsites
        nd, ni = s.ndna, s.nion
        names = s.type_names()
        q = [s.cgnuc if a == "P" else 0.0 for a in names[:nd]] + list(s.ion_cg)
        T = nd + ni
        self.nt = T
        law = {k: np.zeros((T, T)) for k in ("fct", "eps4", "sg2", "c0", "c1", "c2", "c3", "c4")}
        self.tab = np.full((T, T), -1)
        tables = []
        for i in range(T):
            for j in range(T):
                law["fct"][i, j] = CELEC * q[i] * q[j] / s.cdie
                law["eps4"][i, j] = 4 * math.sqrt(s.lj_eps[names[i]] * s.lj_eps[names[j]])
                law["sg2"][i, j] = (0.5 * (s.lj_sigma[names[i]] + s.lj_sigma[names[j]])) ** 2
                sp = s.srpmf.get((names[i], names[j])) or s.srpmf.get((names[j], names[i]))
                if sp:
                    for m in range(5):
                        law["c%d" % m][i, j] = sp[m]
        self.keys = list(s.efpot_knots)
        for (a, b), (r, u) in s.efpot_knots.items():
            i, j = names.index(a), names.index(b)
            self.tab[i, j] = self.tab[j, i] = len(tables)
            tables.append(_table(np.asarray(r, float), np.asarray(u, float), law["fct"][i, j])
                          + (r[0], r[-1], len(r)))
        self.law = {k: _t(v) for k, v in law.items()}
        self.rth = 8.0 if s.srpmf_rth is None else s.srpmf_rth
        self.has_srp = bool(s.srpmf)
        if tables:
            first = np.cumsum([0] + [t[4] for t in tables])
            self.ep, self.sc = _t(np.concatenate([t[0] for t in tables])), _t([t[1] for t in tables])
            self.rlo, self.rhi = _t([t[2] for t in tables]), _t([t[3] for t in tables])
            self.first = torch.tensor(first[:-1], device=_device())
            self.count = torch.tensor([t[4] for t in tables], device=_device())
            self.ires = 1.0 / s.efpot_res
        self.tabt = torch.tensor(self.tab, device=_device())
        self.qtype = _t(q)
        self.phix = _Map(*s.phix) if s.phix is not None else None
        self.phiv = _Map(s.phiv[0], s.phiv[1]) if s.phiv is not None else None
        if s.rfpar is not None:
            self.gs, self.gr = _Map(s.rfpar[0], s.rfpar[1]), _Map(s.rfpar[0], s.rfpar[2])
        D = [0.0] * nd + list(s.ion_diff)
        diffnuc = 0.1
        self.f1 = _t([diffnuc * s.kbt * s.dt] * nd + [d * s.dt / s.kbt for d in D[nd:]])
        self.f2 = _t([math.sqrt(2 * s.dt * diffnuc)] * nd
                     + [math.sqrt(2 * s.dt * d) for d in D[nd:]])
        self.L = _t([s.lx, s.ly, s.lz])

    def start(self):
        s = self.s
        p = _t(np.stack([s.x, s.y, s.z], 1))
        t = np.abs(np.asarray(s.typei)) - 1
        if self.ns:
            t[:self.ns] = s.site_types - 1
        return p, torch.tensor(t, dtype=torch.long, device=_device())

    # -- laws: energies by kind and minus dE/dr over r --------------------------
    def tabulated(self, k, d2, ep, sc):
        """E and -E'/r of table k at squared distance d2 (flat)."""
        r = d2.sqrt()
        with torch.no_grad():
            at = ((r - self.rlo[k]) * self.ires).long()
            at = self.first[k] + torch.minimum(at.clamp_min(0), self.count[k] - 1)
        p, c = ep[at], sc[k]
        core, tail = d2 < self.rlo[k] ** 2, d2 > self.rhi[k] ** 2
        i2 = 1.0 / d2
        i6 = i2 ** 3
        f = self.tabfct[k] / r
        e = torch.where(core, c[:, 0] * i6 * i6 + c[:, 1], torch.where(
            tail, c[:, 2] * i6 + f, p[:, 0] + r * (p[:, 1] + r * p[:, 2])))
        g = torch.where(core, 12 * c[:, 0] * i6 * i6 * i2, torch.where(
            tail, (6 * c[:, 2] * i6 + f) * i2, -p[:, 1] / r - 2 * p[:, 2]))
        return e, g

    @property
    def tabfct(self):
        names = self.s.type_names()
        return torch.stack([self.law["fct"][names.index(a), names.index(b)] for a, b in self.keys])

    def srpmf(self, i, j, d2, interact):
        r = d2.sqrt()
        c0, c1, c2, c3, c4 = (self.law["c%d" % m][i, j] for m in range(5))
        x0, k, y = self.rth - 0.5, 6.90775527898 / 0.5, 0.001
        on = (c2 != 0)
        c2 = torch.where(on, 1.0 / c2, 0 * c2)
        w = c3 * math.pi * (c1 - r)
        e1, e6 = c0 * torch.exp((c1 - r) * c2), c4 * (c1 / r) ** 6
        e = e1 * torch.cos(w) + e6
        de = e1 * (-c2 * torch.cos(w) + c3 * math.pi * torch.sin(w)) - 6 * e6 / r
        t = torch.exp(-k * (r - x0))
        far = r >= x0
        if interact:  # INTERACT ends the law otherwise than ENERGY
            e = torch.where(far, e * t - y, e)
        else:
            de = torch.where(far, de * (t - y) - e * k * t, de)
            e = torch.where(far, e * (t - y), e)
        z = torch.zeros_like(e)
        return torch.where(on, e, z), torch.where(on, -de / r, z)

    def pairs(self, p, t, rows, tr, interact=False, srfe=None, reff=None, same=None):
        """Sums of rows against all of p: energies [coulomb, lj, srpmf, tables]
        and the reaction field's, forces on the rows, and the reaction field's
        derivative sums.  same: the particle that each row is (-1: none)."""
        d2, sep = 0.0, []
        for a in range(3):
            d = rows[:, a, None] - p[None, :, a]
            if self.s.periodic_rcut is not None:
                d -= self.L[a] * torch.round(d / self.L[a])
            sep.append(d)
            d2 = d2 + d * d
        me = torch.arange(len(p), device=p.device)[None] == same[:, None]
        off = me
        if self.s.ndna:
            off = off | (tr[:, None] < self.s.ndna) & (t[None] < self.s.ndna)
        if self.s.periodic_rcut is not None:
            off = off | (d2 >= self.s.periodic_rcut ** 2)
        d2.masked_fill_(me, 1.0)
        if self.keys:
            tab = self.tabt[tr][:, t]
            plain = (~off & (tab < 0)).double()
        else:
            plain = (~off).double()
        i2 = 1.0 / d2
        i1 = i2.sqrt()
        ec = self.law["fct"][tr][:, t] * i1 * plain
        s6 = self.law["sg2"][tr][:, t] * i2
        s6 = s6 * s6 * s6
        e4 = self.law["eps4"][tr][:, t] * plain
        elj = e4 * s6 * (s6 - 1)
        g = (ec + e4 * (2 * s6 - 1) * s6 * 6) * i2
        e = [ec.sum(), elj.sum(), 0.0, 0.0]
        if self.has_srp:
            a, b = torch.nonzero((plain > 0) & (d2 <= self.rth ** 2), as_tuple=True)
            es, gs = self.srpmf(tr[a], t[b], d2[a, b], interact)
            e[2] = es.sum()
            g[a, b] += gs
        if self.keys:
            a, b = torch.nonzero(~off & (tab >= 0), as_tuple=True)
            et, gt = self.tabulated(tab[a, b], d2[a, b], self.ep, self.sc)
            e[3] = et.sum()
            g[a, b] += gt
        A = B = erf = None
        if srfe is not None:
            ions = (t >= self.s.ndna).double()[None] * (~me).double()
            qq = CELEC * self.qtype[tr][:, None] * self.qtype[t][None] * ions
            R = reff[same][:, None] * reff[None] if (same >= 0).all() else None
            rd = (R * R + d2).rsqrt()
            a1 = qq * R * rd
            A = (a1 * srfe[None]).sum(1)
            ss = srfe[same][:, None] * srfe[None]
            erf = (a1 * ss).sum()
            a2 = qq * ss * rd * rd * rd
            B = (a2 * (d2 + 0.5 * R) * reff[None]).sum(1)
            g = g + a2 * R
        return e, erf, torch.stack([(g * d).sum(1) for d in sep], 1), A, B

    def rf(self, p, t):
        """srfe and reff of every particle (0 for sites and off the map)."""
        ok = self.gs.inside(p) & (t >= self.s.ndna)
        z = torch.zeros(len(p), dtype=torch.float64, device=p.device)
        a = z.index_put((torch.nonzero(ok)[:, 0],), self.gs.linear(p[ok])[0])
        b = z.index_put((torch.nonzero(ok)[:, 0],), self.gr.linear(p[ok])[0])
        return a, math.sqrt(self.s.rfpar[3]) * b

    def single(self, p, t, interact=False):
        """Single-particle energies: membrane, static field, repulsion."""
        s = self.s
        q = self.qtype[t]
        em = ex = ev = torch.zeros((), dtype=torch.float64, device=p.device)
        if s.membrane is not None:
            m = s.membrane["types"]["K"]
            h, pz, pr = 0.5 * s.membrane["thick"], m["pmemb"], m["ppore"]
            z, r = p[:, 2], (p[:, 0] ** 2 + p[:, 1] ** 2).sqrt()

            def smooth(d):
                return 1 + (2 * d - 3) * d * d

            d1 = ((z.abs() - h) / pz).clamp(0, 1)
            d2 = ((m["radi"] + pr - r) / pr).clamp(0, 1)
            w1, w2 = smooth(d1), smooth(d2)
            in1, in2 = d1 <= 0, d2 <= 0
            a1, a2 = m["amplmemb"], m["amplpore"]
            full = torch.full_like(w1, 1e10) if interact else a2 * torch.ones_like(w1)
            e = torch.where(in1, torch.where(in2, full, a2 * w2),
                            torch.where(in2, a1 * w1, 0.5 * (a2 * w2 + a1 * w1)))
            em = torch.where((d1 < 1) & (d2 < 1), e, 0 * e).sum()
        if self.phix is not None:
            ok = self.phix.inside(p)
            ex = (CELEC * q[ok] * self.phix.linear(p[ok])[0]).sum()
        if self.phiv is not None:
            o = s.phiv[2]
            ok = self.phiv.inside(p, 0.0 if o["trilinear"] or interact else self.phiv.d)
            ok &= (p[:, 2] <= o["vzmax"]) & (p[:, 2] >= o["vzmin"])
            v, nodes = (self.phiv.linear if o["trilinear"] else self.phiv.spline)(p[ok])
            v = o["svdw"] * v
            if interact:
                v = torch.where(nodes >= (8.0 if o["trilinear"] else 27.0), 1e10 + 0 * v, v)
            ev = v.sum()
        return em, ex, ev

    def basis(self, p, t):
        """The ions' charge times MMIJ basis values [n, functions]."""
        m = self.s.mmij
        half = _t([b[1] for b in m["region"]])
        u = p / half
        leg = []
        for a in range(3):
            v = [torch.ones_like(u[:, a]), u[:, a]]
            for k in range(2, max(3, m["npol"][a])):
                v.append(((2 * k - 1) * u[:, a] * v[-1] - (k - 1) * v[-2]) / k)
            leg.append(torch.stack(v, 1))
        l = [torch.as_tensor(np.asarray(v), device=p.device) for v in m["lstp"]]
        norm = ((2.0 * l[0] + 1) * (2.0 * l[1] + 1) * (2.0 * l[2] + 1)
                / (8.0 * half.prod())).sqrt()
        b = norm * leg[0][:, l[0]] * leg[1][:, l[1]] * leg[2][:, l[2]]
        ok = ((p.abs() <= half).all(1) & (t >= self.s.ndna)).double()
        return b * (ok * self.qtype[t])[:, None]

    def field(self, c):
        m = self.s.mmij
        return 0.5 * CELEC * m.get("rfscal", 1.0) * (c @ _t(m["mmij"]) @ c)

    def bonded(self, p):
        """The strand's energies by kind, and the forces of the angles, which the
        model defines apart from its energy."""
        n, F = self.s.nucl, torch.zeros_like(p)

        def at(lst):
            return torch.tensor([list(v) for v in lst], dtype=torch.long, device=p.device) - 1

        def sep(i):
            return p[i[:, 1]] - p[i[:, 0]]

        e = dict.fromkeys(("ebond", "eang", "edihe", "estack", "ebp", "eex", "eqq"), 0.0 * p.sum())
        eps = n.epsnuc
        if n.bonds:
            i = at([b[0] for b in n.bonds])
            x2 = (sep(i).norm(dim=1) - _t([b[1] for b in n.bonds])) ** 2
            e["ebond"] = (eps * x2 * (1 + 100 * x2)).sum()
        if n.angles:
            i = at([a[0] for a in n.angles])
            u, v = p[i[:, 0]] - p[i[:, 1]], p[i[:, 2]] - p[i[:, 1]]
            u, v = u.detach(), v.detach()
            nn = u.norm(dim=1) * v.norm(dim=1)
            th = torch.acos((u * v).sum(1) / nn)
            dth = th - _t([a[1] for a in n.angles])
            e["eang"] = (700 * eps * dth ** 2).sum()
            de = (1400 * eps * dth / nn / torch.sin(th))[:, None]
            F.index_add_(0, i[:, 0], de * v)
            F.index_add_(0, i[:, 1], -de * (u + v))
            F.index_add_(0, i[:, 2], de * u)
        if n.dihes:
            i = at([a[0] for a in n.dihes])
            a, b, c = p[i[:, 0]] - p[i[:, 1]], p[i[:, 2]] - p[i[:, 1]], p[i[:, 2]] - p[i[:, 3]]
            n1, n2 = torch.linalg.cross(a, b), torch.linalg.cross(b, c)
            phi = torch.atan2(b.norm(dim=1) * (a * n2).sum(1), (n1 * n2).sum(1))
            e["edihe"] = (28 * eps * (1 - torch.cos(phi - _t([v[1] for v in n.dihes])))).sum()
        if n.stacks:
            i = at([a[0] for a in n.stacks])
            c = (_t([a[1] for a in n.stacks]) ** 2 / (sep(i) ** 2).sum(1)) ** 3
            e["estack"] = (4 * eps * c * (c - 1)).sum()
        if n.bps:
            i = at([a[0] for a in n.bps])
            w = eps * n.scalepairing * _t([2.532 if a[2] else 2.0 for a in n.bps])
            c = _t([a[1] for a in n.bps]) ** 2 / (sep(i) ** 2).sum(1)
            e["ebp"] = (w * c ** 5 * (20 * c - 24)).sum()
        if n.exs:
            i = at([a[0] for a in n.exs])
            c = (_t([a[1] for a in n.exs]) ** 2 / (sep(i) ** 2).sum(1))
            near, c = c > 1, c ** 3
            e["eex"] = torch.where(near, 4 * eps * c * (c - 1) + eps, 0 * c).sum()
        if n.qqs:
            i = at(n.qqs)
            e["eqq"] = (n.fctn / sep(i).norm(dim=1)).sum()
        return e, F

    def energy(self, p, t):
        """The 23 ENERGY terms and the forces."""
        s = self.s
        p = p.detach().clone().requires_grad_()
        em, ex, ev = self.single(p, t)
        smooth = em + ex + ev
        e = dict.fromkeys(abi.TERM_NAMES, 0.0)
        F = torch.zeros_like(p)
        if s.mmij is not None:
            gsbp = self.field(self.basis(p, t).sum(0))
            smooth = smooth + gsbp
            e["egsbpb"] = gsbp.item()
        if s.nucl is not None:
            eb, Fb = self.bonded(p)
            F = F + Fb.detach()
            smooth = smooth + sum(v for k, v in eb.items() if k != "eang")
            e.update({k: v.item() for k, v in eb.items()})
        if smooth.requires_grad:
            F = F - torch.autograd.grad(smooth, p)[0]
        srfe = reff = None
        if s.rfpar is not None:
            srfe, reff = self.rf(p, t)
            d1, = torch.autograd.grad(srfe.sum(), p, retain_graph=True)
            d2, = torch.autograd.grad(reff.sum(), p)
            srfe, reff = srfe.detach(), reff.detach()
            q2 = CELEC * self.qtype[t] ** 2 * (t >= s.ndna)
            e["erfpar"] = (0.5 * q2 * srfe ** 2).sum().item()
            F = F - (q2 * srfe)[:, None] * d1
        p = p.detach()
        e.update(ememb=em.item(), egsbpa=ex.item(), evdwgd=ev.item())
        n = len(p)
        sums = torch.zeros(4, dtype=torch.float64, device=p.device)
        rows = max(1, (1 << 23) // n)
        for a in range(0, n, rows):
            own = torch.arange(a, min(n, a + rows), device=p.device)
            ei, erf, f, A, B = self.pairs(p, t, p[own], t[own], srfe=srfe, reff=reff, same=own)
            sums += torch.stack([torch.as_tensor(v, dtype=torch.float64, device=p.device)
                                 for v in ei])
            F[own] += f
            if srfe is not None:
                e["erfpar"] += 0.5 * float(erf)
                F[own] -= A[:, None] * d1[own] + B[:, None] * d2[own]
        e["eelec"], e["evdw"], e["esrpmf"], tables = (0.5 * float(v) for v in sums)
        e["eefpotmx" if s.ndna else "eefpot"] = tables
        if s.rfpar is not None:
            e["egsbpb"] = e["erfpar"]
        e["ener"] = sum(v for k, v in e.items()
                        if k not in ("ener", "egsbpb")) + (e["egsbpb"] if s.mmij is not None else 0)
        return e, F

    def interact(self, p, t, r, tj, j):
        """The energy of a particle of type tj at r among p, where it is j (or,
        with j = len(p), comes in)."""
        s = self.s
        r = r.reshape(1, 3)
        tt = torch.tensor([tj], device=p.device)
        out = sum(self.single(r, tt, interact=True))
        if j < len(p):
            p = p.clone()
            p[j] = r[0]
        else:
            p, t = torch.cat([p, r]), torch.cat([t, tt])
        same = torch.tensor([j], device=p.device)
        srfe = reff = None
        if s.rfpar is not None and bool(self.gs.inside(r)[0]):
            srfe, reff = self.rf(p, t)
            out = out + 0.5 * CELEC * self.qtype[tj] ** 2 * srfe[j] ** 2
        ei, erf, _, _, _ = self.pairs(p, t, r, tt, interact=True, srfe=srfe, reff=reff, same=same)
        out = out + sum(ei) + (erf if erf is not None else 0.0)
        if s.mmij is not None:
            b = self.basis(p, t)
            c = b.sum(0)
            out = out + self.field(c) - self.field(c - b[j])
        return float(out)

    def move(self, p, t, F, seed, step):
        s = self.s
        z = _t(_normals(seed, step, len(p)))
        d = (F * self.f1[t][:, None]).clamp(-s.bdmax, s.bdmax)
        p = p + d + self.f2[t][:, None] * z
        c = _t([s.cx, s.cy, s.cz])
        if s.periodic_rcut is not None:
            lo = c - 0.5 * self.L
            return torch.where(p < lo, p + self.L, torch.where(p >= lo + self.L, p - self.L, p))
        return torch.minimum(torch.maximum(p, c - 0.5 * self.L), c + 0.5 * self.L)

    def steps(self, p, t, k, seed, step0=0):
        for i in range(k):
            p = self.move(p, t, self.energy(p, t)[1], seed, step0 + i)
        return p


class _Gcmc:
    """GRAND and COUNT on a system's ions."""

    def __init__(self, sys):
        s = sys.s
        self.sys, b = sys, s.buffers
        self.p, self.t = sys.start()
        self.type = [s.ion_names.index(x["ion"]) for x in b]
        self.lo, self.hi = [x["lzmin"] for x in b], [x["lzmax"] for x in b]
        self.aver, self.mu = [x["aver"] for x in b], [x["mu"] for x in b]
        self.tag = np.asarray(s.ibuffer).copy()
        self.nat = [x["nat"] for x in b]

    def grand(self, attempts, seed, cycle):
        s, total = self.sys.s, 0.0
        nb = len(self.nat)
        for k in range(attempts):
            u = _uniforms(seed, cycle, k, 2)
            if next(u) < 0.5:
                b = int(nb * next(u))
                r = np.array([s.lx * (next(u) - 0.5) + s.cx, s.ly * (next(u) - 0.5) + s.cy,
                              self.lo[b] + (self.hi[b] - self.lo[b]) * next(u)])
                e = self.sys.interact(self.p, self.t, _t(r), self.type[b], len(self.p))
                w = self.aver[b] / (self.nat[b] + 1) * math.exp(min(-(e - self.mu[b]) / s.kbt, 700))
                if next(u) <= w / (1 + w):
                    total += e
                    self.p = torch.cat([self.p, _t(r)[None]])
                    self.t = torch.cat([self.t, self.t.new_tensor([self.type[b]])])
                    self.tag = np.append(self.tag, b + 1)
                    self.nat[b] += 1
            else:
                b = int(nb * next(u))
                k0 = int(self.nat[b] * next(u))
                if k0 >= self.nat[b]:
                    continue
                i = int(np.nonzero(self.tag == b + 1)[0][k0])
                e = self.sys.interact(self.p, self.t, self.p[i], self.type[b], i)
                w = self.aver[b] / self.nat[b] * math.exp(min(-(e - self.mu[b]) / s.kbt, 700))
                if next(u) <= 1 / (1 + w):
                    total -= e
                    for a in (self.p, self.t, self.tag):
                        a[i] = a[-1].clone() if torch.is_tensor(a) else a[-1]
                    self.p, self.t, self.tag = self.p[:-1], self.t[:-1], self.tag[:-1]
                    self.nat[b] -= 1
        return total

    def count(self):
        z, t = self.p[:, 2].cpu().numpy(), self.t.cpu().numpy()
        self.tag[:] = 0
        for b in range(len(self.nat)):
            at = (self.tag == 0) & (t == self.type[b]) & (z >= self.lo[b]) & (z <= self.hi[b])
            self.tag[at] = b + 1
            self.nat[b] = int(at.sum())


def _metropolis(sys, moves, mcmax, seed, cycle):
    p, t = sys.start()
    s, n, total = sys.s, len(p), 0.0
    half = _t([s.lx, s.ly, s.lz]) * 0.5
    for m in range(moves):
        u = _uniforms(seed, cycle, m, 3)
        while True:
            i = int(n * next(u))
            r = p[i] + mcmax * _t([next(u) - 0.5 for _ in range(3)])
            if bool((r.abs() <= half).all()):
                break
        old = sys.interact(p, t, p[i], int(t[i]), i)
        new = sys.interact(p, t, r, int(t[i]), i)
        if new <= old or next(u) < math.exp(-(new - old) / s.kbt):
            p = p.clone()
            p[i] = r
            total += new - old
    return total, p


def _adjoint(sys, case, seed):
    """Histogram of the segment's pair distances and the gradient of the RDF
    loss with respect to the tables, by automatic differentiation."""
    s, steps = sys.s, case["steps"]
    p, t = sys.start()
    n = len(p)
    kind = torch.nn.functional.one_hot(t, 2).double()
    rb = ADJ_R0 + ADJ_DR * np.arange(ADJ_BINS)
    far = (rb[-1] + 5 * ADJ_SIGMA) ** 2
    which = torch.tensor([[0, 1], [1, 2]], device=p.device)

    def within(x, rmax2):
        """Pairs i < j closer than that."""
        d2 = sum((x[:, a, None] - x[None, :, a]) ** 2 for a in range(3))
        return torch.nonzero(torch.triu(d2 <= rmax2, 1), as_tuple=True)

    def forces(x, ep, sc):
        # the tables' pairs one by one, all others by the analytic tail
        with torch.no_grad():
            i, j = within(x, float(sys.rhi.max()) ** 2)
        d2 = sum((x[:, a, None] - x[None, :, a]) ** 2 for a in range(3))
        d2 = d2 + torch.eye(n, dtype=x.dtype, device=x.device)
        i2 = 1 / d2
        c6 = kind @ torch.stack([sc[0, 2], sc[1, 2], sc[1, 2], sc[2, 2]]).reshape(2, 2) @ kind.T
        fct = sys.law["fct"][t][:, t]
        keep = torch.ones_like(d2)
        keep[i, j] = keep[j, i] = 0
        keep.fill_diagonal_(0)
        g = (6 * c6 * i2 ** 3 + fct * i2.sqrt()) * i2 * keep
        _, near = sys.tabulated(which[t[i], t[j]], d2[i, j], ep, sc)
        g = g + torch.zeros_like(g).index_put((torch.cat([i, j]), torch.cat([j, i])),
                                              torch.cat([near, near]))
        return torch.stack([(g * (x[:, a, None] - x[None, :, a])).sum(1) for a in range(3)], 1)

    def hist(x):
        with torch.no_grad():
            i, j = within(x, far)
        r, pair, rows = ((x[i] - x[j]) ** 2).sum(1).sqrt(), which[t[i], t[j]], []
        centre = _t(rb)
        for k in range(3):
            h = torch.zeros(ADJ_BINS, dtype=torch.float64, device=x.device)
            for part in r[pair == k].split(1 << 17):
                w = (centre[None] - part[:, None]) / ADJ_SIGMA
                w = torch.where(w.abs() <= 5, torch.exp(-0.5 * w * w), 0 * w)
                h = h + w.sum(0) / (math.sqrt(2 * math.pi) * ADJ_SIGMA)
            rows.append(h)
        return torch.stack(rows)

    path, H = [p], torch.zeros((3, ADJ_BINS), dtype=torch.float64, device=p.device)
    with torch.no_grad():
        for k in range(steps):
            p = sys.move(p, t, forces(p, sys.ep, sys.sc), seed, k)
            path.append(p)
            H += hist(p)
    a, b = (n + 1) // 2, n // 2
    npair = _t([a * (a - 1) / 2, a * b, b * (b - 1) / 2])
    norm = steps * npair[:, None] * 4 * math.pi * _t(rb) ** 2 / s.lx ** 3
    dl = 2 * (H / norm - 1) / norm
    g_ep, g_sc, back = torch.zeros_like(sys.ep), torch.zeros_like(sys.sc), torch.zeros_like(p)
    for k in reversed(range(steps)):
        x = path[k + 1].detach().requires_grad_()
        back = back + torch.autograd.grad((dl * hist(x)).sum(), x)[0]
        x, ep, sc = (v.detach().requires_grad_() for v in (path[k], sys.ep, sys.sc))
        y = sys.move(x, t, forces(x, ep, sc), seed, k)
        back, u, v = torch.autograd.grad(y, (x, ep, sc), back)
        g_ep, g_sc = g_ep + u, g_sc + v
    return H, g_ep, g_sc, p


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        _, reps = _replicas(case, seed)
        base = int(seed) % 100003
        dener, frames = [], []
        for r, s in enumerate(reps):
            sys = _System(s) if r == 0 or case["attempts"] else _shared(sys, s)
            if case["attempts"]:
                g = _Gcmc(sys)
                dener.append(g.grand(case["attempts"], base + r, 1))
                p = sys.steps(g.p, g.t, case["steps"], base + r)
                frames.append(_padded(p, 2 * len(s.x) + 64))
            else:
                frames.append(sys.steps(*sys.start(), case["steps"], base + r))
        frames = torch.cat(frames).T
        return [np.array(dener), frames] + [None] * 5 if case["attempts"] else [frames]
    sys = _System(_spec(case, seed))
    if kind == "energy":
        e, F = sys.energy(*sys.start())
        return np.array([e[k] for k in abi.TERM_NAMES]), F, None
    if kind in ("bulk", "ssdna"):
        p, t = sys.start()
        return sys.steps(p, t, case["steps"], seed).T
    if kind == "cycle":
        g = _Gcmc(sys)
        for c in range(case["cycles"]):
            d = g.grand(case["attempts"], seed, c + 1)
            g.p = sys.steps(g.p, g.t, case["nbd"], seed, c * case["nbd"])
            g.count()
        return (np.array([d]), _padded(g.p, 2 * len(sys.s.x) + 64).T) + (None,) * 5
    if kind == "metropolis":
        total, p = _metropolis(sys, case["moves"], 1.0, seed, 1)
        return None, np.array([total]), p.T
    H, g_ep, g_sc, p = _adjoint(sys, case, seed)
    return H, _knots(sys, g_ep.cpu().numpy(), g_sc.cpu().numpy()), p.T


def _padded(p, cap):
    return torch.cat([p, p.new_zeros(cap - len(p), 3)])


def _knots(sys, g_ep, g_sc):
    """The tables' gradient on their knots: a table is linear in the knots."""
    out = []
    for k, (r, u) in enumerate(sys.s.efpot_knots.values()):
        r, u, a = np.asarray(r, float), np.asarray(u, float), int(sys.first[k])
        fct = float(sys.tabfct[k])
        ep, sc = _table(r, u, fct)
        g = np.zeros(len(u))
        for m in range(len(u)):
            v = u.copy()
            v[m] += 1.0
            e1, s1 = _table(r, v, fct)
            g[m] = ((e1 - ep) * g_ep[a:a + len(u)]).sum() + ((s1 - sc) * g_sc[k]).sum()
        out.append(g)
    return np.stack(out)


def _shared(sys, s):
    """Another system with the first one's laws and maps."""
    new = object.__new__(_System)
    new.__dict__.update(sys.__dict__)
    new.s, new.L = s, _t([s.lx, s.ly, s.lz])
    return new
