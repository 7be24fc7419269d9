"""The solver calls that a user's program makes, with the sizes it makes them at.

A case names a call (`kind`) and its sizes.  `prepare` builds what the program
holds before the call: the parameter set, the spectral tables and the
temperature field made from the seed, and the solver context, batch or server
that it keeps between calls.  `run` is one call through the package's entry
points and returns what the program reads back.

kinds
  solve    host field in, host Q and sigma and the FP64 means, variances and
           wall fluxes out: `Solver.solve`
  dnscall  what the channel DNS does with mc_gpu_ / get_results_: host field in,
           float Q and sigma into the caller's own arrays
  slab     one rank's planes of a z-slab solve with the field and the results
           in device memory: `solve_device_async` + `collect_device`
  dnsstep  a whole radiation update of the DNS: the field from its double
           temperature, the solve, and the source terms back in host arrays
  dnssrc   the source-term kernel alone on a finished solve, device arrays
  batch    many small problems of uneven size in one launch: `Batch`
  served   the same mix as single requests to a `Server`
"""
import math

import numpy as np
import torch

from radchan_b200 import api
from radchan_b200 import workloads as W

# mean path of a bundle in metres before it is absorbed or meets a wall, by
# medium (the synthetic tables' decades of k, or grey gas of 1/m); a bundle
# crosses path/2 * (cells per metre of every axis) faces
PATH = {"grey": 2.35, "thin": 0.28, "thick": 0.27}
LOGK = {"thin": -3.0, "thick": -1.0}
FLOPS_STEP, FLOPS_BUNDLE = 60.0, 200.0


def _case(name, kind, nx, ny, nz, photmax, **kw):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, photmax=photmax, nvar=4, gas="thin", nb=100, nq=8, nt=64,
             levels=1, walls=0, specular=0, fp64=0, particles=0, pcol=1, members=1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a grey channel for a quick look or a unit test of the caller, launches and latency
        _case("grey16", "solve", 16, 16, 16, 32, gas="grey"),
        # the reference's grey set-up: 32^3, one level, wall to wall paths
        _case("grey32", "solve", 32, 32, 32, 64, gas="grey"),
        # nothing a power of two: odd edges, bands, g points, bundles and replicates, coarse level of ratio 3
        _case("ragged", "solve", 45, 27, 33, 75, nvar=3, nb=61, nq=5, nt=41, levels=2, walls=1),
        # the headline solve: narrow band, three levels, west wall flux, called as the DNS calls it
        _case("nb64", "dnscall", 64, 64, 64, 256, levels=3, walls=1),
        # one of four ranks of that channel on its own planes, everything in device memory
        _case("slab64", "slab", 64, 64, 64, 128, levels=3, walls=1, pcol=4),
        # the headline solve with suspended particles that scatter
        _case("particles64", "dnscall", 64, 64, 64, 128, levels=3, walls=1, particles=1),
        # the double precision build (floatpoint = 1), used to check a float run
        _case("double32", "solve", 32, 32, 32, 64, levels=2, walls=1, fp64=1),
        # the largest: an optically thick 192x128x128 channel, specular y walls, both wall fluxes
        _case("thick192", "slab", 192, 128, 128, 16, gas="thick", specular=1, walls=2),
        # a radiation update of the DNS, from its temperature to its source terms, at a radStep's bundle count
        _case("dnsstep64", "dnsstep", 64, 64, 64, 32, levels=3, walls=1),
        # the source terms of a large pencil when the DNS's arrays live on the device
        _case("dnssrc192", "dnssrc", 192, 128, 128, 1, walls=1, nvar=2),
        # a parameter study of small uneven problems, half grey and half narrow band, in one launch
        _case("batch24", "batch", 16, 32, 24, 64, members=24),
        # the same study sent to a server as single requests
        _case("served16", "served", 16, 32, 24, 64, members=16),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "dnscall", "dnscall", "slab", "dnsstep", "dnssrc", "batch", "served"])
    if kind == "dnssrc":
        return _plain(_case("", kind, _edge(rng, 24, 192), _edge(rng, 17, 128), _edge(rng, 17, 128), 1, nvar=2,
                            walls=rng.randint(0, 2), nb=rng.randint(20, 100)))
    if kind in ("batch", "served"):
        lo = rng.randint(12, 18)
        return _plain(_case("", kind, lo, rng.randint(24, 34), rng.randint(20, 28), _edge(rng, 20, 96),
                            members=rng.randint(6, 24)))
    levels = rng.choice([1, 1, 2, 3])
    unit = {1: 1, 2: 3, 3: 4}[levels]  # ratios 3, and 2 and 2
    edge = lambda: max(12 // unit, _edge(rng, 12, 96) // unit) * unit
    nx, ny, nz = edge(), edge(), edge()
    pcol = 1
    if kind == "slab":
        pcol = rng.choice([2, 3, 4])
        nz = max(nz // (unit * pcol), 1) * unit * pcol
    gas = rng.choice(["grey", "thin", "thin", "thick"]) if kind in ("solve", "slab") else rng.choice(["thin", "thick"])
    fp64 = 1 if kind == "solve" and rng.random() < 0.2 else 0
    particles = 1 if kind == "dnscall" and rng.random() < 0.4 else 0
    nvar = rng.choice([2, 3, 4, 8])
    # steps of a pass spread over three decades, at most those of the largest listed case
    c = _case("", kind, nx, ny, nz, 1, gas=gas, fp64=fp64, particles=particles, nvar=nvar, levels=levels, pcol=pcol,
              walls=rng.randint(0, 2), specular=rng.randint(0, 1), nb=rng.randint(20, 100), nq=rng.randint(2, 8),
              nt=rng.randint(24, 64))
    target = math.exp(rng.uniform(math.log(3e6), math.log(1.0e9))) / (8 if fp64 else 3 if particles else 1)
    per_photon = _bundles(c) * _steps(c)
    c["photmax"] = max(8, min(400, int(target / per_photon)))
    return _plain(c)


def _plain(c):
    c.pop("name")
    return c


def _bundles(c):
    n = c["nx"] * c["ny"] * (c["nz"] // c["pcol"]) + c["walls"] * c["ny"] * (c["nz"] // c["pcol"])
    return float(n) * c["nvar"] * c["photmax"]


def _steps(c):
    coarse = {1: 1.0, 2: 0.6, 3: 0.55}[c["levels"]]  # coarse cells take fewer steps
    return 1.0 + 0.5 * PATH[c["gas"]] * coarse * (c["nx"] / 2.0 + c["ny"] / (2 * math.pi) + c["nz"] / math.pi)


def _study(c):
    """Edges, medium and bundles of every member of a batch or a served mix, from the case alone."""
    rng = np.random.default_rng(c["nx"] * 1000 + c["members"])
    edges = sorted({c["nx"], c["ny"], c["nz"], (c["nx"] + c["ny"]) // 2})
    out = []
    for i in range(c["members"]):
        nx, ny, nz = (int(rng.choice(edges)) for _ in range(3))
        out.append(dict(c, kind="solve", nx=nx, ny=ny, nz=nz, gas="grey" if i % 2 == 0 else "thin",
                        photmax=int(rng.choice([c["photmax"] // 2, c["photmax"]])), nb=int(rng.integers(20, 101)),
                        members=1))
    return out


def _levels(c):
    n = (c["nx"], c["ny"], c["nz"])
    if c["levels"] == 1:
        return [n], [100000]
    if c["levels"] == 2:
        r = 3 if all(e % 3 == 0 for e in n) else 2
        return [n, tuple(e // r for e in n)], [5, 100000]
    return [n, tuple(e // 2 for e in n), tuple(e // 4 for e in n)], [5, 5, 100000]


def _params(c, seed):
    lev, maxs = _levels(c)
    p = W.channel_params(c["nx"], c["ny"], c["nz"], grey=c["gas"] == "grey", photmax=c["photmax"], nVar=c["nvar"],
                         levels=lev, maxs=maxs, adiabw=int(c["walls"] > 0), adiabe=int(c["walls"] > 1),
                         calcwalls=int(c["walls"] > 0), bd_y=3 if c["specular"] else 1, nB=c["nb"], nQ=c["nq"],
                         nT=c["nt"], eps=0.8 if c["specular"] else 1.0, seed=seed, floatpoint=c["fp64"])
    p.p_col = c["pcol"]
    return p


def _problem(c, seed):
    p = _params(c, 1000003 * seed + 17)
    tabs = None
    if c["gas"] != "grey":
        tabs = W.tables_nb(nB=c["nb"], nQ=c["nq"], nT=c["nt"], logk_lo=LOGK[c["gas"]], seed=20240601 + seed)
    return p, tabs, W.channel_field(p, seed=seed + 7)


def _dns_inputs(c, p, T, tabs, seed):
    """The DNS's own double temperature and its coupling constants."""
    a = tabs.arrays()
    Tin = 955.0
    cpl = api.DnsCoupling(Tin=Tin, Height=0.5, underrelax=0.8, Tnb=a["Tnb"].astype(np.float64),
                          kP=a["kP"].astype(np.float64) * 0.5)
    noise = np.random.default_rng(seed + 99).uniform(-1e-4, 1e-4, T.shape)
    return cpl, T.astype(np.float64) / Tin + noise


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "batch":
        b = api.Batch()
        s = dict(c=c, batch=b, keep=[], out=[])
        for i, m in enumerate(_study(c)):
            p, tabs, T = _problem(m, seed * 31 + i)
            sv = api.Solver(p, tabs)
            b.add(sv, T)
            s["keep"].append((sv, tabs))
            s["out"].append((np.zeros(api.result_shape(p), np.float32), np.zeros(api.result_shape(p), np.float32)))
        return s
    if c["kind"] == "served":
        sv = api.Server(max_inflight=8)
        s = dict(c=c, server=sv, requests=[])
        for i, m in enumerate(_study(c)):
            p, tabs, T = _problem(m, seed * 31 + i)
            s["requests"].append((p, T, sv.add_tables(tabs) if tabs is not None else -1))
        return s
    p, tabs, T = _problem(c, seed)
    sv = api.Solver(p, tabs)
    s = dict(c=c, p=p, T=T, solver=sv, tabs=tabs)
    if c["particles"]:
        sv.set_scattering(api.Scattering.synthetic(nB=c["nb"], nQ=c["nq"], nA=181, ksca_lo=0.1, ksca_hi=1.0,
                                                   g_lo=0.0, g_hi=0.8, seed=3 + seed))
    if c["kind"] == "dnscall":
        s["Q"] = np.zeros(api.result_shape(p), np.float32)
        s["S"] = np.zeros(api.result_shape(p), np.float32)
    elif c["kind"] == "slab":
        kl = p.kmax // p.p_col
        s["zstart"] = 1 + (seed % p.p_col) * kl
        s["Td"] = torch.from_numpy(T).cuda()
        s["out"] = [torch.zeros((kl, p.jmax, p.imax), dtype=torch.float64, device="cuda") for _ in range(2)]
        s["out"] += [torch.zeros((2, kl, p.jmax), dtype=torch.float64, device="cuda") for _ in range(2)]
    elif c["kind"] in ("dnsstep", "dnssrc"):
        s["cpl"], s["T1"] = _dns_inputs(c, p, T, tabs, seed)
        if c["kind"] == "dnssrc":
            s["ticket"] = sv.solve_async(T)
            sv.wait_device(s["ticket"])
            tshape, oshape = s["cpl"].pencil_shapes(p)
            s["T1d"] = torch.from_numpy(s["T1"]).cuda()
            s["out"] = [torch.empty(oshape, dtype=torch.float64, device="cuda") for _ in range(4)]
    return s


def run(s):
    kind = s["c"]["kind"]
    if kind == "batch":
        s["batch"].run()
        s["batch"].wait()
        for i, (Q, S) in enumerate(s["out"]):
            s["batch"].collect_into(i, Q, S)
        return s["out"]
    if kind == "served":
        ids = [s["server"].submit(p, T, ts) for p, T, ts in s["requests"]]
        got = [s["server"].wait(i) for i in ids]
        return [(r.Q, r.sigma) for r in got]
    sv = s["solver"]
    if kind == "solve":
        r = sv.solve(s["T"])
        return dict(Q=r.Q, sigma=r.sigma, q64=r.q64, var64=r.var64, qw64=r.qw64, vw64=r.vw64)
    if kind == "dnscall":
        sv.collect_into(sv.solve_async(s["T"]), s["Q"], s["S"])
        return dict(Q=s["Q"], sigma=s["S"])
    if kind == "slab":
        t = sv.solve_device_async(s["Td"].data_ptr(), s["zstart"])
        sv.collect_device(t, *(o.data_ptr() for o in s["out"]))
        return dict(zip(("q64", "var64", "qw64", "vw64"), s["out"]))
    if kind == "dnsstep":
        T = api.field_from_dns(s["T1"], s["cpl"].Tin)
        return sv.dns_source(sv.solve_async(T), s["cpl"], s["T1"])
    sv.dns_source_device(s["ticket"], s["cpl"], s["T1d"].data_ptr(), *(o.data_ptr() for o in s["out"]),
                         stream=torch.cuda.current_stream().cuda_stream)
    return dict(zip(("Qnew", "Varnew", "Knew", "Gnew"), s["out"]))


def exact(case, seed):
    """The absorption coefficient of the source terms has a value in closed form; a Monte Carlo mean, drawn from
    the package's own counters, has none outside it."""
    c = dict(case)
    if c["kind"] not in ("dnsstep", "dnssrc"):
        return None
    p, tabs, T = _problem(c, seed)
    cpl, T1 = _dns_inputs(c, p, T, tabs, seed)
    x, y = cpl.Tnb, cpl.kP
    x0 = T1[1:-1, 1:-1, :] * cpl.Tin
    t = np.clip((np.trunc(x0 - x[0]) / int(x[1] - x[0])).astype(np.int64), 0, len(x) - 2)
    K = (y[t + 1] - y[t]) / (x[t + 1] - x[t]) * (x0 - x[t]) + y[t]
    out = dict(Qnew=None, Varnew=None, Knew=K, Gnew=None)
    if c["kind"] == "dnsstep":
        out["n_clamped"] = None
    return out


def work(case):
    c = dict(case)
    if c["kind"] in ("batch", "served"):
        parts = [work(m) for m in _study(c)]
        return dict(bytes=sum(w["bytes"] for w in parts), flops=sum(w["flops"] for w in parts))
    field = 4.0 * (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)
    cells = float(c["nx"]) * c["ny"] * (c["nz"] // c["pcol"])
    if c["kind"] == "dnssrc":
        out = (c["nx"] + 2.0) * c["ny"] * c["nz"]
        return dict(bytes=out * (8 + 8 + 32), flops=out * 20)
    tables = 0.0 if c["gas"] == "grey" else 4.0 * c["nb"] * c["nt"] * (c["nq"] * 2 + 2)
    flops = _bundles(c) * (FLOPS_BUNDLE + _steps(c) * FLOPS_STEP)
    if c["particles"]:
        flops *= 1.4
    return dict(bytes=field + tables + 24.0 * cells, flops=flops)
