"""Performance cases of the lattice Boltzmann engine: what its users have it do, over the real range.

A case is one piece of a solve as a program of this framework runs it: a few diagnostic intervals of
lattice steps (`step(every)`, then `diag()`), regrids at their cadence where the grid is adaptive, and
at the end the state or the macroscopic field read into the caller's pinned memory, as a program does
before it writes a frame or hands the state on.  Cadences are the programs' own (steps/240 between
diagnostics of a uniform solve, steps/160 of an AMR solve, regrids every 20 coarse steps).

`prepare` makes the solver (its Reynolds number and velocity amplitude, and where the case says so its
whole state, come from the seed); every `run` goes on from where the last one stopped.
"""
import ctypes as C
import math
import os
import random
import sys

import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jp-solver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import jpsolver as J  # noqa: E402

Q = 19
ELEM = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}
# floating-point operations of one D3Q19 BGK cell update: 45 for the moments, 15 for velocity and
# equilibrium constants, 12 per pair of opposite populations, 12 for the rest population and weights
FLOPS = 180
CX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0)
CY = (0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1)
W = (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12


# ---- the cases ----------------------------------------------------------------------------------------


def uniform(n, storage, samples, every, out, inplace=False):
    return {"kind": "uniform", "n": n, "storage": storage, "samples": samples, "every": every, "out": out,
            "inplace": inplace}


def amr(n, mode, storage, graph, samples, every, frac1=0.3, frac2=0.1):
    return {"kind": "amr", "n": n, "mode": mode, "storage": storage, "graph": graph, "samples": samples,
            "every": every, "frac1": frac1, "frac2": frac2}


def listed():
    return [
        # the smallest calls: two diagnostic intervals of a coarse exploratory solve; launches and
        # latency are all there is to it
        dict(uniform(32, "fp32", 2, 5, "populations"), name="uniform_n32_fp32"),
        # the small validation solve: N=64, 2000 steps, diagnostics every 50 (here four intervals)
        dict(uniform(64, "fp32", 4, 50, "populations"), name="uniform_n64_fp32"),
        # the `uniform` program's default size, t*=12 sampled 240 times (every 20 steps)
        dict(uniform(128, "fp32", 4, 20, "populations"), name="uniform_n128_fp32"),
        # the headline size: one diagnostic interval at N=512 (20 GB of populations)
        dict(uniform(512, "fp32", 1, 81, "fields"), name="uniform_n512_fp32"),
        # the same flow with 16-bit storage, the reduced-memory option at full size
        dict(uniform(512, "fp16", 1, 81, "fields"), name="uniform_n512_fp16"),
        # double-precision storage, the oracle run that the other storages' errors are quoted against
        dict(uniform(256, "fp64", 1, 40, "populations"), name="uniform_n256_fp64"),
        # in-place streaming, for cubes that must live in half the memory; an edge that is no power of two
        dict(uniform(400, "fp32", 1, 64, "fields", True), name="inplace_n400_fp32"),
        # static AMR gold run: coarse 64^3, both levels refined everywhere, one diagnostic interval
        # from a given state of the finest level
        dict(amr(64, "all", "fp32", True, 1, 15), name="amr_static_n64_fp32"),
        # dynamic AMR run: coarse 96^3, sensor-driven levels, regrid and diagnostics every 20 coarse steps
        dict(amr(96, "sensor", "fp32", True, 4, 20), name="amr_dynamic_n96_fp32"),
        # a served dynamic AMR solve with 16-bit storage, stepped by direct launches
        dict(amr(48, "sensor", "fp16", False, 4, 20), name="amr_dynamic_n48_fp16"),
        # an ensemble: uniform cubes of the served sizes and small AMR solves stepped together
        {"kind": "ensemble", "uniform": "32,48,64,96,128", "amr": "16,24,32", "storage": "fp32", "copies": 2, "steps": 24,
         "name": "ensemble_mixed_fp32"},
        # a state in the host's blocked FP32 layout taken in by a 16-bit solver, advanced one diagnostic
        # interval and handed back in the same layout (coupling, restart from another code's state)
        {"kind": "exchange", "n": 96, "storage": "fp16", "layout": "blocked", "every": 15, "name": "exchange_n96_fp16"},
    ]


def _log_size(rng, lo, hi, step):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["uniform"] * 5 + ["amr"] * 3 + ["ensemble", "exchange"])
    if kind == "uniform":
        storage = rng.choice(["fp32", "fp32", "fp32", "fp16", "bf16", "fp64"])
        n = _log_size(rng, 24, 256 if storage == "fp64" else 448, 4)  # multiples of four: odd block counts too
        inplace = storage != "fp64" and rng.random() < 0.25
        out = "populations" if storage == "fp64" or (storage == "fp32" and not inplace and n <= 192) else "fields"
        return uniform(n, storage, rng.randint(1, 4) if n <= 192 else 1, max(1, round(n / 6.4) + rng.randint(-2, 2)), out,
                       inplace)
    if kind == "amr":
        mode = rng.choice(["all", "sensor", "sensor"])
        n = _log_size(rng, 16, 56 if mode == "all" else 88, 8)
        storage = rng.choice(["fp32", "fp32", "fp16", "bf16"]) if mode == "sensor" else "fp32"
        return amr(n, mode, storage, rng.random() < 0.5, rng.randint(1, 4), rng.randint(8, 24),
                   round(rng.uniform(0.2, 0.4), 3), round(rng.uniform(0.05, 0.3), 3))
    if kind == "ensemble":
        u = sorted(rng.choice([32, 48, 64, 96, 128]) for _ in range(rng.randint(2, 5)))
        a = sorted(rng.choice([16, 24, 32]) for _ in range(rng.randint(1, 3)))
        return {"kind": "ensemble", "uniform": ",".join(map(str, u)), "amr": ",".join(map(str, a)),
                "storage": rng.choice(["fp32", "fp32", "fp16"]), "copies": rng.randint(1, 2), "steps": rng.randint(8, 32)}
    return {"kind": "exchange", "n": _log_size(rng, 32, 112, 8), "storage": rng.choice(["fp16", "bf16", "fp32"]),
            "layout": rng.choice(["flat", "blocked"]), "every": rng.randint(5, 20)}


# ---- inputs and states ----------------------------------------------------------------------------------


def _flow(case, seed):
    """Reynolds number and velocity amplitude of a solve, from the seed (a resolved, stable range)."""
    r = random.Random("%d flow" % seed)
    n = case["n"] * (4 if case["kind"] == "amr" else 1)
    top = max(250.0, min(1600.0, 12.0 * n))
    return {"re": math.exp(r.uniform(math.log(200.0), math.log(top))), "u0": r.uniform(0.03, 0.05)}


def _flat_state(n, u0, seed, device, dtype):
    """Equilibrium populations [19, n, n, n] of a Taylor-Green vortex with three weaker modes of random phase."""
    g = random.Random("%d state" % seed)
    x = (torch.arange(n, dtype=torch.float64, device=device) + 0.5) * (2 * math.pi / n)
    zz, yy, xx = x.view(n, 1, 1), x.view(1, n, 1), x.view(1, 1, n)
    p = [g.uniform(0, 2 * math.pi) for _ in range(3)]
    ux = u0 * torch.sin(xx) * torch.cos(yy) * torch.cos(zz) + 0.2 * u0 * torch.sin(2 * zz + p[0]) + 0 * (xx + yy)
    uy = -u0 * torch.cos(xx) * torch.sin(yy) * torch.cos(zz) + 0.2 * u0 * torch.sin(2 * xx + p[1]) + 0 * (zz + yy)
    uz = 0.2 * u0 * torch.sin(3 * yy + p[2]) + 0 * (xx + zz)
    rho = 1 + 3 * (u0 * u0 / 16) * (torch.cos(2 * xx) + torch.cos(2 * yy)) * (torch.cos(2 * zz) + 2)
    return _equilibrium(rho, ux, uy, uz, dtype)


def _equilibrium(rho, ux, uy, uz, dtype=torch.float64):
    n = rho.shape[0]
    f = torch.empty((Q,) + tuple(rho.shape), dtype=dtype, device=rho.device)
    usq = 1.5 * (ux * ux + uy * uy + uz * uz)
    for q in range(Q):
        cu = 3 * (CX[q] * ux + CY[q] * uy + CZ[q] * uz)
        f[q] = W[q] * rho * (1 + cu + 0.5 * cu * cu - usq)
    assert f.shape[1] == n
    return f


def _to_blocked(f, mb=8):
    """[19, n, n, n] -> [block][19][mb^3], blocks and cells with x fastest."""
    n = f.shape[1]
    g = n // mb
    return f.view(Q, g, mb, g, mb, g, mb).permute(1, 3, 5, 0, 2, 4, 6).reshape(g ** 3, Q, mb ** 3)


def _octants(n, mb=8):
    """For each block of a 4n grid (as [bz][by][bx]) its place in the pool when both levels are refined everywhere."""
    g0 = n // mb
    i = torch.arange(4 * g0)
    pos0, o1, o2 = i // 4, (i // 2) % 2, i % 2

    def at(z, y, x):
        return (z.view(-1, 1, 1), y.view(1, -1, 1), x.view(1, 1, -1))

    z, y, x = at(pos0, pos0, pos0)
    b = (z * g0 + y) * g0 + x
    z, y, x = at(o1, o1, o1)
    b = 8 * b + (z * 4 + y * 2 + x)
    z, y, x = at(o2, o2, o2)
    return 8 * b + (z * 4 + y * 2 + x)


def _finest_blocked(f, n):
    """[19, 4n, 4n, 4n] as the level-2 population pool of a solve refined everywhere."""
    b = _to_blocked(f)
    order = _octants(n).reshape(-1).to(f.device)
    out = torch.empty_like(b)
    out[order] = b
    return out


def _pinned(count, dtype=torch.float32):
    return torch.empty(int(count), dtype=dtype, pin_memory=True)


def _check(status):
    if status:
        raise RuntimeError("jp status %d: %s" % (status, J.lib().jp_last_error().decode()))


def _read_populations(s, buf, level=0, layout="flat"):
    count = s.population_count(level)
    if count > buf.numel():  # a regrid grew the pool
        buf = _pinned(count, buf.dtype)
    dt = 1 if buf.dtype == torch.float64 else 0
    if count:
        _check(J.lib().jp_get_populations(s.h, level, J.LAYOUT[layout], dt, C.c_void_p(buf.data_ptr()), count))
    return buf[:count]


def _read_macro(s, buf):
    _check(J.lib().jp_get_macro(s.h, C.cast(buf.data_ptr(), C.POINTER(C.c_float)), buf.numel()))
    return buf


def _solver(case, seed):
    flow = _flow(case, seed)
    if case["kind"] == "uniform":
        flags = J.FLAG_INPLACE if case["inplace"] else 0
        return J.Solver("uniform", n=case["n"], storage=case["storage"], mb=8 if case["n"] % 8 == 0 else 4, flags=flags,
                        **flow)
    kw = dict(l1_mode=case["mode"], l2_mode=case["mode"], frac1=case["frac1"], frac2=case["frac2"], tstar=20.0,
              adapt_every=20, max_gb=16.0, flags=J.FLAG_GRAPH if case["graph"] else 0)
    return J.Solver("amr", n=case["n"], storage=case["storage"], **flow, **kw)


def prepare(case, seed):
    """The solver, set up as its program has it before the next diagnostic interval, and the pinned memory that the
    program reads results into."""
    J.lib()
    k = case["kind"]
    if k == "uniform":
        s = _solver(case, seed)
        cells = case["n"] ** 3
        if case["out"] == "populations":
            buf = _pinned(Q * cells, torch.float64 if case["storage"] == "fp64" else torch.float32)
        else:
            buf = _pinned(4 * cells)
        return {"case": case, "s": s, "buf": buf}
    if k == "amr":
        s = _solver(case, seed)
        n = case["n"]
        if case["mode"] == "all":
            f = _flat_state(4 * n, s.cfg.u0, seed, "cuda", torch.float64)
            p = _finest_blocked(f, n).to(torch.float32).reshape(-1)
            host = _pinned(p.numel())
            host.copy_(p)
            del f, p
            _check(J.lib().jp_set_populations(s.h, 2, J.LAYOUT["blocked"], 0, C.c_void_p(host.data_ptr()), host.numel()))
            s.sync()
            return {"case": case, "s": s, "bufs": [host]}
        if case["storage"] != "fp32":
            m = (4 * n) ** 3
            return {"case": case, "s": s, "bufs": [_pinned(m), _pinned(m), _pinned(3 * m)]}
        c = s.counts()
        sizes = (c["cnb0"], c["cap1"], c["cap2"])
        return {"case": case, "s": s, "bufs": [_pinned(Q * 512 * b) for b in sizes]}
    if k == "ensemble":
        e = J.Ensemble(0)
        members, bufs = [], []
        for c in range(case["copies"]):
            for i, n in enumerate(case["uniform"].split(",")):
                m = uniform(int(n), case["storage"], 1, case["steps"], "fields")
                members.append(_solver(m, seed + 100 * c + i))
                bufs.append(_pinned(4 * int(n) ** 3))
            for i, n in enumerate(case["amr"].split(",")):
                m = amr(int(n), "sensor", case["storage"], False, 1, case["steps"])
                members.append(_solver(m, seed + 100 * c + 50 + i))
                bufs.append(None)
        for s in members:
            e.add(s)
        return {"case": case, "e": e, "members": members, "bufs": bufs}
    n = case["n"]
    s = J.Solver("uniform", n=n, storage=case["storage"], **_flow(case, seed))
    f = _flat_state(n, s.cfg.u0, seed, "cuda", torch.float64)
    if case["layout"] == "blocked":
        f = _to_blocked(f)
    src = _pinned(f.numel())
    src.copy_(f.to(torch.float32).reshape(-1))
    return {"case": case, "s": s, "src": src, "dst": _pinned(src.numel())}


def run(state):
    """One pass: the samples of the case, then the state or field as the program reads it."""
    case = state["case"]
    k = case["kind"]
    if k == "ensemble":
        state["e"].step(case["steps"])
        out = []
        for s, buf in zip(state["members"], state["bufs"]):
            d = list(s.diag())
            out.append(d if buf is None else d + [_read_macro(s, buf)])
        # at most 64 outputs: the diagnostics of all solves in one list of numbers
        return {"diag": torch.tensor([o[:3] for o in out], dtype=torch.float32), "macro": [o[3] for o in out if len(o) > 3]}
    s = state["s"]
    if k == "exchange":
        lay = J.LAYOUT[case["layout"]]
        src, dst = state["src"], state["dst"]
        _check(J.lib().jp_set_populations(s.h, 0, lay, 0, C.c_void_p(src.data_ptr()), src.numel()))
        s.step(case["every"])
        d = s.diag()
        return {"diag": torch.tensor(d, dtype=torch.float32), "populations": _read_populations(s, dst, 0, case["layout"])}
    d = []
    for _ in range(case["samples"]):
        s.step(case["every"])
        if k == "amr" and case["mode"] == "sensor":
            s.regrid()
        d.append(s.diag())
    out = {"diag": torch.tensor(d, dtype=torch.float32)}
    if k == "uniform":
        if case["out"] == "populations":
            out["populations"] = _read_populations(s, state["buf"])
        else:
            out["macro"] = _read_macro(s, state["buf"])
        return out
    bufs = state["bufs"]
    if case["mode"] == "all":
        out["level2"] = _read_populations(s, bufs[0], 2, "blocked")
    elif case["storage"] == "fp32":
        for level in range(3):
            out["level%d" % level] = _read_populations(s, bufs[level], level, "blocked")
    else:
        fp = C.POINTER(C.c_float)
        _check(J.lib().jp_get_output_fields(s.h, *(C.cast(b.data_ptr(), fp) for b in bufs), bufs[0].numel()))
        out["q"], out["speed"], out["velocity"] = bufs
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------


def _state_work(cells, updates, elem):
    """One read and one write of the populations for the whole pass, and the arithmetic of every update."""
    return 2.0 * Q * elem * cells, float(FLOPS) * updates


def _amr_cells(case):
    """(cells of all levels, cell updates per coarse step) of the 1:2:4 subcycle at the requested fractions."""
    n3 = case["n"] ** 3
    n1 = 8 * n3 * (1.0 if case["mode"] == "all" else case["frac1"])
    n2 = 8 * n1 * (1.0 if case["mode"] == "all" else case["frac2"])
    return n3 + n1 + n2, n3 + 2 * n1 + 4 * n2, n1, n2


def work(case):
    k = case["kind"]
    if k == "uniform":
        cells, steps, elem = case["n"] ** 3, case["samples"] * case["every"], ELEM[case["storage"]]
        b, f = _state_work(cells, cells * steps, elem)
        return {"bytes": b + (0 if case["out"] == "populations" else 16 * cells), "flops": f}
    if k == "exchange":
        cells = case["n"] ** 3
        return {"bytes": 2.0 * Q * 4 * cells, "flops": float(FLOPS) * cells * case["every"]}
    if k == "amr":
        cells, per_step, _, _ = _amr_cells(case)
        b, f = _state_work(cells, per_step * case["samples"] * case["every"], ELEM[case["storage"]])
        return {"bytes": b + (0 if case["storage"] == "fp32" else 20 * (4 * case["n"]) ** 3), "flops": f}
    bytes_, flops = 0.0, 0.0
    for n in case["uniform"].split(","):
        b, f = _state_work(int(n) ** 3, int(n) ** 3 * case["steps"], ELEM[case["storage"]])
        bytes_, flops = bytes_ + b + 16 * int(n) ** 3, flops + f
    for n in case["amr"].split(","):
        cells, per_step, _, _ = _amr_cells(amr(int(n), "sensor", case["storage"], False, 1, case["steps"]))
        b, f = _state_work(cells, per_step * case["steps"], ELEM[case["storage"]])
        bytes_, flops = bytes_ + b, flops + f
    return {"bytes": bytes_ * case["copies"], "flops": flops * case["copies"]}


# ---- the same in 64 bits ----------------------------------------------------------------------------------


def _moments(f):
    rho = f.sum(0)
    j = [torch.zeros_like(rho) for _ in range(3)]
    for q in range(1, Q):
        for c, t in zip((CX[q], CY[q], CZ[q]), j):
            if c:
                t.add_(f[q], alpha=c)
    return rho, [t.div_(rho) for t in j]


def _bgk_steps(f, omega, steps):
    """`steps` pull stream-collide steps of [19, z, y, x] populations in place of `f`'s values."""
    g = torch.empty_like(f)
    for _ in range(steps):
        for q in range(Q):
            g[q] = torch.roll(f[q], (CZ[q], CY[q], CX[q]), (0, 1, 2)) if q else f[q]
        rho, (ux, uy, uz) = _moments(g)
        base = 1 - 1.5 * (ux * ux + uy * uy + uz * uz)
        ow = omega * rho
        torch.add((1 - omega) * g[0], ow * base, alpha=W[0], out=f[0])
        for q in range(1, Q, 2):
            a = None
            for c, u in ((CX[q], ux), (CY[q], uy), (CZ[q], uz)):
                if c:
                    a = (u if c > 0 else -u) if a is None else a + c * u
            sym = (a * a).mul_(4.5).add_(base).mul_(ow).mul_(W[q])
            asym = (a * ow).mul_(3 * W[q])
            torch.add(g[q], sym, alpha=1 / (1 - omega), out=f[q])
            f[q].add_(asym, alpha=1 / (1 - omega)).mul_(1 - omega)
            torch.add(g[q + 1], sym, alpha=1 / (1 - omega), out=f[q + 1])
            f[q + 1].sub_(asym, alpha=1 / (1 - omega)).mul_(1 - omega)
    return f


def _diag(rho, u):
    def d(a, axis):
        return (torch.roll(a, -1, axis) - torch.roll(a, 1, axis)) * 0.5

    ux, uy, uz = u
    e = 0.5 * (ux * ux + uy * uy + uz * uz).mean()
    w = [d(uz, 1) - d(uy, 0), d(ux, 0) - d(uz, 2), d(uy, 2) - d(ux, 1)]
    ens = 0.5 * sum((t * t).mean() for t in w)
    return [float(e), float(ens), float(rho.mean())]


def _tau(n, re, u0):
    return 3.0 * u0 * n / (2 * math.pi * re) + 0.5


def _tgv(n, u0, device):
    x = (torch.arange(n, dtype=torch.float64, device=device) + 0.5) * (2 * math.pi / n)
    zz, yy, xx = x.view(n, 1, 1), x.view(1, n, 1), x.view(1, 1, n)
    ux = u0 * torch.sin(xx) * torch.cos(yy) * torch.cos(zz)
    uy = -u0 * torch.cos(xx) * torch.sin(yy) * torch.cos(zz)
    rho = 1 + 3 * (u0 * u0 / 16) * (torch.cos(2 * xx) + torch.cos(2 * yy)) * (torch.cos(2 * zz) + 2)
    return _equilibrium(rho, ux, uy, torch.zeros_like(ux))


def _macro(f):
    rho, u = _moments(f)
    return rho, u, torch.stack([rho] + u, -1).reshape(-1)


def exact(case, seed):
    """The pass in plain 64-bit torch; adaptive grids, whose tables follow the sensor, have no value here."""
    k = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if k == "uniform":
        flow = _flow(case, seed)
        n = case["n"]
        omega = 1.0 / _tau(n, **flow)
        f, d = _tgv(n, flow["u0"], dev), []
        for _ in range(case["samples"]):
            f = _bgk_steps(f, omega, case["every"])
            d.append(_diag(*_moments(f)))
        out = {"diag": torch.tensor(d, dtype=torch.float64)}
        if case["out"] == "populations":
            out["populations"] = f.reshape(-1)
        else:
            out["macro"] = _macro(f)[2]
        return out
    if k == "exchange":
        flow = _flow(case, seed)
        f = _flat_state(case["n"], flow["u0"], seed, dev, torch.float64).to(torch.float32).to(torch.float64)
        f = _bgk_steps(f, 1.0 / _tau(case["n"], **flow), case["every"])
        d = _diag(*_moments(f))
        return {"diag": torch.tensor(d, dtype=torch.float64),
                "populations": (_to_blocked(f) if case["layout"] == "blocked" else f).reshape(-1)}
    if k == "amr" and case["mode"] == "all":
        # refined everywhere, the finest level is a periodic cube of edge 4n at its own relaxation time
        flow = _flow(case, seed)
        n = case["n"]
        tau = _tau(n, **flow)
        tau2 = 2.0 * (2.0 * tau - 0.5) - 0.5
        f = _flat_state(4 * n, flow["u0"], seed, dev, torch.float64).to(torch.float32).to(torch.float64)
        d = []
        for _ in range(case["samples"]):
            f = _bgk_steps(f, 1.0 / tau2, 4 * case["every"])
            d.append(_diag(*_moments(f)))
        return {"diag": torch.tensor(d, dtype=torch.float64), "level2": _finest_blocked(f, n).reshape(-1)}
    if k == "ensemble":
        fields = []
        for c in range(case["copies"]):
            for i, n in enumerate(case["uniform"].split(",")):
                m = uniform(int(n), case["storage"], 1, case["steps"], "fields")
                flow = _flow(m, seed + 100 * c + i)
                f = _bgk_steps(_tgv(int(n), flow["u0"], dev), 1.0 / _tau(int(n), **flow), case["steps"])
                fields.append(_macro(f)[2])
        return {"diag": None, "macro": fields}
    return None
