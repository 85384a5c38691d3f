"""Performance cases: what a user of the library has it do, through its plan objects.

Each case is a plain dict; `prepare` makes the plan and the device buffers a user's
program holds, `run` is one pass through the public entry points, `exact` the same
outputs by full-grid FFTs in FP64 without the library.  Kinds of pass:

  roundtrip  forward KRFFT of B fields and backward of the spectra (plan.forward,
             plan.backward; both directions of the transform)
  contour    Ns diffusion contour steps of B chains (step_diffusion on a centred plan)
  qfused     the same through plan_diffusion's Q-matrix solver (plain lattices)
  fullgrid   fields on the whole grid: gather onto the subgrid, forward, backward and the
             symmetry fill back to the whole grid
  scft       one SCFT evaluation of an AB diblock (both propagators, densities,
             residuals, partition function and free energy)

Fields are random (one N(0,1) value per orbit) or, where they enter an exponential,
Gaussian-smoothed, symmetric under the group's operations about a half-step-shifted
origin, as the transforms require.
"""
import importlib.util
import itertools
import math
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "crystallographicfft.jl_b200")


def _lib():
    name = "crystallographicfft_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PKG, "__init__.py"),
                                                      submodule_search_locations=[PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ----------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest transform in use: one field, launch latency counts
        {"name": "im3m-32-one", "kind": "roundtrip", "group": 229, "N1": 32, "N2": 32, "N3": 32, "precision": 4, "batch": 1},
        # one field at the headline grid: a serial solver's call
        {"name": "im3m-128-one", "kind": "roundtrip", "group": 229, "N1": 128, "N2": 128, "N3": 128, "precision": 4, "batch": 1},
        # the headline workload: a batch of fields resident in device memory
        {"name": "im3m-128-batch", "kind": "roundtrip", "group": 229, "N1": 128, "N2": 128, "N3": 128, "precision": 4, "batch": 128},
        # plain lattice in FP64
        {"name": "pmmm-64-f64", "kind": "roundtrip", "group": 47, "N1": 64, "N2": 64, "N3": 64, "precision": 8, "batch": 256},
        # a large cubic grid, a few fields
        {"name": "im3m-192", "kind": "roundtrip", "group": 229, "N1": 192, "N2": 192, "N3": 192, "precision": 4, "batch": 16},
        # hexagonal cell: the axes differ
        {"name": "p6mmm-60x60x80", "kind": "roundtrip", "group": 191, "N1": 60, "N2": 60, "N3": 80, "precision": 8, "batch": 4},
        # a two-dimensional phase diagram: plane group, many small fields
        {"name": "p4mm-160", "kind": "roundtrip", "group": 11, "N1": 160, "N2": 160, "N3": 1, "precision": 8, "batch": 64},
        # a parameter sweep of chains: the contour loop on a batch
        {"name": "ia3d-96-contour", "kind": "contour", "group": 230, "N1": 96, "N2": 96, "N3": 96, "precision": 4, "batch": 256,
         "steps": 20},
        # the Q-matrix solver for a plain cubic lattice
        {"name": "pm3m-48-qfused", "kind": "qfused", "group": 221, "N1": 48, "N2": 48, "N3": 48, "precision": 8, "batch": 4,
         "steps": 50},
        # fields kept on the whole grid, an edge that is no power of two
        {"name": "fd3m-80-fullgrid", "kind": "fullgrid", "group": 227, "N1": 80, "N2": 80, "N3": 80, "precision": 4, "batch": 8},
        # the SCFT iteration of the gyroid: two propagators, a serial chain of steps
        {"name": "ia3d-64-scft", "kind": "scft", "group": 230, "N1": 64, "N2": 64, "N3": 64, "precision": 8, "batch": 2,
         "steps": 100},
        # the contour loop of one chain pair in FP32, the early phase of such a solve
        {"name": "ia3d-96-pair", "kind": "contour", "group": 230, "N1": 96, "N2": 96, "N3": 96, "precision": 4, "batch": 2,
         "steps": 100},
    ]


# Grid edges in use: factors 2, 3 and 5; groups with quarter translations take multiples
# of 8, the other cubic, orthorhombic and square ones even edges, hexagonal ones any.
_EDGES = [16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 90, 96, 100, 108, 120, 128, 144,
          160, 180, 192]
_FIXED = [8, 12, 16, 24, 32, 48]  # channel edges of the Q-matrix solver


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _supported(c):
    """Whether the library plans the case: its channel planes fit a block's shared memory
    and the phase denominator lcm(N) is at most 8192."""
    N, ops, L = _shape(c)
    M = [n // l for n, l in zip(N, L)]
    fold = c["group"] in (225, 227, 229, 230) and all(l == 2 for l in L) and all(m % 2 == 0 for m in M)
    H = [m // 2 for m in M] if fold else M
    if len(set(H)) == 1 and H[0] in _FIXED[:5] + [4, 6] + [48] * (c["precision"] == 4):
        return True
    if c["kind"] == "qfused":
        return False
    ch = (2 if c["group"] in (225, 227) else 4) if fold else 1
    size = 2 * c["precision"] * max(2 * ch * H[0] * H[1] + H[0] + H[1], 2 * H[0] * H[2] + H[2])
    return size <= 227 * 1024 and math.lcm(*N) <= 8192


def _draw(rng):
    kind = rng.choice(["roundtrip", "roundtrip", "roundtrip", "contour", "qfused", "fullgrid", "scft"])
    form = rng.choice(["cubic", "cubic", "cubic", "plane", "axes"]) if kind == "roundtrip" else "cubic"
    if form == "plane":
        group, n = 11, [rng.choice([18, 32, 50, 54, 64, 90, 96, 128, 144, 150, 160])] * 2 + [1]
    elif form == "axes":
        group = rng.choice([191, 47])
        a, b, d = (rng.choice([e for e in _EDGES if e <= 100 and (group == 191 or e % 2 == 0)]) for _ in range(3))
        n = [a, a if group == 191 else b, d]
    else:
        group = rng.choice([221, 47] if kind == "qfused" else [229, 230, 227] if kind == "scft" else [229, 230, 227, 225, 221, 47])
        lo, hi = (24, 96) if kind in ("qfused", "scft") else (16, 192 if kind == "roundtrip" else 128)
        n = [rng.choice([e for e in _EDGES if lo <= e <= hi and e % (8 if group in (227, 230) else 2) == 0])] * 3
    c = {"kind": kind, "group": group, "N1": n[0], "N2": n[1], "N3": n[2], "precision": rng.choice([4, 4, 8])}
    c["batch"] = 2
    if kind == "scft":  # residuals are differences of near-equal fields: the FP64 phase
        c["precision"], c["steps"] = 8, 100
    elif kind in ("contour", "qfused"):
        c["steps"] = _log(rng, 1, 50)
    if kind != "scft":  # whole-grid points times steps at most about the largest listed case's
        c["batch"] = _log(rng, 1, max(1, min(256, 1.5e8 / (n[0] * n[1] * n[2]) / max(1.0, c.get("steps", 0) / 5))))
    return c


def draw(rng):
    while True:
        c = _draw(rng)
        if _supported(c):
            return c


# ----------------------------------------------------------------- symmetry (generators of the International Tables)

_M3M = ["-x,-y,z", "-x,y,-z", "z,x,y", "y,x,-z", "-x,-y,-z"]
_GENERATORS = {
    47: ["-x,-y,z", "-x,y,-z", "-x,-y,-z"],
    191: ["-y,x-y,z", "-x,-y,z", "y,x,-z", "-x,-y,-z"],
    221: _M3M,
    225: _M3M + ["x,y+1/2,z+1/2", "x+1/2,y,z+1/2"],
    227: ["-x+3/4,-y+1/4,z+1/2", "-x+1/4,y+1/2,-z+3/4", "z,x,y", "y+3/4,x+1/4,-z+1/2", "-x,-y,-z",
          "x,y+1/2,z+1/2", "x+1/2,y,z+1/2"],
    229: _M3M + ["x+1/2,y+1/2,z+1/2"],
    230: ["-x+1/2,-y,z+1/2", "-x,y+1/2,-z+1/2", "z,x,y", "y+3/4,x+1/4,-z+1/4", "-x,-y,-z", "x+1/2,y+1/2,z+1/2"],
    11: ["-x,-y,z", "-y,x,z", "-x,y,z"],
}


def _seitz(text):
    """(R, 12 t) of a coordinate triplet."""
    R, t = np.zeros((3, 3), dtype=np.int64), [0, 0, 0]
    for i, part in enumerate(text.split(",")):
        for term in part.replace("-", "+-").split("+"):
            s = -1 if term.startswith("-") else 1
            term = term.lstrip("-")
            if term in ("x", "y", "z"):
                R[i, "xyz".index(term)] += s
            elif term:
                p, q = term.split("/")
                t[i] += s * 12 * int(p) // int(q)
    return tuple(R.ravel().tolist()), tuple(v % 12 for v in t)


def _closure(gens):
    ident = (tuple(np.eye(3, dtype=np.int64).ravel().tolist()), (0, 0, 0))
    found, front = {ident}, [ident]
    while front:
        new = []
        for (Ra, ta), (Rb, tb) in itertools.product(front, gens):
            A, B = np.reshape(Ra, (3, 3)), np.reshape(Rb, (3, 3))
            op = (tuple((A @ B).ravel().tolist()), tuple(int(v) % 12 for v in A @ np.array(tb) + np.array(ta)))
            if op not in found:
                found.add(op)
                new.append(op)
        front = new
    return [ident] + sorted(found - {ident})


def _operations(case):
    """[(R, t)] in grid units about the origin moved by half a grid step along every axis,
    where that keeps the translations whole (then no point is its own mirror image)."""
    N = np.array([case["N1"], case["N2"], case["N3"]])
    ops = [(np.reshape(R, (3, 3)), np.array(t) * N // 12) for R, t in _closure([_seitz(g) for g in _GENERATORS[case["group"]]])]
    s = np.array([1, 1, 1 if N[2] > 1 else 0])
    move = [np.eye(3, dtype=np.int64) @ s - R @ s for R, _ in ops]
    whole = all((m % 2 == 0).all() for m in move)
    return [(R, (t - m // 2) % N if whole else t % N) for (R, t), m in zip(ops, move)]


def _strides(ops, N):
    """Largest strides (1 or 2 per axis) whose parity classes the translations reach."""
    axes = 3 if N[2] > 1 else 2
    top = [2 if any(t[d] % 2 for _, t in ops) else 1 for d in range(axes)]
    best = [1] * axes
    masks = [tuple(top)] + [tuple(2 if (m >> d) & 1 and top[d] == 2 else 1 for d in range(axes)) for m in range(1, 2 ** axes)]
    for L in masks:
        n = int(np.prod(L))
        if n > int(np.prod(best)) and len({tuple(int(t[d]) % L[d] for d in range(axes)) for _, t in ops}) == n:
            best = list(L)
    return best + [1] * (3 - axes)


def _grid(N, L=(1, 1, 1)):
    z, y, x = torch.meshgrid(*(torch.arange(0, N[d], L[d], device="cuda", dtype=torch.int64) for d in (2, 1, 0)), indexing="ij")
    return x, y, z


def _linear(v, N):
    return (torch.remainder(v[2], N[2]) * N[1] + torch.remainder(v[1], N[1])) * N[0] + torch.remainder(v[0], N[0])


def _apply(M, p, t=(0, 0, 0)):
    return [sum(int(M[i][j]) * p[j] for j in range(3) if int(M[i][j])) + int(t[i]) for i in range(3)]


def _orbits(ops, N, L):
    """Orbit number of every point of the stride-L grid, in memory order (z, y, x)."""
    p = _grid(N, L)
    low = None
    for R, t in ops:
        k = _linear(_apply(R, p, t), N)
        low = k if low is None else torch.minimum(low, k)
    return torch.unique(low, return_inverse=True)[1]


def _spectral_points(ops, N):
    """Grid positions of the independent spectral points: the lowest index of each orbit of
    R^T h that no operation extinguishes, ordered by (h1, h2, h3)."""
    h = _grid(N)
    lin = _linear(h, N)
    keep = torch.ones_like(lin, dtype=torch.bool)
    for R, t in ops:
        k = _linear(_apply(R.T, h), N)
        phase = sum(int(t[d]) * h[d].double() / N[d] for d in range(3))
        dead = (k == lin) & ((phase - torch.round(phase)).abs() > 1e-6)
        keep &= (k >= lin) & ~dead
    x, y, z = (v[keep] for v in h)
    order = torch.argsort((x * N[1] + y) * N[2] + z)
    return lin[keep][order]


# ----------------------------------------------------------------- inputs

def _shape(case):
    N = (case["N1"], case["N2"], case["N3"])
    ops = _operations(case)
    return N, ops, _strides(ops, N)


def _random(case, seed, orbits, count):
    """`count` fields on the points that `orbits` numbers: one normal value per orbit."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    n = int(orbits.max()) + 1
    return (torch.randn(n, generator=g, device="cuda", dtype=torch.float64)[orbits.reshape(-1)].reshape(orbits.shape)
            for _ in range(count))


def _smooth(u, N):
    """Gaussian filter of width 2 grid points, zero mean and unit deviation."""
    k2 = sum((2 * math.pi * torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)).square().reshape(
        [-1 if a == i else 1 for a in range(3)]) for i, n in enumerate((N[2], N[1], N[0])))
    u = torch.fft.ifftn(torch.fft.fftn(u) * torch.exp(-2.0 * k2)).real
    u = u - u.mean()
    return u / u.std()


def _cell(case):
    return 4.0


def _sub(u, L):
    return u[..., ::L[2], ::L[1], ::L[0]]


def _fields(case, seed, N, ops, L, whole):
    """The case's random fields on the whole grid or the subgrid, in FP64, one at a time."""
    return _random(case, seed, _orbits(ops, N, (1, 1, 1) if whole else L), case["batch"])


def _chains(case, seed, N, ops):
    """(q, w) pairs on the whole grid: propagator starts and interaction fields."""
    it = _random(case, seed, _orbits(ops, N, (1, 1, 1)), 2 * case["batch"])
    for u in it:
        yield torch.exp(0.3 * _smooth(u, N)), 5.0 * _smooth(next(it), N)


def _diblock(case, seed, N, ops):
    """(w_A, w_B) on the whole grid: the seeded start of an SCFT solve, f = 0.4, chi N = 20."""
    eta = _smooth(next(_random(case, seed, _orbits(ops, N, (1, 1, 1)), 1)), N)
    return torch.stack([20.0 * 0.6 + eta, 20.0 * 0.4 - eta])


_DT = {4: torch.float32, 8: torch.float64}


def prepare(case, seed):
    cf = _lib()
    N, ops, L = _shape(case)
    dim = 3 if N[2] > 1 else 2
    dt, B, kind = _DT[case["precision"]], case["batch"], case["kind"]
    Nd, lattice = N[:dim], np.eye(dim) * _cell(case)
    _, sym = cf.find_optimal_shift(cf.get_ops(case["group"], dim, Nd), Nd)
    if {(op.R, tuple(v % n for v, n in zip(op.t, Nd))) for op in sym} != {
            (tuple(int(v) for v in R[:dim, :dim].ravel()), tuple(int(v) for v in t[:dim])) for R, t in ops}:
        raise ValueError("the library's operations about its chosen origin are other ones")
    spec = cf.calc_spectral_asu(sym, dim, Nd)
    s = {"kind": kind, "lib": cf}
    if kind == "scft":
        plan, s["solver"] = cf.plan_scft(case["group"], N, 9.0, f=0.4, chiN=20.0, Ns=case["steps"],
                                         precision=case["precision"], ops=sym)
        s["w"] = _sub(_diblock(case, seed, N, ops), L).to(dt).contiguous()
    elif kind in ("contour", "qfused"):
        if kind == "contour":
            plan = cf.plan_centered_scft(spec, sym, Nd, 0.01, lattice, precision=case["precision"], max_batch=B)
        else:
            plan = cf.KRFFTPlan(spec, sym, N=Nd, ds=0.01, lattice=lattice, precision=case["precision"], max_batch=B,
                                path=cf.PATH_M2Q)
        s["solver"] = cf.DiffusionSolver(plan)
        pairs = [(_sub(q, L).to(dt), _sub(w, L).to(dt)) for q, w in _chains(case, seed, N, ops)]
        s["q0"], s["w"] = (torch.stack(v).contiguous() for v in zip(*pairs))
        s["q"], s["steps"] = torch.empty_like(s["q0"]), case["steps"]
    else:
        plan = cf.plan_krfft_centered(spec, sym, precision=case["precision"], max_batch=B)
        u = torch.stack([v.to(dt) for v in _fields(case, seed, N, ops, L, kind == "fullgrid")])
        s["u" if kind == "fullgrid" else "f0"] = u
        M = plan.M
        s["f1"] = torch.empty((B,) + tuple(reversed(M)), dtype=dt, device="cuda")
        s["F"] = torch.empty((B, plan.n_spec), dtype=torch.complex64 if dt == torch.float32 else torch.complex128, device="cuda")
        if kind == "fullgrid":
            s["g0"], s["u1"] = torch.empty_like(s["f1"]), torch.empty_like(u)
    if list(plan.L) != list(L[:dim]):
        raise ValueError("strides %s, the plan has %s" % (L, plan.L))
    s["plan"] = plan
    return s


def run(s):
    plan, kind = s["plan"], s["kind"]
    if kind == "roundtrip":
        plan.forward(s["f0"], out=s["F"])
        plan.backward(s["F"], out=s["f1"])
        return s["F"], s["f1"]
    if kind == "fullgrid":
        plan.fullgrid_to_subgrid(s["u"], out=s["g0"])
        plan.forward(s["g0"], out=s["F"])
        plan.backward(s["F"], out=s["f1"])
        return s["F"], plan.subgrid_to_fullgrid(s["f1"], out=s["u1"])
    if kind == "scft":
        r = s["solver"].evaluate(s["w"])
        return r["phi"], r["d"], r["Q"], r["F"], r["err"]
    s["q"].copy_(s["q0"])  # every solve starts from the chain end
    s["lib"].step_diffusion(s["solver"], s["q"], s["w"], 0.01, s["steps"])
    return s["q"]


def work(case):
    """Inputs read once and outputs written once; the arithmetic of the transforms of the
    independent points (5 n log2 n per complex point pair, two real fields per transform)."""
    N, ops, L = _shape(case)
    B, r = case["batch"], case["precision"]
    vol = N[0] * N[1] * N[2]
    sub = vol // int(np.prod(L))
    spec = 2 * vol // max(1, len(ops))  # complex points of the spectral ASU, about
    flops = 2.5 * sub * math.log2(max(2, sub)) * B  # one transform of the subgrid
    kind = case["kind"]
    if kind == "scft":
        n = case["steps"]
        return {"bytes": r * sub * (2 * 2 * (n + 1) + 2 * 3), "flops": (2 * flops + 4 * sub * B) * n}
    if kind in ("contour", "qfused"):
        return {"bytes": 3 * r * sub * B, "flops": 2 * flops * case["steps"]}
    field = vol if kind == "fullgrid" else sub
    return {"bytes": 2 * r * B * (field + spec), "flops": 2 * flops}


# ----------------------------------------------------------------- the same in FP64 by full-grid FFTs

def _kernel(N, ds, cell):
    """exp(-ds |2 pi h / cell|^2) with h in [-N/2, N/2)."""
    k2 = 0
    for a, n in enumerate((N[2], N[1], N[0])):
        h = torch.arange(n, device="cuda", dtype=torch.float64)
        h = torch.where(h >= n // 2, h - n, h)
        k2 = k2 + (2 * math.pi * h / cell).square().reshape([-1 if i == a else 1 for i in range(3)])
    return torch.exp(-ds * k2)


def _simpson(n):
    w = torch.ones(n + 1, dtype=torch.float64)
    if n % 2:
        w[0] = w[-1] = 0.5
        return w
    w[1:-1:2], w[2:-1:2] = 4.0, 2.0
    return w / 3.0


def exact(case, seed):
    N, ops, L = _shape(case)
    kind = case["kind"]
    dt = _DT[case["precision"]]
    if kind == "scft":
        n = case["steps"]
        wa, wb = _diblock(case, seed, N, ops).to(dt).double()
        K, na, ds = _kernel(N, 1.0 / n, 9.0), round(0.4 * n), 1.0 / n
        ea, eb = torch.exp(-0.5 * ds * wa), torch.exp(-0.5 * ds * wb)
        q, p = [torch.ones_like(wa)], [torch.ones_like(wa)]
        for i in range(n):
            for chain, e in ((q, ea if i < na else eb), (p, ea if n - 1 - i < na else eb)):
                chain.append(e * torch.fft.ifftn(K * torch.fft.fftn(e * chain[-1])).real)
        Q = q[n].mean()
        sa, sb = _simpson(na), _simpson(n - na)
        pa = sum(sa[j] * q[j] * p[n - j] for j in range(na + 1)) * ds / Q
        pb = sum(sb[j - na] * q[j] * p[n - j] for j in range(na, n + 1)) * ds / Q
        da, db = 20.0 * (pb - 0.5) + 0.5 * (wb - wa), 20.0 * (pa - 0.5) + 0.5 * (wa - wb)
        err = torch.sqrt((da.square().sum() + db.square().sum()) / (wa.square().sum() + wb.square().sum()))
        F = -torch.log(Q) + ((wb - wa).square() / 80.0 - 0.5 * (wa + wb)).mean() + 5.0
        return (_sub(torch.stack([pa, pb]), L).contiguous(), _sub(torch.stack([da, db]), L).contiguous(),
                float(Q), float(F), float(err))
    if kind in ("contour", "qfused"):
        K, out = _kernel(N, 0.01, _cell(case)), []
        for q, w in _chains(case, seed, N, ops):
            q, e = q.to(dt).double(), torch.exp(-0.005 * w.to(dt).double())
            for _ in range(case["steps"]):
                q = e * torch.fft.ifftn(K * torch.fft.fftn(e * q)).real
            out.append(_sub(q, L).clone())
        return torch.stack(out)
    at, Fs, us = _spectral_points(ops, N), [], []
    for u in _fields(case, seed, N, ops, L, True):
        u = u.to(dt).double()
        Fs.append(torch.fft.fftn(u).reshape(-1)[at])
        us.append(u if kind == "fullgrid" else _sub(u, L).clone())
    return torch.stack(Fs), torch.stack(us)
