"""Performance cases of the pressure solve: what a host model has the library do.

Every case goes through the public Python entry points (one call each into the
C ABI).  The geometries are the workload generator's own recipes (tank, sloping
beach with obstacles, 2DV flume, 2DH dispersion plan) at the sizes of this
repository's configurations and tests, and at generic ones between them.  The
geometry of a grid is fixed; the seed gives the provisional velocities, hence
the right-hand sides, and the weights of the adjoint.
"""
import functools
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("2clowns-3d_gb300")

MAX_CELLS = 256 * 256 * 96


def listed():
    return [
        # a small basin solved every time step of a small model: launches and latency
        {"name": "fp64_tank_24x16x16", "kind": "solve", "prec": "fp64", "geom": "tank", "nx": 24, "ny": 16, "nz": 16, "eps": 1e-10},
        # the Fortran program's own call (host arrays in, host arrays out) on the plain tank configuration
        {"name": "host_tank_64x64x32", "kind": "host", "geom": "tank", "nx": 64, "ny": 64, "nz": 32, "eps": 1e-12},
        # a vertical section (2DV mode, four columns) as used for flume studies; ragged length
        {"name": "fp64_flume_701x1x45", "kind": "solve", "prec": "fp64", "geom": "flume", "nx": 701, "ny": 1, "nz": 45, "eps": 1e-10},
        # the ordinary size of a basin study: device-resident FP64 and mixed precision
        {"name": "fp64_beach_128x128x48", "kind": "solve", "prec": "fp64", "geom": "beach", "nx": 128, "ny": 128, "nz": 48, "eps": 1e-10},
        {"name": "mixed_beach_128x128x48", "kind": "solve", "prec": "mixed", "geom": "beach", "nx": 128, "ny": 128, "nz": 48, "eps": 1e-10},
        # the headline configuration, plain FP64 and mixed: the largest solves
        {"name": "fp64_beach_256x256x96", "kind": "solve", "prec": "fp64", "geom": "beach", "nx": 256, "ny": 256, "nz": 96, "eps": 1e-10},
        {"name": "mixed_beach_256x256x96", "kind": "solve", "prec": "mixed", "geom": "beach", "nx": 256, "ny": 256, "nz": 96, "eps": 1e-10},
        # an ensemble of uneven half-size members solved together (mixed precision, as configured)
        {"name": "mixed_ensemble_12", "kind": "ensemble", "prec": "mixed", "members": 12, "scale": 0.5, "eps": 1e-10},
        # the 2DH dispersion solve of a plan grid (four columns, few iterations, output post-processing)
        {"name": "will_601x433", "kind": "will", "nx": 601, "ny": 433, "eps": 1e-10},
        # classification, static coefficients, rows, right-hand side and assembly: what a step does before its solve
        {"name": "build_beach_256x256x96", "kind": "build", "geom": "beach", "nx": 256, "ny": 256, "nz": 96},
        # one whole time step through the session: host fields in, classify, the ik loop, host fields out
        {"name": "session_beach_128x128x48", "kind": "session", "geom": "beach", "nx": 128, "ny": 128, "nz": 48, "eps": 1e-10},
        # the adjoint: transpose, adjoint solve and face gradients for gauge weights
        {"name": "adjoint_beach_96x96x48", "kind": "adjoint", "geom": "beach", "nx": 96, "ny": 96, "nz": 48, "eps": 1e-12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "host", "ensemble", "will", "build", "session", "adjoint"])
    if kind == "will":
        nx = _log_int(rng, 40, 1600)
        ny = _log_int(rng, 40, 1200)
        return {"kind": kind, "nx": nx, "ny": ny, "eps": 1e-10}
    if kind == "ensemble":
        return {"kind": kind, "prec": rng.choice(["fp64", "mixed"]), "members": rng.randint(2, 16),
                "scale": round(math.exp(rng.uniform(math.log(0.15), math.log(0.6))), 3), "eps": 1e-10}
    small = kind in ("host", "session", "adjoint")
    top = 128 if small else 256
    geom = rng.choice(["tank", "beach", "beach", "flume"] if kind == "solve" else ["tank", "beach"])
    if geom == "flume":
        c = {"kind": kind, "geom": geom, "nx": _log_int(rng, 60, 2000), "ny": 1, "nz": _log_int(rng, 16, 80)}
    else:
        c = {"kind": kind, "geom": geom, "nx": _log_int(rng, 16, top), "ny": _log_int(rng, 16, top),
             "nz": _log_int(rng, 12, 48 if small else 96)}
    if kind == "solve":
        c["prec"] = rng.choice(["fp64", "fp64", "mixed"])
    if kind != "build":
        c["eps"] = 1e-12 if kind == "adjoint" or (kind == "host" and geom == "tank") else 1e-10
    return c


# ---------------------------------------------------------------------------
# Inputs

@functools.lru_cache(maxsize=3)
def _geometry(geom, nx, ny, nz, eps):
    w = pkg.workload
    if geom == "tank":
        return w.make_case(nx, ny, nz, dz=0.8 / nz, amplitude=0.05, partial=False, noise=0.0, seed=0, eps0=eps)
    if geom == "flume":
        return w.make_case(nx, ny, nz, dz=0.8 / nz, slope=1.0 / 20.0, amplitude=0.05, noise=0.0, seed=1, eps0=eps)
    obstacles = min(40, max(0, nx * ny // 64))
    return w.make_case(nx, ny, nz, dz=0.8 / nz, slope=1.0 / 20.0, n_obstacles=obstacles, amplitude=0.05, noise=0.0,
                       seed=1, eps0=eps)


@functools.lru_cache(maxsize=2)
def _ensemble(members, scale):
    return [pkg.workload.ensemble_case(s) for s in pkg.workload.ensemble_members(members, seed=3, scale=scale)]


@functools.lru_cache(maxsize=2)
def _plan(nx, ny):
    return pkg.workload.dispersion_system(nx, ny, seed=7)


def _velocities(base, seed):
    """The provisional face velocities: the wave's plus N(0, 1e-3) on the wet cells."""
    rng = np.random.default_rng(seed)
    noise = rng.standard_normal(base.un.shape, dtype=np.float32)
    return base.un + np.where((base.f > 0.0)[:, None], 1.0e-3, 0.0) * noise


def _case(case, seed):
    import dataclasses
    base = _geometry(case["geom"], case["nx"], case["ny"], case["nz"], case.get("eps", 1e-10))
    return dataclasses.replace(base, un=_velocities(base, seed))


def _zeros(n):
    return torch.zeros(n, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "will":
        p = _plan(case["nx"], case["ny"])
        rng = np.random.default_rng(seed)
        b = p.b * rng.uniform(0.5, 1.5, p.n)
        st |= {k: torch.from_numpy(v).cuda() for k, v in (("al", p.al), ("ll", p.ll), ("d", p.d), ("b0", b))}
        st["b"] = torch.empty_like(st["b0"])
        st["solver"] = pkg.WillSolver(p.n, 4)
        return st
    if kind == "ensemble":
        import dataclasses
        sys_, xs = [], []
        for m, c in enumerate(_ensemble(case["members"], case["scale"])):
            _, ds = pkg.prepare_dev(dataclasses.replace(c, un=_velocities(c, seed * 101 + m)))
            sys_.append(ds)
            xs.append(_zeros(ds.mm2))
        prec = pkg.PREC_MIXED if case["prec"] == "mixed" else pkg.PREC_FP64
        st |= {"sys": sys_, "xs": xs, "solver": pkg.BatchedSolver([s.mnoe for s in sys_], prec)}
        return st
    c = _case(case, seed)
    if kind == "session":
        p = np.zeros(c.inne2 + 2)
        st |= {"c": c, "p": p, "session": pkg.Session(c)}
        return st
    if kind == "build":
        st["dc"] = pkg.DeviceCase.upload(c)
        return st
    dc, ds = pkg.prepare_dev(c)
    n = ds.mnoe
    if kind == "host":
        st |= {"n": n, "al": ds.alu.cpu().numpy(), "ll": ds.llu.cpu().numpy(), "d": ds.de.cpu().numpy(),
               "b": ds.b.cpu().numpy(), "x": np.zeros(ds.mm2 + 64)}
        return st
    nl = ds.alu.shape[0]
    st |= {"dc": dc, "ds": ds, "x": _zeros(ds.mm2)}
    if kind == "adjoint":
        st["solver"] = pkg.Solver(n, nl)
        st["solver"].solve(ds.alu, ds.llu, ds.de, ds.b, st["x"], eps=1e-12)
        rng = np.random.default_rng(seed)
        w = np.zeros(n)
        w[rng.integers(0, n, 16)] = rng.uniform(0.5, 1.5, 16)       # 16 gauges
        st["djdx"] = torch.from_numpy(w).cuda()
        return st
    st["solver"] = pkg.MixedSolver(n, nl) if case["prec"] == "mixed" else pkg.Solver(n, nl)
    return st


# ---------------------------------------------------------------------------
# One pass

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        ds, x = st["ds"], st["x"]
        x.zero_()                                   # the model starts every solve from xe = 0
        info = st["solver"].solve(ds.alu, ds.llu, ds.de, ds.b, x, eps=case["eps"])
        return {"x": x[:ds.mnoe], "iter": info.iter, "ier": info.ier}
    if kind == "host":
        st["x"][:] = 0.0
        eps, it, ier = pkg.pcgpme(st["al"], st["ll"], st["d"], st["b"], st["x"], st["n"], eps=case["eps"])
        return {"x": st["x"][:st["n"]], "iter": it, "ier": ier}
    if kind == "ensemble":
        for x in st["xs"]:
            x.zero_()
        infos = st["solver"].solve([(s.alu, s.llu, s.de, s.b) for s in st["sys"]], st["xs"], eps=case["eps"])
        return {"x": [x[:s.mnoe] for s, x in zip(st["sys"], st["xs"])], "iter": [i.iter for i in infos]}
    if kind == "will":
        st["b"].copy_(st["b0"])
        info = st["solver"].solve(st["al"], st["ll"], st["d"], st["b"], eps=case["eps"])
        return {"b": st["b"], "iter": info.iter}
    if kind == "build":
        dc = st["dc"]
        fln, ifln, sfn, isfn, passes = pkg.set_nflag_dev(dc)
        mp, alu_c, ll_c, de_c = pkg.init_matrix_dev(dc)
        r = pkg.rows_rhs_assemble_dev(dc, fln, ifln, mp, alu_c, ll_c, de_c)
        n = r["mnoe"]
        return {"nf": dc.nf, "nfb": dc.nfb, "fln": fln, "sfn": sfn, "alu_c": alu_c, "ll_c": ll_c, "de_c": de_c,
                "mno": r["mno"], "mno2mn": r["mno2mn"], "b": r["b"], "de": r["de"][:n], "alu": r["alu"][:, :n],
                "llu": r["llu"][:, :n], "dmax": r["dmax"]}
    if kind == "session":
        c, s = st["c"], st["session"]
        s.set_fields(c.nf, c.nfb, c.f, c.fb, c.a, c.un, c.sp, st["p"])
        s.classify()
        loop = s.pressure_loop(c.dt, eps0=case["eps"])
        out = s.fields()
        return {"nf": out["nf"], "nfb": out["nfb"], "f": out["f"], "p": out["p"], "un": out["un"],
                "ik": loop["ik"], "iter": loop["iter"]}
    lam, grad, info = pkg.adjoint_dev(st["dc"], st["ds"], st["x"], st["djdx"], eps=case["eps"], solver=st["solver"])
    return {"lam": lam, "grad": grad, "iter": info.iter}


# ---------------------------------------------------------------------------
# What a pass cannot do without

def _rows(nx, ny, nz):
    return nx * ny * (0.625 * nz + 1)           # half-metre depth in a 0.8 m domain


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: the reference's arithmetic (37 FP64 multiply-adds
    per row and iteration, 31 in four columns), at about 1.3 iterations per cell of the longest side (27 for the 2DH solve)."""
    kind = case["kind"]
    if kind == "will":
        n = case["nx"] * case["ny"]
        return {"bytes": n * (4 * 12 + 8 + 8 + 8), "flops": n * 31 * 2 * 27}
    if kind == "ensemble":
        s = case["scale"]
        n = case["members"] * _rows(176 * s, 144 * s, 64 * s)
        return {"bytes": n * 96, "flops": n * 37 * 2 * 1.3 * 200 * s}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, cells = _rows(nx, ny, nz), nx * ny * nz
    if kind == "build":
        # in: map, i, j, k, flags, f, fb, a, un, sp; out: static coefficients, lists, map, matrix rows
        return {"bytes": cells * (24 + 96) + cells * 84 + n * 100, "flops": cells * 30}
    flops = n * (31 if case["geom"] == "flume" else 37) * 2 * 1.3 * max(nx, ny)
    if kind == "session":
        return {"bytes": cells * (8 + 96) + cells * 48, "flops": flops}
    if kind == "adjoint":
        return {"bytes": n * 96 + cells * 48, "flops": flops}
    return {"bytes": n * ((4 if case["geom"] == "flume" else 6) * 12 + 8 + 8 + 8), "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits, with plain torch

def _ell(al, ll, d, n):
    a = al[:, :n]
    c = ll[:, :n].long() - 1
    a = torch.where(c >= 0, a, torch.zeros_like(a))
    return a, c.clamp_(min=0), d[:n]


def _apply(mat, x):
    a, c, d = mat
    y = d * x
    for k in range(a.shape[0]):
        y = y + a[k] * x[c[k]]
    return y


def _apply_t(mat, x):
    a, c, d = mat
    y = d * x
    for k in range(a.shape[0]):
        y.index_add_(0, c[k], a[k] * x)
    return y


def _solve(op, d, b, tol=1e-13):
    """x with op(x) = b: diagonally scaled BiCGSTAB, restarted from the true residual."""
    x = torch.zeros_like(b)
    bn = (b / d).norm()
    if bn == 0:
        return x
    for _ in range(12):
        r = (b - op(x)) / d
        start = r.norm()
        if start <= tol * bn:
            break
        r0, p, dx = r.clone(), r.clone(), torch.zeros_like(b)
        rho = r0 @ r
        for it in range(4000):
            v = op(p) / d
            alpha = rho / (r0 @ v)
            s = r - alpha * v
            t = op(s) / d
            omega = (t @ s) / (t @ t)
            dx += alpha * p + omega * s
            r = s - omega * t
            new = r0 @ r
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
            if it % 16 == 0 and not r.norm() > 1e-9 * start:
                break
        if not torch.isfinite(dx).all():
            break
        x = x + dx
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "session":
        return None                             # whole numbers and fields of a loop with its own stop test
    st = prepare(case, seed)
    if kind == "build":
        return _exact_build(st)
    if kind == "host":
        t = {k: torch.from_numpy(st[k]).cuda() for k in ("al", "ll", "d", "b")}
        m = _ell(t["al"], t["ll"], t["d"], st["n"])
        return {"x": _solve(lambda v: _apply(m, v), m[2], t["b"][:st["n"]]), "iter": None, "ier": None}
    if kind == "ensemble":
        xs = []
        for s in st["sys"]:
            m = _ell(s.alu, s.llu, s.de, s.mnoe)
            xs.append(_solve(lambda v: _apply(m, v), m[2], s.b[:s.mnoe]))
        return {"x": xs, "iter": None}
    if kind == "will":
        m = _ell(st["al"], st["ll"], st["d"], st["d"].numel())
        x = _solve(lambda v: _apply(m, v), m[2], st["b0"])
        return {"b": torch.where(st["ll"][0] == 0, torch.zeros_like(x), x), "iter": None}   # rows without neighbours keep the residual
    ds = st["ds"]
    m = _ell(ds.alu, ds.llu, ds.de, ds.mnoe)
    if kind == "adjoint":
        return {"lam": _solve(lambda v: _apply_t(m, v), m[2], st["djdx"]), "grad": None, "iter": None}
    return {"x": _solve(lambda v: _apply(m, v), m[2], ds.b[:ds.mnoe]), "iter": None, "ier": None}


def _exact_build(st):
    """The static coefficients from the input arrays; the rest of the outputs are lists and flags, or copies of these."""
    c = st["dc"].case
    is_, js, ks = (int(v) for v in c.dims[:3])
    n = c.inne
    idx = [c.in_[1:n + 1].astype(np.int64), c.jn[1:n + 1].astype(np.int64), c.kn[1:n + 1].astype(np.int64)]
    pos = c.dx[(c.dx > 0.0)]
    mp = float(pos.min()) ** 2
    open_ = (c.nf[1:n + 1] != -1) & (c.fb[1:n + 1] != 0.0)
    alu = np.zeros((6, n))
    for l in range(3):
        for side in (0, 1):
            at = [v.copy() for v in idx]
            at[l] += 1 if side else -1
            nb = c.mn[at[1] - (js - 2), at[2] - (ks - 2), at[0] - (is_ - 2)]
            own = nb if side else np.arange(1, n + 1)
            face = c.a[own, l]
            use = open_ & ~((c.nf[nb] == -1) & (c.nfb[nb] != 4)) & (face != 0.0) & (c.fb[nb] != 0.0)
            d0, d1 = c.dx[idx[l] - 1, l], c.dx[at[l] - 1, l]
            with np.errstate(divide="ignore", invalid="ignore"):
                v = -mp * 2.0 / (d0 * (d0 + d1)) * face / c.fb[1:n + 1]
            alu[2 * l + side] = np.where(use, v, 0.0)
    return {"nf": None, "nfb": None, "fln": None, "sfn": None, "alu_c": alu, "ll_c": None, "de_c": -alu.sum(0),
            "mno": None, "mno2mn": None, "b": None, "de": None, "alu": None, "llu": None, "dmax": None}
